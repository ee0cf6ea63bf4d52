// chunk_plan.h -- which cells of an octree's top levels the GPU builder takes one
// after another.
#pragma once
#include <cstdint>
#include <vector>

#include "../../include/libsvo_b200.h"

namespace svo {

// Cell `index` (Morton order) of the 8^level cells of a level.
struct Cell {
  uint32_t level;
  uint64_t index;
};

// Of an octree `depth` levels deep, the smallest code inside the cell.
inline uint64_t cell_code(const Cell& c, uint32_t depth) { return c.index << (3 * (depth - c.level)); }

// The coarsest level at which a node that begins in cell b is not one of cell a's,
// the cells being different and neither inside the other: the codes of their voxels
// differ first where the cells' own codes do.
inline uint32_t first_new_level(const Cell& a, const Cell& b, uint32_t depth) {
  uint64_t diff = cell_code(a, depth) ^ cell_code(b, depth);
  uint32_t digit = 0;
  while (diff >>= 3) ++digit;
  return depth - digit;
}

// Cells are not split beyond this level (512 cells): a cell is counted by a pass over
// all triangles, and its children's columns are twice its own in all.
constexpr uint32_t kLastSplit = 3;

// Builds the octree cell by cell, in Morton order, beginning with the cells of
// `level`: a cell of more than max_columns columns, and one whose build finds no
// memory before it has added anything (SVO_ERR_NOMEM with *began false), gives
// way to its eight children.  The last level's cells are built whatever their
// columns.
//   int count(const Cell&, uint64_t* columns)
//   int build(const Cell&, uint64_t columns, bool* began)
template <class Count, class Build>
int for_each_chunk(uint32_t depth, uint32_t level, uint64_t max_columns, Count&& count, Build&& build) {
  std::vector<Cell> todo;
  for (uint64_t i = 1ull << (3 * level); i-- > 0;) todo.push_back({level, i});
  while (!todo.empty()) {
    const Cell c = todo.back();
    todo.pop_back();
    uint64_t columns = 0;
    int rc = count(c, &columns);
    if (rc != SVO_OK) return rc;
    if (columns == 0) continue;
    const bool splits = c.level < kLastSplit && c.level + 1 < depth;
    if (columns <= max_columns || !splits) {
      bool began = false;
      rc = build(c, columns, &began);
      if (rc == SVO_OK) continue;
      if (rc != SVO_ERR_NOMEM || began || !splits) return rc;
    }
    for (uint64_t k = 8; k-- > 0;) todo.push_back({c.level + 1, c.index * 8 + k});
  }
  return SVO_OK;
}

}  // namespace svo
