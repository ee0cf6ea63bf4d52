// builder_host.cpp -- what the GPU builder's tests need of host code: the cells that
// its plan visits (libsvo_b200/csrc/chunk_plan.h), and the voxels of a sliver by the
// host builder's own overlap test (libsvo_b200/csrc/scene.cpp) without the walk over
// the sliver's whole box.  TEST INFRASTRUCTURE ONLY.
#include "../../libsvo_b200/csrc/scene.cpp"

#include "../../libsvo_b200/csrc/chunk_plan.h"

extern "C" {

// Boxes of columns, lo and hi inclusive (u, v, w per box: every (u, v) of a box is a
// column in each cell that the box's w range meets).  A build holds `memory` columns
// at most.  Writes {level, index, columns, first_new_level against the last built
// cell} per built cell; returns their number, or minus the status.
int64_t plan(const int32_t* boxes, uint64_t num_boxes, uint32_t depth, uint32_t level, uint64_t max_columns,
             uint64_t memory, uint64_t* out, uint64_t cap) {
  uint64_t n = 0;
  svo::Cell last = {0, 0};
  const int rc = svo::for_each_chunk(
      depth, level, max_columns,
      [&](const svo::Cell& c, uint64_t* columns) {
        int32_t at[3] = {0, 0, 0};
        for (uint32_t b = 0; b < c.level; ++b)
          for (int k = 0; k < 3; ++k) at[k] |= (int32_t)((c.index >> (3 * b + 2 - k)) & 1u) << b;
        const int32_t side = (int32_t)((1u << depth) >> c.level);
        *columns = 0;
        for (uint64_t i = 0; i < num_boxes; ++i) {
          uint64_t size[3];
          for (int k = 0; k < 3; ++k) {
            const int32_t lo = std::max(boxes[6 * i + k], at[k] * side);
            const int32_t hi = std::min(boxes[6 * i + 3 + k], (at[k] + 1) * side - 1);
            size[k] = lo > hi ? 0 : (uint64_t)(hi - lo + 1);
          }
          if (size[2]) *columns += size[0] * size[1];
        }
        return SVO_OK;
      },
      [&](const svo::Cell& c, uint64_t columns, bool* began) {
        if (columns > memory) return SVO_ERR_NOMEM;
        *began = true;
        if (n == cap) return SVO_ERR_NOMEM;  // after it has begun: the end
        uint64_t* o = out + 4 * n++;
        o[0] = c.level;
        o[1] = c.index;
        o[2] = columns;
        o[3] = n == 1 ? 0 : svo::first_new_level(last, c, depth);
        last = c;
        return SVO_OK;
      });
  return rc == SVO_OK ? (int64_t)n : (int64_t)rc;
}

// The codes of the voxels that triangle t (a, b, c: nine floats) overlaps, looked for
// within `margin` voxels of its edges ab and cb at every x; t must be longest along x.
uint64_t near_voxels(const float* t, uint32_t depth, int margin, uint64_t* codes, uint64_t cap) {
  const uint32_t R = 1u << depth;
  const float inv = 1.0f / (float)R, h = 0.5f * inv;
  double lo[3], hi[3];
  for (int k = 0; k < 3; ++k) {
    lo[k] = std::min({t[k], t[3 + k], t[6 + k]});
    hi[k] = std::max({t[k], t[3 + k], t[6 + k]});
  }
  auto cell = [&](double x) { return (int)std::floor((x + 0.5) * R); };
  uint64_t n = 0;
  for (int x = std::max(0, cell(lo[0]) - margin); x <= std::min((int)R - 1, cell(hi[0]) + margin); ++x) {
    double from[2] = {1e9, 1e9}, to[2] = {-1e9, -1e9};
    for (int edge = 0; edge < 2; ++edge)
      for (int side = 0; side < 2; ++side) {
        const float* a = t + 6 * edge;
        const float* b = t + 3;
        const double px = -0.5 + (double)(x + side) / R;
        const double s = std::min(1.0, std::max(0.0, (px - a[0]) / ((double)b[0] - a[0])));
        for (int k = 0; k < 2; ++k) {
          const double p = a[1 + k] + s * ((double)b[1 + k] - a[1 + k]);
          from[k] = std::min(from[k], p);
          to[k] = std::max(to[k], p);
        }
      }
    for (int y = std::max(0, cell(from[0]) - margin); y <= std::min((int)R - 1, cell(to[0]) + margin); ++y)
      for (int z = std::max(0, cell(from[1]) - margin); z <= std::min((int)R - 1, cell(to[1]) + margin); ++z) {
        const float bc[3] = {-0.5f + ((float)x + 0.5f) * inv, -0.5f + ((float)y + 0.5f) * inv,
                             -0.5f + ((float)z + 0.5f) * inv};
        if (!svo::tri_box_overlap(bc, h, t, t + 3, t + 6)) continue;
        if (n < cap) codes[n] = svo::morton3((uint32_t)x, (uint32_t)y, (uint32_t)z, depth);
        ++n;
      }
  }
  return n;
}

}  // extern "C"
