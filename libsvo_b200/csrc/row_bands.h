// row_bands.h -- a frame's rows in pieces of one launch each.
#pragma once
#include <algorithm>
#include <cstdint>

#include "../../include/libsvo_b200.h"

namespace svo {

constexpr uint32_t kGridRows = 65535u;  // blocks along y of one launch

// int launch(uint32_t y0, uint32_t rows, uint32_t grid_rows), for blocks of block_h
// rows.  The next band's first row may lie beyond 2^32 where the last band of a
// frame does not, so it is counted in 64 bits.
template <class Launch>
int for_each_band(uint32_t height, uint32_t block_h, Launch&& launch) {
  const uint32_t most = kGridRows * block_h;
  for (uint64_t y0 = 0; y0 < height; y0 += most) {
    const uint32_t rows = (uint32_t)std::min<uint64_t>(height - y0, most);
    const int rc = launch((uint32_t)y0, rows, (rows + block_h - 1) / block_h);
    if (rc != SVO_OK) return rc;
  }
  return SVO_OK;
}

}  // namespace svo
