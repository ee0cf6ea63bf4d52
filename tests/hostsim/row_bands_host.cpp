// row_bands_host.cpp -- the bands of a frame's rows (libsvo_b200/csrc/row_bands.h).
// TEST INFRASTRUCTURE ONLY.
#include "../../libsvo_b200/csrc/row_bands.h"

// Writes {first row, rows, blocks} per band; stops with -1 after `cap` of them.
extern "C" int64_t bands(uint32_t height, uint32_t block_h, uint32_t* out, int64_t cap) {
  int64_t n = 0;
  const int rc = svo::for_each_band(height, block_h, [&](uint32_t y0, uint32_t rows, uint32_t gy) {
    if (n == cap) return (int)SVO_ERR_RANGE;
    out[3 * n] = y0;
    out[3 * n + 1] = rows;
    out[3 * n++ + 2] = gy;
    return (int)SVO_OK;
  });
  return rc == SVO_OK ? n : -1;
}
