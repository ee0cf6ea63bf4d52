// ray_order.cuh -- whether a set of explicit rays comes in an order that keeps
// neighbours together (pixel rays, rays sorted by the caller), asked of a few of
// its pairs.  It decides which kernel casts the set, never what a ray hits.
#pragma once
#include <cstdint>

namespace svo {

// Pairs asked, evenly spread over the set, and how many of them must be close:
// some fall on the end of an image's row.
constexpr uint32_t kOrderPairs = 8;
constexpr uint32_t kOrderClose = 6;

// The first ray of pair k; the second is the next one.
__device__ __forceinline__ uint64_t order_pair(uint32_t k, uint64_t n) { return k * (n / kOrderPairs); }

__device__ __forceinline__ bool close_by(const float* a, const float* b, float limit) {
  const float x = b[0] - a[0], y = b[1] - a[1], z = b[2] - a[2];
  return x * x + y * y + z * z <= limit;
}

// Whether rays i and i + 1 are close: directions within 1/32 of their length,
// origins within 1/32 of the root box's side (not with a NaN).  The line: a million
// pixel rays moved at random, lanes that take further rays against a thread a ray,
// us: directions by 1/128 193 against 178 over a depth-11 icosphere, 102 against 82
// over a depth-10 terrain, by 1/32 204 against 213 and 111 against 99, by 1/8 205
// against 282 and 123 against 150; origins of parallel rays by 1/128 260 against
// 239 and 151 against 113, by 1/32 273 against 278 and 158 against 128, by 1/8 278
// against 360 and 169 against 159.  (A move by a lies between neighbours that
// differ by 1.4 a.)
__device__ __forceinline__ bool pair_close(const float* origins, const float* dirs, uint64_t i) {
  const float *o = origins + 3 * i, *d = dirs + 3 * i;
  constexpr float kNear = 1.0f / 1024.0f;
  return close_by(o, o + 3, kNear) && close_by(d, d + 3, kNear * (d[0] * d[0] + d[1] * d[1] + d[2] * d[2]));
}

}  // namespace svo
