// ray_order_host.cpp -- the question whether rays come in order
// (libsvo_b200/csrc/ray_order.cuh), built for the host.  TEST INFRASTRUCTURE ONLY:
// see host_shim.h.
#include "host_shim.h"

#include "../../libsvo_b200/csrc/ray_order.cuh"

// The close pairs among those that the kernels ask; last is the largest ray
// index that is read.
extern "C" uint32_t host_close_pairs(const float* origins, const float* dirs, uint64_t n, uint64_t* last) {
  uint32_t close = 0;
  *last = 0;
  for (uint32_t k = 0; k < svo::kOrderPairs; ++k) {
    const uint64_t i = svo::order_pair(k, n);
    close += svo::pair_close(origins, dirs, i) ? 1u : 0u;
    if (i + 1 > *last) *last = i + 1;
  }
  return close;
}
extern "C" uint32_t host_close_needed() { return svo::kOrderClose; }
