// yield_host.cpp -- the descent that can be left and taken up again
// (libsvo_b200/csrc/traverse.cuh), built for the host as stream_rays_kernel uses
// it.  A host call is one lane, so every number of lanes to keep asks for a yield
// at each opportunity.  TEST INFRASTRUCTURE ONLY: see host_shim.h.
#include "host_shim.h"

#include "../../libsvo_b200/csrc/traverse.cuh"

// The rays' hit records, and in calls the most calls that one ray took; returns
// the number of calls that neither ended their ray nor moved it on by a pass (a
// ray is given up there).
template <bool kFlat>
static uint64_t cast(const svo::GlobalFetch& fetch, uint64_t num_nodes, const float* origins, const float* dirs,
                     uint64_t n, float tsr, int S, int keep, uint32_t* out, uint32_t* calls) {
  uint2 stack[svo::kMaxStack];
  uint64_t idle = 0;
  *calls = 0;
  for (uint64_t i = 0; i < n; ++i) {
    const float o[3] = {origins[3 * i], origins[3 * i + 1], origins[3 * i + 2]};
    svo::RayHit h;
    svo::Ray r;
    float t_min = 0.0f;
    const svo::RayKind kind =
        svo::setup_ray<kFlat>(o, dirs[3 * i], dirs[3 * i + 1], dirs[3 * i + 2], tsr, r, t_min, h);
    svo::RayState st = {0u, t_min, r.t_max, 0.0f, 0.0f, 0.0f, 0.5f, 0u, 0u};
    svo::Outcome end = kind == svo::kGeneral ? svo::kLeaves : svo::kEnded;
    if (kind == svo::kFast) {
      const uint32_t limit = svo::pass_limit(S);
      svo::Descent w = svo::descent_start(fetch, num_nodes, r, t_min, limit, stack);
      uint32_t used = 0;
      for (;;) {
        const uint32_t before = w.passes;
        h = svo::no_hit();
        end = svo::descend<kFlat, true>(fetch, num_nodes, r, S, stack, 1, limit, keep, w, st, h);
        ++used;
        if (end != svo::kYields) break;
        if (w.passes == before) {
          ++idle;
          end = svo::kEnded;
          break;
        }
      }
      if (used > *calls) *calls = used;
    }
    if (end == svo::kLeaves)
      svo::descend_general<kFlat>(fetch, num_nodes, r, S, stack, 1, st, h, 0u);
    uint32_t* q = out + 4 * i;  // the 16-byte svo_hit record
    q[0] = h.node;
    q[1] = __float_as_uint(h.t);
    q[2] = (h.depth & 0xFFFFu) | ((h.hit & 0xFFu) << 16) | ((h.flags & 0xFFu) << 24);
    q[3] = (h.loops & 0xFFFFu) | (h.fetches << 16);
  }
  return idle;
}

extern "C" uint64_t host_cast_yielding(const uint32_t* nodes, uint64_t num_nodes, const float* origins,
                                       const float* dirs, uint64_t n, float tsr, int S, int flat, int keep,
                                       uint32_t* hits, uint32_t* calls) {
  const svo::GlobalFetch fetch{reinterpret_cast<const uint2*>(nodes)};
  return flat ? cast<true>(fetch, num_nodes, origins, dirs, n, tsr, S, keep, hits, calls)
              : cast<false>(fetch, num_nodes, origins, dirs, n, tsr, S, keep, hits, calls);
}
