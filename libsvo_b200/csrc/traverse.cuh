// traverse.cuh -- per-ray sparse-voxel-octree descent for sm_100a.
//
// Restates the reference's two traversals bit for bit:
//   * treelet: sample() in opencl/treeletRenderer_rgba.cl:201-382 over the
//     TreeletMemoryManager incore pool (first-child indices relative to the
//     node, added mod 2^32; src/TreeletMemoryManager.cpp:531-539);
//   * flat:    CpuRaycasterSingleRay3::traversSvo
//     (src/incore/CpuRaycasterSingleRay3.cpp:159-387) over a breadth-first
//     pool with absolute first-child indices.
//
// Every FP32 operation is an explicit round-to-nearest intrinsic, so no
// multiply-add is ever contracted and the operation order is the
// reference's.  Divisions, reciprocals and the square root are the IEEE
// correctly rounded ones.  OpenCL's max(a, b) is (a < b) ? b : a.
//
// Storage.  The reference keeps {node, tMin, tMax, centre} per stack level.
// Two facts shrink that to {node, tMax}:
//   - a level's tMin is only read again after popping back to it, and at the
//     push it was set to the pushed child's tcMax, which is the child frame's
//     tMax and never changes afterwards; so on a pop tMin := popped tMax;
//   - node centres are exact dyadic numbers (-0.5 + (2i+1) 2^-(k+1) for a
//     depth-k node with lattice coordinate i), so any ancestor's centre is a
//     prefix of the bits of a node's own (ancestor_center).
// The stack lives in shared memory, one 8-byte word per level per thread,
// laid out [level][thread] so a warp's accesses are contiguous.
#pragma once
#include <cstdint>

#include "../../include/libsvo_b200.h"

namespace svo {

constexpr int kMaxStack = 24;  // largest supported stack_size / flat depth

struct RayHit {
  uint32_t node;
  float t;
  uint32_t depth;
  uint32_t hit;
  uint32_t flags;
  uint32_t loops;
  uint32_t fetches;  // loop iterations that read the parent node
  // set on a leaf or LOD stop, for the analysis pass and the quality view:
  // the hit child's entry distance, the child size, and whether the child was
  // a leaf (the watchdog stop sets tMin, the current size and leaf = 1, so
  // that quality = sx2 - tScaleRatio * tc_min holds for both)
  float tc_min;
  float sx2;
  uint32_t leaf;
  // SampleResult.nodeCenter: the hit child's centre, or the current node's
  // when the watchdog ends the ray (shadow rays start there)
  float cx, cy, cz;
  float t_enter, t_exit;  // the root box (both 0 when the ray misses it)
};

__device__ __forceinline__ RayHit no_hit() {
  RayHit h;
  h.node = 0u;
  h.t = 0.0f;
  h.depth = 0u;
  h.hit = 0u;
  h.flags = 0u;
  h.loops = 0u;
  h.fetches = 0u;
  h.tc_min = 0.0f;
  h.sx2 = 0.0f;
  h.leaf = 0u;
  h.cx = 0.0f;
  h.cy = 0.0f;
  h.cz = 0.0f;
  h.t_enter = 0.0f;
  h.t_exit = 0.0f;
  return h;
}

__device__ __forceinline__ float cl_max(float a, float b) { return (a < b) ? b : a; }
__device__ __forceinline__ float cl_min(float a, float b) { return (b < a) ? b : a; }

// OpenCL sign(): +-1, the argument itself for +-0, 0 for NaN.
__device__ __forceinline__ float cl_sign(float v) {
  return v > 0.0f ? 1.0f : (v < 0.0f ? -1.0f : (v == 0.0f ? v : 0.0f));
}

// 2^e for -126 <= e <= 0, exact.
__device__ __forceinline__ float pow2i(int e) { return __int_as_float((127 + e) << 23); }

// intersectAABB (opencl/treeletRenderer_rgba.cl:100-178) against [-0.5,0.5]^3.
__device__ __forceinline__ bool root_slab(const float o[3], const float d[3], float& t_min,
                                          float& t_max) {
  float t_near = -10000000.0f;
  float t_far = 10000000.0f;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    if (d[i] == 0.0f && (-0.5f > o[i] || 0.5f < o[i])) return false;
    float t1 = __fdiv_rn(__fsub_rn(-0.5f, o[i]), d[i]);
    float t2 = __fdiv_rn(__fsub_rn(0.5f, o[i]), d[i]);
    if (t1 > t2) {
      const float s = t1;
      t1 = t2;
      t2 = s;
    }
    if (t1 > t_near) t_near = t1;
    if (t2 < t_far) t_far = t2;
    if (t_near > t_far) return false;
    if (t_far < 0.0f) return false;
  }
  t_min = t_near;
  t_max = t_far;
  return true;
}

// Node-record fetch policies.  GlobalFetch reads through the read-only
// cache; StagedFetch serves the first `count` records (the top levels of a
// breadth-first treelet pool) from a shared-memory copy.
struct GlobalFetch {
  const uint2* __restrict__ nodes;
  __device__ __forceinline__ uint2 operator()(uint32_t i) const { return __ldg(nodes + i); }
};
struct StagedFetch {
  const uint2* __restrict__ nodes;
  const uint2* top;
  uint32_t count;
  __device__ __forceinline__ uint2 operator()(uint32_t i) const {
    return i < count ? top[i] : __ldg(nodes + i);
  }
};

// A saved traversal state for the cycle search of rays that do not advance
// (descend_general): frame node, size and tMin bits, the stacked frames, and
// the loop and fetch counts when it was saved.  Lives in local memory
// (volatile, so no registers are spent on it).
constexpr uint32_t kSearchFrom = 128;  // rays that run descend_general from the root
constexpr uint32_t kFirstGap = 32;
struct CycleMark {
  uint32_t node, size, tmin, loops, fetches, next_save, gap;
  uint32_t stack[2 * kMaxStack];
};

// Bit 31 set exactly when pos > c.  The sign of c - pos says so: with
// subnormals the difference rounds to zero only when the two are equal, x - x
// is +0, and a NaN the hardware produces is positive (the comparison is false).
__device__ __forceinline__ uint32_t above(float pos, float c) {
#if defined(__CUDACC__)
  return __float_as_uint(__fsub_rn(c, pos));
#else
  return pos > c ? 0x80000000u : 0u;
#endif
}

// v with the sign that `above` gives: v where bit 31 is set, else -v.  v > 0.
__device__ __forceinline__ float with_side(uint32_t side, float v) {
  return __uint_as_float((~side & 0x80000000u) | __float_as_uint(v));
}

// (acc << 1) | bit 31 of side: one funnel shift.
__device__ __forceinline__ uint32_t shift_in(uint32_t acc, uint32_t side) {
#if defined(__CUDACC__)
  return __funnelshift_l(side, acc, 1);
#else
  return (acc << 1) | (side >> 31);
#endif
}

// The lanes that run a piece of code together at this moment.  Only a hint: CUDA
// does not promise when lanes that parted come together again, so nothing may
// wait for this number to change.  (A host caller is one lane.)
__device__ __forceinline__ int lanes_together() {
#if defined(__CUDACC__)
  return __popc(__activemask());
#else
  return 1;
#endif
}

// The valid bits of a node's children before child ci.
__device__ __forceinline__ uint32_t valid_below(uint32_t ci) {
#if defined(__CUDACC__)
  uint32_t mask;
  asm("bmsk.clamp.b32 %0, 8, %1;" : "=r"(mask) : "r"(ci));
  return mask;
#else
  return (0x100u << ci) - 0x100u;
#endif
}

// The centre coordinate of the ancestor at the level whose child size is sx2,
// from a descendant's: as c + 1.5, in [1, 2), the coordinate's fraction is the
// lattice coordinate in fixed point, so the ancestor's is its leading bits with
// the bit of weight sx2 set (one = the bits of 1 + sx2, keep = the mask of the
// bits above).  The sum is rounded down: the one centre that needs 24 bits
// (depth 23) then loses a bit below those that are kept.
__device__ __forceinline__ float ancestor_center(float c, uint32_t one, uint32_t keep) {
#if defined(__CUDACC__)
  const uint32_t x = __float_as_uint(__fadd_rz(c, 1.5f));
#else
  const uint32_t x = 0x3f800000u | (uint32_t)(int32_t)(((double)c + 0.5) * 8388608.0);
#endif
  return __fadd_rn(__uint_as_float((x & keep) | one), -1.5f);
}

// Two floats for the packed FP32 instructions, each half rounded as the scalar
// ones round.  A product and a sum of two packed operations may be contracted
// into one rounding where the compiler sees them side by side (add.rn.f32x2 of
// mul.rn.f32x2 came out one bit off on 1.7 % of a frame's rays), so a sum of
// products multiplies the product by a one that it cannot know: constant memory
// belongs to the host.
#if defined(__CUDACC__)
typedef unsigned long long Pair;
static __constant__ Pair kPairOfOnes = 0x3f8000003f800000ull;
__device__ __forceinline__ Pair pair_of(float a, float b) {
  Pair r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void halves(Pair v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ Pair pair_mul(Pair a, Pair b) {
  Pair r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ Pair pair_add(Pair a, Pair b) {
  Pair r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ Pair pair_fma(Pair a, Pair b, Pair c) {
  Pair r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// a * b + c, rounded twice
__device__ __forceinline__ Pair pair_mul_add(Pair a, Pair b, Pair c) {
  return pair_fma(pair_mul(a, b), kPairOfOnes, c);
}
// ancestor_center of both halves
__device__ __forceinline__ Pair ancestor_centers(Pair c, uint32_t one, uint32_t keep) {
  Pair q;
  asm("add.rz.f32x2 %0, %1, %2;" : "=l"(q) : "l"(c), "l"(0x3fc000003fc00000ull));
  float a, b;
  halves(q, a, b);
  return pair_add(pair_of(__uint_as_float((__float_as_uint(a) & keep) | one),
                          __uint_as_float((__float_as_uint(b) & keep) | one)),
                  0xbfc00000bfc00000ull);
}
// c - a: a times -1 is exact
__device__ __forceinline__ Pair pair_sub_from(Pair a, Pair c) {
  return pair_fma(a, 0xbf800000bf800000ull, c);
}
#else
struct Pair {
  float a, b;
};
inline Pair pair_of(float a, float b) { return Pair{a, b}; }
inline void halves(Pair v, float& a, float& b) { a = v.a, b = v.b; }
inline Pair pair_mul(Pair x, Pair y) { return Pair{x.a * y.a, x.b * y.b}; }
inline Pair pair_add(Pair x, Pair y) { return Pair{x.a + y.a, x.b + y.b}; }
inline Pair pair_mul_add(Pair x, Pair y, Pair z) { return pair_add(pair_mul(x, y), z); }
inline Pair ancestor_centers(Pair c, uint32_t one, uint32_t keep) {
  return Pair{ancestor_center(c.a, one, keep), ancestor_center(c.b, one, keep)};
}
// (the host's `above` compares; 1 stands for a negative difference)
inline Pair pair_sub_from(Pair x, Pair z) { return Pair{x.a > z.a ? -1.0f : 1.0f, x.b > z.b ? -1.0f : 1.0f}; }
#endif

// Where a ray stands between two iterations of the reference: its frame (node,
// interval, centre, child size: 2^-(k+1) at depth k) and what it has counted.
struct RayState {
  uint32_t node;
  float tmin, tmax, cx, cy, cz, sx2;
  uint32_t loops, fetches;
};

// The ray against the root box, set up once per ray.
struct Ray {
  float ox, oy, oz, dx, dy, dz;  // origin, clamped direction
  float rx, ry, rz, px, py, pz;  // 1 / d and -o / d
  float t_max, tsr;              // exit from the root box, tScaleRatio
};

// The frame's level counted as the reference's S - scale: 1 at the root.
__device__ __forceinline__ uint32_t level_of(float sx2) {
  return 127u - (__float_as_uint(sx2) >> 23);
}

// The reference's pop test.
template <bool kFlat>
__device__ __forceinline__ bool interval_done(float tmin, float tmax) {
  const float eps = 0.00001f;
  if (kFlat) return (tmax < 0.0f) || (fabsf(__fsub_rn(tmin, tmax)) < eps) || !(tmin < tmax);
  return (tmax < 0.0f) || !(fabsf(__fsub_rn(tmin, tmax)) > eps);
}

// The child size at which the treelet rules stop (the reference's scale 1) or,
// in a flat pool, below which no child may be an inner node (scale 0).
template <bool kFlat>
__device__ __forceinline__ float last_size(int S) {
  return pow2i(kFlat ? -S : 1 - S);
}

__device__ __forceinline__ void ray_missed(bool flat, const Ray& r, uint32_t loops,
                                           uint32_t fetches, RayHit& h) {
  h.hit = 0u;
  h.node = 0u;
  h.depth = 0u;
  h.t = flat ? 0.0f : r.t_max;
  h.loops = loops;
  h.fetches = fetches;
}

// The reference's loop as it is written, from any state on: every frame is
// stacked, a child's slab distances are compared and swapped, and the watchdog
// is looked at in every iteration.  Rays that `descend` cannot take (an
// infinite reciprocal, an origin that is not finite, or -0: see cast_ray) run it from
// the root, and those that stop advancing or come near the watchdog finish in
// it.  A pass is one child test and the pops that follow it.
template <bool kFlat, class Fetch>
__device__ __forceinline__ void descend_general(const Fetch& fetch, uint64_t num_nodes,
                                                const Ray& r, int S, uint2* stack, int stride,
                                                const RayState& from, RayHit& h,
                                                uint32_t loop_cap) {
  const float eps = 0.00001f;
  // the reference's watchdog, or the caller's smaller cap (cost estimates)
  const uint32_t watchdog = (uint32_t)((S + 1) * (S + 1) * 5);
  const uint32_t max_loops = loop_cap && loop_cap < watchdog ? loop_cap : watchdog;
  const float sx2_last = last_size<kFlat>(S);
  const uint32_t last_node = num_nodes ? (uint32_t)(num_nodes - 1u) : 0u;
  uint32_t node = 0u;
  float tmin = from.tmin, tmax = r.t_max;
  float cx = 0.0f, cy = 0.0f, cz = 0.0f;
  float sx2 = 0.5f;
  uint32_t loops = from.loops, fetches = from.fetches;
  uint2* sp = stack;  // the next free stack word
  bool in_pool = num_nodes > 0u;
  uint2 nd = in_pool ? fetch(0u) : make_uint2(0u, 0u);
  // the first iteration of the cycle search
  const uint32_t search_from = from.loops ? from.loops + 1u : kSearchFrom;
  uint32_t check_at = max_loops < search_from ? max_loops : search_from;
  volatile CycleMark mark;
  mark.loops = 0u;  // none saved
  mark.next_save = search_from;
  mark.gap = kFirstGap;

  uint32_t ci = 0u;            // the child on the given side of the centre,
  float tc_min, tc_max, half;  // its slab and half size
  auto slab = [&](uint32_t bx, uint32_t by, uint32_t bz) {
    ci = shift_in(shift_in(bx >> 31, by), bz);
    half = __fmul_rn(sx2, 0.5f);
    // child centre (-0.5 + b) * sx2 + c = c +- half; faces ccx -+ half
    const float ccx = __fadd_rn(with_side(bx, half), cx);
    const float ccy = __fadd_rn(with_side(by, half), cy);
    const float ccz = __fadd_rn(with_side(bz, half), cz);
    float tx0 = __fadd_rn(__fmul_rn(r.rx, __fsub_rn(ccx, half)), r.px);
    float tx1 = __fadd_rn(__fmul_rn(r.rx, __fadd_rn(ccx, half)), r.px);
    if (tx0 > tx1) {
      const float s = tx0;
      tx0 = tx1;
      tx1 = s;
    }
    float ty0 = __fadd_rn(__fmul_rn(r.ry, __fsub_rn(ccy, half)), r.py);
    float ty1 = __fadd_rn(__fmul_rn(r.ry, __fadd_rn(ccy, half)), r.py);
    if (ty0 > ty1) {
      const float s = ty0;
      ty0 = ty1;
      ty1 = s;
    }
    float tz0 = __fadd_rn(__fmul_rn(r.rz, __fsub_rn(ccz, half)), r.pz);
    float tz1 = __fadd_rn(__fmul_rn(r.rz, __fadd_rn(ccz, half)), r.pz);
    if (tz0 > tz1) {
      const float s = tz0;
      tz0 = tz1;
      tz1 = s;
    }
    tc_min = cl_max(tx0, cl_max(ty0, tz0));
    tc_max = cl_min(tx1, cl_min(ty1, tz1));
  };
  auto push = [&](uint32_t bx, uint32_t by, uint32_t bz) {
    *sp = make_uint2(node, __float_as_uint(tmax));
    sp += stride;
    node = (kFlat ? 0u : node) + nd.x + __popc(nd.y & ((0x100u << ci) - 0x100u));
    in_pool = node <= last_node;
    if (in_pool) nd = fetch(node);
    tmax = tc_max;
    cx = __fadd_rn(with_side(bx, half), cx);
    cy = __fadd_rn(with_side(by, half), cy);
    cz = __fadd_rn(with_side(bz, half), cz);
    sx2 = half;
  };
  // the frames above the given one: a frame's interval end depends only on its
  // box and the ray, so they are pushed again from the root
  while (sx2 != from.sx2) {
    const uint32_t bx = above(from.cx, cx), by = above(from.cy, cy), bz = above(from.cz, cz);
    slab(bx, by, bz);
    push(bx, by, bz);
  }

  auto capped = [&]() {
    h.flags = SVO_HITFLAG_CAPPED;
    h.loops = loops;
    h.fetches = fetches;
    h.tc_min = tmin;
    if (!kFlat) {  // sample() reports the current node as a hit (:268-277)
      h.hit = 1u;
      h.node = node;
      h.depth = level_of(sx2);
      h.t = tmin;
      h.cx = cx;
      h.cy = cy;
      h.cz = cz;
      // quality = scale_exp2 - tScaleRatio * tMin, as for a leaf
      h.sx2 = sx2;
      h.leaf = 1u;
    }
  };

  bool pop = interval_done<kFlat>(tmin, tmax);  // whether the next iteration pops
  for (;;) {                                    // ends by a return
    ++loops;
    if (loops >= check_at) {
      if (loops >= max_loops) {
        capped();
        return;
      }
      // The state at the start of an iteration is the frame's node, size and
      // tMin and the stacked frames.  Once that state recurs, the ray repeats
      // the same iterations with period p until the watchdog, so whole periods
      // are skipped (loop and fetch counts advanced by them) and the
      // iterations left run as usual: the watchdog then stops the ray in the
      // state, and with the counts, the reference reaches.  Every iteration is
      // compared with a saved state, which is replaced after 32, 64, 128, ...
      // of them (Brent's cycle search); check_at = loops + 1 keeps a pass to one
      // iteration meanwhile.
      const uint32_t depth = level_of(sx2) - 1u;
      bool same = mark.loops != 0u && mark.node == node && mark.size == __float_as_uint(sx2) &&
                  mark.tmin == __float_as_uint(tmin);
      for (uint32_t j = 0; same && j < depth; ++j) {
        const uint2 a = stack[j * stride];
        same = a.x == mark.stack[2 * j] && a.y == mark.stack[2 * j + 1];
      }
      if (same) {
        const uint32_t period = loops - mark.loops;
        const uint32_t skip = (max_loops - loops) / period;
        fetches += skip * (fetches - mark.fetches);
        loops += skip * period;
        check_at = max_loops;
        if (loops == max_loops) {
          capped();
          return;
        }
      } else {
        if (loops >= mark.next_save) {
          mark.node = node;
          mark.size = __float_as_uint(sx2);
          mark.tmin = __float_as_uint(tmin);
          mark.loops = loops;
          mark.fetches = fetches;
          mark.next_save = loops + mark.gap;
          mark.gap = 2u * mark.gap;
          for (uint32_t j = 0; j < depth; ++j) {
            const uint2 a = stack[j * stride];
            mark.stack[2 * j] = a.x;
            mark.stack[2 * j + 1] = a.y;
          }
        }
        check_at = loops + 1u;
      }
    }
    if (!pop) {
      // childEntryPoint = (o + (tMin + eps) d) - centre and its sign test
      const float te = __fadd_rn(tmin, eps);
      const uint32_t bx = above(__fadd_rn(r.ox, __fmul_rn(te, r.dx)), cx);
      const uint32_t by = above(__fadd_rn(r.oy, __fmul_rn(te, r.dy)), cy);
      const uint32_t bz = above(__fadd_rn(r.oz, __fmul_rn(te, r.dz)), cz);
      slab(bx, by, bz);
      if (!in_pool) {
        h.flags = SVO_HITFLAG_BOUNDS;
        h.loops = loops;
        h.fetches = fetches;
        return;
      }
      ++fetches;
      const uint32_t sh = nd.y >> ci;  // bit 8: valid, bit 0: leaf
      if (sh & 0x100u) {
        const bool leaf = sh & 1u;
        const bool lod = kFlat ? (__fmul_rn(r.tsr, tc_max) > sx2)
                               : (__fmul_rn(r.tsr, tc_min) > sx2 || sx2 == sx2_last);
        if (leaf || lod) {
          h.hit = 1u;
          h.node = (kFlat ? 0u : node) + nd.x + __popc(nd.y & ((0x100u << ci) - 0x100u));
          h.depth = (leaf || kFlat) ? level_of(sx2) : level_of(sx2) + 1u;
          h.t = tmin;
          h.loops = loops;
          h.fetches = fetches;
          h.tc_min = tc_min;
          h.sx2 = sx2;
          h.leaf = leaf ? 1u : 0u;
          h.cx = __fadd_rn(with_side(bx, half), cx);
          h.cy = __fadd_rn(with_side(by, half), cy);
          h.cz = __fadd_rn(with_side(bz, half), cz);
          return;
        }
        if (kFlat && sx2 == sx2_last) {  // non-leaf below the octree's depth: corrupt pool
          h.flags = SVO_HITFLAG_BOUNDS;
          h.loops = loops;
          h.fetches = fetches;
          return;
        }
        // the current frame's tMin becomes tc_max (recovered on pop)
        push(bx, by, bz);
        tmin = tc_min;
      } else {
        tmin = tc_max;  // advance to the next sibling
      }
      pop = interval_done<kFlat>(tmin, tmax);
      if (!pop || loops + 1u >= check_at) continue;
      ++loops;
    }
    for (;;) {  // one level a turn; each is one iteration of the reference
      if (sx2 == 0.5f) {  // above the root: the ray leaves the octree
        ray_missed(kFlat, r, loops, fetches, h);
        return;
      }
      sp -= stride;
      tmin = tmax;
      tmax = __uint_as_float(sp->y);
      sx2 = __fmul_rn(sx2, 2.0f);
      pop = interval_done<kFlat>(tmin, tmax);
      if (!pop || loops + 1u >= check_at) break;
      ++loops;
    }
    // a stacked node passed the in-pool test before its children were tested
    node = sp->x;
    in_pool = true;
    nd = fetch(node);
    const uint32_t one = __float_as_uint(__fadd_rn(1.0f, sx2));
    const uint32_t keep = 0x7f000000u - 2u * one;
    cx = ancestor_center(cx, one, keep);
    cy = ancestor_center(cy, one, keep);
    cz = ancestor_center(cz, one, keep);
  }
}

// The descent of a ray with finite reciprocals, until it ends (true), or until
// it has run `limit` passes or is seen not to advance (false: `st` holds where
// it stands).
// kFlat selects the CpuRaycasterSingleRay3 rules; S is the stack size
// (treelet) or the octree depth (flat).  `stack` points at this thread's column
// of the shared-memory stack, `stride` words apart.
//
// A pass of the loop is one child test of the reference and every pop that
// follows it.  A warp whose lanes each spend a pass on a single pop runs the
// test for the other lanes beside it: on the 1080p icosphere frame 21 of 32
// lanes took part in an average test and 11 in an average pop, and a pop took
// 1.8 turns.  With the pops behind the test the frame takes 1.35 M warp passes
// instead of 1.91 M, and 27 lanes take part in a test.  The loop is bound by
// instruction issue where warps fill the GPU (a 3840x2160 primary + shadow frame
// 1738 -> 1248 us, a million explicit rays 573 -> 446 us against one event a
// pass) and by the chain of its longest ray elsewhere (a 1920x1080 frame 283 ->
// 225 us, 641x479 with hit records 82 -> 55 us).  What the loop keeps per level
// was chosen for few instructions and 48 registers (10 blocks of 128 threads an
// SM; 55 and 9 before): no lattice coordinates, no test counter beside the pass
// counter, no in-pool flag.
//
// A child that ends where its parent does -- it leaves through the same plane,
// so the two tMax have the same bits -- is popped together with it, so the
// parent is not stacked: popping the child goes to the nearest ancestor that
// ends later, in one stack read.  `open` has the bit of weight sx2 set for each
// stacked frame (over the exponent bits of 1.0f, so that a bit and those are
// the float 1 + sx2); the level it names gives the size, the centre
// (ancestor_center) and the number of iterations the pops count as.
//
// A few rays of a frame never end: they advance in place, or repeat a short
// cycle of pushes and pops, until the watchdog stops them at (S+1)^2*5
// iterations.  tMin grows along every other ray, so a ray whose tMin has not
// grown over kProgressPasses passes leaves for descend_general, which looks for
// the cycle and skips it.  (The lanes of a warp begin together and a pass is
// one test for each, so they all look in the same pass.)
//
// The reference orders each child's slab distances with a compare and swap
// (tx0 > tx1).  When the reciprocal r is finite, rounding is monotone, so the
// swap happens exactly when r < 0 (equal values swap to themselves): the near
// face is lo when r > 0 and hi when r < 0.  A child's two faces along an axis
// are the parent's mid plane c and its outer face c +- sx2 (exact dyadic
// numbers, the values the reference's childCenter +- childSizeHalf produce), so
// each axis costs the distance to the mid plane, the distance to the outer
// face and the max of the two (the far face); the min (the near face) is taken
// only for a valid child, the one case that reads tcMin.  There is no NaN and
// no -0 among the distances (see cast_ray), so the hardware min/max give the
// reference's order bit for bit.
//
// With kYield the ray goes on from `w` and the loop also ends (kYields, with the
// ray in `w` again) once no more than `keep` lanes of the warp are still in it.
// It is asked behind a pass, never before the first one: every call moves its ray
// on by a pass or ends it, however few lanes run together, so a caller that calls
// again until its rays have ended comes to an end.  (A million rays without order
// 320 us when asked ahead of each pass, the first one too; 315 us behind it; 331 us
// ahead of each but the first.)
constexpr uint32_t kProgressPasses = 32;
enum Outcome { kEnded, kLeaves, kYields };

// A ray between two passes of the loop.
struct Descent {
  uint32_t node;
  float tmin, tmax, cx, cy, cz, sx2;
  uint2 nd;
  uint32_t passes, pops, check_at;
  float seen;
  uint32_t open;
  uint2* sp;
};

template <class Fetch>
__device__ __forceinline__ Descent descent_start(const Fetch& fetch, uint64_t num_nodes,
                                                 const Ray& r, float t_min, uint32_t limit,
                                                 uint2* stack) {
  Descent w;
  w.node = 0u;
  w.tmin = t_min;
  w.tmax = r.t_max;
  w.cx = w.cy = w.cz = 0.0f;
  w.sx2 = 0.5f;
  w.nd = num_nodes ? fetch(0u) : make_uint2(0u, 0xFFFFu);
  w.passes = w.pops = 0u;
  w.check_at = kProgressPasses < limit ? kProgressPasses : limit;
  w.seen = t_min;
  w.open = 0x3f800000u;
  w.sp = stack;
  return w;
}

template <bool kFlat, bool kYield, class Fetch>
__device__ __forceinline__ Outcome descend(const Fetch& fetch, uint64_t num_nodes, const Ray& r,
                                           int S, uint2* stack, int stride, uint32_t limit,
                                           int keep, Descent& w, RayState& st, RayHit& h) {
  // Packed x and y take the issue slots of one: 1920x1080 icosphere 224 -> 214 us,
  // 3840x2160 726 -> 703, with shadow rays 1227 -> 1211, 48 batched views 983 -> 923,
  // 1920x1080 flat pool 176 -> 170.  Lanes that take further rays have no registers
  // left for aligned pairs (320 -> 329 us with them).
  constexpr bool kPairs = !kYield;
  const float eps = 0.00001f;
  const float sx2_last = last_size<kFlat>(S);
  // Pools hold at most 2^32 nodes, so the in-pool test of a 32-bit index is one
  // compare against the last index.  A node outside gets a record of valid
  // leaves only: its test then ends the ray, where the index is looked at again.
  const uint32_t last_node = num_nodes ? (uint32_t)(num_nodes - 1u) : 0u;
  constexpr uint32_t kOne = 0x3f800000u;
  if (!kYield) w = descent_start(fetch, num_nodes, r, st.tmin, limit, stack);
  uint32_t node = w.node;
  float tmin = w.tmin, tmax = w.tmax;
  float cx = w.cx, cy = w.cy, cz = w.cz;
  float sx2 = w.sx2;
  uint2 nd = w.nd;
  uint32_t passes = w.passes, pops = w.pops;  // tests (the reference's fetches), popped levels
  uint32_t check_at = w.check_at;
  float seen = w.seen;  // tMin when it was last looked at
  uint32_t open = w.open;
  uint2* sp = w.sp;  // the next free stack word
  if (passes == 0u && interval_done<kFlat>(tmin, tmax)) {
    ray_missed(kFlat, r, 1u, 0u, h);
    return kEnded;
  }
  for (;;) {
    if (passes == check_at) {
      if (passes == limit || tmin <= seen) break;
      seen = tmin;
      check_at = check_at + kProgressPasses < limit ? check_at + kProgressPasses : limit;
    }
    ++passes;
    // childEntryPoint = (o + (tMin + eps) d) - centre and its sign test
    const float te = __fadd_rn(tmin, eps);
    uint32_t bx, by;
    float mx, my, ox, oy;  // the distances to the mid planes and the outer faces
    float fx = 0.0f, fy = 0.0f;
    Pair cxy, fxy;
    if (kPairs) {  // x and y in packed instructions, z beside them
      cxy = pair_of(cx, cy);
      const Pair rxy = pair_of(r.rx, r.ry), pxy = pair_of(r.px, r.py);
      float ux, uy;
      halves(pair_sub_from(pair_mul_add(pair_of(te, te), pair_of(r.dx, r.dy), pair_of(r.ox, r.oy)), cxy), ux, uy);
      bx = __float_as_uint(ux);
      by = __float_as_uint(uy);
      halves(pair_mul_add(rxy, cxy, pxy), mx, my);
      fxy = pair_add(cxy, pair_of(with_side(bx, sx2), with_side(by, sx2)));
      halves(pair_mul_add(rxy, fxy, pxy), ox, oy);
    } else {
      bx = above(__fadd_rn(r.ox, __fmul_rn(te, r.dx)), cx);
      by = above(__fadd_rn(r.oy, __fmul_rn(te, r.dy)), cy);
      mx = __fadd_rn(__fmul_rn(r.rx, cx), r.px);
      my = __fadd_rn(__fmul_rn(r.ry, cy), r.py);
      fx = __fadd_rn(cx, with_side(bx, sx2));
      fy = __fadd_rn(cy, with_side(by, sx2));
      ox = __fadd_rn(__fmul_rn(r.rx, fx), r.px);
      oy = __fadd_rn(__fmul_rn(r.ry, fy), r.py);
    }
    const uint32_t bz = above(__fadd_rn(r.oz, __fmul_rn(te, r.dz)), cz);
    const float mz = __fadd_rn(__fmul_rn(r.rz, cz), r.pz);
    const float fz = __fadd_rn(cz, with_side(bz, sx2));
    const float oz = __fadd_rn(__fmul_rn(r.rz, fz), r.pz);
    const float tc_max = fminf(fmaxf(mx, ox), fminf(fmaxf(my, oy), fmaxf(mz, oz)));
    const uint32_t ci = shift_in(shift_in(bx >> 31, by), bz);
    const uint32_t masks = nd.y;
    const uint32_t sh = masks >> ci;  // bit 8: valid, bit 0: leaf
    if (sh & 0x100u) {
      const float tc_min = fmaxf(fminf(mx, ox), fmaxf(fminf(my, oy), fminf(mz, oz)));
      const float half = __fmul_rn(sx2, 0.5f);
      const uint32_t below = __popc(masks & valid_below(ci));
      const uint32_t child = (kFlat ? 0u : node) + nd.x + below;
      const bool leaf = sh & 1u;
      const bool lod = kFlat ? (__fmul_rn(r.tsr, tc_max) > sx2)
                             : (__fmul_rn(r.tsr, tc_min) > sx2 || sx2 == sx2_last);
      if (leaf || lod || (kFlat && sx2 == sx2_last)) {
        h.loops = passes + pops;
        h.fetches = passes;
        if (node > last_node || num_nodes == 0u) {  // the frame's node is outside the pool
          h.flags = SVO_HITFLAG_BOUNDS;
          h.fetches = passes - 1u;
          return kEnded;
        }
        if (kFlat && !leaf && !lod) {  // non-leaf below the octree's depth: corrupt pool
          h.flags = SVO_HITFLAG_BOUNDS;
          return kEnded;
        }
        h.hit = 1u;
        h.node = child;
        h.depth = (leaf || kFlat) ? level_of(sx2) : level_of(sx2) + 1u;
        h.t = tmin;
        h.tc_min = tc_min;
        h.sx2 = sx2;
        h.leaf = leaf ? 1u : 0u;
        h.cx = __fadd_rn(with_side(bx, half), cx);
        h.cy = __fadd_rn(with_side(by, half), cy);
        h.cz = __fadd_rn(with_side(bz, half), cz);
        return kEnded;
      }
      // push: the current frame's tMin becomes tc_max (recovered on pop)
      if (tc_max != tmax) {
        *sp = make_uint2(node, __float_as_uint(tmax));
        sp += stride;
        open |= __float_as_uint(__fadd_rn(1.0f, sx2));
      }
      node = child;
      nd = make_uint2(0u, 0xFFFFu);
      if (node <= last_node) nd = fetch(node);
      tmin = tc_min;
      tmax = tc_max;
      // the child's centre, between its faces (exact): an add and a multiply, not
      // a select and an add, as the selects' pipe is the busier one (a 3840x2160
      // frame 770 -> 726 us, 48 batched views 1010 -> 960 us with the mask below)
      if (kPairs) {
        halves(pair_mul(pair_add(cxy, fxy), pair_of(0.5f, 0.5f)), cx, cy);
      } else {
        cx = __fmul_rn(__fadd_rn(cx, fx), 0.5f);
        cy = __fmul_rn(__fadd_rn(cy, fy), 0.5f);
      }
      cz = __fmul_rn(__fadd_rn(cz, fz), 0.5f);
      sx2 = half;
    } else {
      tmin = tc_max;  // advance to the next sibling
    }
    if (interval_done<kFlat>(tmin, tmax)) {
      uint32_t bit;
      do {
        if (open == kOne) {  // above the root: the ray leaves the octree
          ray_missed(kFlat, r, passes + pops + level_of(sx2), passes, h);
          return kEnded;
        }
        sp -= stride;
        const uint2 e = *sp;
        tmin = tmax;
        node = e.x;
        tmax = __uint_as_float(e.y);
        bit = open & (0u - open);
        open ^= bit;
      } while (interval_done<kFlat>(tmin, tmax));
      // a stacked node passed the in-pool test before its children were tested
      nd = fetch(node);
      const uint32_t one = kOne | bit;
      const uint32_t keep = 0u - 2u * bit;
      if (kPairs) {
        halves(ancestor_centers(pair_of(cx, cy), one, keep), cx, cy);
      } else {
        cx = ancestor_center(cx, one, keep);
        cy = ancestor_center(cy, one, keep);
      }
      cz = ancestor_center(cz, one, keep);
      const float size = __fadd_rn(__uint_as_float(one), -1.0f);
      pops += (__float_as_uint(size) - __float_as_uint(sx2)) >> 23;
      sx2 = size;
    }
    if (kYield && lanes_together() <= keep) {
      w = Descent{node, tmin, tmax, cx, cy, cz, sx2, nd, passes, pops, check_at, seen, open, sp};
      return kYields;
    }
  }
  st = RayState{node, tmin, tmax, cx, cy, cz, sx2, passes + pops, passes};
  return kLeaves;
}

// The ray set up against the root box: kMissesBox, kFast where `descend` can
// take it, else kGeneral.
enum RayKind { kMissesBox, kFast, kGeneral };
template <bool kFlat>
__device__ __forceinline__ RayKind setup_ray(const float o[3], float dx, float dy, float dz,
                                             float tsr, Ray& r, float& t_min, RayHit& h) {
  h = no_hit();
  float t_max;
  {
    const float d0[3] = {dx, dy, dz};
    if (!root_slab(o, d0, t_min, t_max)) {
      h.flags = SVO_HITFLAG_BOXMISS;
      return kMissesBox;
    }
  }
  h.t_enter = t_min;
  h.t_exit = t_max;
  // Direction clamp: sample() replaces |d| < 1e-4 by 1e-4 * sign(d)
  // (:231-239); traversSvo replaces |d| < 1e-5 by 1e-5 * sign(d) * 10 (:184-186).
  if (kFlat) {
    const float eps = 0.00001f;
    if (fabsf(dx) < eps) dx = __fmul_rn(__fmul_rn(eps, cl_sign(dx)), 10.0f);
    if (fabsf(dy) < eps) dy = __fmul_rn(__fmul_rn(eps, cl_sign(dy)), 10.0f);
    if (fabsf(dz) < eps) dz = __fmul_rn(__fmul_rn(eps, cl_sign(dz)), 10.0f);
  } else {
    const float mn = 0.0001f;
    if (fabsf(dx) < mn) dx = __fmul_rn(mn, cl_sign(dx));
    if (fabsf(dy) < mn) dy = __fmul_rn(mn, cl_sign(dy));
    if (fabsf(dz) < mn) dz = __fmul_rn(mn, cl_sign(dz));
  }
  r.ox = o[0];
  r.oy = o[1];
  r.oz = o[2];
  r.dx = dx;
  r.dy = dy;
  r.dz = dz;
  r.rx = __frcp_rn(dx);
  r.ry = __frcp_rn(dy);
  r.rz = __frcp_rn(dz);
  r.px = __fmul_rn(-o[0], r.rx);
  r.py = __fmul_rn(-o[1], r.ry);
  r.pz = __fmul_rn(-o[2], r.rz);
  r.t_max = t_max;
  r.tsr = tsr;
  // `descend` needs finite 1 / d and -o / d (the second is finite only with the
  // first, and with a finite origin), so that no slab distance is a NaN.  It
  // also takes the hardware min/max: a distance r * plane + p is -0 only for
  // the plane at 0 when the origin coordinate is -0 and r < 0 (x + (-x) rounds
  // to +0), so rays with a -0 origin coordinate keep the compare/select.
  const bool neg_zero = __float_as_uint(o[0]) == 0x80000000u ||
                        __float_as_uint(o[1]) == 0x80000000u ||
                        __float_as_uint(o[2]) == 0x80000000u;
  return isfinite(r.px) && isfinite(r.py) && isfinite(r.pz) && !neg_zero ? kFast : kGeneral;
}

// Passes of the fast loop: n passes are n tests, at most as many pushes, and so
// at most n pops plus the root's, so below this many no ray comes to the watchdog.
__device__ __forceinline__ uint32_t pass_limit(int S) {
  return ((uint32_t)((S + 1) * (S + 1) * 5) - 2u) / 2u;
}

// One ray: root box test, direction clamp, then the descent.  pass_cap > 0
// stops the ray after that many child tests instead of the watchdog's
// (S+1)^2*5 iterations (used only to estimate costs; results under a cap are
// not the reference's: h.tc_min is how far the ray has come).
template <bool kFlat, class Fetch>
__device__ __forceinline__ RayHit cast_ray(const Fetch& fetch, uint64_t num_nodes,
                                           const float o[3], float dx, float dy, float dz,
                                           float tsr, int S, uint2* stack, int stride,
                                           uint32_t pass_cap = 0u) {
  RayHit h;
  Ray r;
  float t_min = 0.0f;
  const RayKind kind = setup_ray<kFlat>(o, dx, dy, dz, tsr, r, t_min, h);
  if (kind == kMissesBox) return h;
  RayState st = {0u, t_min, r.t_max, 0.0f, 0.0f, 0.0f, 0.5f, 0u, 0u};
  Descent w;
  if (kind == kFast) {
    if (pass_cap) {
      if (descend<kFlat, false>(fetch, num_nodes, r, S, stack, stride, pass_cap, 0, w, st, h) != kEnded) {
        h.flags = SVO_HITFLAG_CAPPED;
        h.loops = st.loops;
        h.tc_min = st.tmin;
      }
      return h;
    }
    if (descend<kFlat, false>(fetch, num_nodes, r, S, stack, stride, pass_limit(S), 0, w, st, h) == kEnded)
      return h;
  }
  descend_general<kFlat>(fetch, num_nodes, r, S, stack, stride, st, h, pass_cap);
  return h;
}

}  // namespace svo
