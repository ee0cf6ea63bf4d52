// gpu_builder.cu -- mesh -> octree -> treelets -> fully resident incore pool,
// on the GPU.
//
// The same scene the host builder produces (csrc/scene.cpp:
// build_mesh_leaves, octree_from_leaves, cut_treelets) followed by
// TreeletMemoryManager::insert_all (csrc/memory_manager.cpp), bit for bit,
// for the scale of the largest configuration (about 10^9 leaves), where the
// host path would need tens of GB of host memory and hours of CPU time.  It
// stands in for the reference's TreeletBuilderFromFaces::buildFromQueue
// (src/TreeletBuilderFromFaces.cpp:189-365), TreeletBuildManager
// (src/TreeletBuildManager.cpp:150-258) and the insertion loop of
// TreeletMemoryManager (src/TreeletMemoryManager.cpp:518-545).
//
// Pipeline, all in device memory:
//  1. per-triangle records: what a leaf needs of a triangle that does not depend
//     on the voxel (the interpolation's vectors, or the face normal);
//  2. voxelisation: one thread per column of voxels along a triangle's dominant
//     normal axis, walked exactly like the host builder with the separating-axis
//     triangle/box test; the columns of all triangles are numbered one after
//     another, so a triangle of two voxels and one of a thousand fill the GPU
//     alike.  A first pass keeps each column's hits as a mask, a second writes
//     the overlaps as 64-bit keys (code << tri_bits | triangle), triangles
//     ascending;
//  3. a stable radix sort of the keys by code (CUB), so equal codes are grouped
//     with their triangles ascending;
//  4. the octree from the sorted keys in two passes: where a key differs from the
//     one before it says which levels begin a node there, so one count per block
//     and level, and one pass that writes every level's first children and each
//     leaf's attributes (summed over its triangles in order, as the host does);
//  5. attributes of the inner levels bottom-up, one thread per parent over its
//     <= 8 children;
//  6. the treelet cut in closed form: treelet boundaries sit on fixed levels
//     (stop_level), each treelet is the breadth-first fill of its root's
//     subtree down to the next boundary, so its nodes at a level are one
//     contiguous range of that level, its local positions are range offsets,
//     and the treelet ids are range offsets of the boundary levels; one block
//     per treelet writes its slot, with every sub-treelet root patched into
//     its parent's leaf as insert_all does.
// Octrees whose keys would not fit 64 bits, whose columns number more than
// kMaxColumns or whose scratch does not fit run 2 to 4 once per spatial chunk: cells
// of the top levels, split further where one has too much (for_each_chunk), and
// chunks that still have too many columns are walked pass by pass.
//
// Scratch comes from a stream-ordered memory pool of the library's own; the host
// waits three times a chunk for a size, and once more for the slots' size.  An
// 81,920-triangle icosphere at depth 11 (13 M leaves, 17.3 M nodes, a 628 MB pool)
// takes 3.2 ms while another scene keeps scratch and a destroyed scene's pool on the
// device (kept_memory.h), 5.5 ms with no other scene alive (69 before the columns);
// a 131,072-triangle terrain at depth 9 0.9 and 1.7 ms (20); the first build of a
// process 13 ms (25); the 5.2 M-triangle depth-14 octree 0.70 s (1.61).  A triangle
// takes 228 bytes of scratch with vertex attributes, 112 without, a column 4 and an
// overlap 16: 1.0 GB at the peak for the icosphere, its pool among it (0.8 before),
// 2.1 GB for a depth-12 terrain with a 1.2 GB pool (1.5).
//
// FP32 arithmetic uses explicit round-to-nearest intrinsics in the host
// builder's operation order (the library is built with -fmad=false), so the
// attributes and the voxel sets match the host builder's bit for bit.
#include <cuda_runtime.h>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cstdint>
#include <utility>
#include <vector>

#include "../../include/libsvo_b200.h"
#include "chunk_plan.h"
#include "errors.h"
#include "gpu_builder.h"
#include "kept_memory.h"

namespace svo {

namespace {

// ---- shared arithmetic (host builder: csrc/scene.cpp) ----------------------

__device__ __forceinline__ float smin(float a, float b) { return (b < a) ? b : a; }  // std::min
__device__ __forceinline__ float smax(float a, float b) { return (a < b) ? b : a; }  // std::max

__device__ __forceinline__ uint64_t split3(uint32_t a) {
  uint64_t x = a & 0x1fffffu;
  x = (x | x << 32) & 0x1f00000000ffffull;
  x = (x | x << 16) & 0x1f0000ff0000ffull;
  x = (x | x << 8) & 0x100f00f00f00f00full;
  x = (x | x << 4) & 0x10c30c30c30c30c3ull;
  x = (x | x << 2) & 0x1249249249249249ull;
  return x;
}
__device__ __forceinline__ uint64_t morton3(uint32_t x, uint32_t y, uint32_t z) {
  return (split3(x) << 2) | (split3(y) << 1) | split3(z);
}

__device__ __forceinline__ uint32_t unorm8(float c) {
  if (!(c > 0.0f)) return 0u;
  if (c >= 1.0f) return 255u;
  return __float2uint_rz(__fadd_rn(__fmul_rn(c, 255.0f), 0.5f));
}
__device__ __forceinline__ uint32_t pack_color(float r, float g, float b) {
  return (unorm8(r) << 24) | (unorm8(g) << 16) | (unorm8(b) << 8) | 255u;
}
__device__ __forceinline__ uint32_t pack_normal(float x, float y, float z) {
  return pack_color(__fadd_rn(__fmul_rn(x, 0.5f), 0.5f), __fadd_rn(__fmul_rn(y, 0.5f), 0.5f),
                    __fadd_rn(__fmul_rn(z, 0.5f), 0.5f));
}
__device__ __forceinline__ float len3(float x, float y, float z) {
  return __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z)));
}

// cell_floor of the host builder: floor(x) clamped to [-2, R + 1], NaN -> -2.
__device__ __forceinline__ int cell_floor(float x, uint32_t R) {
  const float hi = __fadd_rn((float)R, 1.0f);
  if (!(x >= -2.0f)) return -2;
  if (x > hi) return (int)R + 1;
  return __float2int_rz(floorf(x));
}

__device__ __forceinline__ float dot3(float ax, float ay, float az, const float v[3]) {
  return __fadd_rn(__fadd_rn(__fmul_rn(ax, v[0]), __fmul_rn(ay, v[1])), __fmul_rn(az, v[2]));
}

// ---- 1. triangle records -------------------------------------------------------

__device__ __forceinline__ void face_normal(const float* a, const float* b, const float* c,
                                            float n[3]) {
  n[0] = __fsub_rn(__fmul_rn(__fsub_rn(b[1], a[1]), __fsub_rn(c[2], a[2])),
                   __fmul_rn(__fsub_rn(b[2], a[2]), __fsub_rn(c[1], a[1])));
  n[1] = __fsub_rn(__fmul_rn(__fsub_rn(b[2], a[2]), __fsub_rn(c[0], a[0])),
                   __fmul_rn(__fsub_rn(b[0], a[0]), __fsub_rn(c[2], a[2])));
  n[2] = __fsub_rn(__fmul_rn(__fsub_rn(b[0], a[0]), __fsub_rn(c[1], a[1])),
                   __fmul_rn(__fsub_rn(b[1], a[1]), __fsub_rn(c[0], a[0])));
}

__global__ void face_normals_kernel(const float* __restrict__ V, const uint32_t* __restrict__ T,
                                    uint64_t nt, float* __restrict__ fn) {
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  float n[3];
  face_normal(V + 3 * (uint64_t)T[3 * t], V + 3 * (uint64_t)T[3 * t + 1],
              V + 3 * (uint64_t)T[3 * t + 2], n);
  const float len = len3(n[0], n[1], n[2]);
  if (len > 0.0f) {
    fn[3 * t] = __fdiv_rn(n[0], len);
    fn[3 * t + 1] = __fdiv_rn(n[1], len);
    fn[3 * t + 2] = __fdiv_rn(n[2], len);
  } else {
    fn[3 * t] = 0.0f;
    fn[3 * t + 1] = 0.0f;
    fn[3 * t + 2] = 1.0f;
  }
}

// The part of leaf_contribution (host builder, csrc/scene.cpp) that is the same
// for every voxel of a triangle: 128 bytes, read by each of the triangle's
// leaves (160 on average in the depth-11 icosphere) instead of computed there.
struct __align__(16) TriRecord {
  float p0[3], inv;   // vertex 0; 1 / det, 0 where the ray is parallel
  float pv[3], e1[3], d[3];
  float n0[3], n1[3], n2[3], c0[3], c1[3], c2[3];
  float hits;         // 1: the ray meets the plane, 0: u = v = 0
};
static_assert(sizeof(TriRecord) == 128, "eight 16-byte loads");

__global__ void tri_records_kernel(const float* __restrict__ V, const float* __restrict__ N,
                                   const float* __restrict__ C, const uint32_t* __restrict__ T,
                                   uint64_t nt, TriRecord* __restrict__ out) {
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  TriRecord r;
  float p1[3], p2[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const uint64_t i0 = 3 * (uint64_t)T[3 * t] + k, i1 = 3 * (uint64_t)T[3 * t + 1] + k,
                   i2 = 3 * (uint64_t)T[3 * t + 2] + k;
    r.p0[k] = V[i0];
    p1[k] = V[i1];
    p2[k] = V[i2];
    r.n0[k] = N[i0];
    r.n1[k] = N[i1];
    r.n2[k] = N[i2];
    r.c0[k] = C[i0];
    r.c1[k] = C[i1];
    r.c2[k] = C[i2];
    r.d[k] = __fdiv_rn(__fadd_rn(__fadd_rn(r.n0[k], r.n1[k]), r.n2[k]), 3.0f);
  }
  const float len = len3(r.d[0], r.d[1], r.d[2]);
  if (len > 0.0f) {
#pragma unroll
    for (int k = 0; k < 3; ++k) r.d[k] = __fdiv_rn(r.d[k], len);
  }
  float e2[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    r.e1[k] = __fsub_rn(p1[k], r.p0[k]);
    e2[k] = __fsub_rn(p2[k], r.p0[k]);
  }
  r.pv[0] = __fsub_rn(__fmul_rn(r.d[1], e2[2]), __fmul_rn(r.d[2], e2[1]));
  r.pv[1] = __fsub_rn(__fmul_rn(r.d[2], e2[0]), __fmul_rn(r.d[0], e2[2]));
  r.pv[2] = __fsub_rn(__fmul_rn(r.d[0], e2[1]), __fmul_rn(r.d[1], e2[0]));
  const float det = dot3(r.e1[0], r.e1[1], r.e1[2], r.pv);
  const bool hits = !(det > -1e-8f && det < 1e-8f);
  r.hits = hits ? 1.0f : 0.0f;
  r.inv = hits ? __fdiv_rn(1.0f, det) : 0.0f;
  out[t] = r;
}

// ---- 2. voxelisation ---------------------------------------------------------

struct Chunk {
  int lo[3], hi[3];    // voxel range of the chunk, inclusive
  uint32_t shift;      // 3 * (depth - chunk_levels): bits of a code inside the chunk
  uint32_t tri_bits;   // bits of the triangle index in a key
};

// A triangle as the voxeliser walks it: columns of voxels along axis w (the
// dominant one of its normal), iu in [ulo, ulo + nu), iv in [vlo, vlo + nv).  Its
// coordinates are kept in the order (u, v, w), a cyclic turn of (x, y, z).
struct __align__(16) TriWalk {
  float a[3], b[3], c[3], n[3], pd;  // pd: dot(n, a), in the order x, y, z
  int w, ulo, vlo, wlo, whi;
  uint32_t nv, pad;
};
static_assert(sizeof(TriWalk) == 80, "five 16-byte loads");

__device__ __forceinline__ float turned(const float* x, int w, int k) {  // k: 0 u, 1 v, 2 w
  const int i = k == 2 ? w : (k == 0 ? (w == 2 ? 0 : w + 1) : (w == 0 ? 2 : w - 1));
  return i == 0 ? x[0] : (i == 1 ? x[1] : x[2]);
}
__device__ __forceinline__ int turned(const int* x, int w, int k) {
  const int i = k == 2 ? w : (k == 0 ? (w == 2 ? 0 : w + 1) : (w == 0 ? 2 : w - 1));
  return i == 0 ? x[0] : (i == 1 ? x[1] : x[2]);
}

// Returns the number of columns with candidate voxels in the chunk.
__device__ __forceinline__ uint64_t tri_walk(const float* __restrict__ V,
                                             const uint32_t* __restrict__ T, uint64_t t,
                                             uint32_t depth, const Chunk& ch, TriWalk& s) {
  const uint32_t R = 1u << depth;
  const float Rf = (float)R;
  const uint64_t i0 = 3 * (uint64_t)T[3 * t], i1 = 3 * (uint64_t)T[3 * t + 1],
                 i2 = 3 * (uint64_t)T[3 * t + 2];
  const float a[3] = {V[i0], V[i0 + 1], V[i0 + 2]}, b[3] = {V[i1], V[i1 + 1], V[i1 + 2]},
              c[3] = {V[i2], V[i2 + 1], V[i2 + 2]};
  float n[3];
  face_normal(a, b, c, n);
  int lo[3], hi[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float mn = smin(a[k], smin(b[k], c[k]));
    const float mx = smax(a[k], smax(b[k], c[k]));
    lo[k] = max(0, cell_floor(__fmul_rn(__fadd_rn(mn, 0.5f), Rf), R));
    hi[k] = min((int)R - 1, cell_floor(__fmul_rn(__fadd_rn(mx, 0.5f), Rf), R));
  }
  int w = 0;
  if (fabsf(n[1]) > fabsf(n[0])) w = 1;
  if (fabsf(n[2]) > fabsf(w == 1 ? n[1] : n[0])) w = 2;
  s.w = w;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    s.a[k] = turned(a, w, k);
    s.b[k] = turned(b, w, k);
    s.c[k] = turned(c, w, k);
    s.n[k] = turned(n, w, k);
  }
  s.pd = dot3(n[0], n[1], n[2], a);
  // the chunk restricts the (u, v) range and each column's w range
  s.ulo = max(turned(lo, w, 0), turned(ch.lo, w, 0));
  s.vlo = max(turned(lo, w, 1), turned(ch.lo, w, 1));
  const int uhi = min(turned(hi, w, 0), turned(ch.hi, w, 0)), vhi = min(turned(hi, w, 1), turned(ch.hi, w, 1));
  s.wlo = turned(lo, w, 2);
  s.whi = turned(hi, w, 2);
  s.pad = 0;
  const bool none = lo[0] > hi[0] || lo[1] > hi[1] || lo[2] > hi[2] || s.ulo > uhi || s.vlo > vhi ||
                    max(s.wlo, turned(ch.lo, w, 2)) > min(s.whi, turned(ch.hi, w, 2));
  s.nv = none ? 0u : (uint32_t)(vhi - s.vlo + 1);
  return none ? 0ull : (uint64_t)(uint32_t)(uhi - s.ulo + 1) * s.nv;
}

// The candidate voxels of column (iu, iv), w from *wlo to *whi.
__device__ __forceinline__ void column_range(const TriWalk& s, uint32_t depth, const Chunk& ch,
                                             int iu, int iv, int* wlo, int* whi) {
  const uint32_t R = 1u << depth;
  const float Rf = (float)R;
  const float inv = __fdiv_rn(1.0f, Rf);
  *wlo = s.wlo;
  *whi = s.whi;
  if (s.n[2] != 0.0f) {
    const float u0 = __fadd_rn(-0.5f, __fmul_rn((float)iu, inv)), u1 = __fadd_rn(u0, inv);
    const float v0 = __fadd_rn(-0.5f, __fmul_rn((float)iv, inv)), v1 = __fadd_rn(v0, inv);
    float wmin = 1e30f, wmax = -1e30f;
    const float us[2] = {u0, u1}, vs[2] = {v0, v1};
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float ww = __fdiv_rn(
            __fsub_rn(__fsub_rn(s.pd, __fmul_rn(s.n[0], us[i])), __fmul_rn(s.n[1], vs[j])), s.n[2]);
        wmin = smin(wmin, ww);
        wmax = smax(wmax, ww);
      }
    *wlo = max(*wlo, cell_floor(__fmul_rn(__fadd_rn(wmin, 0.5f), Rf), R) - 1);
    *whi = min(*whi, cell_floor(__fmul_rn(__fadd_rn(wmax, 0.5f), Rf), R) + 1);
  }
  *wlo = max(*wlo, turned(ch.lo, s.w, 2));
  *whi = min(*whi, turned(ch.hi, s.w, 2));
}

// The host builder's tri_box_overlap (Akenine-Moeller 2001, restated there) in
// two parts.  A voxel overlaps when no axis separates it from the triangle, in
// whatever order the axes are tried, and the axes without a w component see the
// same values in every voxel of a column, bit for bit: they are tried once a
// column (half of the columns of a triangle's box end there), the others per
// voxel.  An axis is the cross product of an edge and a coordinate axis, so it
// has a zero and two components, whose products may be summed in any order; the
// zero's product is kept for coordinates that are not finite.
__device__ __forceinline__ bool separated(float s, float t, float p0s, float p0t, float p0z, float p1s,
                                          float p1t, float p1z, float p2s, float p2t, float p2z, float h) {
  const float p0 = __fadd_rn(__fadd_rn(__fmul_rn(s, p0s), __fmul_rn(t, p0t)), __fmul_rn(0.0f, p0z));
  const float p1 = __fadd_rn(__fadd_rn(__fmul_rn(s, p1s), __fmul_rn(t, p1t)), __fmul_rn(0.0f, p1z));
  const float p2 = __fadd_rn(__fadd_rn(__fmul_rn(s, p2s), __fmul_rn(t, p2t)), __fmul_rn(0.0f, p2z));
  const float mn = smin(p0, smin(p1, p2)), mx = smax(p0, smax(p1, p2));
  const float r = __fmul_rn(h, __fadd_rn(fabsf(s), fabsf(t)));
  return mn > r || mx < -r;
}

__device__ __forceinline__ float center_of(int i, float inv) {
  return __fadd_rn(-0.5f, __fmul_rn(__fadd_rn((float)i, 0.5f), inv));
}

__device__ __forceinline__ bool column_may_overlap(const TriWalk& s, uint32_t depth, int iu, int iv) {
  const float inv = __fdiv_rn(1.0f, (float)(1u << depth));
  const float h = __fmul_rn(0.5f, inv);
  const float bu = center_of(iu, inv), bv = center_of(iv, inv);
  const float u[3] = {__fsub_rn(s.a[0], bu), __fsub_rn(s.b[0], bu), __fsub_rn(s.c[0], bu)};
  const float v[3] = {__fsub_rn(s.a[1], bv), __fsub_rn(s.b[1], bv), __fsub_rn(s.c[1], bv)};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float eu = __fsub_rn(u[(k + 1) % 3], u[k]), ev = __fsub_rn(v[(k + 1) % 3], v[k]);
    if (separated(ev, -eu, u[0], v[0], s.a[2], u[1], v[1], s.b[2], u[2], v[2], s.c[2], h)) return false;
  }
  if (smin(u[0], smin(u[1], u[2])) > h || smax(u[0], smax(u[1], u[2])) < -h) return false;
  return !(smin(v[0], smin(v[1], v[2])) > h || smax(v[0], smax(v[1], v[2])) < -h);
}

// u, v and w products summed in the order x, y, z.
__device__ __forceinline__ float sum_xyz(float u, float v, float w, int axis) {
  const float x = axis == 0 ? w : (axis == 1 ? v : u), y = axis == 0 ? u : (axis == 1 ? w : v),
              z = axis == 0 ? v : (axis == 1 ? u : w);
  return __fadd_rn(__fadd_rn(x, y), z);
}

__device__ __forceinline__ bool voxel_overlaps(const TriWalk& s, uint32_t depth, int iu, int iv, int iw) {
  const float inv = __fdiv_rn(1.0f, (float)(1u << depth));
  const float h = __fmul_rn(0.5f, inv);
  const float bc[3] = {center_of(iu, inv), center_of(iv, inv), center_of(iw, inv)};
  float p[3][3];  // vertex, coordinate
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    p[0][k] = __fsub_rn(s.a[k], bc[k]);
    p[1][k] = __fsub_rn(s.b[k], bc[k]);
    p[2][k] = __fsub_rn(s.c[k], bc[k]);
  }
  if (smin(p[0][2], smin(p[1][2], p[2][2])) > h || smax(p[0][2], smax(p[1][2], p[2][2])) < -h) return false;
  float e[3][3];
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int i = 0; i < 3; ++i) e[k][i] = __fsub_rn(p[(k + 1) % 3][i], p[k][i]);
  float n[3], f[3], g[3], m[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int j = (i + 1) % 3, k = (i + 2) % 3;
    n[i] = __fsub_rn(__fmul_rn(e[0][j], e[1][k]), __fmul_rn(e[0][k], e[1][j]));
    f[i] = __fmul_rn(n[i], p[0][i]);
    g[i] = __fmul_rn(n[i], n[i] > 0.0f ? -h : h);
    m[i] = __fmul_rn(n[i], n[i] > 0.0f ? h : -h);
  }
  const float d = -sum_xyz(f[0], f[1], f[2], s.w);
  if (__fadd_rn(sum_xyz(g[0], g[1], g[2], s.w), d) > 0.0f) return false;
  if (!(__fadd_rn(sum_xyz(m[0], m[1], m[2], s.w), d) >= 0.0f)) return false;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (separated(e[k][2], -e[k][1], p[0][1], p[0][2], p[0][0], p[1][1], p[1][2], p[1][0], p[2][1], p[2][2],
                  p[2][0], h))
      return false;
    if (separated(e[k][0], -e[k][2], p[0][2], p[0][0], p[0][1], p[1][2], p[1][0], p[1][1], p[2][2], p[2][0],
                  p[2][1], h))
      return false;
  }
  return true;
}

__device__ __forceinline__ uint64_t voxel_code(int w, int iu, int iv, int iw) {
  const uint32_t x = (uint32_t)(w == 0 ? iw : (w == 1 ? iv : iu)), y = (uint32_t)(w == 0 ? iu : (w == 1 ? iw : iv)),
                 z = (uint32_t)(w == 0 ? iv : (w == 1 ? iu : iw));
  return morton3(x, y, z);
}

// walks[t], and cols[t]: the columns of triangle t inside the chunk; cols[nt] =
// 0, so that an exclusive sum over nt + 1 entries ends with the total.
__global__ void column_count_kernel(const float* __restrict__ V, const uint32_t* __restrict__ T,
                                    uint64_t nt, uint32_t depth, Chunk ch,
                                    TriWalk* __restrict__ walks, uint64_t* __restrict__ cols) {
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t > nt) return;
  if (t == nt) {
    cols[t] = 0;
    return;
  }
  TriWalk s;
  cols[t] = tri_walk(V, T, t, depth, ch, s);
  walks[t] = s;
}

// The last index of off[lo..hi] whose value is <= x (off[lo] <= x).
__device__ __forceinline__ uint64_t last_at_most(const uint64_t* __restrict__ off, uint64_t lo,
                                                 uint64_t hi, uint64_t x) {
  while (lo < hi) {
    const uint64_t mid = (lo + hi + 1) / 2;
    if (off[mid] <= x)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

constexpr int kColThreads = 256;

// The columns first .. first + count - 1 of a chunk, of one pass over them.
struct ColumnWindow {
  uint64_t first, count;
};

// A column's hits: bit i of the low byte for the voxel i above the first
// candidate, whose w is in the bits above; columns of more than eight candidates
// (a triangle without a dominant axis) are tested again where they are emitted.
constexpr uint32_t kTestAgain = 0xFFFFFFFFu;

// block_tri[b]: the triangle of the first column of block b, and of the last
// column behind the last block.  (Looked up by one thread of each block, the
// search was a third of the test and half of the emission.)
__global__ void block_triangles_kernel(const uint64_t* __restrict__ off, uint64_t nt, ColumnWindow win,
                                       uint64_t blocks, uint32_t* __restrict__ block_tri) {
  const uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (b <= blocks)
    block_tri[b] = (uint32_t)last_at_most(off, 0, nt - 1, win.first + min(b * kColThreads, win.count - 1));
}

// The triangle of column c, and the column's place (iu, iv) in it.
__device__ __forceinline__ uint64_t column_triangle(const uint64_t* __restrict__ off,
                                                    const uint32_t* __restrict__ block_tri, uint64_t c) {
  return last_at_most(off, block_tri[blockIdx.x], block_tri[blockIdx.x + 1], c);
}
__device__ __forceinline__ void column_place(const TriWalk& s, uint64_t k, int* iu, int* iv) {
  uint64_t row;
  if (k >> 32)  // a triangle of more than 2^32 columns
    row = k / s.nv;
  else
    row = (uint32_t)k / s.nv;
  *iu = s.ulo + (int)row;
  *iv = s.vlo + (int)(uint32_t)(k - row * s.nv);
}

__global__ void __launch_bounds__(kColThreads) column_test_kernel(
    const TriWalk* __restrict__ walks, uint32_t depth, Chunk ch,
    const uint64_t* __restrict__ off, const uint32_t* __restrict__ block_tri, ColumnWindow win,
    uint32_t* __restrict__ rec, uint64_t* __restrict__ block_hits) {
  const uint64_t i = (uint64_t)blockIdx.x * kColThreads + threadIdx.x, c = win.first + i;
  uint32_t hits = 0;
  if (i < win.count) {
    const uint64_t t = column_triangle(off, block_tri, c);
    const TriWalk s = walks[t];
    int iu, iv;
    column_place(s, c - off[t], &iu, &iv);
    int wlo = 0, whi = -1;
    uint32_t mask = 0;
    if (column_may_overlap(s, depth, iu, iv)) {
      column_range(s, depth, ch, iu, iv, &wlo, &whi);
      for (int iw = wlo; iw <= whi; ++iw)
        if (voxel_overlaps(s, depth, iu, iv, iw)) {
          ++hits;
          mask |= 1u << ((iw - wlo) & 31);
        }
    }
    rec[i] = hits == 0 ? 0u : (whi - wlo >= 8 ? kTestAgain : ((uint32_t)wlo << 8) | mask);
  }
  __shared__ uint32_t warp_hits[kColThreads / 32];
  const uint32_t sum = __reduce_add_sync(0xFFFFFFFFu, hits);
  if (threadIdx.x % 32 == 0) warp_hits[threadIdx.x / 32] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint64_t n = 0;
    for (int i = 0; i < kColThreads / 32; ++i) n += warp_hits[i];
    block_hits[blockIdx.x] = n;
    if (blockIdx.x == gridDim.x - 1) block_hits[gridDim.x] = 0;  // the sum's total lands here
  }
}

__global__ void __launch_bounds__(kColThreads) column_emit_kernel(
    const TriWalk* __restrict__ walks, uint32_t depth, Chunk ch,
    const uint64_t* __restrict__ off, const uint32_t* __restrict__ block_tri, ColumnWindow win,
    const uint32_t* __restrict__ rec,
    const uint64_t* __restrict__ block_off, uint64_t* __restrict__ keys) {
  const uint64_t i = (uint64_t)blockIdx.x * kColThreads + threadIdx.x, c = win.first + i;
  const uint32_t r = i < win.count ? rec[i] : 0u;
  uint64_t t = 0;
  int w = 0, iu = 0, iv = 0, wlo = 0, whi = -1;
  uint32_t n = 0;
  if (r != 0u) {
    t = column_triangle(off, block_tri, c);
    const TriWalk& s = walks[t];
    w = s.w;
    column_place(s, c - off[t], &iu, &iv);
    if (r == kTestAgain) {
      column_range(s, depth, ch, iu, iv, &wlo, &whi);
      for (int iw = wlo; iw <= whi; ++iw) n += voxel_overlaps(s, depth, iu, iv, iw) ? 1u : 0u;
    } else {
      wlo = (int)(r >> 8);
      n = (uint32_t)__popc(r & 0xFFu);
    }
  }
  // exclusive position inside the block
  __shared__ uint32_t warp_sum[kColThreads / 32];
  const uint32_t lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  uint32_t x = n;
  for (uint32_t d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, d);
    if (lane >= d) x += y;
  }
  if (lane == 31) warp_sum[warp] = x;
  __syncthreads();
  uint64_t pos = block_off[blockIdx.x] + (x - n);
  for (uint32_t i = 0; i < warp; ++i) pos += warp_sum[i];
  if (r == 0u) return;
  const uint64_t low = ch.shift >= 64 ? ~0ull : ((1ull << ch.shift) - 1ull);
  auto put = [&](int iw) { keys[pos++] = ((voxel_code(w, iu, iv, iw) & low) << ch.tri_bits) | t; };
  if (r == kTestAgain) {
    for (int iw = wlo; iw <= whi; ++iw)
      if (voxel_overlaps(walks[t], depth, iu, iv, iw)) put(iw);
  } else {
    for (uint32_t m = r & 0xFFu; m != 0u; m &= m - 1u) put(wlo + __ffs((int)m) - 1);
  }
}

// ---- 3. levels from the sorted keys ------------------------------------------------

constexpr int kMaxLevels = 22;

// The coarsest level that begins a node at key i: a node of level d holds the
// keys with the same leading d octal digits of their codes.  depth + 1 where
// the code is the one before (another triangle of the same voxel).
struct KeyLevels {
  const uint64_t* keys;
  uint64_t n;
  uint32_t tri_bits, depth;
  uint32_t first_level;  // at the chunk's first key
  __device__ __forceinline__ uint32_t operator()(uint64_t i) const {
    if (i >= n) return depth + 1u;
    if (i == 0) return first_level;
    const uint64_t diff = (keys[i] ^ keys[i - 1]) >> tri_bits;
    return diff == 0 ? depth + 1u : depth - (uint32_t)(63 - __clzll((long long)diff)) / 3u;
  }
};

constexpr int kKeyThreads = 256;
constexpr int kKeyRows = 4;  // a block takes 4 rows of 256 keys
constexpr int kKeyBlock = kKeyThreads * kKeyRows;

// counts[d * nblocks + block]: the nodes of level d that begin in the block.
__global__ void __launch_bounds__(kKeyThreads) level_count_kernel(KeyLevels kl, uint64_t nblocks,
                                                                  uint32_t* __restrict__ counts) {
  __shared__ uint32_t sums[kMaxLevels];
  if (threadIdx.x < kMaxLevels) sums[threadIdx.x] = 0;
  __syncthreads();
  uint32_t k[kKeyRows];
#pragma unroll
  for (int r = 0; r < kKeyRows; ++r)
    k[r] = kl((uint64_t)blockIdx.x * kKeyBlock + r * kKeyThreads + threadIdx.x);
  // few warps begin a node of the upper levels
  for (uint32_t d = __reduce_min_sync(0xFFFFFFFFu, min(min(k[0], k[1]), min(k[2], k[3]))); d <= kl.depth; ++d) {
    uint32_t n = 0;
#pragma unroll
    for (int r = 0; r < kKeyRows; ++r) n += (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, k[r] <= d));
    if (threadIdx.x % 32 == 0 && n) atomicAdd(&sums[d], n);
  }
  __syncthreads();
  if (threadIdx.x <= kl.depth) counts[threadIdx.x * nblocks + blockIdx.x] = sums[threadIdx.x];
}

// One block per level: counts become the level's node index at each key block,
// on from totals[level], which is advanced by the chunk's nodes.
__global__ void __launch_bounds__(1024) level_scan_kernel(uint32_t* __restrict__ counts,
                                                          uint64_t nblocks,
                                                          uint64_t* __restrict__ totals) {
  uint32_t* c = counts + (uint64_t)blockIdx.x * nblocks;
  __shared__ uint32_t warp_sum[32];
  __shared__ uint64_t carry;
  const uint32_t lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  if (threadIdx.x == 0) carry = totals[blockIdx.x];
  constexpr uint32_t kItems = 4;
  for (uint64_t base = 0; base < nblocks; base += 1024 * kItems) {
    uint32_t v[kItems], sum = 0;
    for (uint32_t k = 0; k < kItems; ++k) {
      const uint64_t i = base + threadIdx.x * kItems + k;
      v[k] = i < nblocks ? c[i] : 0u;
      sum += v[k];
    }
    uint32_t x = sum;
    for (uint32_t d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, d);
      if (lane >= d) x += y;
    }
    if (lane == 31) warp_sum[warp] = x;
    __syncthreads();
    if (warp == 0) {
      uint32_t y = warp_sum[lane];
      for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t z = __shfl_up_sync(0xFFFFFFFFu, y, d);
        if (lane >= d) y += z;
      }
      warp_sum[lane] = y;
    }
    __syncthreads();
    uint64_t at = carry + (warp ? warp_sum[warp - 1] : 0u) + (x - sum);
    for (uint32_t k = 0; k < kItems; ++k) {
      const uint64_t i = base + threadIdx.x * kItems + k;
      if (i < nblocks) c[i] = (uint32_t)at;  // below 2^32: the totals are looked at before use
      at += v[k];
    }
    __syncthreads();
    if (threadIdx.x == 0) carry += warp_sum[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// A chunk's part of the levels, indexed by a level's node index less base[level].
struct LevelOut {
  uint32_t* first[kMaxLevels];  // a node's first child; levels above the leaves
  uint8_t* octant[kMaxLevels];  // a node's place in its parent
  svo_attrib* leaf_attribs;
  uint32_t base[kMaxLevels];
};

__device__ __forceinline__ uint32_t compact3(uint64_t x) {
  x &= 0x1249249249249249ull;
  x = (x ^ (x >> 2)) & 0x10c30c30c30c30c3ull;
  x = (x ^ (x >> 4)) & 0x100f00f00f00f00full;
  x = (x ^ (x >> 8)) & 0x1f0000ff0000ffull;
  x = (x ^ (x >> 16)) & 0x1f00000000ffffull;
  x = (x ^ (x >> 32)) & 0x1fffffull;
  return (uint32_t)x;
}

// What the leaves' attributes are made of: face normals, or the triangles'
// records where the mesh has vertex normals and colours (records != nullptr).
struct LeafInput {
  const float* face_normals;
  const TriRecord* records;
  uint64_t chunk_base;  // the code bits above the key's
};

// The reference's interpolated vertex normal and colour of one triangle at the
// voxel centre c (leaf_contribution of the host builder, operation for
// operation; the voxel-independent part is in the record).
__device__ __forceinline__ void leaf_contribution(const TriRecord& r, const float c[3],
                                                  float n_out[3], float c_out[3]) {
  float u = 0.0f, v = 0.0f;
  if (r.hits != 0.0f) {
    const float tv[3] = {__fsub_rn(c[0], r.p0[0]), __fsub_rn(c[1], r.p0[1]),
                         __fsub_rn(c[2], r.p0[2])};
    u = __fmul_rn(dot3(tv[0], tv[1], tv[2], r.pv), r.inv);
    const float qv[3] = {__fsub_rn(__fmul_rn(tv[1], r.e1[2]), __fmul_rn(tv[2], r.e1[1])),
                         __fsub_rn(__fmul_rn(tv[2], r.e1[0]), __fmul_rn(tv[0], r.e1[2])),
                         __fsub_rn(__fmul_rn(tv[0], r.e1[1]), __fmul_rn(tv[1], r.e1[0]))};
    v = __fmul_rn(dot3(r.d[0], r.d[1], r.d[2], qv), r.inv);
  }
  u = u < 0.0f ? 0.0f : (u > 1.0f ? 1.0f : u);
  v = v < 0.0f ? 0.0f : (v > 1.0f ? 1.0f : v);
  const float w = __fsub_rn(__fsub_rn(1.0f, u), v);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    n_out[k] = __fadd_rn(__fadd_rn(__fmul_rn(r.n0[k], w), __fmul_rn(r.n1[k], u)), __fmul_rn(r.n2[k], v));
    c_out[k] = __fadd_rn(__fadd_rn(__fmul_rn(r.c0[k], w), __fmul_rn(r.c1[k], u)), __fmul_rn(r.c2[k], v));
  }
  const float len = len3(n_out[0], n_out[1], n_out[2]);
  if (len > 0.0f) {
#pragma unroll
    for (int k = 0; k < 3; ++k) n_out[k] = __fdiv_rn(n_out[k], len);
  }
}

// One triangle's contribution to the leaf `code`.
struct LeafPart {
  float n[3], c[3];
};
__device__ __forceinline__ LeafPart leaf_part(const LeafInput& in, uint32_t depth, uint64_t code,
                                              uint64_t t) {
  LeafPart p;
  if (in.records != nullptr) {
    const float inv = __fdiv_rn(1.0f, (float)(1u << depth));
    const float c[3] = {center_of((int)compact3(code >> 2), inv), center_of((int)compact3(code >> 1), inv),
                        center_of((int)compact3(code), inv)};
    leaf_contribution(in.records[t], c, p.n, p.c);
  } else {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      p.n[k] = in.face_normals[3 * t + k];
      p.c[k] = 0.0f;
    }
  }
  return p;
}

// The attributes of the leaf whose first key is i: over its triangles in order,
// the mean of the interpolated normals (normalised) and colours, or the
// normalised sum of the face normals.  The contributions of the keys up to `end`
// are in `part`; a run that crosses it has the others made here.
__device__ __forceinline__ svo_attrib leaf_attrib(const KeyLevels& kl, const LeafInput& in, uint64_t code,
                                                  uint64_t i, uint64_t end,
                                                  const LeafPart* __restrict__ part) {
  const uint64_t own = kl.keys[i] >> kl.tri_bits;
  float sn[3] = {0.0f, 0.0f, 0.0f}, sc[3] = {0.0f, 0.0f, 0.0f};
  uint64_t j = i;
  do {
    const LeafPart p = j < end ? part[kKeyThreads - (end - j)]
                               : leaf_part(in, kl.depth, code, kl.keys[j] & ((1ull << kl.tri_bits) - 1ull));
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      sn[k] = __fadd_rn(sn[k], p.n[k]);
      sc[k] = __fadd_rn(sc[k], p.c[k]);
    }
    ++j;
  } while (j < kl.n && (kl.keys[j] >> kl.tri_bits) == own);
  if (in.records != nullptr && j - i > 1) {  // x / 1 is x
    const float cnt = (float)(j - i);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      sn[k] = __fdiv_rn(sn[k], cnt);
      sc[k] = __fdiv_rn(sc[k], cnt);
    }
  }
  const float len = len3(sn[0], sn[1], sn[2]);
  if (len > 0.0f) {
#pragma unroll
    for (int k = 0; k < 3; ++k) sn[k] = __fdiv_rn(sn[k], len);
  } else {
    sn[0] = 0.0f;
    sn[1] = 0.0f;
    sn[2] = 1.0f;
  }
  const uint32_t normal = pack_normal(sn[0], sn[1], sn[2]);
  // without vertex colours, colour = normal * 0.5 + 0.5 = the packed normal
  return svo_attrib{normal, in.records != nullptr ? pack_color(sc[0], sc[1], sc[2]) : normal};
}

// Every level's nodes that begin in the block, and the leaves' attributes.
__global__ void __launch_bounds__(kKeyThreads) level_write_kernel(
    KeyLevels kl, LeafInput in, uint64_t nblocks, const uint32_t* __restrict__ counts, LevelOut out) {
  // before[d][g]: the nodes of level d that begin in the block ahead of group g
  // (a row's warp)
  constexpr int kGroups = kKeyRows * kKeyThreads / 32;
  static_assert(kGroups == 32, "one warp scans the groups of a level");
  __shared__ uint32_t before[kMaxLevels][kGroups];
  __shared__ LeafPart part[kKeyThreads];
  const uint32_t lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  uint32_t k[kKeyRows];
#pragma unroll
  for (int r = 0; r < kKeyRows; ++r)
    k[r] = kl((uint64_t)blockIdx.x * kKeyBlock + r * kKeyThreads + threadIdx.x);
  for (uint32_t i = threadIdx.x; i < (kl.depth + 1) * kGroups; i += kKeyThreads) (&before[0][0])[i] = 0u;
  __syncthreads();
  uint32_t top[kKeyRows];  // the coarsest level that begins in the row's warp
#pragma unroll
  for (int r = 0; r < kKeyRows; ++r) {
    top[r] = __reduce_min_sync(0xFFFFFFFFu, k[r]);
    for (uint32_t d = top[r]; d <= kl.depth; ++d) {
      const uint32_t b = __ballot_sync(0xFFFFFFFFu, k[r] <= d);
      if (lane == 0) before[d][r * (kKeyThreads / 32) + warp] = (uint32_t)__popc(b);
    }
  }
  __syncthreads();
  for (uint32_t d = warp; d <= kl.depth; d += kKeyThreads / 32) {
    const uint32_t n = before[d][lane];
    uint32_t x = n;
    for (uint32_t s = 1; s < 32; s <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, s);
      if (lane >= s) x += y;
    }
    before[d][lane] = counts[d * nblocks + blockIdx.x] - out.base[d] + x - n;
  }
  __syncthreads();
#pragma unroll 1
  for (int r = 0; r < kKeyRows; ++r) {
    const uint64_t row = (uint64_t)blockIdx.x * kKeyBlock + r * kKeyThreads, i = row + threadIdx.x;
    const uint32_t kr = k[0], from = top[0];
    k[0] = k[1];
    k[1] = k[2];
    k[2] = k[3];
    top[0] = top[1];
    top[1] = top[2];
    top[2] = top[3];
    const uint64_t key = i < kl.n ? kl.keys[i] : 0;
    const uint64_t code = in.chunk_base | (key >> kl.tri_bits);
    uint32_t up = 0;  // the node's index one level up
    for (uint32_t d = from; d <= kl.depth; ++d) {
      const uint32_t b = __ballot_sync(0xFFFFFFFFu, kr <= d);
      if (kr > d) continue;
      const uint32_t at = before[d][r * (kKeyThreads / 32) + warp] + __popc(b & ((1u << lane) - 1u));
      if (kr < d) out.first[d - 1][up] = at + out.base[d];
      out.octant[d][at] = (uint8_t)((code >> (3 * (kl.depth - d))) & 7u);
      up = at;
    }
    // every key's contribution, then the leaves' sums over theirs
    if (i < kl.n) part[threadIdx.x] = leaf_part(in, kl.depth, code, key & ((1ull << kl.tri_bits) - 1ull));
    __syncthreads();
    if (kr <= kl.depth) out.leaf_attribs[up] = leaf_attrib(kl, in, code, i, row + kKeyThreads, part);
    __syncthreads();
  }
}

// ---- 4. inner attributes ---------------------------------------------------------

// One thread per parent (host: octree_from_leaves' inner loop): the valid mask
// and the mean of the children's attributes, in order.  An attribute byte is one
// of 256 values, so its unpacked forms (a division by 255 each on the host) are
// read from two tables.
constexpr int kParentThreads = 256;
__global__ void __launch_bounds__(kParentThreads) parent_kernel(
    const uint32_t* __restrict__ first, uint32_t n, uint32_t children,
    const uint8_t* __restrict__ octant, const svo_attrib* __restrict__ ca,
    uint8_t* __restrict__ masks, svo_attrib* __restrict__ pa) {
  __shared__ float col[256], nrm[256];
  col[threadIdx.x] = __fdiv_rn((float)threadIdx.x, 255.0f);
  nrm[threadIdx.x] = __fmul_rn(__fsub_rn(col[threadIdx.x], 0.5f), 2.0f);
  __syncthreads();
  const uint32_t p = blockIdx.x * kParentThreads + threadIdx.x;
  if (p >= n) return;
  const uint32_t f = first[p], end = p + 1 < n ? first[p + 1] : children;
  uint32_t mask = 0;
  float n0 = 0.0f, n1 = 0.0f, n2 = 0.0f, c0 = 0.0f, c1 = 0.0f, c2 = 0.0f;
  for (uint32_t j = f; j < end; ++j) {
    mask |= 1u << octant[j];
    const svo_attrib a = ca[j];
    n0 = __fadd_rn(n0, nrm[a.packed_normal >> 24]);
    n1 = __fadd_rn(n1, nrm[(a.packed_normal >> 16) & 255u]);
    n2 = __fadd_rn(n2, nrm[(a.packed_normal >> 8) & 255u]);
    c0 = __fadd_rn(c0, col[a.packed_color >> 24]);
    c1 = __fadd_rn(c1, col[(a.packed_color >> 16) & 255u]);
    c2 = __fadd_rn(c2, col[(a.packed_color >> 8) & 255u]);
  }
  const float cnt = (float)(end - f);
  n0 = __fdiv_rn(n0, cnt);
  n1 = __fdiv_rn(n1, cnt);
  n2 = __fdiv_rn(n2, cnt);
  c0 = __fdiv_rn(c0, cnt);
  c1 = __fdiv_rn(c1, cnt);
  c2 = __fdiv_rn(c2, cnt);
  const float len = len3(n0, n1, n2);
  if (len > 0.0f) {
    n0 = __fdiv_rn(n0, len);
    n1 = __fdiv_rn(n1, len);
    n2 = __fdiv_rn(n2, len);
  } else {
    n0 = 0.0f;
    n1 = 0.0f;
    n2 = 1.0f;
  }
  masks[p] = (uint8_t)mask;
  pa[p] = svo_attrib{pack_normal(n0, n1, n2), pack_color(c0, c1, c2)};
}

// ---- 5. treelet cut ------------------------------------------------------------

struct LevelPtrs {
  const uint8_t* masks[kMaxLevels];
  const uint32_t* first[kMaxLevels];
  const svo_attrib* attribs[kMaxLevels];
};

struct Partition {           // treelets rooted at one boundary level
  uint32_t root_level;
  uint32_t stop_level;
  uint32_t gid_base;         // gid of the partition's first treelet
  uint32_t count;            // treelets in the partition (nodes at root_level)
};

struct CutParams {
  Partition parts[kMaxLevels];
  uint32_t num_parts;
  uint32_t depth;
  uint64_t N;                // nodes per slot
};

// Subtree ranges of treelet (part, root index): lo/hi per level and the
// treelet's local offset of each level.  Returns the node count.
__device__ uint64_t treelet_ranges(const LevelPtrs& L, uint32_t r, uint32_t s, uint64_t root,
                                   uint64_t* lo, uint64_t* hi, uint64_t* off) {
  lo[0] = root;
  hi[0] = root + 1;
  off[0] = 0;
  uint64_t total = 1;
  for (uint32_t l = r; l < s; ++l) {
    const uint32_t k = l - r;
    const uint64_t last = hi[k] - 1;
    lo[k + 1] = L.first[l][lo[k]];
    hi[k + 1] = (uint64_t)L.first[l][last] + (uint64_t)__popc(L.masks[l][last]);
    off[k + 1] = total;
    total += hi[k + 1] - lo[k + 1];
  }
  return total;
}

__global__ void treelet_sizes_kernel(LevelPtrs L, CutParams cp, uint32_t num_treelets,
                                     unsigned long long* __restrict__ stats) {
  const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= num_treelets) return;
  uint32_t p = 0;
  while (p + 1 < cp.num_parts && gid >= cp.parts[p + 1].gid_base) ++p;
  const Partition& P = cp.parts[p];
  uint64_t lo[kMaxLevels], hi[kMaxLevels], off[kMaxLevels];
  const uint64_t n = treelet_ranges(L, P.root_level, P.stop_level, gid - P.gid_base, lo, hi, off);
  atomicMax(stats, (unsigned long long)n);
  atomicAdd(stats + 1, (unsigned long long)n);
}

// One block per treelet: its slot (slot = gid, as insert_all fills an empty
// pool) with every sub-treelet root copied into this treelet's leaf and
// re-pointed (insert_treelet's patch), leaf flags of resident sub-treelets
// cleared, tail zero.
__global__ void __launch_bounds__(256) cut_kernel(LevelPtrs L, CutParams cp,
                                                  uint32_t num_treelets,
                                                  uint2* __restrict__ nodes,
                                                  svo_attrib* __restrict__ attribs) {
  const uint32_t gid = blockIdx.x;
  if (gid >= num_treelets) return;
  __shared__ uint64_t lo[kMaxLevels], hi[kMaxLevels], off[kMaxLevels];
  __shared__ uint32_t part;
  if (threadIdx.x == 0) {
    uint32_t p = 0;
    while (p + 1 < cp.num_parts && gid >= cp.parts[p + 1].gid_base) ++p;
    part = p;
    treelet_ranges(L, cp.parts[p].root_level, cp.parts[p].stop_level, gid - cp.parts[p].gid_base,
                   lo, hi, off);
  }
  __syncthreads();
  const Partition& P = cp.parts[part];
  const uint32_t r = P.root_level, s = P.stop_level, D = cp.depth;
  const uint64_t base = (uint64_t)gid * cp.N;
  // the sub-treelets' partition and its stop level (their roots' leaf flags)
  const bool has_sub = s < D;
  const uint32_t sub_base = has_sub ? cp.parts[part + 1].gid_base : 0u;
  const uint32_t sub_stop = has_sub ? cp.parts[part + 1].stop_level : 0u;
  for (uint32_t l = r; l <= s; ++l) {
    const uint32_t k = l - r;
    const uint64_t lo_l = lo[k], cnt = hi[k] - lo[k];
    for (uint64_t e = threadIdx.x; e < cnt; e += blockDim.x) {
      const uint64_t g = lo_l + e;
      const uint64_t p = off[k] + e;
      attribs[base + p] = L.attribs[l][g];
      uint2 rec;
      if (l < s) {
        const uint32_t m = L.masks[l][g];
        const uint64_t child = off[k + 1] + ((uint64_t)L.first[l][g] - lo[k + 1]);
        const uint32_t leaf = (l + 1 == s && s == D) ? m : 0u;
        rec = make_uint2((uint32_t)(child - p), (m << 8) | leaf);
      } else if (!has_sub) {
        rec = make_uint2(0u, 0u);
      } else {
        // leaf holding a copy of sub-treelet c's root, first child at c's slot + 1;
        // the copy is taken when c is inserted, before c's own sub-treelets
        // clear the leaf flags in c's slot, so it keeps them
        const uint64_t c = (uint64_t)sub_base + g;
        const uint32_t m = L.masks[l][g];
        const uint32_t leaf = (l + 1 == sub_stop) ? m : 0u;
        rec = make_uint2((uint32_t)((c * cp.N + 1u) - (base + p)), (m << 8) | leaf);
      }
      nodes[base + p] = rec;
    }
  }
  // the rest of the slot: the pool is written once, without clearing it first
  const uint64_t used = off[s - r] + (hi[s - r] - lo[s - r]);
  for (uint64_t p = used + threadIdx.x; p < cp.N; p += blockDim.x) {
    nodes[base + p] = make_uint2(0u, 0u);
    attribs[base + p] = svo_attrib{0u, 0u};
  }
}

// ---- host side -----------------------------------------------------------------------

// Columns of one pass, at most: 2 GB of records.  A chunk of more is split while it
// can be (for_each_chunk), then taken in several passes.
constexpr uint64_t kMaxColumns = 1ull << 29;
static_assert(kMaxColumns % kColThreads == 0 && kMaxColumns / kColThreads <= 0x7FFFFFFF, "whole blocks, one grid");

// Scratch of one build, ordered on its stream.
struct Scratch {
  cudaMemPool_t pool = nullptr;
  cudaStream_t st = nullptr;
};

template <class T>
struct DevBuf {
  T* p = nullptr;
  cudaStream_t st = nullptr;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  DevBuf(DevBuf&& o) noexcept : p(o.p), st(o.st) { o.p = nullptr; }
  DevBuf& operator=(DevBuf&& o) noexcept {
    if (this != &o) {
      reset();
      p = o.p;
      st = o.st;
      o.p = nullptr;
    }
    return *this;
  }
  ~DevBuf() { reset(); }
  void reset() {
    if (p) cudaFreeAsync(p, st);
    p = nullptr;
  }
  cudaError_t alloc(const Scratch& s, size_t count) {
    reset();
    st = s.st;
    return scratch_alloc(s.pool, (count ? count : 1) * sizeof(T), s.st, (void**)&p);
  }
};

// The levels of a chunk, or of the whole octree.
struct Levels {
  uint64_t size[kMaxLevels] = {};
  DevBuf<uint32_t> first[kMaxLevels];
  DevBuf<uint8_t> octant[kMaxLevels];
  DevBuf<svo_attrib> leaf_attribs;
};

uint32_t bits_for(uint64_t v) {
  uint32_t b = 1;
  while (b < 64 && (1ull << b) < v) ++b;
  return b;
}

// The host builder's stop_level (csrc/scene.cpp).
uint32_t stop_level_of(uint32_t D, uint32_t L, uint32_t r) {
  if (L == 0) return D;
  const uint32_t m = (D - r) % L;
  uint32_t stop = r + (m == 0 ? L : m);
  if (stop == r + 1 && stop < D && r > 0) stop = std::min(D, stop + L);
  return stop;
}

#define GB_TRY(x)                                              \
  do {                                                         \
    const cudaError_t e_ = (x);                                \
    if (e_ != cudaSuccess) return cuda_status(e_);             \
  } while (0)

unsigned grid_of(uint64_t n, unsigned threads) {
  return (unsigned)((n + threads - 1) / threads);
}

// In-place exclusive sum of n + 1 counts, the last of them 0; returns the total.
int sum_counts(const Scratch& sc, uint64_t* counts, uint64_t n, uint64_t* total) {
  size_t bytes = 0;
  GB_TRY(cub::DeviceScan::ExclusiveSum(nullptr, bytes, counts, counts, n + 1, sc.st));
  DevBuf<uint8_t> tmp;
  GB_TRY(tmp.alloc(sc, bytes));
  GB_TRY(cub::DeviceScan::ExclusiveSum(tmp.p, bytes, counts, counts, n + 1, sc.st));
  GB_TRY(cudaMemcpyAsync(total, counts + n, 8, cudaMemcpyDeviceToHost, sc.st));
  GB_TRY(cudaStreamSynchronize(sc.st));
  return SVO_OK;
}

template <class Count>
int sort_keys(const Scratch& sc, cub::DoubleBuffer<uint64_t>& kb, Count n, int lo_bit, int hi_bit) {
  size_t bytes = 0;
  GB_TRY(cub::DeviceRadixSort::SortKeys(nullptr, bytes, kb, n, lo_bit, hi_bit, sc.st));
  DevBuf<uint8_t> tmp;
  GB_TRY(tmp.alloc(sc, bytes));
  GB_TRY(cub::DeviceRadixSort::SortKeys(tmp.p, bytes, kb, n, lo_bit, hi_bit, sc.st));
  return SVO_OK;
}

Chunk chunk_of(const Cell& cell, uint32_t depth, uint32_t tri_bits) {
  uint32_t cxyz[3] = {0, 0, 0};
  for (uint32_t b = 0; b < cell.level; ++b)
    for (int k = 0; k < 3; ++k) cxyz[k] |= (uint32_t)((cell.index >> (3 * b + 2 - k)) & 1u) << b;
  const uint32_t cs = (1u << depth) >> cell.level;  // voxels per chunk per axis
  Chunk ch;
  for (int k = 0; k < 3; ++k) {
    ch.lo[k] = (int)(cxyz[k] * cs);
    ch.hi[k] = (int)((cxyz[k] + 1) * cs) - 1;
  }
  ch.shift = 3 * (depth - cell.level);
  ch.tri_bits = tri_bits;
  return ch;
}

}  // namespace

int DeviceScene::build_mesh(const float* h_vertices, const float* h_normals,
                            const float* h_colors, uint64_t nv, const uint32_t* h_triangles,
                            uint64_t nt, uint32_t depth_, uint32_t treelet_levels,
                            cudaStream_t st) {
  if (depth_ < 1 || depth_ > 21) return SVO_ERR_RANGE;
  if (nt == 0 || nv == 0) return SVO_ERR_INVALID;
  if ((h_normals == nullptr) != (h_colors == nullptr)) return SVO_ERR_INVALID;
  uint32_t largest = 0;
  for (uint64_t i = 0; i < 3 * nt; ++i) largest = std::max(largest, h_triangles[i]);
  if (largest >= nv) return SVO_ERR_INVALID;
  depth = depth_;
  const uint32_t tri_bits = bits_for(nt);
  // chunk levels: enough that a key (code inside the chunk, triangle) fits 64 bits
  uint32_t chunk_levels = 0;
  while (chunk_levels < depth && 3 * (depth - chunk_levels) + tri_bits > 64) ++chunk_levels;
  if (chunk_levels > 3 || 3 * (depth - chunk_levels) + tri_bits > 64) return SVO_ERR_RANGE;
  int dev = 0;
  GB_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return SVO_ERR_RANGE;
  device = dev;
  user_begins(dev);  // until this scene is destroyed
  Scratch sc;
  sc.st = st;
  GB_TRY(scratch_pool(dev, &sc.pool));

  DevBuf<float> dV, dFn, dN, dC;
  DevBuf<uint32_t> dT;
  DevBuf<TriRecord> dRec;
  GB_TRY(dV.alloc(sc, 3 * nv));
  GB_TRY(dT.alloc(sc, 3 * nt));
  GB_TRY(cudaMemcpyAsync(dV.p, h_vertices, 3 * nv * sizeof(float), cudaMemcpyHostToDevice, st));
  GB_TRY(cudaMemcpyAsync(dT.p, h_triangles, 3 * nt * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
  LeafInput leaf_in = {nullptr, nullptr, 0};
  if (h_normals != nullptr) {
    GB_TRY(dN.alloc(sc, 3 * nv));
    GB_TRY(dC.alloc(sc, 3 * nv));
    GB_TRY(dRec.alloc(sc, nt));
    GB_TRY(cudaMemcpyAsync(dN.p, h_normals, 3 * nv * sizeof(float), cudaMemcpyHostToDevice, st));
    GB_TRY(cudaMemcpyAsync(dC.p, h_colors, 3 * nv * sizeof(float), cudaMemcpyHostToDevice, st));
    tri_records_kernel<<<grid_of(nt, 128), 128, 0, st>>>(dV.p, dN.p, dC.p, dT.p, nt, dRec.p);
    leaf_in.records = dRec.p;
  } else {
    GB_TRY(dFn.alloc(sc, 3 * nt));
    face_normals_kernel<<<grid_of(nt, 256), 256, 0, st>>>(dV.p, dT.p, nt, dFn.p);
    leaf_in.face_normals = dFn.p;
  }
  GB_TRY(cudaGetLastError());
  dN.reset();
  dC.reset();

  // -- voxels and levels, chunk by chunk; a chunk's leaves are sorted and unique
  DevBuf<uint64_t> cols, d_totals;
  DevBuf<TriWalk> walks;
  GB_TRY(walks.alloc(sc, nt));
  GB_TRY(cols.alloc(sc, nt + 1));
  GB_TRY(d_totals.alloc(sc, kMaxLevels));
  GB_TRY(cudaMemsetAsync(d_totals.p, 0, kMaxLevels * sizeof(uint64_t), st));
  std::vector<Levels> parts;
  uint64_t totals[kMaxLevels] = {};
  auto count_columns = [&](const Cell& cell, uint64_t* n) -> int {
    column_count_kernel<<<grid_of(nt + 1, 128), 128, 0, st>>>(dV.p, dT.p, nt, depth,
                                                              chunk_of(cell, depth, tri_bits), walks.p, cols.p);
    GB_TRY(cudaGetLastError());
    return sum_counts(sc, cols.p, nt, n);
  };
  Cell last_cell = {0, 0};  // the last one with leaves
  auto build_chunk = [&](const Cell& cell, uint64_t columns, bool* began) -> int {
    const Chunk ch = chunk_of(cell, depth, tri_bits);
    int rc = SVO_OK;
    DevBuf<uint64_t> keys, keys2;
    uint64_t P = 0;
    {
      // pass by pass over the columns where they are more than a pass may have:
      // the overlaps are counted first, and each pass's test made again for them
      const uint64_t pass = std::min(columns, kMaxColumns);
      const uint64_t col_blocks = (pass + kColThreads - 1) / kColThreads;
      DevBuf<uint32_t> rec;
      DevBuf<uint64_t> block_hits;
      DevBuf<uint32_t> block_tri;
      GB_TRY(rec.alloc(sc, pass));
      GB_TRY(block_hits.alloc(sc, col_blocks + 1));
      GB_TRY(block_tri.alloc(sc, col_blocks + 1));
      ColumnWindow win = {0, 0};
      unsigned blocks = 0;
      auto test_columns = [&](uint64_t first, uint64_t* hits) -> int {
        win = {first, std::min(pass, columns - first)};
        blocks = grid_of(win.count, kColThreads);
        block_triangles_kernel<<<grid_of(blocks + 1, 256), 256, 0, st>>>(cols.p, nt, win, blocks, block_tri.p);
        GB_TRY(cudaGetLastError());
        column_test_kernel<<<blocks, kColThreads, 0, st>>>(walks.p, depth, ch, cols.p, block_tri.p, win, rec.p,
                                                           block_hits.p);
        GB_TRY(cudaGetLastError());
        return sum_counts(sc, block_hits.p, blocks, hits);
      };
      uint64_t hits = 0;
      for (uint64_t first = 0; first < columns; first += pass) {
        rc = test_columns(first, &hits);
        if (rc != SVO_OK) return rc;
        P += hits;
      }
      if (P == 0) return SVO_OK;
      GB_TRY(keys.alloc(sc, P));
      uint64_t at = 0;
      for (uint64_t first = 0; first < columns; first += pass) {
        if (pass < columns) {
          rc = test_columns(first, &hits);
          if (rc != SVO_OK) return rc;
        }
        column_emit_kernel<<<blocks, kColThreads, 0, st>>>(walks.p, depth, ch, cols.p, block_tri.p, win, rec.p,
                                                           block_hits.p, keys.p + at);
        GB_TRY(cudaGetLastError());
        at += hits;
      }
    }
    // stable, by code alone: the triangles of a code are ascending already
    GB_TRY(keys2.alloc(sc, P));
    cub::DoubleBuffer<uint64_t> kb(keys.p, keys2.p);
    const int lo_bit = (int)tri_bits, hi_bit = (int)(ch.shift + tri_bits);
    rc = P <= 0x7FFFFFFFull ? sort_keys(sc, kb, (int)P, lo_bit, hi_bit) : sort_keys(sc, kb, P, lo_bit, hi_bit);
    if (rc != SVO_OK) return rc;
    if (kb.Current() == keys.p)
      keys2.reset();
    else
      keys = std::move(keys2);
    KeyLevels kl;
    kl.keys = keys.p;
    kl.n = P;
    kl.tri_bits = tri_bits;
    kl.depth = depth;
    kl.first_level = 0;
    if (!parts.empty()) kl.first_level = first_new_level(last_cell, cell, depth);
    const uint64_t key_blocks = (P + kKeyBlock - 1) / kKeyBlock;
    if (key_blocks > 0x7FFFFFFFull) return SVO_ERR_RANGE;
    DevBuf<uint32_t> counts;
    GB_TRY(counts.alloc(sc, (depth + 1) * key_blocks));
    level_count_kernel<<<(unsigned)key_blocks, kKeyThreads, 0, st>>>(kl, key_blocks, counts.p);
    GB_TRY(cudaGetLastError());
    level_scan_kernel<<<depth + 1, 1024, 0, st>>>(counts.p, key_blocks, d_totals.p);
    GB_TRY(cudaGetLastError());
    uint64_t now[kMaxLevels];
    GB_TRY(cudaMemcpyAsync(now, d_totals.p, sizeof(now), cudaMemcpyDeviceToHost, st));
    GB_TRY(cudaStreamSynchronize(st));
    if (now[depth] > 0xFFFFFFFFull) return SVO_ERR_RANGE;
    Levels lv;
    LevelOut out = {};
    auto alloc_levels = [&]() -> int {
      for (uint32_t d = 0; d <= depth; ++d) {
        lv.size[d] = now[d] - totals[d];
        out.base[d] = (uint32_t)totals[d];
        GB_TRY(lv.octant[d].alloc(sc, lv.size[d]));
        out.octant[d] = lv.octant[d].p;
        if (d == depth) continue;
        GB_TRY(lv.first[d].alloc(sc, lv.size[d]));
        out.first[d] = lv.first[d].p;
      }
      GB_TRY(lv.leaf_attribs.alloc(sc, lv.size[depth]));
      out.leaf_attribs = lv.leaf_attribs.p;
      return SVO_OK;
    };
    rc = alloc_levels();
    if (rc != SVO_OK) {  // the totals as they were, for the cell's children
      GB_TRY(cudaMemcpyAsync(d_totals.p, totals, sizeof(totals), cudaMemcpyHostToDevice, st));
      return rc;
    }
    *began = true;
    std::copy(now, now + kMaxLevels, totals);
    last_cell = cell;
    pairs += P;
    parts.push_back(std::move(lv));
    leaf_in.chunk_base = cell_code(cell, depth);
    level_write_kernel<<<(unsigned)key_blocks, kKeyThreads, 0, st>>>(kl, leaf_in, key_blocks, counts.p,
                                                                    out);
    GB_TRY(cudaGetLastError());
    return SVO_OK;
  };
  int rc = for_each_chunk(depth, chunk_levels, kMaxColumns, count_columns, build_chunk);
  if (rc != SVO_OK) return rc;
  cols.reset();
  walks.reset();
  dV.reset();
  dT.reset();
  dFn.reset();
  dRec.reset();
  if (parts.empty()) return SVO_ERR_INVALID;
  leaf_voxels = totals[depth];
  if (totals[0] != 1) return SVO_ERR_INVALID;

  // -- the chunks' levels one after another
  if (parts.size() > 1) {
    Levels all;
    auto join = [&](auto get, uint32_t d, auto& to) -> int {
      GB_TRY(to.alloc(sc, totals[d]));
      uint64_t at = 0;
      for (Levels& lv : parts) {
        auto& from = get(lv);
        GB_TRY(cudaMemcpyAsync(to.p + at, from.p, lv.size[d] * sizeof(*to.p), cudaMemcpyDeviceToDevice, st));
        at += lv.size[d];
        from.reset();
      }
      return SVO_OK;
    };
    for (uint32_t d = 0; d <= depth && rc == SVO_OK; ++d) {
      rc = join([d](Levels& lv) -> auto& { return lv.octant[d]; }, d, all.octant[d]);
      if (rc == SVO_OK && d < depth)
        rc = join([d](Levels& lv) -> auto& { return lv.first[d]; }, d, all.first[d]);
    }
    if (rc == SVO_OK) rc = join([](Levels& lv) -> auto& { return lv.leaf_attribs; }, depth, all.leaf_attribs);
    if (rc != SVO_OK) return rc;
    parts.clear();
    parts.push_back(std::move(all));
  }
  Levels& lv = parts[0];

  // -- attributes and masks, bottom-up
  DevBuf<uint8_t> masks[kMaxLevels];
  DevBuf<svo_attrib> attribs[kMaxLevels];
  attribs[depth] = std::move(lv.leaf_attribs);
  octree_nodes = totals[depth];
  for (int d = (int)depth - 1; d >= 0; --d) {
    const uint32_t n = (uint32_t)totals[d];
    octree_nodes += n;
    GB_TRY(masks[d].alloc(sc, n));
    GB_TRY(attribs[d].alloc(sc, n));
    parent_kernel<<<grid_of(n, kParentThreads), kParentThreads, 0, st>>>(
        lv.first[d].p, n, (uint32_t)totals[d + 1], lv.octant[d + 1].p, attribs[d + 1].p, masks[d].p,
        attribs[d].p);
    GB_TRY(cudaGetLastError());
    lv.octant[d + 1].reset();
  }

  // -- partitions (treelet boundary levels) and gids
  CutParams cp{};
  cp.depth = depth;
  uint64_t gid_next = 0;
  uint32_t np = 0;
  for (uint32_t r = 0; r < depth; r = stop_level_of(depth, treelet_levels, r)) {
    if (np >= (uint32_t)kMaxLevels) return SVO_ERR_RANGE;
    Partition& P = cp.parts[np++];
    P.root_level = r;
    P.stop_level = stop_level_of(depth, treelet_levels, r);
    P.gid_base = (uint32_t)gid_next;
    P.count = (uint32_t)totals[r];
    gid_next += totals[r];
    if (gid_next > 0x7FFFFFFFull) return SVO_ERR_RANGE;
  }
  cp.num_parts = np;
  num_treelets = (uint32_t)gid_next;
  LevelPtrs L{};
  for (uint32_t d = 0; d <= depth; ++d) {
    L.masks[d] = masks[d].p;
    L.first[d] = lv.first[d].p;
    L.attribs[d] = attribs[d].p;
  }

  // -- slot size: the largest treelet + 8 (cut_treelets' automatic size)
  {
    DevBuf<unsigned long long> stats;  // {largest treelet, sum of treelet sizes}
    GB_TRY(stats.alloc(sc, 2));
    GB_TRY(cudaMemsetAsync(stats.p, 0, 16, st));
    treelet_sizes_kernel<<<grid_of(num_treelets, 128), 128, 0, st>>>(L, cp, num_treelets, stats.p);
    GB_TRY(cudaGetLastError());
    unsigned long long h[2] = {0, 0};
    GB_TRY(cudaMemcpyAsync(h, stats.p, 16, cudaMemcpyDeviceToHost, st));
    GB_TRY(cudaStreamSynchronize(st));
    nodes_per_slot = h[0] + 8;
    treelet_nodes = h[1];
  }
  if (nodes_per_slot < 16 || nodes_per_slot * 8 > 0xFFFFFFFFull) return SVO_ERR_RANGE;
  if ((uint64_t)num_treelets * nodes_per_slot > 0x100000000ull) return SVO_ERR_RANGE;
  cp.N = nodes_per_slot;
  pool_nodes = (uint64_t)num_treelets * nodes_per_slot;

  // -- the pool: nodes, then attributes, in one allocation
  const uint64_t half = (pool_nodes * sizeof(svo_node) + 255u) & ~255ull;
  void* mem = nullptr;
  GB_TRY(pool_alloc(dev, 2 * half, &mem, &pool_bytes_));
  d_nodes = (svo_node*)mem;
  d_attribs = (svo_attrib*)((char*)mem + half);
  cut_kernel<<<num_treelets, 256, 0, st>>>(L, cp, num_treelets, reinterpret_cast<uint2*>(d_nodes),
                                           d_attribs);
  GB_TRY(cudaGetLastError());
  GB_TRY(cudaStreamSynchronize(st));
  return SVO_OK;
}

DeviceScene::~DeviceScene() {
  if (device < 0) return;
  int now = device;
  const bool other = cudaGetDevice(&now) == cudaSuccess && now != device;
  if (other) cudaSetDevice(device);
  pool_free(device, d_nodes, pool_bytes_);
  user_ends(device);
  if (other) cudaSetDevice(now);
}

}  // namespace svo
