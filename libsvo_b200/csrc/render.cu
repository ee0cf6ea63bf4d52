// render.cu -- the per-frame ray cast (renderToBuffer) and explicit-ray cast.
//
// Replaces the OpenCL kernel renderToBuffer (opencl/treeletRenderer_rgba.cl:
// 610-734) and its enqueue (projects/raycast_serialized_opencl/src/
// raycast_serialized_opencl.cpp:729-747).  One thread per pixel; a warp
// covers an 8x4 pixel tile so neighbouring rays walk the same nodes; a block
// of 128 threads covers 16x8 pixels (smaller blocks than 16x16 measured 3 %
// faster on a 1080p frame and 10 % on 512x512: the last wave is shorter).
// The RGBA8 epilogue is fused.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "render.h"
#include "ray_order.cuh"
#include "row_bands.h"
#include "shade.cuh"
#include "traverse.cuh"

namespace svo {

namespace {

constexpr int kBlockW = 16;  // 128 threads: finer blocks balance the tail of a frame
constexpr int kBlockH = 8;
constexpr int kThreads = kBlockW * kBlockH;

// ---- longest-first dispatch ------------------------------------------------
// A frame's blocks differ in cost by two orders of magnitude (rays that graze
// a surface run hundreds of iterations, most rays a dozen), and raster order
// starts some of the longest blocks last, where they run on after the other
// SMs are done.  Frames of one to four million pixels therefore estimate each
// 16x8 block's cost first (its two 8x8 cells' centre rays) and append the block
// to the list of its cost bucket; block r of the frame kernel then casts the
// r-th block of the buckets taken costliest first.  Every pixel is still cast by
// the same code: only the order the blocks start in changes.
//
// The estimate is a chain of dependent node reads per ray, so its time grows
// with the cap on its passes, and a low cap ranks the blocks worse.  A ray at the
// cap counts for what its progress says about the rest of its way through the root
// box, so that the long blocks are told from one another (with the capped counts as
// they are, the 1920x1080 icosphere took 255 us against 226 us, as long as in raster
// order).  The cap (us, 32 / 40 / 48 / 56 passes, six views each):
//   depth-9 icosphere   1280x1024 140 / 143 / 146 / 149  1920x1080 155 / 158 / 161 / 164
//   depth-11 icosphere  1280x1024 180 / 173 / 175 / 177  1920x1080 196 / 194 / 198 / 203
//   the same, near      1920x1080 255 / 249 / 249 / 252
//   depth-10 terrain    1280x1024 161 / 162 / 163 / 165  1920x1080 218 / 222 / 224 / 227
//   depth-12 terrain    1280x1024 182 / 183 / 185 / 188  1920x1080 247 / 252 / 255 / 258
// so 40 is the lowest that ranks the deep icosphere's blocks, for about 1.5 % of a
// terrain.  Measured with the loop before the present one: one sample a block 235 us
// against 226; all 32 of a warp's lanes casting samples instead of 16 (the paths of
// more cells diverge in each of its passes) 248 against 241 us.
//
// The lines: the tail that the order removes is a few long rays, so it does not
// grow with the frame, while the estimate is a share of it.  In raster order and
// ordered (us): the depth-11 icosphere 1024x768 148 / 140, 1280x1024 192 / 173,
// 1920x1080 215 / 194, 2560x1440 366 / 318, 3840x2160 653 / 636; the depth-9 one 113 /
// 107, 153 / 143, 170 / 158, 252 / 250, 473 / 513; the depth-12 terrain 109 / 124,
// 162 / 184, 238 / 252, 416 / 436, 918 / 969.  A terrain has no such tail and is
// faster in raster order throughout, by 5 to 14 %; what a frame will show is not
// known before it is cast.
constexpr uint32_t kCostCap = 40;  // passes of an estimate ray
constexpr uint32_t kCostBuckets = 49;
constexpr uint32_t kCostTop = kCostBuckets - 1;
constexpr uint32_t kCostSamples = kBlockW / 8;  // one ray per 8x8 cell of a block
constexpr uint32_t kCostLanes = 16;             // lanes of a warp that cast a sample
constexpr uint64_t kOrderMinPixels = 1ull << 20;
constexpr uint64_t kOrderMaxPixels = 1ull << 22;
static_assert(kCostSamples == 2, "a block's cost is the larger of two adjacent lanes' samples");
static_assert(kCostBuckets > 32 && kCostBuckets <= 64, "one warp scans the buckets, two per lane");

// count[k]: blocks of estimated cost k; list[k * nblocks + j]: the j-th of
// them.  count == nullptr: raster order.
struct BlockOrder {
  const uint32_t* count;
  const uint32_t* list;
  uint32_t nblocks;
};

// The lanes of the warp whose key equals this lane's, for keys below 128:
// seven ballots, one per key bit.  All 32 lanes take part.
__device__ __forceinline__ uint32_t same_key_lanes(uint32_t k) {
  uint32_t peers = 0xFFFFFFFFu;
#pragma unroll
  for (int bit = 0; bit < 7; ++bit) {
    const bool set = (k >> bit) & 1u;
    const uint32_t b = __ballot_sync(0xFFFFFFFFu, set);
    peers &= set ? b : ~b;
  }
  return peers;
}

// The r-th block in cost order (buckets kCostTop down to 0, each in the
// order its blocks were appended).  Called by one whole warp; every lane
// returns the block.
__device__ __forceinline__ uint32_t ordered_block(const BlockOrder& o, uint32_t r, uint32_t lane) {
  const uint32_t k1 = lane + 32 < kCostBuckets ? kCostTop - 32 - lane : 0u;
  const uint32_t c0 = __ldg(o.count + (kCostTop - lane));
  const uint32_t c1 = lane + 32 < kCostBuckets ? __ldg(o.count + k1) : 0u;
  uint32_t p0 = c0, p1 = c1;  // inclusive prefix sums, bucket kCostTop first
  for (uint32_t d = 1; d < 32; d <<= 1) {
    const uint32_t y0 = __shfl_up_sync(0xFFFFFFFFu, p0, d);
    const uint32_t y1 = __shfl_up_sync(0xFFFFFFFFu, p1, d);
    if (lane >= d) {
      p0 += y0;
      p1 += y1;
    }
  }
  p1 += __shfl_sync(0xFFFFFFFFu, p0, 31);
  uint32_t m = __ballot_sync(0xFFFFFFFFu, p0 > r);
  uint32_t bucket, before;
  if (m != 0u) {
    const int l = __ffs(m) - 1;
    bucket = kCostTop - (uint32_t)l;
    before = __shfl_sync(0xFFFFFFFFu, p0 - c0, l);
  } else {
    m = __ballot_sync(0xFFFFFFFFu, p1 > r);
    if (m == 0u) return r;  // not reached: the buckets hold every block once
    const int l = __ffs(m) - 1;
    bucket = kCostTop - 32 - (uint32_t)l;
    before = __shfl_sync(0xFFFFFFFFu, p1 - c1, l);
  }
  return __ldg(o.list + (uint64_t)bucket * o.nblocks + (r - before));
}

// The thread's pixel; false outside the frame.  Warp w of a block covers 8
// columns and rays / 8 rows of it, two warps side by side (16x8 pixels at 32
// rays a warp); rows start at y0 (frames taller than one grid's rows take
// several launches).
__device__ __forceinline__ bool block_pixel(const svo_frame_params& p, uint32_t bx, uint32_t by,
                                            uint32_t y0, uint32_t rays, uint32_t* x, uint32_t* y) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, rows = rays / 8;
  *x = bx * kBlockW + (warp % (kBlockW / 8)) * 8 + (lane & 7);
  *y = y0 + by * (kBlockH / 4 * rows) + (warp / (kBlockW / 8)) * rows + (lane >> 3);
  return lane < rays && *x < p.width && *y < p.height;
}

// kExt: view modes 2, 6 and 7 (shade_ext); the other modes compile without
// the extra exit state.  With `order` (1-D grid) block r casts the r-th block
// in estimated-cost order of a frame gx blocks wide; without it the grid is
// the frame's blocks in raster order.
// kHost: rgba is page-locked host memory, written as the blocks end instead of
// being copied after the last one.  A block's colours go through shared memory
// so that its rows cross PCIe in 64-byte pieces (a warp's own tile has 32).
template <bool kFlat, bool kExt, bool kHost>
__global__ void __launch_bounds__(kThreads) render_frame_kernel(
    const uint2* __restrict__ nodes, const uint2* __restrict__ attribs, uint64_t num_nodes,
    const svo_frame_params p, int S, uint32_t* __restrict__ rgba, svo_hit* __restrict__ hits,
    svo_stats* __restrict__ stats, uint32_t y0, const BlockOrder order, uint32_t gx, uint32_t rays) {
  extern __shared__ uint2 stack_smem[];
  const int t = threadIdx.x;
  const int warp = t >> 5, lane = t & 31;
  uint32_t bx = blockIdx.x, by = blockIdx.y;
  if (order.count != nullptr) {
    __shared__ uint32_t block;
    // launched as a programmatic dependent of the estimate: wait until its
    // bucket lists are complete and visible
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (warp == 0) {
      const uint32_t b = ordered_block(order, blockIdx.x, (uint32_t)lane);
      if (lane == 0) block = b;
    }
    __syncthreads();
    bx = block % gx;
    by = block / gx;
  }
  uint32_t x, y;
  const bool inside = block_pixel(p, bx, by, y0, rays, &x, &y);
  if (!kHost && !inside) return;
  uint32_t colour = 0u;
  if (inside) {
    float o[3], dx, dy, dz;
    pixel_ray(p, x, y, o, dx, dy, dz);
    const RayHit h = cast_ray<kFlat>(GlobalFetch{nodes}, num_nodes, o, dx, dy, dz, p.t_scale_ratio,
                                     S, stack_smem + t, kThreads);
    const uint64_t pix = (uint64_t)y * p.width + x;
    colour = kExt ? shade_ext(p.mode, h, attribs, num_nodes, S, p.t_scale_ratio, dx, dy, dz)
                  : shade(p.mode, h, attribs, num_nodes, S);
    if (!kHost) rgba[pix] = colour;
    if (hits != nullptr) store_hit(hits, pix, h);
    count_stats(stats, h);
  }
  if (kHost) {
    __shared__ uint32_t tile[kThreads];
    const uint32_t rows = kBlockH / 4 * (rays / 8);  // of the block
    const uint32_t bx0 = bx * kBlockW, by0 = y0 + by * rows;
    if (lane < (int)rays) tile[(y - by0) * kBlockW + (x - bx0)] = colour;
    __syncthreads();
    const uint32_t px = bx0 + t % kBlockW, py = by0 + t / kBlockW;
    if (t < (int)(rows * kBlockW) && px < p.width && py < p.height) rgba[(uint64_t)py * p.width + px] = tile[t];
  }
}

// The bucket of a sample ray: six to a doubling of its expected iterations.
__device__ __forceinline__ uint32_t cost_bucket(const RayHit& h) {
  float n = (float)h.loops;
  if (h.flags == SVO_HITFLAG_CAPPED) {
    const float enter = fmaxf(h.t_enter, 0.0f);
    const float done = __fdividef(h.tc_min - enter, h.t_exit - enter);
    n = __fdividef(n, fminf(fmaxf(done, 0.02f), 1.0f));
  }
  return min((uint32_t)(__log2f(fmaxf(n, 1.0f)) * 6.0f), kCostBuckets - 1u);
}

// The cost estimate: one thread per sample ray, the two samples of block b
// in adjacent lanes.  The larger of its two buckets is the block's, and the
// block is appended to that bucket's list
// (one atomic per bucket and warp, so neighbouring blocks of a bucket stay
// together).
template <bool kFlat>
__global__ void __launch_bounds__(kThreads) block_cost_kernel(
    const uint2* __restrict__ nodes, uint64_t num_nodes, const svo_frame_params p, int S,
    uint32_t gx, uint32_t nblocks, uint32_t* __restrict__ count, uint32_t* __restrict__ list) {
  extern __shared__ uint2 stack_smem[];
  const uint32_t lane = threadIdx.x % 32;
  const uint64_t i = ((uint64_t)blockIdx.x * (kThreads / 32) + threadIdx.x / 32) * kCostLanes + lane;
  // the frame kernel may be scheduled once every block of this grid has
  // started (it waits for this grid's completion before reading the lists)
  asm volatile("griddepcontrol.launch_dependents;");
  const bool live = lane < kCostLanes && i < (uint64_t)nblocks * kCostSamples;
  const uint32_t b = (uint32_t)(i / kCostSamples), c = (uint32_t)(i % kCostSamples);
  // the cell's centre pixel (pixel 4, 4 of the 8x8 cell; clamped to the
  // frame in cells cut by its edge)
  const uint32_t x0 = (b % gx) * kBlockW + c * 8, y0 = (b / gx) * kBlockH;
  const uint32_t x = min(x0 + 4u, p.width - 1u), y = min(y0 + 4u, p.height - 1u);
  uint32_t cost = 0u;
  if (live && x0 < p.width && y0 < p.height) {
    float o[3], dx, dy, dz;
    pixel_ray(p, x, y, o, dx, dy, dz);
    const RayHit h = cast_ray<kFlat>(GlobalFetch{nodes}, num_nodes, o, dx, dy, dz, p.t_scale_ratio,
                                     S, stack_smem + threadIdx.x, kThreads, kCostCap);
    cost = cost_bucket(h);
  }
  cost = max(cost, __shfl_xor_sync(0xFFFFFFFFu, cost, 1));
  const bool appends = live && c == 0;
  const uint32_t peers = same_key_lanes(appends ? cost : kCostBuckets) & 0x55555555u;
  if (appends) {
    const int first = __ffs(peers) - 1;
    uint32_t base = 0u;
    if ((int)lane == first) base = atomicAdd(count + cost, (uint32_t)__popc(peers));
    base = __shfl_sync(peers, base, first);
    list[(uint64_t)cost * nblocks + base + __popc(peers & ((1u << lane) - 1u))] = b;
  }
}

// Primary ray plus one shadow ray per hit, shaded as shade_diffuse_color_shadow
// (opencl/fillFrameBuffer_rgba.cl:494-529) with the live renderer's attribute
// addressing (attribute index = node index, :388-404):
//   n = getNormal, c = getColor, nDotL = max(0, dot(n, L)),
//   shadow = sample(nodeCenter + n * offset, L, tsr_shadow) ? 1 : 0,
//   colour = c * nDotL * (1 - shadow) + c * 0.2, alpha 1; misses, and hits
//   outside the pool, (0.2, 0.3, 0.2).
// The shadow ray reuses the primary ray's stack columns.
__global__ void __launch_bounds__(kThreads) render_shadow_kernel(
    const uint2* __restrict__ nodes, const uint2* __restrict__ attribs, uint64_t num_nodes,
    const svo_frame_params p, const svo_shadow_cfg sc, int S, uint32_t* __restrict__ rgba,
    svo_hit* __restrict__ hits, svo_hit* __restrict__ shadow_hits,
    svo_stats* __restrict__ stats, uint32_t y0, uint32_t rays) {
  extern __shared__ uint2 stack_smem[];
  const int t = threadIdx.x;
  uint32_t x, y;
  if (!block_pixel(p, blockIdx.x, blockIdx.y, y0, rays, &x, &y)) return;
  float o[3], dx, dy, dz;
  pixel_ray(p, x, y, o, dx, dy, dz);
  const RayHit h = cast_ray<false>(GlobalFetch{nodes}, num_nodes, o, dx, dy, dz, p.t_scale_ratio,
                                   S, stack_smem + t, kThreads);
  const uint64_t pix = (uint64_t)y * p.width + x;
  uint32_t out = pack_rgba8(0.2f, 0.3f, 0.2f, 1.0f);
  RayHit sh;
  sh.node = 0u;
  sh.t = 0.0f;
  sh.depth = sh.hit = sh.flags = sh.loops = sh.fetches = 0u;
  if (h.hit && (uint64_t)h.node < num_nodes) {
    {
      const uint2 a = __ldg(attribs + h.node);
      float nx, ny, nz, c[4];
      unpack_normal(a.x, nx, ny, nz);
      unpack_color(a.y, c);
      const float lx = sc.light_direction[0], ly = sc.light_direction[1],
                  lz = sc.light_direction[2];
      const float ndl = cl_max(0.0f, dot3(nx, ny, nz, lx, ly, lz));
      const float so[3] = {__fadd_rn(h.cx, __fmul_rn(nx, sc.normal_offset)),
                           __fadd_rn(h.cy, __fmul_rn(ny, sc.normal_offset)),
                           __fadd_rn(h.cz, __fmul_rn(nz, sc.normal_offset))};
      sh = cast_ray<false>(GlobalFetch{nodes}, num_nodes, so, lx, ly, lz, sc.t_scale_ratio, S,
                           stack_smem + t, kThreads);
      const float lit = __fsub_rn(1.0f, sh.hit ? 1.0f : 0.0f);
      float r[3];
      for (int i = 0; i < 3; ++i)
        r[i] = __fadd_rn(__fmul_rn(__fmul_rn(c[i], ndl), lit), __fmul_rn(c[i], 0.2f));
      out = pack_rgba8(r[0], r[1], r[2], 1.0f);
      count_stats(stats, sh);
    }
  }
  rgba[pix] = out;
  if (hits != nullptr) store_hit(hits, pix, h);
  if (shadow_hits != nullptr) store_hit(shadow_hits, pix, sh);
  count_stats(stats, h);
}

// Whether a set's rays come in order (ray_order.cuh): every block asks the same
// eight pairs, which its SM then has in L1.  Called by the whole block.
__device__ __forceinline__ bool rays_in_order(const float* origins, const float* dirs, uint64_t n) {
  __shared__ bool in_order;
  if (threadIdx.x < 32) {
    const bool close = threadIdx.x < kOrderPairs && pair_close(origins, dirs, order_pair(threadIdx.x, n));
    const uint32_t pairs = __ballot_sync(0xFFFFFFFFu, close);
    if (threadIdx.x == 0) in_order = (uint32_t)__popc(pairs) >= kOrderClose;
  }
  __syncthreads();
  return in_order;
}

// kAsk: casts the rays only if they come in order; launched as a programmatic
// dependent of stream_rays_kernel, which casts them if they do not.  Behind it, not
// ahead of it: the blocks that find nothing to cast come and go while the last rays
// end (ahead of it a million rays without order took 267 against 260 us, four
// million 883 against 854).  Held to the 10 blocks an SM of the plain kernel.
template <bool kFlat, bool kAsk>
__global__ void __launch_bounds__(kThreads, kAsk ? 10 : 0) trace_rays_kernel(
    const uint2* __restrict__ nodes, uint64_t num_nodes, const float* __restrict__ origins,
    const float* __restrict__ dirs, uint64_t n, float tsr, int S, svo_hit* __restrict__ hits,
    svo_stats* __restrict__ stats, uint32_t rays) {
  extern __shared__ uint2 stack_smem[];
  if (kAsk) {
    // what comes behind this grid waits for it, and so for the grids before it
    if (blockIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (!rays_in_order(origins, dirs, n)) return;
  }
  const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const uint64_t i = ((uint64_t)blockIdx.x * (kThreads / 32) + warp) * rays + lane;
  if (lane >= rays || i >= n) return;
  const float o[3] = {origins[3 * i], origins[3 * i + 1], origins[3 * i + 2]};
  const RayHit h = cast_ray<kFlat>(GlobalFetch{nodes}, num_nodes, o, dirs[3 * i], dirs[3 * i + 1],
                                   dirs[3 * i + 2], tsr, S, stack_smem + threadIdx.x, kThreads);
  store_hit(hits, i, h);
  count_stats(stats, h);
}

// The ray counter of stream_rays_kernel, which need not wait for it until it casts
// (a cleared counter by cudaMemsetAsync: 256,000 pixel rays over a terrain 46 us,
// so 43).
__global__ void clear_kernel(uint32_t* next) {
  asm volatile("griddepcontrol.launch_dependents;");
  *next = 0u;
}

// The same rays with lanes that take the next ray as soon as enough of their
// warp's have ended (kKeepLanes or fewer still run).  Rays without order differ in
// length by an order of magnitude within a warp, and lanes of ended rays idled
// through two thirds of the warp's passes.  `next` is the next ray to take, 0 at
// launch.  A million rays without order, a thread a ray against this (us): depth-9
// icosphere 341 -> 258, depth-11 icosphere 399 -> 302, depth-10 terrain 342 -> 237;
// with 8 lanes kept 266, 312, 266, with 14 266, 314, 246, with 26 275, 319, 252.
// Rays in order end together anyway, and a thread a ray is the faster one by up to
// a third (921,600 pixel rays 148 against 164 us over the icospheres, 65 against 84
// over the terrain), so they are left to trace_rays_kernel.  72 registers; bounded to
// 64 for an eighth block an SM it was slower (336 against 326 us).
constexpr int kKeepLanes = 20;
template <bool kFlat>
__global__ void __launch_bounds__(kThreads) stream_rays_kernel(
    const uint2* __restrict__ nodes, uint64_t num_nodes, const float* __restrict__ origins,
    const float* __restrict__ dirs, uint32_t n, float tsr, int S, svo_hit* __restrict__ hits,
    svo_stats* __restrict__ stats, uint32_t* next) {
  extern __shared__ uint2 stack_smem[];
  // trace_rays_kernel may be scheduled once every block of this grid has started
  asm volatile("griddepcontrol.launch_dependents;");
  const bool in_order = rays_in_order(origins, dirs, n);
  if (!in_order || blockIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");  // for the counter
  if (in_order) return;
  uint2* stack = stack_smem + threadIdx.x;
  const uint32_t lane = threadIdx.x % 32;
  const GlobalFetch fetch{nodes};
  const uint32_t limit = pass_limit(S);
  Descent w;
  Ray r;
  uint32_t ray = 0u;
  bool alive = false, more = true;
  auto finish = [&](const RayHit& h) {
    store_hit(hits, ray, h);
    count_stats(stats, h);
  };
  for (;;) {
    uint32_t live = __ballot_sync(0xFFFFFFFFu, alive);
    if (more) {
      const uint32_t idle = ~live, count = (uint32_t)__popc(idle);
      uint32_t base = 0u;
      if (lane == 0) base = atomicAdd(next, count);
      base = __shfl_sync(0xFFFFFFFFu, base, 0);
      more = base < n && n - base > count;
      const uint32_t mine = base + __popc(idle & ((1u << lane) - 1u));
      if (!alive && mine < n) {
        ray = mine;
        const uint64_t k = 3 * (uint64_t)ray;
        const float o[3] = {origins[k], origins[k + 1], origins[k + 2]};
        RayHit h;
        float t_min = 0.0f;
        const RayKind kind = setup_ray<kFlat>(o, dirs[k], dirs[k + 1], dirs[k + 2], tsr, r, t_min, h);
        if (kind == kFast) {
          w = descent_start(fetch, num_nodes, r, t_min, limit, stack);
          alive = true;
        } else if (kind == kGeneral) {
          const RayState st = {0u, t_min, r.t_max, 0.0f, 0.0f, 0.0f, 0.5f, 0u, 0u};
          descend_general<kFlat>(fetch, num_nodes, r, S, stack, kThreads, st, h, 0u);
        }
        if (!alive) finish(h);
      }
      live = __ballot_sync(0xFFFFFFFFu, alive);
    }
    if (live == 0u && !more) return;
    if (alive) {
      RayHit h = no_hit();
      RayState st;
      const Outcome out =
          descend<kFlat, true>(fetch, num_nodes, r, S, stack, kThreads, limit, more ? kKeepLanes : 0, w, st, h);
      if (out == kLeaves)
        descend_general<kFlat>(fetch, num_nodes, r, S, stack, kThreads, st, h, 0u);
      if (out != kYields) {
        finish(h);
        alive = false;
      }
    }
  }
}

}  // namespace

size_t render_smem_bytes(int S) { return (size_t)S * kThreads * sizeof(uint2); }

namespace {

// The scratch of a cast -- longest-first dispatch's lists, 196 bytes per block,
// and the ray counter of stream_rays_kernel -- comes from a memory pool of the
// library's own, one per device, in stream order: calls on different streams get
// different scratch, and the pool keeps up to 64 MB between calls instead of
// returning it at every synchronisation.
constexpr int kMaxDevices = 64;
cudaMemPool_t g_scratch_pool[kMaxDevices] = {};
std::mutex g_scratch_pool_mu;

cudaMemPool_t scratch_pool() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lock(g_scratch_pool_mu);
  if (!g_scratch_pool[dev]) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) return nullptr;
    uint64_t keep = 64ull << 20;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    g_scratch_pool[dev] = pool;
  }
  return g_scratch_pool[dev];
}

// Longest-first order of the frame's blocks into *order (stream-ordered
// scratch the caller frees with cudaFreeAsync(order->count)); false when the
// frame is too small or too large for it or scratch is not available, and the raster launch is used
// instead.
bool order_blocks(const uint2* nodes, uint64_t num_nodes, const svo_frame_params& p, int S,
                  bool flat, uint32_t gx, uint32_t nblocks, cudaStream_t stream, BlockOrder* order) {
  const uint64_t pixels = (uint64_t)p.width * p.height;
  if (pixels < kOrderMinPixels || pixels > kOrderMaxPixels) return false;
  cudaMemPool_t pool = scratch_pool();
  if (!pool) {
    cudaGetLastError();
    return false;
  }
  // scratch: the bucket counts (256 bytes), then the bucket lists
  constexpr size_t kCountBytes = 256;
  static_assert(kCostBuckets * sizeof(uint32_t) <= kCountBytes, "counts fit their header");
  uint32_t* scratch = nullptr;
  const size_t bytes = kCountBytes + (size_t)kCostBuckets * nblocks * sizeof(uint32_t);
  if (cudaMallocFromPoolAsync((void**)&scratch, bytes, pool, stream) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  uint32_t* list = scratch + kCountBytes / sizeof(uint32_t);
  const uint64_t samples = (uint64_t)nblocks * kCostSamples;
  constexpr uint32_t kPerBlock = kThreads / 32 * kCostLanes;
  const unsigned grid = (unsigned)((samples + kPerBlock - 1) / kPerBlock);
  const size_t smem = render_smem_bytes(S);
  bool ok = cudaMemsetAsync(scratch, 0, kCountBytes, stream) == cudaSuccess;
  if (ok) {
    if (flat)
      block_cost_kernel<true><<<grid, kThreads, smem, stream>>>(nodes, num_nodes, p, S, gx, nblocks, scratch, list);
    else
      block_cost_kernel<false><<<grid, kThreads, smem, stream>>>(nodes, num_nodes, p, S, gx, nblocks, scratch, list);
    ok = cudaGetLastError() == cudaSuccess;
  }
  if (!ok) {
    cudaFreeAsync(scratch, stream);
    cudaGetLastError();
    return false;
  }
  *order = BlockOrder{scratch, list, nblocks};
  return true;
}

}  // namespace

int launch_render(const svo_node* nodes, const svo_attrib* attribs, uint64_t num_nodes,
                  const svo_frame_params& p, const svo_trace_cfg& cfg, uint32_t* rgba,
                  svo_hit* hits, svo_stats* stats, cudaStream_t stream, bool host_image) {
  if (p.width == 0 || p.height == 0) return SVO_OK;
  if (p.height > 0xFFFFFFF0u) return SVO_ERR_RANGE;  // row indices stay below 2^32
  const int S = cfg.stack_size;
  const size_t smem = render_smem_bytes(S);
  const uint2* n2 = reinterpret_cast<const uint2*>(nodes);
  const uint2* a2 = reinterpret_cast<const uint2*>(attribs);
  const bool ext = p.mode == 2 || p.mode == 6 || p.mode == 7;
  const bool flat = cfg.traversal == SVO_TRAVERSAL_FLAT;
  auto* fn = host_image
                 ? (flat ? (ext ? render_frame_kernel<true, true, true> : render_frame_kernel<true, false, true>)
                         : (ext ? render_frame_kernel<false, true, true> : render_frame_kernel<false, false, true>))
                 : (flat ? (ext ? render_frame_kernel<true, true, false> : render_frame_kernel<true, false, false>)
                         : (ext ? render_frame_kernel<false, true, false> : render_frame_kernel<false, false, false>));
  const uint32_t gx = (p.width + kBlockW - 1) / kBlockW;
  const uint64_t nblocks64 = (uint64_t)gx * ((p.height + kBlockH - 1) / kBlockH);
  BlockOrder order{nullptr, nullptr, 0u};
  if (nblocks64 <= 0x7FFFFFFFull &&
      order_blocks(n2, num_nodes, p, S, flat, gx, (uint32_t)nblocks64, stream, &order)) {
    // programmatic dependent launch: the frame kernel's launch and first
    // blocks overlap the estimate's last microseconds (0.5 % on the 1080p frame)
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)nblocks64);
    lc.blockDim = dim3(kThreads);
    lc.dynamicSmemBytes = smem;
    lc.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&lc, fn, n2, a2, num_nodes, p, S, rgba, hits, stats, 0u, order, gx, 32u);
    const cudaError_t last = cudaGetLastError();  // clears a launch error
    if (e == cudaSuccess) e = last;
    cudaFreeAsync(const_cast<uint32_t*>(order.count), stream);
    return e == cudaSuccess ? SVO_OK : SVO_ERR_CUDA;
  }
  const uint32_t rays = rays_per_warp((uint64_t)p.width * p.height), block_h = kBlockH / 4 * rays / 8;
  return for_each_band(p.height, block_h, [&](uint32_t y0, uint32_t, uint32_t gy) -> int {
    fn<<<dim3(gx, gy), kThreads, smem, stream>>>(n2, a2, num_nodes, p, S, rgba, hits, stats, y0,
                                                 BlockOrder{nullptr, nullptr, 0u}, gx, rays);
    return cudaGetLastError() == cudaSuccess ? SVO_OK : SVO_ERR_CUDA;
  });
}

int launch_render_shadow(const svo_node* nodes, const svo_attrib* attribs, uint64_t num_nodes,
                         const svo_frame_params& p, const svo_shadow_cfg& sc, int S,
                         uint32_t* rgba, svo_hit* hits, svo_hit* shadow_hits, svo_stats* stats,
                         cudaStream_t stream) {
  if (p.width == 0 || p.height == 0) return SVO_OK;
  if (p.height > 0xFFFFFFF0u) return SVO_ERR_RANGE;  // row indices stay below 2^32
  const uint2* n2 = reinterpret_cast<const uint2*>(nodes);
  const uint2* a2 = reinterpret_cast<const uint2*>(attribs);
  // One pass in raster order.  Measured with the loop of one event a pass (a
  // 3840x2160 frame 1.79 ms, 1.07 to 1.21 with the present one): ordered by
  // primary-ray cost 2.02 ms, the shadow rays' cost being unknown to the estimate
  // and neighbouring blocks no longer sharing the caches; in two passes (the primary
  // rays longest first, each hit appended to a job list, then one shadow ray per
  // job in full warps) 2.22 ms, and 0.626 against 0.529 ms at 1920x1080, where the
  // shadow pass alone took 330 us for 504 k rays.  A shadow ray cast right after its
  // primary ray finds the nodes of its descent in L1; cast in a later pass it reads
  // them from L2 again.
  const uint32_t gx = (p.width + kBlockW - 1) / kBlockW;
  const uint32_t rays = rays_per_warp((uint64_t)p.width * p.height), block_h = kBlockH / 4 * rays / 8;
  return for_each_band(p.height, block_h, [&](uint32_t y0, uint32_t, uint32_t gy) -> int {
    render_shadow_kernel<<<dim3(gx, gy), kThreads, render_smem_bytes(S), stream>>>(
        n2, a2, num_nodes, p, sc, S, rgba, hits, shadow_hits, stats, y0, rays);
    return cudaGetLastError() == cudaSuccess ? SVO_OK : SVO_ERR_CUDA;
  });
}

namespace {

// From here on lanes have rays to take: a third more than all lanes of
// stream_rays_kernel hold at once (us, a thread a ray against it, rays without order
// over depth-9 and depth-11 icospheres and a depth-10 terrain: 131,072 rays 73 / 98 /
// 79 against 87 / 113 / 89, 170,000 87 / 112 / 97 against 99 / 115 / 104, 200,000 104 /
// 133 / 108 against 102 / 126 / 105, 262,144 121 / 146 / 127 against 114 / 140 / 119).
constexpr uint64_t kStreamRays = 3ull << 16;

// A set of rays whose order is not known: stream_rays_kernel, as many blocks as are
// resident at once, and behind it trace_rays_kernel; one of them casts the set, the
// other finds that it need not.  SVO_ERR_NOTSUP, with nothing launched, where there
// is no scratch for the counter or the stream is being captured.
int stream_or_trace(const uint2* nodes, uint64_t num_nodes, const float* origins, const float* dirs,
                    uint32_t n, float tsr, int S, bool flat, svo_hit* hits, svo_stats* stats,
                    cudaStream_t stream) {
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    return SVO_ERR_NOTSUP;
  }
  auto* fn = flat ? stream_rays_kernel<true> : stream_rays_kernel<false>;
  auto* trace = flat ? trace_rays_kernel<true, true> : trace_rays_kernel<false, true>;
  const size_t smem = render_smem_bytes(S);
  int dev = 0, sms = 0, per_sm = 0;
  uint32_t* next = nullptr;
  cudaMemPool_t pool = scratch_pool();
  if (!pool || cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kThreads, smem) != cudaSuccess || per_sm < 1 ||
      cudaMallocFromPoolAsync((void**)&next, sizeof(uint32_t), pool, stream) != cudaSuccess) {
    cudaGetLastError();
    return SVO_ERR_NOTSUP;
  }
  const unsigned blocks = (n + kThreads - 1) / kThreads;
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(std::min(blocks, (unsigned)(sms * per_sm)));
  lc.blockDim = dim3(kThreads);
  lc.dynamicSmemBytes = smem;
  lc.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = attr;
  lc.numAttrs = 1;
  clear_kernel<<<1, 1, 0, stream>>>(next);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess)
    e = cudaLaunchKernelEx(&lc, fn, nodes, num_nodes, origins, dirs, n, tsr, S, hits, stats, next);
  if (e == cudaSuccess) {
    lc.gridDim = dim3(blocks);
    e = cudaLaunchKernelEx(&lc, trace, nodes, num_nodes, origins, dirs, (uint64_t)n, tsr, S, hits, stats, 32u);
  }
  const cudaError_t last = cudaGetLastError();  // clears a launch error
  if (e == cudaSuccess) e = last;
  cudaFreeAsync(next, stream);
  return e == cudaSuccess ? SVO_OK : SVO_ERR_CUDA;
}

}  // namespace

int launch_trace_rays(const svo_node* nodes, uint64_t num_nodes, const float* origins,
                      const float* dirs, uint64_t n, float tsr, const svo_trace_cfg& cfg,
                      svo_hit* hits, svo_stats* stats, cudaStream_t stream) {
  if (n == 0) return SVO_OK;
  // (us, 32 / 16 / 8 lanes, rays without order over the depth-11 icosphere: 1,000
  // rays 62 / 60 / 56, 8,000 72 / 61 / 58, 16,000 75 / 69 / 69, 30,000 79 / 77 / 85,
  // 50,000 93 / 84 / 102; over a depth-9 terrain 40 / 36 / 35, 50 / 44 / 44, 50 / 48 /
  // 49, 54 / 50 / 55, 56 / 57 / 73)
  const uint32_t rays = n <= (1u << 15) ? rays_per_warp(n) : 32u;
  const uint64_t per_block = kThreads / 32 * rays, blocks = (n + per_block - 1) / per_block;
  if (blocks > 0x7FFFFFFFull) return SVO_ERR_RANGE;
  const int S = cfg.stack_size;
  const size_t smem = render_smem_bytes(S);
  const uint2* n2 = reinterpret_cast<const uint2*>(nodes);
  if (n >= kStreamRays && n <= 0x7FFFFFFFull) {
    const int rc = stream_or_trace(n2, num_nodes, origins, dirs, (uint32_t)n, tsr, S,
                                   cfg.traversal == SVO_TRAVERSAL_FLAT, hits, stats, stream);
    if (rc != SVO_ERR_NOTSUP) return rc;
  }
  if (cfg.traversal == SVO_TRAVERSAL_FLAT)
    trace_rays_kernel<true, false><<<(unsigned)blocks, kThreads, smem, stream>>>(
        n2, num_nodes, origins, dirs, n, tsr, S, hits, stats, rays);
  else
    trace_rays_kernel<false, false><<<(unsigned)blocks, kThreads, smem, stream>>>(
        n2, num_nodes, origins, dirs, n, tsr, S, hits, stats, rays);
  return cudaGetLastError() == cudaSuccess ? SVO_OK : SVO_ERR_CUDA;
}

}  // namespace svo
