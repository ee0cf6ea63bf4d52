// render.h -- host-side launchers of the ray-cast kernels.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

#include "../../include/libsvo_b200.h"

namespace svo {

size_t render_smem_bytes(int stack_size);

// Rays of one warp in a frame, an analysis pass or a set of rays.  A set too
// small to fill the GPU takes as long as its slowest warp, and a warp with fewer
// rays takes fewer of the loop's paths in each pass, so it is cast with 8 or 16
// of a warp's lanes (us, 32 / 16 / 8 lanes, eight views each): a depth-11 icosphere
// 64x64 22.9 / 22.4 / 21.1, with shadow rays 77 / 71 / 63; 128x128 33.6 / 32.4 / 31.1
// and 105 / 98 / 89; 160x160 40.0 / 38.5 / 38.2; 192x192 43.6 / 42.3 / 44.9 and 110 /
// 105 / 107; 224x224 47.7 / 47.6 / 50.3; 256x256 55.7 / 55.2 / 62.2 and 125 / 122 /
// 131; a depth-9 terrain 128x128 25.5 / 24.7 / 24.4, 192x192 32.1 / 31.4 / 33.1,
// 224x224 33.3 / 33.9 / 37.3.
inline uint32_t rays_per_warp(uint64_t rays) {
  return rays <= (1u << 14) ? 8u : (rays <= (3u << 14) ? 16u : 32u);
}

// host_image: rgba is the device-side address of page-locked host memory.
int launch_render(const svo_node* nodes, const svo_attrib* attribs, uint64_t num_nodes,
                  const svo_frame_params& p, const svo_trace_cfg& cfg, uint32_t* rgba,
                  svo_hit* hits, svo_stats* stats, cudaStream_t stream, bool host_image = false);

int launch_render_shadow(const svo_node* nodes, const svo_attrib* attribs, uint64_t num_nodes,
                         const svo_frame_params& p, const svo_shadow_cfg& sc, int stack_size,
                         uint32_t* rgba, svo_hit* hits, svo_hit* shadow_hits, svo_stats* stats,
                         cudaStream_t stream);

int launch_trace_rays(const svo_node* nodes, uint64_t num_nodes, const float* origins,
                      const float* dirs, uint64_t n, float tsr, const svo_trace_cfg& cfg,
                      svo_hit* hits, svo_stats* stats, cudaStream_t stream);

}  // namespace svo
