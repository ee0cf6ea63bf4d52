// upload.cu -- scatter of packed incore slots into the device pools.
//
// The packed upload (TreeletMemoryManagerCuda::upload_packed) replaces the
// reference's per-range buffer writes (src/TreeletMemoryManagerCl.cpp:
// 177-236): only dirty slots cross PCIe, in one copy per 32 MB, and this
// kernel places them at HBM bandwidth.  One block per slot; 8-byte records,
// coalesced on both sides.
#include <cuda_runtime.h>

#include "upload.h"

namespace svo {

namespace {

__global__ void __launch_bounds__(256) slot_scatter_kernel(const uint2* __restrict__ stage,
                                                           const uint32_t* __restrict__ ids,
                                                           uint64_t N, uint2* __restrict__ nodes,
                                                           uint2* __restrict__ attribs) {
  const uint2* src = stage + (uint64_t)blockIdx.x * 2 * N;
  const uint64_t dst = (uint64_t)ids[blockIdx.x] * N;
  for (uint64_t i = threadIdx.x; i < N; i += blockDim.x) {
    nodes[dst + i] = src[i];
    attribs[dst + i] = src[N + i];
  }
}

// PCIe bounds the gather: the bytes that cross it, and enough of them in flight.
// A slot holds a third of its records on average (slots have the size of the
// largest treelet), and a leaf written into a resident treelet changes two
// records, so only the records held are read, in 16-byte loads, eight of a
// thread's in flight, by kSlotParts blocks a slot; the slot's tail is written as
// zeros.  Bringing in 46 treelets of the
// depth-10 icosphere took 266 us with whole slots, 31 us so.
constexpr uint32_t kSlotParts = 4;
constexpr uint32_t kGatherThreads = 256;

// Records [lo, hi), in pairs from an even index on where both sides can take
// 16-byte accesses there (pools are at least 16-byte aligned unless a caller
// attached others).
__device__ __forceinline__ void gather_range(const uint2* __restrict__ src, uint2* __restrict__ dst,
                                             uint64_t lo, uint64_t hi) {
  constexpr int kUnroll = 8;
  if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) != 0u) {
    for (uint64_t i = lo + threadIdx.x; i < hi; i += kGatherThreads) dst[i] = src[i];
    return;
  }
  if ((lo & 1u) && lo < hi) {
    if (threadIdx.x == 0) dst[lo] = src[lo];
    ++lo;
  }
  if ((hi & 1u) && lo < hi) {
    --hi;
    if (threadIdx.x == 32) dst[hi] = src[hi];
  }
  const uint4* s4 = reinterpret_cast<const uint4*>(src);
  uint4* d4 = reinterpret_cast<uint4*>(dst);
  for (uint64_t i0 = lo / 2 + threadIdx.x; i0 < hi / 2; i0 += kGatherThreads * kUnroll) {
    uint4 v[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const uint64_t i = i0 + (uint64_t)u * kGatherThreads;
      if (i < hi / 2) v[u] = s4[i];
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const uint64_t i = i0 + (uint64_t)u * kGatherThreads;
      if (i < hi / 2) d4[i] = v[u];
    }
  }
}

__global__ void __launch_bounds__(kGatherThreads) slot_gather_kernel(
    const uint2* __restrict__ hn, const uint2* __restrict__ ha, const uint2* __restrict__ jobs,
    uint32_t count, uint64_t N, const uint4* __restrict__ patches, uint32_t num_patches,
    uint2* __restrict__ nodes, uint2* __restrict__ attribs) {
  const uint32_t bodies = count * kSlotParts;
  if (blockIdx.x >= bodies) {
    const uint32_t i = (blockIdx.x - bodies) * kGatherThreads + threadIdx.x;
    if (i >= num_patches) return;
    const uint4 p = patches[i];
    nodes[p.x] = make_uint2(p.z, p.w);
    return;
  }
  const uint2 job = jobs[blockIdx.x / kSlotParts];
  const uint32_t part = blockIdx.x % kSlotParts;
  const uint64_t base = (uint64_t)job.x * N, used = base + job.y;
  // the parts share what is read, and what is cleared, evenly
  const uint64_t lo = base + (uint64_t)job.y * part / kSlotParts,
                 hi = base + (uint64_t)job.y * (part + 1) / kSlotParts;
  gather_range(hn, nodes, lo, hi);
  gather_range(ha, attribs, lo, hi);
  const uint64_t tail = N - job.y;
  for (uint64_t i = used + tail * part / kSlotParts + threadIdx.x, end = used + tail * (part + 1) / kSlotParts;
       i < end; i += kGatherThreads) {
    nodes[i] = make_uint2(0u, 0u);
    attribs[i] = make_uint2(0u, 0u);
  }
}

}  // namespace

int launch_slot_gather(const svo_node* host_nodes, const svo_attrib* host_attribs,
                       const uint32_t* jobs, uint32_t count, uint64_t N, const uint32_t* patches,
                       uint32_t num_patches, svo_node* nodes, svo_attrib* attribs,
                       cudaStream_t stream) {
  const uint64_t blocks =
      (uint64_t)count * kSlotParts + (num_patches + kGatherThreads - 1) / kGatherThreads;
  if (blocks == 0) return SVO_OK;
  if (blocks > 0x7FFFFFFFull) return SVO_ERR_RANGE;
  slot_gather_kernel<<<(unsigned)blocks, kGatherThreads, 0, stream>>>(
      reinterpret_cast<const uint2*>(host_nodes), reinterpret_cast<const uint2*>(host_attribs),
      reinterpret_cast<const uint2*>(jobs), count, N, reinterpret_cast<const uint4*>(patches),
      num_patches, reinterpret_cast<uint2*>(nodes), reinterpret_cast<uint2*>(attribs));
  return cudaGetLastError() == cudaSuccess ? SVO_OK : SVO_ERR_CUDA;
}

int launch_slot_scatter(const void* stage, const uint32_t* ids, uint32_t count, uint64_t N,
                        svo_node* nodes, svo_attrib* attribs, cudaStream_t stream) {
  if (count == 0) return SVO_OK;
  slot_scatter_kernel<<<count, 256, 0, stream>>>(reinterpret_cast<const uint2*>(stage), ids, N,
                                                 reinterpret_cast<uint2*>(nodes),
                                                 reinterpret_cast<uint2*>(attribs));
  return cudaGetLastError() == cudaSuccess ? SVO_OK : SVO_ERR_CUDA;
}

}  // namespace svo
