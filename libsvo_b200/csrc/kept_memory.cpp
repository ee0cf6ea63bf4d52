// kept_memory.cpp -- see kept_memory.h.
#include "kept_memory.h"

#include <mutex>
#include <vector>

namespace svo {

namespace {

constexpr uint64_t kScratchKeep = 1ull << 30;
constexpr uint64_t kPoolKeep = 1ull << 30;

struct KeptPool {
  void* p;
  uint64_t bytes;
};
struct Kept {
  std::mutex mu;
  cudaMemPool_t scratch = nullptr;  // once made, as long as the process
  std::vector<KeptPool> pools;
  uint64_t pool_bytes = 0;
  uint64_t users = 0;  // scenes alive and builds running
};
Kept g_kept[kMaxDevices];

// What is kept, taken out of the books; freed by the caller without the lock
// (cudaFree waits for the device).
std::vector<KeptPool> take_pools(Kept& k) {  // k.mu is held
  std::vector<KeptPool> out;
  out.swap(k.pools);
  k.pool_bytes = 0;
  return out;
}

void give_back(const std::vector<KeptPool>& pools, cudaMemPool_t scratch) {
  for (const KeptPool& p : pools) cudaFree(p.p);
  if (scratch) cudaMemPoolTrimTo(scratch, 0);
}

}  // namespace

void user_begins(int dev) {
  std::lock_guard<std::mutex> lock(g_kept[dev].mu);
  ++g_kept[dev].users;
}

void user_ends(int dev) {
  Kept& k = g_kept[dev];
  {
    std::lock_guard<std::mutex> lock(k.mu);
    if (--k.users) return;
  }
  cudaDeviceSynchronize();  // scratch still in use by a failed build
  std::unique_lock<std::mutex> lock(k.mu);
  if (k.users) return;  // a build has begun meanwhile: what is kept is its
  const std::vector<KeptPool> pools = take_pools(k);
  cudaMemPool_t scratch = k.scratch;
  lock.unlock();
  give_back(pools, scratch);
}

cudaError_t scratch_pool(int dev, cudaMemPool_t* out) {
  Kept& k = g_kept[dev];
  std::lock_guard<std::mutex> lock(k.mu);
  if (!k.scratch) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    cudaError_t e = cudaMemPoolCreate(&pool, &props);
    if (e != cudaSuccess) return e;
    uint64_t keep = kScratchKeep;
    e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    if (e != cudaSuccess) {
      cudaMemPoolDestroy(pool);
      return e;
    }
    k.scratch = pool;
  }
  *out = k.scratch;
  return cudaSuccess;
}

cudaError_t scratch_alloc(cudaMemPool_t pool, uint64_t bytes, cudaStream_t stream, void** out) {
  cudaError_t e = cudaMallocFromPoolAsync(out, bytes, pool, stream);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    // what the stream has still to free goes back only once it has come to it
    e = cudaStreamSynchronize(stream);
    if (e == cudaSuccess) {
      give_back_kept_memory();
      e = cudaMallocFromPoolAsync(out, bytes, pool, stream);
    }
  }
  if (e != cudaSuccess) {
    cudaGetLastError();  // the caller has it; the next launch's check must not
    *out = nullptr;
  }
  return e;
}

cudaError_t pool_alloc(int dev, uint64_t bytes, void** out, uint64_t* got) {
  Kept& k = g_kept[dev];
  {
    std::lock_guard<std::mutex> lock(k.mu);
    size_t best = k.pools.size();
    for (size_t i = 0; i < k.pools.size(); ++i)
      if (k.pools[i].bytes >= bytes && k.pools[i].bytes - bytes <= bytes / 4 &&
          (best == k.pools.size() || k.pools[i].bytes < k.pools[best].bytes))
        best = i;
    if (best < k.pools.size()) {
      *out = k.pools[best].p;
      *got = k.pools[best].bytes;
      k.pool_bytes -= *got;
      k.pools.erase(k.pools.begin() + (ptrdiff_t)best);
      return cudaSuccess;
    }
  }
  *got = bytes;
  return device_alloc(out, bytes);
}

void pool_free(int dev, void* p, uint64_t bytes) {
  if (!p) return;
  Kept& k = g_kept[dev];
  auto keeps = [&] { return k.users > 1 && k.pool_bytes + bytes <= kPoolKeep; };  // k.mu is held
  std::unique_lock<std::mutex> lock(k.mu);
  if (keeps()) {
    lock.unlock();  // cudaFree waits for the device; a block that is kept must wait as well
    const bool idle = cudaDeviceSynchronize() == cudaSuccess;
    lock.lock();
    if (idle && keeps()) {  // still
      try {
        k.pools.push_back({p, bytes});
        k.pool_bytes += bytes;
        return;
      } catch (...) {
      }
    }
  }
  lock.unlock();
  cudaFree(p);
}

void give_back_kept_memory() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return;
  Kept& k = g_kept[dev];
  std::unique_lock<std::mutex> lock(k.mu);
  const std::vector<KeptPool> pools = take_pools(k);
  cudaMemPool_t scratch = k.scratch;
  lock.unlock();
  give_back(pools, scratch);
}

cudaError_t device_alloc(void** out, uint64_t bytes) {
  cudaError_t e = cudaMalloc(out, bytes);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    give_back_kept_memory();
    e = cudaMalloc(out, bytes);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    *out = nullptr;
  }
  return e;
}

}  // namespace svo
