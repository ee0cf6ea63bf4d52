// kept_memory_host.cpp -- libsvo_b200/csrc/kept_memory.cpp over a device that
// this file pretends to be: a number of bytes, plain allocations, one
// stream-ordered pool that keeps what is freed to it.  TEST INFRASTRUCTURE ONLY.
#include KEPT_MEMORY_SOURCE

#include <chrono>
#include <condition_variable>
#include <map>
#include <mutex>
#include <thread>

namespace {

struct Device {
  std::mutex mu;
  std::condition_variable cv;
  uint64_t size = 0, plain = 0;     // bytes there are, bytes of plain allocations
  uint64_t pool_used = 0;           // of the pool: in use,
  uint64_t pool_pending = 0;        // freed, but the stream has not come to it,
  uint64_t pool_free = 0;           // kept for the next allocation
  uint64_t next = 4096;
  std::map<uint64_t, uint64_t> bytes;
  int last = cudaSuccess;
  uint64_t stream_waits = 0;
  bool hold = false, waiting = false;  // cudaDeviceSynchronize: told to wait, waits
} g;

cudaError_t failed() {
  g.last = cudaErrorMemoryAllocation;
  return cudaErrorMemoryAllocation;
}
uint64_t used() { return g.plain + g.pool_used + g.pool_pending + g.pool_free; }

}  // namespace

extern "C" {

cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() {
  std::lock_guard<std::mutex> l(g.mu);
  const int e = g.last;
  g.last = cudaSuccess;
  return (cudaError_t)e;
}
cudaError_t cudaMalloc(void** p, size_t n) {
  std::lock_guard<std::mutex> l(g.mu);
  if (used() + n > g.size) return failed();
  g.plain += n;
  *p = (void*)g.next;
  g.bytes[g.next] = n;
  g.next += n + 4096;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::lock_guard<std::mutex> l(g.mu);
  if (!p) return cudaSuccess;
  g.plain -= g.bytes.at((uint64_t)p);
  g.bytes.erase((uint64_t)p);
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* out, const cudaMemPoolProps*) {
  *out = (cudaMemPool_t)16;
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t n) {
  std::lock_guard<std::mutex> l(g.mu);
  if (g.pool_free > n) g.pool_free = n;
  return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
  std::lock_guard<std::mutex> l(g.mu);
  // memory of the pool's, else more from the device (kept pieces are not joined
  // to new ones)
  if (g.pool_free >= n)
    g.pool_free -= n;
  else if (used() + n > g.size)
    return failed();
  g.pool_used += n;
  *p = (void*)g.next;
  g.bytes[g.next] = n;
  g.next += n + 4096;
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
  std::lock_guard<std::mutex> l(g.mu);
  const uint64_t n = g.bytes.at((uint64_t)p);
  g.bytes.erase((uint64_t)p);
  g.pool_used -= n;
  g.pool_pending += n;
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
  std::lock_guard<std::mutex> l(g.mu);
  ++g.stream_waits;
  g.pool_free += g.pool_pending;
  g.pool_pending = 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
  std::unique_lock<std::mutex> l(g.mu);
  g.waiting = true;
  g.cv.notify_all();
  g.cv.wait(l, [] { return !g.hold; });
  g.waiting = false;
  g.pool_free += g.pool_pending;
  g.pool_pending = 0;
  return cudaSuccess;
}

// ---- what the test calls -----------------------------------------------------

void fake_device(uint64_t size) { g.size = size; }
uint64_t fake_used() { return used(); }
uint64_t fake_plain() { return g.plain; }
int fake_last_error() { return g.last; }

// 1 when `other`, on a second thread, comes back while the device is busy and
// `end` waits for it on this thread's behalf; 0 when it has not after two seconds.
// end: 0 a scene that is kept, 1 the last user.  other: 0 a build begins and
// allocates a pool, 1 a scene that nobody waits for.
int runs_beside(int end, int other) {
  void* p = nullptr;
  uint64_t got = 0;
  svo::user_begins(0);
  if (end == 0) svo::user_begins(0);
  if (svo::pool_alloc(0, 1000, &p, &got) != cudaSuccess) return -1;
  g.hold = true;
  std::thread ending([&] {
    if (end == 0) svo::pool_free(0, p, got);
    svo::user_ends(0);
  });
  {
    std::unique_lock<std::mutex> l(g.mu);
    g.cv.wait(l, [] { return g.waiting; });
  }
  bool done = false;
  std::thread second([&] {
    void* q = nullptr;
    uint64_t n = 0;
    svo::user_begins(0);
    cudaMemPool_t pool;
    if (other == 0) svo::scratch_pool(0, &pool);
    svo::pool_alloc(0, 5000, &q, &n);
    {
      std::lock_guard<std::mutex> l(g.mu);
      done = true;
    }
    g.cv.notify_all();
    cudaFree(q);
  });
  int beside;
  {
    std::unique_lock<std::mutex> l(g.mu);
    beside = g.cv.wait_for(l, std::chrono::seconds(2), [&] { return done; }) ? 1 : 0;
    g.hold = false;
  }
  g.cv.notify_all();
  ending.join();
  second.join();
  if (end == 1) svo::pool_free(0, p, got);
  svo::user_ends(0);
  if (end == 0) svo::user_ends(0);
  return beside;
}

uint64_t block_alloc(uint64_t bytes, uint64_t* got) {
  void* p = nullptr;
  return svo::pool_alloc(0, bytes, &p, got) == cudaSuccess ? (uint64_t)p : 0u;
}
void block_free(uint64_t p, uint64_t bytes) { svo::pool_free(0, (void*)p, bytes); }
uint64_t scratch(uint64_t bytes) {
  cudaMemPool_t pool;
  void* p = nullptr;
  if (svo::scratch_pool(0, &pool) != cudaSuccess) return 0;
  return svo::scratch_alloc(pool, bytes, nullptr, &p) == cudaSuccess ? (uint64_t)p : 0u;
}
void scratch_free(uint64_t p) { cudaFreeAsync((void*)p, nullptr); }
uint64_t words(uint64_t n) {
  uint32_t* p = nullptr;
  return svo::device_array(&p, n) == cudaSuccess ? (uint64_t)p : 0u;
}
void begin() { svo::user_begins(0); }
void end() { svo::user_ends(0); }

}  // extern "C"
