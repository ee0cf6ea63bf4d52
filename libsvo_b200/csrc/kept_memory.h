// kept_memory.h -- device memory that octree builds keep for the next one, and
// the allocations that it is given back to.
//
// Per device: a stream-ordered pool of scratch that holds on to 1 GB (allocating
// and freeing device memory took 50 of the 70 ms of a depth-11 build), and the
// memory of destroyed scenes up to 1 GB, plain cudaMalloc memory like every
// scene's pool, for the next scene of about that size.  Both are kept while a
// scene lives or a build runs on the device, and go back to it when the last one
// ends.  Every function may be called from any thread; none waits for the device
// or allocates while it holds the lock, so that a scene's end does not hold up
// another thread's build.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace svo {

constexpr int kMaxDevices = 64;

// Scenes alive and builds running on the device: what they keep goes back to it
// when the last one ends.
void user_begins(int dev);
void user_ends(int dev);

// The device's pool of scratch memory.
cudaError_t scratch_pool(int dev, cudaMemPool_t* out);

// Scratch memory from it, in the stream's order; on the current device.  Where it
// does not fit, what is kept is given back and it is tried once more.
cudaError_t scratch_alloc(cudaMemPool_t pool, uint64_t bytes, cudaStream_t stream, void** out);

// Scene pool memory: a kept block of at most a quarter more than asked for, else
// new memory.  *got is the block's size.
cudaError_t pool_alloc(int dev, uint64_t bytes, void** out, uint64_t* got);
// ... and its end, from a user of the device; waits until nothing reads it.
void pool_free(int dev, void* p, uint64_t bytes);

// Gives what is kept on the current device back to it.
void give_back_kept_memory();

// Every other allocation of device memory in the library: on the current device;
// where it does not fit, what builds keep is given back and it is tried once more.
cudaError_t device_alloc(void** out, uint64_t bytes);
template <class T>
cudaError_t device_array(T** out, uint64_t count) {
  return device_alloc((void**)out, count * sizeof(T));
}

}  // namespace svo
