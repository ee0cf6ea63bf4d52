// host_image_host.cpp -- libsvo_b200/csrc/host_image.cpp over registrations of host
// memory that this file pretends.  TEST INFRASTRUCTURE ONLY.
#include HOST_IMAGE_SOURCE

#include <map>

#include <cuda.h>
#include <cuda_runtime.h>

namespace {

struct Registered {
  uint64_t size;
  int type;
};
std::map<uint64_t, Registered> g_ranges;  // by first byte; the device sees the host's addresses

const std::pair<const uint64_t, Registered>* find(uint64_t p) {
  auto it = g_ranges.upper_bound(p);
  if (it == g_ranges.begin()) return nullptr;
  --it;
  return p < it->first + it->second.size ? &*it : nullptr;
}

CUresult fake_attributes(unsigned n, CUpointer_attribute* what, void** to, CUdeviceptr p) {
  const auto* r = find(p);
  for (unsigned i = 0; i < n; ++i) {
    if (what[i] == CU_POINTER_ATTRIBUTE_RANGE_START_ADDR)
      *(CUdeviceptr*)to[i] = r ? r->first : 0;
    else if (what[i] == CU_POINTER_ATTRIBUTE_RANGE_SIZE)
      *(size_t*)to[i] = r ? r->second.size : 0;
    else
      return CUDA_ERROR_INVALID_VALUE;
  }
  return CUDA_SUCCESS;
}
int g_no_driver = 0;

}  // namespace

extern "C" {

cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  const auto* r = find((uint64_t)p);
  *a = cudaPointerAttributes{};
  a->type = r ? (cudaMemoryType)r->second.type : cudaMemoryTypeUnregistered;
  a->devicePointer = r ? (void*)p : nullptr;
  a->hostPointer = (void*)p;
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** fn, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* found) {
  *fn = (void*)fake_attributes;
  *found = g_no_driver ? cudaDriverEntryPointSymbolNotFound : cudaDriverEntryPointSuccess;
  return cudaSuccess;
}

void no_driver() { g_no_driver = 1; }
void registered(uint64_t at, uint64_t size, int type) { g_ranges[at] = {size, type}; }
uint64_t mapped(uint64_t at, uint64_t pixels) { return (uint64_t)svo::mapped_image((uint32_t*)at, pixels); }

}  // extern "C"
