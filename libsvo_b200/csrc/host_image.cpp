// host_image.cpp -- see host_image.h.
#include "host_image.h"

#include <cuda.h>
#include <cuda_runtime.h>

namespace svo {

namespace {

// The allocation or registration that an address belongs to.  The runtime tells of
// single addresses only, and memory between two registrations need not be mapped,
// so the driver is asked for its range.
bool range_of(CUdeviceptr p, CUdeviceptr* start, size_t* size) {
  using Fn = CUresult (*)(unsigned, CUpointer_attribute*, void**, CUdeviceptr);
  static const Fn get = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &fn, 7000, cudaEnableDefault, &found) !=
            cudaSuccess ||
        found != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      return Fn(nullptr);
    }
    return (Fn)fn;
  }();
  CUpointer_attribute what[2] = {CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE};
  void* to[2] = {start, size};
  *start = 0;
  *size = 0;
  return get && get(2, what, to, p) == CUDA_SUCCESS && *size != 0;
}

}  // namespace

uint32_t* mapped_image(uint32_t* h, uint64_t pixels) {
  const uint64_t at = (uintptr_t)h;
  if ((at & 3u) != 0u || pixels > (UINT64_MAX - at) / sizeof(uint32_t)) return nullptr;
  const uint64_t end = at + pixels * sizeof(uint32_t);
  CUdeviceptr first = 0;
  for (uint64_t p = at; p < end;) {  // a registration a turn
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, (const void*)(uintptr_t)p) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    if (a.type != cudaMemoryTypeHost || !a.devicePointer) return nullptr;
    const CUdeviceptr d = (CUdeviceptr)a.devicePointer;
    if (p == at) first = d;
    if (d - first != p - at) return nullptr;  // the device sees a gap, or another order
    CUdeviceptr start = 0;
    size_t size = 0;
    if (!range_of(d, &start, &size) || d < start || d - start >= size) return nullptr;
    p += size - (d - start);
  }
  return (uint32_t*)first;
}

}  // namespace svo
