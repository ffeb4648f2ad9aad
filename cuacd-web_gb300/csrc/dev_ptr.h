// dev_ptr.h — whether a mesh buffer lives in device memory. The entry points
// that take meshes accept device buffers of the handle's device as well as
// host buffers: a device mesh is copied on the device (no host round trip);
// a host mesh is staged and uploaded.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace cuacd {

// device or managed allocations are device memory; host memory, registered
// or not, is not
inline bool is_device_ptr(const void* p) {
  if (!p) return false;
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

// whether every index is below n: the largest of them is (a search that stops
// at the first bad index cannot be vectorised and took 0.7 ns per index)
inline bool indices_below(const uint32_t* idx, uint64_t count, uint32_t n) {
  uint32_t mx = 0;
  for (uint64_t k = 0; k < count; k++) mx = idx[k] > mx ? idx[k] : mx;
  return count == 0 || mx < n;
}

}  // namespace cuacd
