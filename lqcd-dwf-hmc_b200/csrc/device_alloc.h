// Device memory of the library's plans and workspaces.
#pragma once

#include <cuda_runtime.h>

namespace b200 {

// cudaMalloc; where it would fail, once more after the scratch that the gauge
// force keeps between calls has been given up (gauge.cu).
cudaError_t device_malloc_bytes(void** p, size_t n);
template <typename T>
cudaError_t device_malloc(T** p, size_t n) {
  return device_malloc_bytes(reinterpret_cast<void**>(p), n);
}

}  // namespace b200
