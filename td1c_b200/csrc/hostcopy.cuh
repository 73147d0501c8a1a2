// hostcopy.cuh -- large copies between pageable host buffers and the device.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace td1c {

cudaError_t host_to_device(void* dst, const void* src, size_t n, cudaStream_t st);
cudaError_t device_to_host(void* dst, const void* src, size_t n, cudaStream_t st);
void host_copy_release();

}  // namespace td1c
