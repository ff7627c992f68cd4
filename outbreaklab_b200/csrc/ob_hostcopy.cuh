// ob_hostcopy.cuh — device-to-host copies into pageable memory (ob_hostcopy.cu).
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace ob {

// copies bytes of device memory, as the work queued on s leaves it, into dst and waits for it
cudaError_t copy_to_host(void* dst, const void* src, size_t bytes, cudaStream_t s);
// the owners of the copies' pinned ring: it is freed with the last of them
void host_copy_retain();
void host_copy_release();

}  // namespace ob
