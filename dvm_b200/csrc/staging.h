// Copies between pageable host memory and the device (staging.cc).
#ifndef DVM_B200_STAGING_H_
#define DVM_B200_STAGING_H_

#include <cstddef>

#include <cuda_runtime.h>

namespace dvmb {

// Copy `bytes` with the semantics of cudaMemcpyAsync: host -> device returns when the source may be reused, device -> host
// from pageable memory when the data has arrived; pinned host memory is copied asynchronously.
cudaError_t CopyToDevice(void *dst, const void *src, size_t bytes, cudaStream_t stream);
cudaError_t CopyToHost(void *dst, const void *src, size_t bytes, cudaStream_t stream);

}  // namespace dvmb

#endif  // DVM_B200_STAGING_H_
