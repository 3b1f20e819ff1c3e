#include "runtime.h"

#include <cuda_runtime.h>

#include <atomic>
#include <string>

#include "../../include/dvm.h"
#include "bounded_wait.cuh"

namespace dvmb {

// One word for the whole process, mapped into every device's address space; null when it could not be had.
static volatile uint32_t *ExpiryFlag() {
  static volatile uint32_t *const flag = []() -> volatile uint32_t * {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;   // (the first launch may happen inside somebody's capture)
    cudaThreadExchangeStreamCaptureMode(&mode);
    void *p = nullptr;
    if (cudaHostAlloc(&p, sizeof(uint32_t), cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
      cudaGetLastError();
      p = nullptr;
    } else {
      *static_cast<volatile uint32_t *>(p) = 0;
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
    return static_cast<volatile uint32_t *>(p);
  }();
  return flag;
}

LaunchTag NextLaunchEpoch() {
  static std::atomic<uint32_t> counter{0};
  uint32_t e = counter.fetch_add(1, std::memory_order_relaxed) + 1;
  if (e == 0) e = counter.fetch_add(1, std::memory_order_relaxed) + 1;   // 0 means "no launch has failed yet"
  return {e, 0u, ExpiryFlag()};
}
bool ExpiryFlagRaised() { return ExpiryFlag() == nullptr || *ExpiryFlag() != 0; }
void LowerExpiryFlag() {
  if (ExpiryFlag() != nullptr) *ExpiryFlag() = 0;
}
void RaiseExpiryFlag() {
  if (ExpiryFlag() != nullptr) *ExpiryFlag() = 1;
}

Runtime &Runtime::Get() {
  static Runtime rt;
  return rt;
}

void Runtime::EnsureInit() {
  if (initialized_) return;
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) {
    std::string msg = std::string("no usable CUDA device: ") + cudaGetErrorString(err);
    cudaGetLastError();
    dvm::DvmException(msg.c_str());
  }
  cudaDeviceProp prop;
  err = cudaGetDeviceProperties(&prop, dev);
  if (err != cudaSuccess) {
    std::string msg = std::string("cudaGetDeviceProperties failed: ") + cudaGetErrorString(err);
    dvm::DvmException(msg.c_str());
  }
  if (prop.major < 10) {
    std::string msg = std::string("dvm-b200 needs an sm_100 class GPU, found ") + prop.name;
    dvm::DvmException(msg.c_str());
  }
  device_ = dev;
  sm_count_ = prop.multiProcessorCount;
  initialized_ = true;
}

}  // namespace dvmb
