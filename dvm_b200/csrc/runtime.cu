#include "runtime.h"

#include <cuda_runtime.h>

#include <atomic>
#include <string>

#include "../../include/dvm.h"
#include "bounded_wait.cuh"

namespace dvmb {

constexpr int kMaxFlagDevices = 64;

// One word per device, mapped into every device's address space; null when they could not be had.
static volatile uint32_t *ExpiryFlags() {
  static volatile uint32_t *const flags = []() -> volatile uint32_t * {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;   // (the first launch may happen inside somebody's capture)
    cudaThreadExchangeStreamCaptureMode(&mode);
    void *p = nullptr;
    if (cudaHostAlloc(&p, kMaxFlagDevices * sizeof(uint32_t), cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
      cudaGetLastError();
      p = nullptr;
    } else {
      for (int i = 0; i < kMaxFlagDevices; ++i) static_cast<volatile uint32_t *>(p)[i] = 0;
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
    return static_cast<volatile uint32_t *>(p);
  }();
  return flags;
}
// The word of the current device; null: none.
static volatile uint32_t *ExpiryFlag() {
  volatile uint32_t *const flags = ExpiryFlags();
  int dev = -1;
  if (flags == nullptr || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxFlagDevices) return nullptr;
  return flags + dev;
}

LaunchTag NextLaunchEpoch() {
  static std::atomic<uint32_t> counter{0};
  uint32_t e = counter.fetch_add(1, std::memory_order_relaxed) + 1;
  if (e == 0) e = counter.fetch_add(1, std::memory_order_relaxed) + 1;   // 0 means "no launch has failed yet"
  return {e, 0u, ExpiryFlag()};
}
bool TakeExpiryFlag() {
  volatile uint32_t *const flag = ExpiryFlag();
  if (flag == nullptr) return true;
  if (*flag == 0) return false;
  *flag = 0;
  return true;
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
