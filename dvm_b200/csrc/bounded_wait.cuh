// Bounded device-side waits shared by the three interpreters / tensor-core kernels.
//
// Every spin on an mbarrier gives up after a time limit (about two seconds): the thread then records
// (code << 24 | block index) in the kernel family's status record and returns, so the kernel always runs to its
// end (with wrong results) and the host reports the failure instead of the GPU hanging.  Once one wait of a launch
// has expired, the other waits of THAT launch return as soon as they reach their slow path; launches are told
// apart by an epoch number the host hands to each launch, so an expiry neither shortens the waits of later
// launches nor of launches running next to it on another stream.  `first_error` keeps the first expiry until
// the host reads and clears it.
#ifndef DVM_B200_BOUNDED_WAIT_CUH_
#define DVM_B200_BOUNDED_WAIT_CUH_

#include <cstdint>

namespace dvmb {

struct WaitStatus {
  unsigned int first_error;   // 0 = ok; else (code << 24 | block index) of the first wait that expired
  unsigned int abort_epoch;   // epoch of the launch whose wait expired last (0 = none yet)
};

constexpr unsigned long long kWaitLimitNs = 2000000000ull;

// What a launch carries for its waits: its epoch, and a word of pinned host memory (null: none could be had) that an expiry
// sets, so that the host learns without a device copy whether there is a record to read - reading the records cost five
// copies of 12 us each at every synchronisation.
struct LaunchTag {
  uint32_t epoch;
  uint32_t pad;
  volatile uint32_t *host_flag;
};
// Host side (runtime.cu): a tag with a fresh non-zero epoch; and whether a wait of a launch on the current device may have
// expired since the last look, which lowers the device's flag.  To be called before the records are read: an expiry writes its
// record first, so one that comes later raises the flag again, and a flag whose record has been read with others is lowered
// by the next look.
LaunchTag NextLaunchEpoch();
bool TakeExpiryFlag();

#ifdef __CUDACC__
__device__ __forceinline__ void record_expiry(WaitStatus *st, uint32_t code, const LaunchTag &tag) {
  atomicCAS(&st->first_error, 0u, (code << 24) | (blockIdx.x & 0xffffffu));
  atomicExch(&st->abort_epoch, tag.epoch);
  __threadfence_system();
  if (tag.host_flag != nullptr) *tag.host_flag = 1u;
}
__device__ __forceinline__ bool launch_aborted(WaitStatus *st, const LaunchTag &tag) {
  return *reinterpret_cast<volatile unsigned int *>(&st->abort_epoch) == tag.epoch;
}
// Spins on `try_once()` until it succeeds, the launch has been marked as failed, or `limit_ns` have passed.
template <typename TryFn>
__device__ __forceinline__ void bounded_spin(TryFn try_once, uint32_t code, WaitStatus *st, LaunchTag epoch,
                                             unsigned long long limit_ns) {
  for (int i = 0; i < 4096; ++i)
    if (try_once()) return;
  unsigned long long t0, t1;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  for (;;) {
    if (launch_aborted(st, epoch)) return;
    for (int i = 0; i < 1024; ++i)
      if (try_once()) return;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
    if (t1 - t0 > limit_ns) {
      record_expiry(st, code, epoch);
      return;
    }
  }
}
#endif

}  // namespace dvmb

#endif  // DVM_B200_BOUNDED_WAIT_CUH_
