// Programmatic dependent launch: a kernel of this library may be set up on the SMs (blocks placed, barriers initialised)
// while the kernel before it on the stream still runs its last blocks; it touches global memory only behind chain_wait(),
// which returns when that kernel has completed and its writes are visible.  Back to back, small launches took 3.6-4.1 us
// each without it and 2.1-2.5 us with it (empty kernels), large ones lose the gap between one's tail and the next one's head.
//
// Rules that every kernel launched with ChainAttribute() follows:
//   - every thread calls chain_wait() before its first access to global memory, and no block leaves without it (a kernel
//     counts as complete for the one after the next only because it has itself waited); prefetches to L2 may come earlier
//     (attn_decode.cu, mm_tile.cu): they deliver nothing to the kernel, and L2 sees the writes that follow;
//   - operands are read by ordinary loads (gload() of vm_ops.cuh), which stay behind the wait, not by non-coherent ones;
//   - chain_launch() comes after the point from which the block needs nothing that a block of the next kernel could hold.
#ifndef DVM_B200_CHAIN_CUH_
#define DVM_B200_CHAIN_CUH_

#include <cuda_runtime.h>

#include <cstdlib>

namespace dvmb {

#ifdef __CUDACC__
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

// Appends the launch attribute to `cfg` (whose attrs array has room for one more).  DVM_B200_NO_CHAIN switches it off.
inline void ChainAttribute(cudaLaunchConfig_t *cfg, cudaLaunchAttribute *attrs) {
  static const bool off = getenv("DVM_B200_NO_CHAIN") != nullptr;
  cfg->attrs = attrs;
  if (off) return;
  attrs[cfg->numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[cfg->numAttrs].val.programmaticStreamSerializationAllowed = 1;
  ++cfg->numAttrs;
}

}  // namespace dvmb

#endif  // DVM_B200_CHAIN_CUH_
