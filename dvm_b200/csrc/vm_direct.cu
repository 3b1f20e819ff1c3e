// Direct kernel for reduce-free programs over dense tensors that do not keep the chip busy for long.
//
// What bounds it: latency.  The vector interpreter (vm_vector.cu) copies its program to shared memory, sets up a ring and
// starts a producer warp before the first element moves - about 7 us on 16000 elements, whose own work is a microsecond.
// Here a thread loads its eight elements of every input at once, straight into registers, and walks the instruction words
// where they are, in the launch's parameter space (a few hundred bytes instead of 4 KB).
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "chain.cuh"
#include "runtime.h"
#include "vm_direct.h"
#include "vm_ops.cuh"

namespace dvmb {
namespace {

constexpr uint32_t kThreads = 128;
constexpr int kE = 8;   // elements per thread: two granules of four, kThreads granules apart

__device__ __forceinline__ void copy_lanes(uint32_t (&d)[kE], const uint32_t (&s)[kE]) {
#pragma unroll
  for (int i = 0; i < kE; ++i) d[i] = s[i];
}

}  // namespace

__global__ void __launch_bounds__(kThreads, 4) dvm_b200_vm_direct(const __grid_constant__ DirectParam P) {
  chain_wait();
  chain_launch();
  const uint32_t n = P.elems;
  for (uint32_t tile = blockIdx.x * (kE * kThreads); tile < n; tile += gridDim.x * (kE * kThreads)) {
    const uint32_t e[2] = {tile + 4u * threadIdx.x, tile + 4u * (threadIdx.x + kThreads)};
    uint32_t x[kDirectInputs][kE];
#pragma unroll
    for (uint32_t s = 0; s < kDirectInputs; ++s) {
      if (s < P.n_in) {
        const uint8_t *const base = reinterpret_cast<const uint8_t *>(P.ptr[s]);
        const uint32_t dt = P.dtype[s];
        uint4 raw[2];
#pragma unroll
        for (int g = 0; g < 2; ++g) raw[g] = e[g] + 4u <= n ? gload4(dt, base, e[g]) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          unpack4(dt, raw[g], &x[s][4 * g]);
          if (e[g] < n && e[g] + 4u > n) {   // the last granule of a length that is no multiple of four
#pragma unroll
            for (uint32_t i = 0; i < 3; ++i)
              if (e[g] + i < n) x[s][4 * g + i] = load_elem(dt, base, e[g] + i);
          }
        }
      }
    }
    uint32_t acc[kE], t0[kE], t1[kE];
#pragma unroll
    for (int i = 0; i < kE; ++i) acc[i] = t0[i] = t1[i] = 0;
    auto fetch = [&](uint32_t kind, uint32_t idx, uint32_t imm, uint32_t (&b)[kE]) {
      if (kind == K_TENSOR) {
        switch (idx) {
          case 0: copy_lanes(b, x[0]); break;
          case 1: copy_lanes(b, x[1]); break;
          case 2: copy_lanes(b, x[2]); break;
          default: copy_lanes(b, x[3]); break;
        }
      } else if (kind == K_TEMP) {
        if (idx == 0) copy_lanes(b, t0); else copy_lanes(b, t1);
      } else if (kind == K_ACC) {
        copy_lanes(b, acc);
      } else {
#pragma unroll
        for (int i = 0; i < kE; ++i) b[i] = imm;
      }
    };
#pragma unroll 1
    for (uint32_t pc = 0;; ++pc) {
      const uint64_t w = P.code[pc];
      const uint32_t opc = DVMB_OPC(w), sub = DVMB_SUB(w), rnd = DVMB_RND(w);
      if (opc == OP_END) break;
      uint32_t b[kE];
      if (opc == OP_COPY || opc == OP_BIN || opc == OP_CMP || opc == OP_SEL) fetch(DVMB_OKIND(w), DVMB_OIDX(w), DVMB_IMM(w), b);
      const VecOperand<kE> bo{b};
      switch (opc) {
        case OP_ST: {
          const uint32_t dt = P.dtype[sub];
          uint8_t *const base = reinterpret_cast<uint8_t *>(P.ptr[sub]);
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            if (e[g] + 4u <= n) {
              gstore4(dt, base, e[g], &acc[4 * g]);
            } else {
#pragma unroll
              for (uint32_t i = 0; i < 3; ++i)
                if (e[g] + i < n) store_elem(dt, base, e[g] + i, acc[4 * g + i]);
            }
          }
          break;
        }
        case OP_COPY: copy_lanes(acc, b); break;
        case OP_MOV:
          if (DVMB_DST(w) == 0) copy_lanes(t0, acc); else copy_lanes(t1, acc);
          break;
        case OP_UN: apply_un<kE>(sub, acc); apply_round<kE>(rnd, acc); break;
        case OP_BIN: apply_bin<kE>(sub, acc, bo); apply_round<kE>(rnd, acc); break;
        case OP_CMP: apply_cmp<kE>(sub, DVMB_ISINT(w), acc, bo); break;
        case OP_SEL: {
          uint32_t c[kE];
          fetch(sub >> 4, sub & 15u, 0, c);
          apply_sel<kE>(DVMB_ISINT(w), DVMB_DST(w) & 1u, acc, bo, c);
          break;
        }
        case OP_CVT: apply_cvt<kE>(sub, acc); apply_round<kE>(rnd, acc); break;
        default: break;
      }
    }
  }
}

int LaunchDirect(const DirectParam &p, void *stream) {
  const uint32_t tiles = (p.elems + kE * kThreads - 1) / (kE * kThreads);
  const uint32_t most = static_cast<uint32_t>(Runtime::Get().sm_count_or_default()) * 16u;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attrs[1];
  cfg.gridDim = dim3(tiles < most ? tiles : most, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.stream = static_cast<cudaStream_t>(stream);
  ChainAttribute(&cfg, attrs);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, dvm_b200_vm_direct, p);
  return e != cudaSuccess ? static_cast<int>(e) : static_cast<int>(cudaGetLastError());
}

}  // namespace dvmb
