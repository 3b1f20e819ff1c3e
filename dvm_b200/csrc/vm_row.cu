// Row kernels: the two normalisation shapes of a vector stage (row_match.cc) as straight-line kernels.
//
// The vector interpreter spends its time on such a graph dispatching (a [64, 256, 56, 56] batch-norm ran at 0.47 of the copy
// bandwidth), and where rows do not start on 16 bytes it falls back to loads and stores of single elements ([32, 200, 27, 27]:
// 131 us for 19 MB).  Here a thread works on 16-byte units at aligned addresses: a run of a tensor is the units that hold at
// least one of its elements, lanes outside the run are masked, and since every streamed tensor of a group lies alike
// relative to 16 bytes, an element is at the same place of its unit in all of them - no shifting, whatever the row length.
//
//   dvm_b200_row_stats_affine  a group (a channel of an NCHW tensor, a row) is shared by a cluster of CTAs; its units stay
//                              in shared memory between the pass that takes the sums and the pass that writes the result,
//                              so memory is read once.  Sums are combined by shuffles and through distributed shared
//                              memory, always in the same order.
//   dvm_b200_row_rms_gate      a row per group of 32 to 512 threads, every load of the row in flight before the first use.
//
// The scalar sections (means, reciprocal roots, what is stored per group) are the usual ones, computed in closed form; stages with
// others run on the interpreter.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <vector>

#include "bounded_wait.cuh"
#include "chain.cuh"
#include "runtime.h"
#include "vm_ops.cuh"
#include "vm_row.h"

namespace dvmb {

__device__ WaitStatus g_row_status = {0u, 0u};

namespace {

constexpr uint32_t kMaxRowThreads = 512;
constexpr uint32_t kMaxWarps = kMaxRowThreads / 32;

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint4 ld_unit(const uint8_t *p) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// ---- units: 16 bytes at an aligned address, kE elements of 16 bits -----------------------------------------
constexpr uint32_t kE = 8;

template <uint32_t DT>
__device__ __forceinline__ void unpack_unit(const uint4 &q, float (&x)[kE]) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if constexpr (DT == T_BF16) {
      x[2 * i] = u2f(w[i] << 16);
      x[2 * i + 1] = u2f(w[i] & 0xffff0000u);
    } else {
      const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
      x[2 * i] = f.x;
      x[2 * i + 1] = f.y;
    }
  }
}
template <uint32_t DT>
__device__ __forceinline__ uint4 pack_unit(const float (&x)[kE]) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if constexpr (DT == T_BF16) {
      w[i] = pack_bf16x2(x[2 * i], x[2 * i + 1]);
    } else {
      const __half2 h = __floats2half2_rn(x[2 * i], x[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t *>(&h);
    }
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
// Two neighbouring elements as one 64-bit register pair (one issue slot per packed operation).
struct F2 {
  uint64_t v;
};
__device__ __forceinline__ F2 f2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 halves(F2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
  return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
template <uint32_t DT>
__device__ __forceinline__ void unpack_pairs(const uint4 &q, F2 (&x)[kE / 2]) {
  float f[kE];
  unpack_unit<DT>(q, f);
#pragma unroll
  for (uint32_t i = 0; i < kE / 2; ++i) x[i] = f2(f[2 * i], f[2 * i + 1]);
}
template <uint32_t DT>
__device__ __forceinline__ uint4 pack_pairs(const F2 (&x)[kE / 2]) {
  float f[kE];
#pragma unroll
  for (uint32_t i = 0; i < kE / 2; ++i) {
    const float2 h = halves(x[i]);
    f[2 * i] = h.x;
    f[2 * i + 1] = h.y;
  }
  return pack_unit<DT>(f);
}
// Zero outside lanes [lo, hi).
__device__ __forceinline__ void mask_pairs(F2 (&x)[kE / 2], uint32_t lo, uint32_t hi) {
#pragma unroll
  for (uint32_t i = 0; i < kE / 2; ++i) {
    const float2 h = halves(x[i]);
    x[i] = f2(2 * i >= lo && 2 * i < hi ? h.x : 0.0f, 2 * i + 1 >= lo && 2 * i + 1 < hi ? h.y : 0.0f);
  }
}
// Lanes [lo, hi) of a unit to memory: whole units as one store, the ends of a run element by element.
__device__ __forceinline__ void store_unit(uint8_t *p, const uint4 &q, uint32_t lo, uint32_t hi) {
  if (lo == 0 && hi == kE) {
    *reinterpret_cast<uint4 *>(p) = q;
    return;
  }
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (uint32_t i = 0; i < kE; ++i)
    if (i >= lo && i < hi) reinterpret_cast<unsigned short *>(p)[i] = (unsigned short)(w[i >> 1] >> (16u * (i & 1u)));
}

__device__ __forceinline__ void group_coords(const RowParam &P, uint32_t g, uint32_t (&k)[kMaxKept]) {
#pragma unroll
  for (int j = kMaxKept - 1; j > 0; --j) {
    const uint32_t q = g / P.kept_size[j];
    k[j] = g - q * P.kept_size[j];
    g = q;
  }
  k[0] = g;
}
__device__ __forceinline__ uint32_t group_offset(const uint32_t (&stride)[kMaxKept], const uint32_t (&k)[kMaxKept]) {
  return k[0] * stride[0] + k[1] * stride[1] + k[2] * stride[2];
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---- statistics, then an affine map ------------------------------------------------------------------------
// Warps 0-7 work, warp 8 streams: a CTA's share of a group is a range of its units, copied to shared memory unit by unit in
// their order (a bulk copy per run), the next group's while this one is worked on.
constexpr uint32_t kWorkThreads = 256, kWorkWarps = kWorkThreads / 32;
constexpr uint32_t kStatsThreads = kWorkThreads + 32;
constexpr uint32_t kMaxBuffers = 2;
// shared memory: the header below, then the buffers
struct StatsShared {
  uint64_t full[kMaxBuffers], empty[kMaxBuffers], sums[2];
  float2 sum[2][8 * kWorkWarps];   // every warp's sums of every CTA of the cluster, in turn for one group and the next
};
constexpr uint32_t kStatsHeader = (sizeof(StatsShared) + 127u) & ~127u;

__device__ __forceinline__ uint32_t saddr_of(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ bool try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
    "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
    : "=r"(ok)
    : "r"(bar), "r"(parity)
    : "memory");
  return ok != 0;
}
__device__ __noinline__ void wait_slow(uint32_t bar, uint32_t parity, uint32_t code, LaunchTag epoch) {
  bounded_spin([&]() { return try_wait(bar, parity); }, code, &g_row_status, epoch, kWaitLimitNs);
}
__device__ __forceinline__ void wait_for(uint32_t bar, uint32_t parity, uint32_t code, LaunchTag epoch) {
  if (!try_wait(bar, parity)) wait_slow(bar, parity, code, epoch);
}
__device__ __forceinline__ void expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void arrive(uint32_t bar) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void work_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kWorkThreads) : "memory"); }

// kWhole: every run starts and ends on 16 bytes, so that every unit belongs to its run with all lanes.
template <uint32_t DT, bool kWhole>
__device__ __forceinline__ void stats_affine_body(const RowParam &P, const LaunchTag epoch) {
  constexpr uint32_t E = kE, SH = 1;
  extern __shared__ __align__(128) uint8_t smem[];
  StatsShared &sm = *reinterpret_cast<StatsShared *>(smem);
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
  const uint32_t CL = P.cluster, rank = CL > 1 ? cluster_rank() : 0u;
  const uint32_t spr = P.slots_per_run, u_begin = min(P.runs * spr, rank * P.per_cta), u_end = min(P.runs * spr, u_begin + P.per_cta);
  const uint32_t run_bytes = P.run_len << SH;
  const uint64_t run_step = (uint64_t)P.run_stride << SH;
  const uint32_t g_first = blockIdx.x / CL, g_step = gridDim.x / CL;
  const uint32_t buffer_bytes = P.buffer_bytes, NB = P.buffers;
  auto buffer = [&](uint32_t b) { return kStatsHeader + b * buffer_bytes; };
  auto group_base = [&](uint32_t g, uint32_t i, uint32_t (&k)[kMaxKept]) {
    group_coords(P, g, k);
    return reinterpret_cast<uint8_t *>(P.stream[i].ptr) + ((uint64_t)group_offset(P.stream[i].kstride, k) << SH);
  };

  if (tid == 0) {
    for (uint32_t i = 0; i < kMaxBuffers; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr_of(&sm.full[i])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr_of(&sm.empty[i])), "r"(kWorkWarps));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr_of(&sm.sums[i])));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (CL > 1) {   // every CTA's barriers exist before a peer signals them
    cluster_arrive();
    cluster_wait();
  }
  chain_wait();
  chain_launch();

  if (warp == kWorkWarps) {
    // ------------------------------ streaming warp ------------------------------
    const uint32_t r_begin = u_begin / spr, r_end = u_end == u_begin ? r_begin : (u_end - 1u) / spr + 1u;
    uint32_t b = 0, parity = 1;
    for (uint32_t g = g_first; g < P.groups; g += g_step) {
      uint32_t k[kMaxKept];
      const uint8_t *const x0 = group_base(g, 0, k);
      // the units of run r in this CTA's share that hold at least one element: source address and bytes
      auto piece = [&](uint32_t r, const uint8_t *&src, uint32_t &dst) {
        const uint8_t *const s = x0 + r * run_step;
        const uint32_t mis = (uint32_t)reinterpret_cast<uint64_t>(s) & 15u;
        const uint32_t n = (mis + run_bytes + 15u) >> 4;   // units the run has
        const uint32_t c0 = r * spr < u_begin ? u_begin - r * spr : 0u, c1 = min(n, u_end - r * spr);
        src = s - mis + 16u * c0;
        dst = 16u * (r * spr + c0 - u_begin);
        return c1 > c0 ? 16u * (c1 - c0) : 0u;
      };
      uint32_t total = 0;
      for (uint32_t r = r_begin + lane; r < r_end; r += 32u) {
        const uint8_t *src;
        uint32_t dst;
        total += piece(r, src, dst);
      }
      total = __reduce_add_sync(0xffffffffu, total);
      const uint32_t full = saddr_of(&sm.full[b]);
      wait_for(saddr_of(&sm.empty[b]), parity, 1, epoch);
      if (lane == 0) expect_tx(full, total);
      __syncwarp();
      for (uint32_t r = r_begin + lane; r < r_end; r += 32u) {
        const uint8_t *src;
        uint32_t dst;
        const uint32_t bytes = piece(r, src, dst);
        if (bytes != 0)
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(saddr_of(smem + buffer(b)) + dst),
                       "l"(src), "r"(bytes), "r"(full)
                       : "memory");
      }
      if (++b == NB) {
        b = 0;
        parity ^= 1u;
      }
    }
    __syncwarp();
  } else {
    // ------------------------------ working warps ------------------------------
    const uint32_t n_units = u_end - u_begin;
    const uint32_t r_first = (u_begin + tid) / spr, c_first = u_begin + tid - r_first * spr;
    const uint32_t step_r = kWorkThreads / spr, step_c = kWorkThreads - step_r * spr;
    uint32_t b = 0, parity = 0, turn = 0, turn_parity = 0;
    for (uint32_t g = g_first; g < P.groups; g += g_step) {
      uint32_t k[kMaxKept];
      uint8_t *const y0 = group_base(g, 1, k);
      const uint8_t *const x0 = group_base(g, 0, k);
      float shift = 0.0f, gamma = 1.0f, beta = -0.0f;
      auto scalar_in = [&](uint32_t i) {
        const TensorDesc &td = P.scalar[i];
        return load_elem(td.dtype, reinterpret_cast<const uint8_t *>(td.ptr), group_offset(td.kstride, k));
      };
      if (P.at_shift != kRowNone) shift = u2f(scalar_in(P.at_shift));
      if (P.at_gamma != kRowNone) gamma = u2f(scalar_in(P.at_gamma));
      if (P.at_beta != kRowNone) beta = u2f(scalar_in(P.at_beta));
      uint8_t *const data = smem + buffer(b);
      wait_for(saddr_of(&sm.full[b]), parity, 2, epoch);
      if (!kWhole) {
        // Lanes of a run's first and last units that lie outside it take the shift's value (x's own first element), whose
        // deviation is zero: the sums then need no masks.
        for (uint32_t i = tid; i < 2u * P.runs; i += kWorkThreads) {
          const uint32_t r = i >> 1, mis = (uint32_t)(reinterpret_cast<uint64_t>(x0) + r * run_step) & 15u;
          const uint32_t head = mis >> SH, stop = (mis + run_bytes) >> SH;   // elements from the run's first unit on
          const uint32_t from = (i & 1u) ? stop : 0u, to = (i & 1u) ? spr * E : head;
          for (uint32_t e = from; e < to; ++e) {
            const uint32_t u = r * spr + e / E;
            if (u < u_begin || u >= u_end) continue;
            uint8_t *const at = data + 16u * (u - u_begin);
            if constexpr (DT == T_F16) {
              reinterpret_cast<__half *>(at)[e % E] = __float2half_rn(shift);
            } else {
              reinterpret_cast<unsigned short *>(at)[e % E] = (unsigned short)(f2u(shift) >> 16);
            }
          }
        }
        work_sync();
      }
      // sums of d and d * d, in eight partial sums per thread
      F2 s1[E / 2], s2[E / 2];
#pragma unroll
      for (uint32_t i = 0; i < E / 2; ++i) s1[i] = s2[i] = f2(0.0f, 0.0f);
      const F2 minus_shift = f2(-shift, -shift);
#pragma unroll 4
      for (uint32_t u = tid; u < n_units; u += kWorkThreads) {
        F2 d[E / 2];
        unpack_pairs<DT>(*reinterpret_cast<const uint4 *>(data + 16u * u), d);
#pragma unroll
        for (uint32_t i = 0; i < E / 2; ++i) {
          d[i] = add2(d[i], minus_shift);
          s1[i] = add2(s1[i], d[i]);
          s2[i] = fma2(d[i], d[i], s2[i]);
        }
      }
#pragma unroll
      for (uint32_t h = E / 4; h > 0; h >>= 1)
#pragma unroll
        for (uint32_t i = 0; i < h; ++i) {
          s1[i] = add2(s1[i], s1[i + h]);
          s2[i] = add2(s2[i], s2[i + h]);
        }
      const float2 h1 = halves(s1[0]), h2 = halves(s2[0]);
      float2 t = make_float2(warp_sum(h1.x + h1.y), warp_sum(h2.x + h2.y));
      // every warp sends its sums to every CTA of the cluster; then each warp adds all of them, in the same order everywhere
      if (CL > 1) {
        const uint32_t bar = saddr_of(&sm.sums[turn]);
        if (tid == 0) expect_tx(bar, CL * kWorkWarps * 8u);
        if (lane < CL) {
          uint32_t to, to_bar;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(saddr_of(&sm.sum[turn][rank * kWorkWarps + warp])), "r"(lane));
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to_bar) : "r"(bar), "r"(lane));
          asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(to), "l"(f2(t.x, t.y).v), "r"(to_bar) : "memory");
        }
        __syncwarp();
        wait_for(bar, turn_parity, 3, epoch);
      } else {
        if (lane == 0) sm.sum[turn][warp] = t;
        work_sync();
      }
      {
        const uint32_t n = CL * kWorkWarps;
        t = lane < n ? sm.sum[turn][lane] : make_float2(0.0f, 0.0f);
        if (lane + 32u < n) {
          const float2 q = sm.sum[turn][lane + 32u];
          t.x += q.x;
          t.y += q.y;
        }
        t.x = warp_sum(t.x);
        t.y = warp_sum(t.y);
      }
      turn ^= 1u;
      if (turn == 0) turn_parity ^= 1u;
      const float ti = __fmul_rn(t.x, P.i1);
      const float mean = __fadd_rn(ti, shift), var = __fmul_rn(__fsub_rn(t.y, __fmul_rn(t.x, ti)), P.i2);
      const float rstd = fast_div(1.0f, sqrtf(__fadd_rn(var, P.eps)));
      // (an absent gamma or beta is an identity that changes no bit: * 1, + (-0))
      const F2 m0 = f2(-mean, -mean), m1 = f2(rstd, rstd), m2 = f2(gamma, gamma), m3 = f2(beta, beta);
      uint8_t *run = y0 + r_first * run_step;   // the run's start in the result, the unit's number in the run
      uint32_t c = c_first;
#pragma unroll 4
      for (uint32_t u = tid; u < n_units; u += kWorkThreads) {
        F2 d[E / 2];
        unpack_pairs<DT>(*reinterpret_cast<const uint4 *>(data + 16u * u), d);
#pragma unroll
        for (uint32_t i = 0; i < E / 2; ++i) d[i] = fma2(mul2(add2(d[i], m0), m1), m2, m3);
        const uint4 q = pack_pairs<DT>(d);
        if (kWhole) {
          *reinterpret_cast<uint4 *>(run + 16u * c) = q;
        } else {
          const uint32_t mis = (uint32_t)reinterpret_cast<uint64_t>(run) & 15u;
          uint8_t *const at = run - mis + 16u * c;
          if (c != 0 && c + 2u < spr) {
            *reinterpret_cast<uint4 *>(at) = q;
          } else {
            const int32_t left = (int32_t)(mis + run_bytes) - (int32_t)(16u * c);
            store_unit(at, q, c == 0 ? mis >> SH : 0u, left <= 0 ? 0u : min(E, (uint32_t)left >> SH));
          }
        }
        run += step_r * run_step;
        c += step_c;
        if (c >= spr) {
          c -= spr;
          run += run_step;
        }
      }
      // the buffer is free for the next copies (whose writes come through the async proxy, behind the edge lanes' writes)
      if (!kWhole) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) arrive(saddr_of(&sm.empty[b]));
      if (++b == NB) {
        b = 0;
        parity ^= 1u;
      }
      if (tid == 0 && rank == 0) {
        auto put = [&](uint32_t i, float f) {
          if (i == kRowNone) return;
          const TensorDesc &td = P.scalar[i];
          store_elem(td.dtype, reinterpret_cast<uint8_t *>(td.ptr), group_offset(td.kstride, k), f2u(f));
        };
        put(P.at_mean, mean);
        put(P.at_var, var);
      }
    }
    __syncwarp();
  }
  if (CL > 1) {   // no CTA leaves while a peer may still send to it
    cluster_arrive();
    cluster_wait();
  }
}

// ---- residual RMS norm beside a gated product ----------------------------------------------------------------
// Eight 16-bit elements that start `mis` elements in front of element 0 of `base` plus 8 c (a vector shared by all rows, read
// against the row's own alignment).
__device__ __forceinline__ uint4 shifted_unit(const unsigned short *base, int32_t first, uint32_t len) {
  const uint64_t s = reinterpret_cast<uint64_t>(base) + (int64_t)first * 2;
  const uint64_t a = s & ~15ull, b0 = reinterpret_cast<uint64_t>(base), b1 = b0 + 2ull * len;
  const uint32_t off = (uint32_t)(s & 15ull) >> 1;
  uint4 lo = make_uint4(0, 0, 0, 0), hi = lo;
  if (a + 16 > b0 && a < b1) lo = gload(reinterpret_cast<const uint4 *>(a));
  if (off == 0) return lo;
  if (a + 16 < b1) hi = gload(reinterpret_cast<const uint4 *>(a) + 1);
  const uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
  uint32_t p[6], q[5];
#pragma unroll
  for (int i = 0; i < 6; ++i) p[i] = (off & 4u) ? w[i + 2] : w[i];
#pragma unroll
  for (int i = 0; i < 5; ++i) q[i] = (off & 2u) ? p[i + 1] : p[i];
  const uint32_t bits = (off & 1u) * 16u;
  return make_uint4(__funnelshift_r(q[0], q[1], bits), __funnelshift_r(q[1], q[2], bits), __funnelshift_r(q[2], q[3], bits),
                    __funnelshift_r(q[3], q[4], bits));
}
__device__ __forceinline__ float rcp_fast(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

template <uint32_t DT, int K>
__device__ __forceinline__ void rms_gate_body(const RowParam &P) {
  __shared__ float part[kMaxWarps];   // sum of each warp
  chain_wait();
  chain_launch();
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
  const uint32_t tg = P.tg, rows = blockDim.x / tg, row_in_cta = tid / tg, t = tid - row_in_cta * tg;
  const uint32_t g = blockIdx.x * rows + row_in_cta;
  const bool live = g < P.groups;
  uint32_t k[kMaxKept];
  group_coords(P, live ? g : 0u, k);
  auto base_of = [&](uint32_t i) { return reinterpret_cast<uint8_t *>(P.stream[i].ptr) + ((uint64_t)group_offset(P.stream[i].kstride, k) << 1); };
  const uint8_t *const a0 = base_of(0);
  const uint32_t mis = (uint32_t)reinterpret_cast<uint64_t>(a0) & 15u, row_bytes = P.run_len * 2u;
  auto lanes = [&](uint32_t c, uint32_t &lo, uint32_t &hi) {
    lo = c == 0 ? mis >> 1 : 0u;
    const int32_t left = (int32_t)(mis + row_bytes) - (int32_t)(16u * c);
    hi = !live || left <= 0 ? 0u : min(8u, (uint32_t)left >> 1);
  };
  uint4 va[K], vb[K], vg[K], vu[K], vw[K];
#pragma unroll
  for (int j = 0; j < K; ++j) {
    const uint32_t c = t + j * tg;
    uint32_t lo, hi;
    lanes(c, lo, hi);
    va[j] = vb[j] = vg[j] = vu[j] = vw[j] = make_uint4(0, 0, 0, 0);
    if (hi > lo) {
      const uint64_t off = 16ull * c - mis;
      va[j] = ld_unit(a0 + off);
      if (P.have_b) vb[j] = ld_unit(base_of(1) + off);
      if (P.have_gate) {
        vg[j] = ld_unit(base_of(4) + off);
        vu[j] = ld_unit(base_of(5) + off);
      }
      if (P.have_w) vw[j] = shifted_unit(reinterpret_cast<const unsigned short *>(P.stream[2].ptr), (int32_t)(8u * c) - (int32_t)(mis >> 1), P.run_len);
    }
  }
  // the residual sum, and the sum of its squares
  F2 x[K][4];
  float s = 0.0f;
#pragma unroll
  for (int j = 0; j < K; ++j) {
    uint32_t lo, hi;
    lanes(t + j * tg, lo, hi);
    unpack_pairs<DT>(va[j], x[j]);
    if (P.have_b) {
      F2 b[4];
      unpack_pairs<DT>(vb[j], b);
#pragma unroll
      for (int i = 0; i < 4; ++i) x[j][i] = add2(x[j][i], b[i]);
    }
    if (lo != 0 || hi != 8u) mask_pairs(x[j], lo, hi);
    F2 q = mul2(x[j][0], x[j][0]);
#pragma unroll
    for (int i = 1; i < 4; ++i) q = fma2(x[j][i], x[j][i], q);
    const float2 h = halves(q);
    s += h.x + h.y;
  }
  s = warp_sum(s);
  if (tg > 32u) {
    if (lane == 0) part[warp] = s;
  }
  // the gated product does not need the row's sum: it fills the time until every warp has delivered its part
  if (P.have_gate) {
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const uint32_t c = t + j * tg;
      uint32_t lo, hi;
      lanes(c, lo, hi);
      if (hi > lo) {
        float gg[8];
        F2 uu[4], y[4];
        unpack_unit<DT>(vg[j], gg);
        unpack_pairs<DT>(vu[j], uu);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float e0 = __fadd_rn(fast_exp(-gg[2 * i]), 1.0f), e1 = __fadd_rn(fast_exp(-gg[2 * i + 1]), 1.0f);
          y[i] = mul2(mul2(f2(rcp_fast(e0), rcp_fast(e1)), f2(gg[2 * i], gg[2 * i + 1])), uu[i]);
        }
        store_unit(base_of(6) + (16ull * c - mis), pack_pairs<DT>(y), lo, hi);
      }
    }
  }
  if (tg > 32u) {
    __syncthreads();
    const uint32_t nw = tg >> 5;
    s = warp_sum(lane < nw ? part[row_in_cta * nw + lane] : 0.0f);
  }
  const float scale = fast_div(1.0f, sqrtf(__fadd_rn(__fmul_rn(s, P.i1), P.eps)));
  const F2 scale2 = f2(scale, scale);
#pragma unroll
  for (int j = 0; j < K; ++j) {
    const uint32_t c = t + j * tg;
    uint32_t lo, hi;
    lanes(c, lo, hi);
    if (hi > lo) {
      F2 y[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) y[i] = mul2(x[j][i], scale2);
      if (P.have_w) {
        F2 w[4];
        unpack_pairs<DT>(vw[j], w);
#pragma unroll
        for (int i = 0; i < 4; ++i) y[i] = mul2(y[i], w[i]);
      }
      store_unit(base_of(3) + (16ull * c - mis), pack_pairs<DT>(y), lo, hi);
    }
  }
}

}  // namespace

#define DVMB_ROW_STATS(NAME, DT, WHOLE)                                                                             \
  __global__ void __launch_bounds__(kStatsThreads, 2) NAME(const __grid_constant__ RowParam P, const LaunchTag epoch) { \
    stats_affine_body<DT, WHOLE>(P, epoch);                                                                           \
  }
DVMB_ROW_STATS(dvm_b200_row_stats_affine_f16, T_F16, false)
DVMB_ROW_STATS(dvm_b200_row_stats_affine_bf16, T_BF16, false)
DVMB_ROW_STATS(dvm_b200_row_stats_affine_f16_whole, T_F16, true)
DVMB_ROW_STATS(dvm_b200_row_stats_affine_bf16_whole, T_BF16, true)
#undef DVMB_ROW_STATS
#define DVMB_ROW_RMS(NAME, DT, K)                                                                    \
  __global__ void __launch_bounds__(kMaxRowThreads) NAME(const __grid_constant__ RowParam P) { rms_gate_body<DT, K>(P); }
DVMB_ROW_RMS(dvm_b200_row_rms_gate_f16_1, T_F16, 1)
DVMB_ROW_RMS(dvm_b200_row_rms_gate_bf16_1, T_BF16, 1)
DVMB_ROW_RMS(dvm_b200_row_rms_gate_f16_2, T_F16, 2)
DVMB_ROW_RMS(dvm_b200_row_rms_gate_bf16_2, T_BF16, 2)
#undef DVMB_ROW_RMS

namespace {

// Every run starts on 16 bytes.
bool RunsAligned(const RowParam &p) {
  uint64_t m = p.stream[0].ptr | (static_cast<uint64_t>(p.run_stride) << 1);
  for (int j = 0; j < kMaxKept; ++j)
    if (p.kept_size[j] != 1) m |= static_cast<uint64_t>(p.stream[0].kstride[j]) << 1;
  return (m & 15u) == 0;
}
// 16-byte units a run touches at most: one more where runs may start inside a unit
uint32_t UnitsPerRun(const RowParam &p) {
  const uint64_t bytes = static_cast<uint64_t>(p.run_len) << 1;
  return static_cast<uint32_t>(RunsAligned(p) ? (bytes + 15) / 16 : (bytes + 15 + 14) / 16);
}

// Clusters of `cl` CTAs that run at a time, as the driver says; asked once per kernel and launch shape.
uint32_t ResidentClusters(const void *fn, uint32_t threads, uint32_t smem, uint32_t cl, uint32_t sms) {
  struct Fit { const void *fn; uint32_t threads, smem, cl, n; int dev; };
  static std::mutex lock;
  static Fit known[64];
  static uint32_t count = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> guard(lock);
  for (uint32_t i = 0; i < std::min(count, 64u); ++i) {
    const Fit &f = known[i];
    if (f.fn == fn && f.threads == threads && f.smem == smem && f.cl == cl && f.dev == dev) return f.n;
  }
  int n = 0;
  if (cl > 1) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sms * cl, 1, 1);
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cl;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) n = 0;
  } else if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, static_cast<int>(threads), smem) == cudaSuccess) {
    n *= static_cast<int>(sms);
  }
  if (n <= 0) {
    cudaGetLastError();
    n = static_cast<int>(std::max(1u, sms / cl));
  }
  known[count++ & 63u] = {fn, threads, smem, cl, static_cast<uint32_t>(n), dev};
  return static_cast<uint32_t>(n);
}

// Shared memory of a CTA: two per SM, or one.
constexpr uint32_t kHalfSm = 112 * 1024, kWholeSm = 226 * 1024;
// A group of `units` units in at most eight CTAs: the cluster, the buffers of each CTA and their size.  False: it does not fit.
bool StatsPlan(uint32_t units, uint32_t groups, uint32_t sms, RowParam *p, uint32_t *smem) {
  const uint32_t half = kHalfSm - kStatsHeader - 1024u, whole = kWholeSm - kStatsHeader - 1024u;
  // The smallest cluster that holds a group with two buffers per CTA, two CTAs per SM (the next group on its way while this one is
  // worked on), then with one (the other CTA's copies overlap), then one CTA with one.  Layouts are not compared by the CTA slots
  // that they fill: a [64, 256, 56, 56] batch-norm runs in 33 clusters of eight, 264 of 296 slots.
  uint32_t cl = 1, room = half / 2, buffers = 2;
  auto fits = [&]() { return (static_cast<uint64_t>(units) + cl - 1) / cl * 16u <= room; };
  while (cl < 8u && !fits()) cl *= 2;
  if (!fits()) {
    room = half;
    buffers = 1;
  }
  if (!fits()) room = whole;
  if (!fits()) return false;
  // more CTAs per group while SMs would stay idle and every thread still has a unit
  while (cl < 8u && static_cast<uint64_t>(groups) * cl * 2 <= 2ull * sms && units / (2 * cl) >= kWorkThreads) cl *= 2;
  p->cluster = cl;
  p->per_cta = (units + cl - 1) / cl;
  p->buffers = buffers;
  p->buffer_bytes = (p->per_cta * 16u + 127u) & ~127u;
  *smem = kStatsHeader + buffers * p->buffer_bytes;
  return true;
}

constexpr uint32_t kRmsMaxUnits = 2 * kMaxRowThreads;
static_assert(kRowRmsMaxElems == kRmsMaxUnits * 8, "two units of eight elements per thread");

}  // namespace

bool RowAddressesOk(const RowParam &p) {
  if (p.form == ROW_OFF || p.stream[0].ptr == 0) return false;
  const uint32_t n = p.form == ROW_STATS_AFFINE ? 2u : static_cast<uint32_t>(kRowMaxStreams);
  for (uint32_t i = 0; i < n; ++i) {
    if (p.form == ROW_RMS_GATE && i == 2) {   // (the row vector is read at any element address)
      if (p.have_w && (p.stream[2].ptr & 1u)) return false;
      continue;
    }
    if (p.form == ROW_RMS_GATE && p.stream[i].ptr == 0) continue;   // an absent stream
    if (((p.stream[i].ptr ^ p.stream[0].ptr) & 15u) != 0 || (p.stream[i].ptr & 1u) != 0) return false;
  }
  if ((static_cast<uint64_t>(p.run_len) << 1) >= (1ull << 30)) return false;   // (32-bit byte counts inside a run)
  if (p.form == ROW_RMS_GATE && UnitsPerRun(p) > kRmsMaxUnits) return false;   // (a row that does not fit a CTA's registers)
  if (p.form == ROW_RMS_GATE) return true;
  const uint64_t units = static_cast<uint64_t>(p.runs) * UnitsPerRun(p);
  RowParam plan = {};
  uint32_t smem = 0;
  const uint32_t sms = static_cast<uint32_t>(Runtime::Get().sm_count_or_default());
  return units < (1ull << 20) && StatsPlan(static_cast<uint32_t>(units), p.groups, sms, &plan, &smem);
}

// Estimates of both kernels in microseconds, a fit to about 1200 launches of 16 to 400 000 groups of 4 to 200 000 elements timed back
// to back in either (runs of 1 to 256, aligned and not).  What decides:
//  - A statistics CTA takes 1.3 us for a group (2.3 with edges) however short it is; the interpreter gives short groups a slice of
//    a CTA: [100000, 64] fp16 432 us here and 62 there, [1200, 64] 7.7 and 10.7, [5000, 512] 23 and 31, [5000, 4096] 29 and 68.
//  - An RMS row of up to 32 units takes a warp about 0.35 ns in all: [400000, 16] bf16 138 us and 37, [400000, 64] 148 and 144.
//  - RMS rows of more than 512 units leave two CTAs on an SM: from 12 rows per SM on, rows that the interpreter's chunks divide
//    are faster there ([5000, 6144] 78 and 58, [600, 6144] 9.6 and 10.3), others are not ([5000, 5120] 74 and 154).
bool RowKernelPays(const RowParam &p, uint32_t chunk_elems) {
  const uint32_t sms = static_cast<uint32_t>(Runtime::Get().sm_count_or_default()), units = UnitsPerRun(p);
  const double groups = p.groups, n = static_cast<double>(p.runs) * p.run_len;
  const bool single = p.runs == 1;
  const bool even = chunk_elems != 0 && static_cast<uint64_t>(p.runs) * p.run_len % chunk_elems == 0;   // no chunk is partly filled
  // runs in whole units of 16 bytes, and in whole granules of four elements (what the interpreter loads at a time)
  const bool whole = RunsAligned(p) && ((p.run_len << 1) & 15u) == 0;
  uint64_t m = p.stream[0].ptr | (static_cast<uint64_t>(p.run_stride | p.run_len) << 1);
  for (int j = 0; j < kMaxKept; ++j)
    if (p.kept_size[j] != 1) m |= static_cast<uint64_t>(p.stream[0].kstride[j]) << 1;
  const bool granules = (m & 7u) == 0;
  double padded = 16.0;   // a short group's slice: a power of two of elements
  while (padded < n) padded *= 2.0;

  if (p.form == ROW_RMS_GATE) {
    if (units <= 32u) {
      const double w = p.have_w != 0, b = p.have_b != 0, g = p.have_gate != 0;
      const double row = 1.5 + groups * 1e-3 * (0.345 + 0.035 * w + 0.015 * b + 0.095 * g);
      const double per_elem = 1e-6 * (5.0 + 1.5 * w + 3.3 * b + 6.2 * g) * (granules ? 1.0 : 2.2);
      return row <= std::max(7.0 + 5.0 * b + 5.0 * g, 5.0 + groups * padded * per_elem);
    }
    return !whole || !even || units <= kMaxRowThreads || groups <= 12.0 * sms;
  }

  RowParam plan = {};
  uint32_t smem = 0;
  if (!StatsPlan(p.runs * units, p.groups, sms, &plan, &smem)) return false;
  const uint32_t slots = std::max(1u, (smem <= kHalfSm ? 2u : 1u) * sms / plan.cluster);
  const double rounds = std::ceil(groups / slots);
  if (rounds <= 1.0) return true;   // (a single round answers sooner than the interpreter)
  const double per_group = std::max(whole ? 1.3 : 2.3, 0.6 + 0.035 * p.runs);
  double base, ns;   // the interpreter: a launch, and every group
  if (n <= 512.0) {
    base = granules ? 10.0 : (single ? 15.0 : 25.0);
    ns = padded * 1e-3 * (single ? (granules ? 10.0 : 20.0) : (granules ? 15.0 : 22.0));
  } else if (single) {
    base = granules ? (!even && n > 2048.0 ? 12.5 : 4.5) : 11.0;
    ns = granules ? 3.0 + 3.5 * std::ceil(n / 2048.0) + (even ? 0.0 : 14.0) : 11.0 + 0.0125 * n;
  } else if (granules) {
    base = p.run_len >= 512u ? 9.0 : 10.0;
    ns = p.run_len >= 512u ? 5.0 + n * (p.run_len >= 2048u ? 2.5e-3 : 4.6e-3) : 9.0 + 0.0115 * n + (even ? 0.0 : 10.0);
  } else {
    base = 25.0;
    ns = 30.0 + 0.022 * n;
  }
  return 1.3 + rounds * per_group <= base + groups * ns * 1e-3;
}

int LaunchRow(const RowParam &p_in, void *stream) {
  RowParam p = p_in;
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  const uint32_t units = UnitsPerRun(p);
  p.slots_per_run = units;
  const uint32_t sms = static_cast<uint32_t>(Runtime::Get().sm_count_or_default());
  if (p.form == ROW_RMS_GATE) {
    // two units per thread keep more loads in flight; one unit and more threads answer sooner while there are few rows
    const bool few = static_cast<uint64_t>(p.groups) < 4ull * sms;
    const uint32_t per_thread = units > kMaxRowThreads || (!few && units > 64u) ? 2u : 1u;
    uint32_t tg = 32;
    while (tg * per_thread < units) tg *= 2;
    p.tg = tg;
    const uint32_t block = tg < 128u ? 128u : tg, rows = block / tg;
    using Fn = void (*)(const RowParam);
    const Fn fn = p.dtype == T_F16 ? (per_thread == 1 ? dvm_b200_row_rms_gate_f16_1 : dvm_b200_row_rms_gate_f16_2)
                                   : (per_thread == 1 ? dvm_b200_row_rms_gate_bf16_1 : dvm_b200_row_rms_gate_bf16_2);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = dim3((p.groups + rows - 1) / rows, 1, 1);
    cfg.blockDim = dim3(block, 1, 1);
    cfg.stream = s;
    ChainAttribute(&cfg, attr);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, fn, p);
    return e != cudaSuccess ? static_cast<int>(e) : static_cast<int>(cudaGetLastError());
  }
  uint32_t smem = 0;
  if (!StatsPlan(p.runs * units, p.groups, sms, &p, &smem)) return -7;
  const bool whole = RunsAligned(p) && ((p.run_len << 1) & 15u) == 0;
  using Fn = void (*)(const RowParam, const LaunchTag);
  static const Fn table[2][2] = {{dvm_b200_row_stats_affine_f16, dvm_b200_row_stats_affine_bf16},
                                 {dvm_b200_row_stats_affine_f16_whole, dvm_b200_row_stats_affine_bf16_whole}};
  int dev = 0;
  cudaGetDevice(&dev);
  static bool attr_set[64] = {false};
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    for (auto &row : table)
      for (auto fn : row) {
        const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kWholeSm);
        if (e != cudaSuccess) return static_cast<int>(e);
      }
    attr_set[dev] = true;
  }
  const Fn fn = table[whole ? 1 : 0][p.dtype == T_F16 ? 0 : 1];
  // persistent clusters, as many as are resident at a time
  const uint32_t resident = std::max(1u, ResidentClusters(reinterpret_cast<const void *>(fn), kStatsThreads, smem, p.cluster, sms));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(std::min(p.groups, resident) * p.cluster, 1, 1);
  cfg.blockDim = dim3(kStatsThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.cluster > 1 ? 1 : 0;
  ChainAttribute(&cfg, attr);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, fn, p, NextLaunchEpoch());
  return e != cudaSuccess ? static_cast<int>(e) : static_cast<int>(cudaGetLastError());
}

unsigned int ReadRowStatus() {
  WaitStatus v = {0u, 0u};
  const unsigned int zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_row_status, sizeof(v)) != cudaSuccess) return 0xffffffffu;
  if (v.first_error != 0) cudaMemcpyToSymbol(g_row_status, &zero, sizeof(zero), offsetof(WaitStatus, first_error));
  return v.first_error;
}

}  // namespace dvmb
