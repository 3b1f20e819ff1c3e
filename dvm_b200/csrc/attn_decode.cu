// Fused attention for a few query rows (decode): O = softmax(scale * Q K^T) V with at most 16 rows of Q per (batch, head).
//
// What bounds it is the read of the key/value cache: [2, 32] heads of 3999 keys of 128 elements are 131 MB, 20 us at the
// measured copy bandwidth.  The 256-row tiles of attn_tcgen05.cu gave that 64 CTAs with 96 KB each in flight and a chain of
// barriers per 128 keys (84 us).  Here the keys of a head are cut over the warps of a cluster of CTAs; a warp streams
// its own keys straight from global memory into the operand registers of mma.sync (16 query rows: the matrix instructions
// cost a tenth of the time the bytes take, so the tensor memory path would gain nothing):
//   - K: contraction order is free as long as Q has the same, so a thread takes 16 consecutive bytes of a key and feeds two
//     K = 16 steps with them; a load instruction of the warp covers 64 bytes of each of eight keys.
//   - V: a thread takes 16 bytes of four keys and pairs neighbouring keys by byte permutes; result column j of n-tile t is
//     element 8 j + t, so that the columns a thread ends up with are consecutive.
// Warps keep their own running maximum and sum; they are combined through shared memory, CTAs through distributed shared
// memory in rank order.  Rounding follows the graph as in attn_tcgen05.cu.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

#include "chain.cuh"
#include "mm_launch.h"
#include "runtime.h"
#include "vm_ops.cuh"

namespace dvmb {
namespace {

constexpr uint32_t kWarps = 4, kThreads = 32 * kWarps;
constexpr uint32_t kRows = 16, kTile = 16;   // query rows of an MMA, keys of a step
constexpr uint32_t kAhead = 2;   // 128-byte lines of K (and of V) per lane that are prefetched
constexpr float kLog2e = 1.4426950408889634f;

struct DecodeArgs {
  uint32_t cluster;
  uint32_t keys_per_warp;   // a multiple of kTile
  uint32_t prefetch;        // the cache comes from memory
};

__device__ __forceinline__ uint32_t rank_in_cluster() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_peer(const float *p, uint32_t rank) {
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float exp2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// C (16 x 8) += A (16 x 16) B (16 x 8).  `lo` are the thread's results of row lane / 4, `hi` of the row eight further.
template <uint32_t DT>
__device__ __forceinline__ void mma16816(float (&lo)[2], float (&hi)[2], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
#define DVMB_MMA(T)                                                                                                        \
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32." T "." T ".f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};" \
               : "+f"(lo[0]), "+f"(lo[1]), "+f"(hi[0]), "+f"(hi[1])                                                        \
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1))
  if (DT == T_BF16) {
    DVMB_MMA("bf16");
  } else {
    DVMB_MMA("f16");
  }
#undef DVMB_MMA
}
template <uint32_t DT>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if (DT == T_BF16) return pack_bf16x2(lo, hi);
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&h);
}
template <uint32_t DT>
__device__ __forceinline__ float2 unpack2(uint32_t p) {
  if (DT == T_BF16) return make_float2(u2f(p << 16), u2f(p & 0xffff0000u));
  return __half22float2(*reinterpret_cast<const __half2 *>(&p));
}
// Two scores as the graph rounds them, in the log2 domain.
template <uint32_t DT, bool SCALE_FIRST>
__device__ __forceinline__ float2 score2(float a, float b, float scale, uint32_t scale2) {
  uint32_t p = pack2<DT>(a, b);
  if (SCALE_FIRST) {
    if (DT == T_BF16) {
      asm("mul.rn.bf16x2 %0, %0, %1;" : "+r"(p) : "r"(scale2));
    } else {
      asm("mul.rn.f16x2 %0, %0, %1;" : "+r"(p) : "r"(scale2));
    }
  }
  float2 x = unpack2<DT>(p);
  const float f = SCALE_FIRST ? kLog2e : scale * kLog2e;
  x.x *= f;
  x.y *= f;
  return x;
}

// Factor of a partial result whose scores had the maximum `m`, in one of maximum `top`.  A partial without a finite score
// counts nothing, but is multiplied all the same: its sums are 0, or NaN where a score was NaN, which the result has to show.
__device__ __forceinline__ float weight_of(float m, float top) { return m == -CUDART_INF_F ? 0.0f : exp2_fast(m - top); }

template <uint32_t D>
struct Combine {
  float m[kWarps][kRows], l[kWarps][kRows];
  float o[kWarps][kRows][D];
};

// (A form for at most eight rows that kept no accumulators for the upper half of the MMA, 168 instead of 233 registers and
// three CTAs per SM, measured 36 us against 25 on [2, 32] heads of 3999 keys.)
// NT: tiles of 16 keys per step.
template <uint32_t DT, uint32_t D, bool SCALE_FIRST, uint32_t NT>
__device__ __forceinline__ void decode_body(const AttnParam &P, const DecodeArgs &A) {
  constexpr uint32_t JK = D / 32, HV = D / 64;   // 16-byte pieces of a key row per thread, 64-element halves of a value row
  constexpr uint32_t kStep = NT * kTile;
  extern __shared__ __align__(16) uint8_t smem[];
  Combine<D> &sm = *reinterpret_cast<Combine<D> *>(smem);
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, q4 = lane & 3u, q8 = lane >> 2;
  const uint32_t CL = A.cluster, rank = CL > 1 ? rank_in_cluster() : 0u;
  const uint32_t head = blockIdx.x / CL;
  const unsigned short *const Q = reinterpret_cast<const unsigned short *>(P.q_ptr) + (uint64_t)head * P.sq * D;
  const unsigned short *const Kh = reinterpret_cast<const unsigned short *>(P.k_ptr) + (uint64_t)head * P.skv * D;
  const unsigned short *const Vh = reinterpret_cast<const unsigned short *>(P.v_ptr) + (uint64_t)head * P.skv * D;
  const uint32_t k_begin = min(P.skv, (rank * kWarps + warp) * A.keys_per_warp), k_end = min(P.skv, k_begin + A.keys_per_warp);

  auto load16 = [](const unsigned short *p, bool ok) {
    uint4 v = make_uint4(0, 0, 0, 0);
    if (ok) asm volatile("ld.global.L1::no_allocate.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
  };
  uint4 kf[NT][2][JK], vf[NT][4][HV];
  auto key_at = [&](uint32_t base, uint32_t u, uint32_t n) { return base + u * kTile + 8u * n + q8; };
  auto value_at = [&](uint32_t base, uint32_t u, uint32_t i) { return base + u * kTile + 2u * q4 + (i & 1u) + (i >> 1) * 8u; };
  auto load_k = [&](uint32_t base) {
#pragma unroll
    for (uint32_t u = 0; u < NT; ++u)
#pragma unroll
      for (uint32_t n = 0; n < 2; ++n) {
        const uint32_t key = key_at(base, u, n);
#pragma unroll
        for (uint32_t j = 0; j < JK; ++j) kf[u][n][j] = load16(Kh + (uint64_t)key * D + j * 32u + q4 * 8u, key < k_end);
      }
  };
  auto load_v = [&](uint32_t base) {
#pragma unroll
    for (uint32_t u = 0; u < NT; ++u)
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i) {
        const uint32_t key = value_at(base, u, i);
#pragma unroll
        for (uint32_t h = 0; h < HV; ++h) vf[u][i][h] = load16(Vh + (uint64_t)key * D + h * 64u + q8 * 8u, key < k_end);
      }
  };
  // The first keys and values are on their way to L2 while the kernel before this one still runs (a prefetch reads nothing
  // that could be stale: L2 holds whatever is written to them meanwhile).
#pragma unroll
  for (uint32_t i = 0; i < kAhead && A.prefetch != 0; ++i) {
    const uint32_t line = i * 32u + lane, key = k_begin + line / (D / 64u), at = line % (D / 64u) * 64u;
    if (key < k_end) {
      asm volatile("prefetch.global.L2 [%0];" ::"l"(Kh + (uint64_t)key * D + at));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(Vh + (uint64_t)key * D + at));
    }
  }
  chain_wait();
  chain_launch();
  load_k(k_begin);
  load_v(k_begin);
  uint32_t qf[2 * JK][4];   // A fragments of Q in K's order of elements
#pragma unroll
  for (uint32_t j = 0; j < JK; ++j) {
#pragma unroll
    for (uint32_t r = 0; r < 2; ++r) {
      const uint32_t row = q8 + 8u * r;
      const uint4 v = load16(Q + row * D + j * 32u + q4 * 8u, row < P.sq);
      qf[2 * j][r] = v.x, qf[2 * j][2 + r] = v.y;
      qf[2 * j + 1][r] = v.z, qf[2 * j + 1][2 + r] = v.w;
    }
  }
  const float scale = u2f(P.scale_bits);
  const uint32_t scale2 = pack2<DT>(scale, scale);
  float o[2][HV][8][2];
#pragma unroll
  for (uint32_t r = 0; r < 2; ++r)
#pragma unroll
    for (uint32_t h = 0; h < HV; ++h)
#pragma unroll
      for (uint32_t t = 0; t < 8; ++t) o[r][h][t][0] = o[r][h][t][1] = 0.0f;
  float m[2], l[2];   // rows q8 and q8 + 8
#pragma unroll
  for (uint32_t r = 0; r < 2; ++r) m[r] = -CUDART_INF_F, l[r] = 0.0f;

#pragma unroll 1
  for (uint32_t base = k_begin; base < k_end; base += kStep) {
    float s[NT][2][2][2];   // [tile][row half][n-tile]
#pragma unroll
    for (uint32_t u = 0; u < NT; ++u)
#pragma unroll
      for (uint32_t n = 0; n < 2; ++n) {
#pragma unroll
        for (uint32_t r = 0; r < 2; ++r) s[u][r][n][0] = s[u][r][n][1] = 0.0f;
#pragma unroll
        for (uint32_t j = 0; j < 2 * JK; ++j) {
          const uint4 &k = kf[u][n][j >> 1];
          const uint32_t b0 = (j & 1u) ? k.z : k.x, b1 = (j & 1u) ? k.w : k.y;
          mma16816<DT>(s[u][0][n], s[u][1][n], qf[j], b0, b1);
        }
      }
    load_k(base + kStep);   // (past the warp's keys: nothing is read)
    // columns of this thread: keys 2 q4 + {0, 1} of each tile and eight further
    float2 x[NT][2][2];
#pragma unroll
    for (uint32_t u = 0; u < NT; ++u)
#pragma unroll
      for (uint32_t n = 0; n < 2; ++n) {
        const uint32_t key = base + u * kTile + 8u * n + 2u * q4;
#pragma unroll
        for (uint32_t r = 0; r < 2; ++r) {
          x[u][r][n] = score2<DT, SCALE_FIRST>(s[u][r][n][0], s[u][r][n][1], scale, scale2);
          if (key >= k_end) x[u][r][n].x = -CUDART_INF_F;
          if (key + 1u >= k_end) x[u][r][n].y = -CUDART_INF_F;
        }
      }
    bool raise = false;
    float top[2];
#pragma unroll
    for (uint32_t r = 0; r < 2; ++r) {
      top[r] = fmaxf(fmaxf(x[0][r][0].x, x[0][r][0].y), fmaxf(x[0][r][1].x, x[0][r][1].y));
#pragma unroll
      for (uint32_t u = 1; u < NT; ++u)
        top[r] = fmaxf(top[r], fmaxf(fmaxf(x[u][r][0].x, x[u][r][0].y), fmaxf(x[u][r][1].x, x[u][r][1].y)));
      top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], 1));
      top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], 2));
      raise |= top[r] > m[r] + 8.0f * kLog2e || m[r] == -CUDART_INF_F;
    }
    // the maximum is only raised when a row exceeds it by more than 8 (a factor e^8 of head-room in P)
    if (__any_sync(0xffffffffu, raise)) {
#pragma unroll
      for (uint32_t r = 0; r < 2; ++r) {
        const float next = fmaxf(m[r], top[r]), f = m[r] == -CUDART_INF_F ? 0.0f : exp2_fast(m[r] - next);
        m[r] = next;
        l[r] *= f;
#pragma unroll
        for (uint32_t h = 0; h < HV; ++h)
#pragma unroll
          for (uint32_t t = 0; t < 8; ++t) {
            o[r][h][t][0] *= f;
            o[r][h][t][1] *= f;
          }
      }
    }
    // (while every score of a row has been -inf its maximum is -inf too, and -inf - -inf would be NaN: nothing is subtracted then)
    const float from[2] = {m[0] == -CUDART_INF_F ? 0.0f : m[0], m[1] == -CUDART_INF_F ? 0.0f : m[1]};
#pragma unroll
    for (uint32_t u = 0; u < NT; ++u) {
      uint32_t pf[4] = {0, 0, 0, 0};   // P as the A operand: rows q8 / q8 + 8, keys of n-tile 0 / 1
#pragma unroll
      for (uint32_t n = 0; n < 2; ++n)
#pragma unroll
        for (uint32_t r = 0; r < 2; ++r) {
          const float p0 = exp2_fast(x[u][r][n].x - from[r]), p1 = exp2_fast(x[u][r][n].y - from[r]);
          l[r] += p0 + p1;
          pf[2 * n + r] = pack2<DT>(p0, p1);
        }
#pragma unroll
      for (uint32_t h = 0; h < HV; ++h) {
        const uint32_t a[4] = {vf[u][0][h].x, vf[u][0][h].y, vf[u][0][h].z, vf[u][0][h].w}, b[4] = {vf[u][1][h].x, vf[u][1][h].y, vf[u][1][h].z, vf[u][1][h].w};
        const uint32_t c[4] = {vf[u][2][h].x, vf[u][2][h].y, vf[u][2][h].z, vf[u][2][h].w}, d[4] = {vf[u][3][h].x, vf[u][3][h].y, vf[u][3][h].z, vf[u][3][h].w};
#pragma unroll
        for (uint32_t t = 0; t < 8; ++t) {
          const uint32_t sel = (t & 1u) ? 0x7632u : 0x5410u;   // element t of the even and of the odd key
          const uint32_t b0 = __byte_perm(a[t >> 1], b[t >> 1], sel), b1 = __byte_perm(c[t >> 1], d[t >> 1], sel);
          mma16816<DT>(o[0][h][t], o[1][h][t], pf, b0, b1);
        }
      }
    }
    load_v(base + kStep);
  }

  // ---- combine: warps of the CTA, then CTAs of the cluster ----
#pragma unroll
  for (uint32_t r = 0; r < 2; ++r) {
    l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
    l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
    const uint32_t row = q8 + 8u * r;
    if (row < P.sq) {
      if (q4 == 0) {
        sm.m[warp][row] = m[r];
        sm.l[warp][row] = l[r];
      }
      // columns h * 64 + 16 q4 + t (first register of the pair) and 8 further (second)
#pragma unroll
      for (uint32_t h = 0; h < HV; ++h)
#pragma unroll
        for (uint32_t i = 0; i < 2; ++i)
#pragma unroll
          for (uint32_t t = 0; t < 8; t += 4)
            *reinterpret_cast<float4 *>(&sm.o[warp][row][h * 64u + 16u * q4 + 8u * i + t]) =
              make_float4(o[r][h][t][i], o[r][h][t + 1][i], o[r][h][t + 2][i], o[r][h][t + 3][i]);
    }
  }
  __syncthreads();
  // (warp 0's slots receive the CTA's own totals: each thread rewrites only elements that it alone reads)
  for (uint32_t i = tid; i < P.sq * D; i += kThreads) {
    const uint32_t row = i / D, col = i - row * D;
    float top = sm.m[0][row];
#pragma unroll
    for (uint32_t w = 1; w < kWarps; ++w) top = fmaxf(top, sm.m[w][row]);
    float sum = 0.0f;
#pragma unroll
    for (uint32_t w = 0; w < kWarps; ++w) sum += sm.o[w][row][col] * weight_of(sm.m[w][row], top);
    sm.o[0][row][col] = sum;
  }
  __syncthreads();
  if (tid < P.sq) {
    float top = sm.m[0][tid], sum = 0.0f;
#pragma unroll
    for (uint32_t w = 1; w < kWarps; ++w) top = fmaxf(top, sm.m[w][tid]);
#pragma unroll
    for (uint32_t w = 0; w < kWarps; ++w) sum += sm.l[w][tid] * weight_of(sm.m[w][tid], top);
    sm.m[0][tid] = top;
    sm.l[0][tid] = sum;
  }
  __syncthreads();
  if (CL > 1) cluster_sync();
  // this CTA's share of the head's result
  unsigned short *const O = reinterpret_cast<unsigned short *>(P.o_ptr) + (uint64_t)head * P.sq * D;
  const uint32_t pairs = P.sq * D / 2u, p_begin = pairs * rank / CL, p_end = pairs * (rank + 1u) / CL;
  for (uint32_t i = p_begin + tid; i < p_end; i += kThreads) {
    const uint32_t row = 2u * i / D, col = 2u * i - row * D;
    float a, b, sum;
    if (CL == 1) {
      a = sm.o[0][row][col];
      b = sm.o[0][row][col + 1];
      sum = sm.l[0][row];
    } else {
      float top = -CUDART_INF_F;
      for (uint32_t c = 0; c < CL; ++c) top = fmaxf(top, ld_peer(&sm.m[0][row], c));
      a = b = sum = 0.0f;
      for (uint32_t c = 0; c < CL; ++c) {
        const float f = weight_of(ld_peer(&sm.m[0][row], c), top);
        a += ld_peer(&sm.o[0][row][col], c) * f;
        b += ld_peer(&sm.o[0][row][col + 1], c) * f;
        sum += ld_peer(&sm.l[0][row], c) * f;
      }
    }
    const float inv = 1.0f / sum;
    *reinterpret_cast<uint32_t *>(O + 2u * i) = pack2<DT>(a * inv, b * inv);
  }
  __syncwarp();
  if (CL > 1) cluster_sync();   // no CTA leaves while a peer may still read its partial result
}

}  // namespace

#define DVMB_DECODE(NAME, DT, D, SF, NT)                                                                                              \
  __global__ void __launch_bounds__(kThreads, D == 128 ? 2 : 3) NAME(const __grid_constant__ AttnParam P, const __grid_constant__ DecodeArgs A) { \
    decode_body<DT, D, SF, NT>(P, A);                                                                                                 \
  }
#define DVMB_DECODE_TYPE(T, DT)                                           \
  DVMB_DECODE(dvm_b200_attention_decode_##T##_d64, DT, 64, false, 1)      \
  DVMB_DECODE(dvm_b200_attention_decode_##T##_d64_sf, DT, 64, true, 1)    \
  DVMB_DECODE(dvm_b200_attention_decode_##T##_d64x2, DT, 64, false, 2)    \
  DVMB_DECODE(dvm_b200_attention_decode_##T##_d64x2_sf, DT, 64, true, 2)  \
  DVMB_DECODE(dvm_b200_attention_decode_##T##_d128, DT, 128, false, 1)    \
  DVMB_DECODE(dvm_b200_attention_decode_##T##_d128_sf, DT, 128, true, 1)
DVMB_DECODE_TYPE(bf16, T_BF16)
DVMB_DECODE_TYPE(f16, T_F16)
#undef DVMB_DECODE_TYPE
#undef DVMB_DECODE

int LaunchAttentionDecode(const AttnParam &p, void *stream) {
  using Fn = void (*)(const AttnParam, const DecodeArgs);
#define DVMB_DECODE_FNS(T) {{dvm_b200_attention_decode_##T##_d64, dvm_b200_attention_decode_##T##_d64_sf}, \
                            {dvm_b200_attention_decode_##T##_d64x2, dvm_b200_attention_decode_##T##_d64x2_sf}, \
                            {dvm_b200_attention_decode_##T##_d128, dvm_b200_attention_decode_##T##_d128_sf}}
  static const Fn table[2][3][2] = {DVMB_DECODE_FNS(bf16), DVMB_DECODE_FNS(f16)};
#undef DVMB_DECODE_FNS
  int dev = 0;
  cudaGetDevice(&dev);
  static bool attr_set[64] = {false};
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    for (auto &t : table)
      for (int d = 0; d < 3; ++d)
        for (auto fn : t[d]) {
          cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, d == 2 ? sizeof(Combine<128>) : sizeof(Combine<64>));
          if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
          if (e != cudaSuccess) return static_cast<int>(e);
        }
    attr_set[dev] = true;
  }
  const uint32_t sms = static_cast<uint32_t>(Runtime::Get().sm_count_or_default()), tiles = (p.skv + kTile - 1) / kTile;
  const uint64_t slots = static_cast<uint64_t>(sms) * (p.d == 128 ? 2u : 3u);
  // CTAs per head: as many as run in one wave, while every warp has a step of keys (measured on 4 to 512 heads: a second,
  // partly filled wave costs more than the SMs a single one leaves idle); two where the heads alone fill more than a wave
  // and their caches are long, which shortens the last one.
  //   A first cut costs 1 us (one row of 64) to 4 (16 rows of 128, many heads: results read from one CTA by the other) and pays where
  // it saves more steps than that: a CTA alone | two, in us, 16 rows of 128: 1 head of 128 keys 5.4 | 6.4, of 256 6.6 | 5.7 (four);
  // 100 heads of 128 keys 5.5 | 8.5, of 512 9.1 | 11.0; one row: 100 heads of 192 keys 4.1 | 5.3.
  //   Clusters of sixteen find room for eight at a time: 16 heads of 2048 keys of 128 10.9 us in them, 7.1 in clusters of eight.
  const uint32_t first_cut = 16u + (4u * p.batch < sms ? 0u : p.sq > 8u ? 24u : p.sq > 4u ? 16u : 8u);   // in steps of 16 keys
  uint32_t cl = 1;
  while (cl < (p.batch <= 8u ? 16u : 8u) && p.batch * 2ull * cl <= slots && tiles >= (cl == 1u ? first_cut : 2u * cl * kWarps * (cl < 8u ? 1u : 2u))) cl *= 2;
  if (p.batch > slots && tiles >= 2u * kWarps * 8u) cl = 2;
  DecodeArgs a;
  a.cluster = cl;
  a.keys_per_warp = (tiles + cl * kWarps - 1) / (cl * kWarps) * kTile;
  // Keys of 64 elements in steps of 32: what a warp has in flight is one step's keys and values, 8 KB as with 128 elements
  // ([8, 32] heads of 4217 keys 64 -> 54.6 us).  Two steps of 16 answer sooner where that is all a warp has.
  const uint32_t form = p.d == 128 ? 2u : (a.keys_per_warp > 32u ? 1u : 0u);
  // Prefetched from 32 MB on: a smaller cache mostly is in L2 already, and the prefetches only delay its loads ([1, 8] heads of
  // 8192 keys of 64, 17 MB, 8.6 -> 9.05 us; [2, 32] of 3999 of 128, 131 MB, 25.4 -> 24.3, [4, 32] of 700 of 128, 46 MB, 11.5 -> 10.8).
  a.prefetch = static_cast<uint64_t>(p.batch) * p.skv * p.d * 4u >= (32ull << 20) ? 1u : 0u;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.batch * cl, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = p.d == 128 ? sizeof(Combine<128>) : sizeof(Combine<64>);
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cl > 1 ? 1 : 0;
  ChainAttribute(&cfg, attr);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, table[p.dtype == T_BF16 ? 0 : 1][form][p.scale_first ? 1 : 0], p, a);
  return e != cudaSuccess ? static_cast<int>(e) : static_cast<int>(cudaGetLastError());
}

}  // namespace dvmb
