// Row kernel: the RMS norm of a vector stage (row_match.cc), with its residual and a gated product beside it, as a straight-line
// kernel: dvm_b200_row_rms_gate.
//
// The vector interpreter spends its time on such a graph dispatching, and where rows do not start on 16 bytes it falls back to
// loads and stores of single elements.  Here a row belongs to 32 to 512 threads, every load of it in flight before the first use,
// and a thread works on 16-byte units at aligned addresses: a row is the units that hold at least one of its elements, lanes
// outside it are masked, and since every streamed tensor of a row lies alike relative to 16 bytes, an element is at the same
// place of its unit in all of them - no shifting, whatever the row length.
//
// The scale of a row is the usual one, computed in closed form; stages with other scalar sections run on the interpreter.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "chain.cuh"
#include "runtime.h"
#include "units.cuh"
#include "vm_row.h"

namespace dvmb {

namespace {

constexpr uint32_t kMaxRowThreads = 512;
constexpr uint32_t kMaxWarps = kMaxRowThreads / 32;
constexpr uint32_t kFewRegisters = 72;   // of a thread in the kernels named _few

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

// kStream: results that exceed L2 anyway leave it before anything else does.
template <bool kStream>
__device__ __forceinline__ void put_unit(uint8_t *p, const uint4 &q, uint32_t lo, uint32_t hi) {
  if (kStream && lo == 0 && hi == kE) {
    asm volatile("st.global.cs.v4.b32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(q.x), "r"(q.y), "r"(q.z), "r"(q.w) : "memory");
  } else {
    store_lanes(p, q, lo, hi);
  }
}

template <uint32_t DT, int K, bool kStream>
__device__ __forceinline__ void rms_gate_body(const RowParam &P) {
  __shared__ float part[kMaxWarps];   // sum of each warp
  chain_wait();
  chain_launch();
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
  const uint32_t tg = P.tg, rows = blockDim.x / tg, row_in_cta = tid / tg, t = tid - row_in_cta * tg;
  const uint32_t g = blockIdx.x * rows + row_in_cta;
  const bool live = g < P.groups;
  uint32_t k[kMaxKept];
  group_coords(P.kept_size, live ? g : 0u, k);
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
        put_unit<kStream>(base_of(6) + (16ull * c - mis), pack_pairs<DT>(y), lo, hi);
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
      put_unit<kStream>(base_of(3) + (16ull * c - mis), pack_pairs<DT>(y), lo, hi);
    }
  }
}

}  // namespace

// Two units per thread: at most 64 registers, so that an SM holds four CTAs of 256 threads and two of 512 (with 72 it was three and one).
// In us, with 72 | 64 registers: [16384, 4096] with residual and gate 129 | 122, [9000, 7000] 184 | 127, [5000, 6144] 98 | 67 (82 in the
// interpreter), [8192, 8192] 177 | 127 (161), a plain norm of [16384, 4096] 81 | 70.  _few has 72, for launches that are on the chip at
// once with those as well.
#define DVMB_ROW_RMS(NAME, DT, K, STREAM, REGISTERS)                                                 \
  __global__ void REGISTERS NAME(const __grid_constant__ RowParam P) { rms_gate_body<DT, K, STREAM>(P); }
DVMB_ROW_RMS(dvm_b200_row_rms_gate_f16_1, T_F16, 1, false, __launch_bounds__(kMaxRowThreads))
DVMB_ROW_RMS(dvm_b200_row_rms_gate_bf16_1, T_BF16, 1, false, __launch_bounds__(kMaxRowThreads))
DVMB_ROW_RMS(dvm_b200_row_rms_gate_f16_2, T_F16, 2, false, __launch_bounds__(kMaxRowThreads, 2))
DVMB_ROW_RMS(dvm_b200_row_rms_gate_bf16_2, T_BF16, 2, false, __launch_bounds__(kMaxRowThreads, 2))
DVMB_ROW_RMS(dvm_b200_row_rms_gate_f16_2_few, T_F16, 2, false, __maxnreg__(kFewRegisters))
DVMB_ROW_RMS(dvm_b200_row_rms_gate_bf16_2_few, T_BF16, 2, false, __maxnreg__(kFewRegisters))
DVMB_ROW_RMS(dvm_b200_row_rms_gate_f16_2_large, T_F16, 2, true, __launch_bounds__(kMaxRowThreads, 2))
DVMB_ROW_RMS(dvm_b200_row_rms_gate_bf16_2_large, T_BF16, 2, true, __launch_bounds__(kMaxRowThreads, 2))
#undef DVMB_ROW_RMS

namespace {

// Every row starts on 16 bytes.
bool RowsAligned(const RowParam &p) {
  uint64_t m = p.stream[0].ptr;
  for (int j = 0; j < kMaxKept; ++j)
    if (p.kept_size[j] != 1) m |= static_cast<uint64_t>(p.stream[0].kstride[j]) << 1;
  return (m & 15u) == 0;
}
// 16-byte units a row touches at most: one more where rows may start inside a unit
uint32_t UnitsPerRow(const RowParam &p) {
  const uint64_t bytes = static_cast<uint64_t>(p.run_len) << 1;
  return static_cast<uint32_t>(RowsAligned(p) ? (bytes + 15) / 16 : (bytes + 15 + 14) / 16);
}

constexpr uint32_t kRmsMaxUnits = 2 * kMaxRowThreads;
static_assert(kRowRmsMaxElems == kRmsMaxUnits * 8, "two units of eight elements per thread");

}  // namespace

bool RowAddressesOk(const RowParam &p) {
  if (p.form == ROW_OFF || p.stream[0].ptr == 0) return false;
  for (int i = 0; i < kRowMaxStreams; ++i) {
    if (i == 2) {   // (the row vector is read at any element address)
      if (p.have_w && (p.stream[2].ptr & 1u)) return false;
      continue;
    }
    if (p.stream[i].ptr == 0) continue;   // an absent stream
    if (((p.stream[i].ptr ^ p.stream[0].ptr) & 15u) != 0 || (p.stream[i].ptr & 1u) != 0) return false;
  }
  return UnitsPerRow(p) <= kRmsMaxUnits;   // (a longer row does not fit a CTA's registers)
}

// Estimates of both kernels in microseconds, a fit to launches of 16 to 400 000 rows timed back to back in either, aligned and not.
// What decides:
//  - A row of up to 32 units takes a warp about 0.35 ns in all; the interpreter gives short rows a slice of a warp: [400000, 16]
//    bf16 138 us here and 37 there, [400000, 64] 148 and 144.
//  - Longer rows are faster here in any number: plain norms of [16384, 4096] 70 and 135, [5000, 6144] 44 and 62, [8192, 8192] 79 and 119,
//    [600, 6144] 7.1 and 13.0.
bool RowKernelPays(const RowParam &p) {
  if (UnitsPerRow(p) > 32u) return true;
  const double groups = p.groups;
  // rows in whole granules of four elements (what the interpreter loads at a time)
  uint64_t m = p.stream[0].ptr | (static_cast<uint64_t>(p.run_len) << 1);
  for (int j = 0; j < kMaxKept; ++j)
    if (p.kept_size[j] != 1) m |= static_cast<uint64_t>(p.stream[0].kstride[j]) << 1;
  double padded = 16.0;   // a short row's slice: a power of two of elements
  while (padded < p.run_len) padded *= 2.0;
  const double w = p.have_w != 0, b = p.have_b != 0, g = p.have_gate != 0;
  const double row = 1.5 + groups * 1e-3 * (0.345 + 0.035 * w + 0.015 * b + 0.095 * g);
  const double per_elem = 1e-6 * (5.0 + 1.5 * w + 3.3 * b + 6.2 * g) * ((m & 7u) == 0 ? 1.0 : 2.2);
  return row <= std::max(7.0 + 5.0 * b + 5.0 * g, 5.0 + groups * padded * per_elem);
}

int LaunchRow(const RowParam &p_in, void *stream) {
  RowParam p = p_in;
  const uint32_t units = UnitsPerRow(p), sms = static_cast<uint32_t>(Runtime::Get().sm_count_or_default());
  // two units per thread keep more loads in flight; one unit and more threads answer sooner while there are few rows
  const bool few = static_cast<uint64_t>(p.groups) < 4ull * sms;
  const uint32_t per_thread = units > kMaxRowThreads || (!few && units > 64u) ? 2u : 1u;
  uint32_t tg = 32;
  while (tg * per_thread < units) tg *= 2;
  p.tg = tg;
  // (L2 holds 126 MB; [16384, 4096] with residual and gate, 268 MB of results: 122 us by ordinary stores, 116 by those of _large)
  const bool large = (2ull * p.groups * p.run_len << (p.have_gate ? 1 : 0)) > (128ull << 20);
  const uint32_t block = tg < 128u ? 128u : tg, rows = block / tg;
  using Fn = void (*)(const RowParam);
  const uint32_t ctas = (p.groups + rows - 1) / rows;
  // 72 registers where all CTAs are on the chip at once with those too: in us, with 64 | 72, [148, 5000] 3.40 | 3.28, [148, 8192] 3.95 | 3.87,
  // [1000, 1024] 3.86 | 3.63, [2000, 1024] 5.00 | 4.53; beyond that 64 ([149, 8192] 4.92 | 6.10, [4000, 1024] 7.48 | 7.80).  Except where only
  // with 64 the CTAs of the next launch find room beside these of 128 threads: [1060 to 1184, 768] 3.4 to 3.6 | 4.0 to 4.1, [1036, 768] 3.30 |
  // 3.26, [1200, 768] 4.31 | 4.11 (CTAs of 512 threads show no such step).
  const uint32_t slots = sms * (65536u / (kFewRegisters * block)), slots64 = sms * (65536u / (64u * block));
  const bool at_once = ctas <= slots && (block == kMaxRowThreads || 2 * ctas <= slots || 2 * ctas > slots64);
  static const Fn fns[2][4] = {
    {dvm_b200_row_rms_gate_f16_1, dvm_b200_row_rms_gate_f16_2, dvm_b200_row_rms_gate_f16_2_few, dvm_b200_row_rms_gate_f16_2_large},
    {dvm_b200_row_rms_gate_bf16_1, dvm_b200_row_rms_gate_bf16_2, dvm_b200_row_rms_gate_bf16_2_few, dvm_b200_row_rms_gate_bf16_2_large}};
  const Fn fn = fns[p.dtype == T_F16 ? 0 : 1][per_thread == 1 ? 0 : (large ? 3 : (at_once ? 2 : 1))];
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3(ctas, 1, 1);
  cfg.blockDim = dim3(block, 1, 1);
  cfg.stream = static_cast<cudaStream_t>(stream);
  ChainAttribute(&cfg, attr);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, fn, p);
  return e != cudaSuccess ? static_cast<int>(e) : static_cast<int>(cudaGetLastError());
}

}  // namespace dvmb
