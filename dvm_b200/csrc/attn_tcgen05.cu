// Fused attention  O = softmax(scale * Q K^T) V  on the sm_100a tensor cores.
//
// The reference has no attention operator: its example (examples/03_attention.py:31-52) builds
// MatMul -> scale -> softmax -> MatMul from API ops, which its splitter turns into several kernels with the full
// score matrix in global memory (src/xkernel.cc:1980-2119).  Here the stage planner recognises that pattern and
// runs it as one launch with the scores kept on chip (online softmax over key/value tiles).
//
// One CTA owns 256 query rows of one (batch, head) at a time - two tiles of 128 rows that take turns on the tensor core, or one where
// there are few - and is persistent over such units.
//   warp 0      TMA producer: K and V tiles of 128 keys through a 4-slot ring
//   warp 1      MMA issuer: S_g = Q_g K^T into TMEM, O_g += P_g V with P_g read from TMEM; the two row tiles g = 0, 1 alternate, so that
//               one tile's softmax overlaps the other tile's MMAs
//   warp 2      TMA producer of Q: a tile's next rows as soon as its last scores of the unit before have been computed
//   warps 4-11  softmax of tile 0, 16 rows each (two rows to four lanes), warps 12-19 of tile 1: scores TMEM -> registers, running
//               maximum, exp2, row sum, P as bf16/fp16 back to TMEM in two halves, P V starting on the first; at the end of a unit
//               O / l through shared memory and a TMA store
// What bounds it: the chain of a row tile, about 3450 cycles per 128 keys where both tiles' MMAs take 2064 and their exponentials 2048:
// wait 100, scores out of TMEM and rounded 340, maximum 260, exponentials 560 and 900 (the other tile's run meanwhile), the slowest
// warp and the issuer 400, the rest of P V and the next scores 900.  On [8, 32, 2048, 128] the power cap comes first: 482 us in short
// runs (490 with P in shared memory and eight softmax warps of 32 rows, on the same GPU), 557 to 570 among other work (563); with little
// else on the chip [1, 4, 4096, 128] 41 us (54), [1, 8, 1024, 128] 13.5 (16.8), with d = 64 [8, 32, 2048, 64] 394 (490).
// 640 threads leave 96 registers each; 12 bytes a thread are spilled, read twice per unit and not per key tile.
//  - P stays in TMEM: as a tile in shared memory it cost a write and a read of 32 KB per MMA of 512 cycles, which alone fill the 128
//    bytes a cycle.  With d = 128 it lies over the scores it came from, so the next scores follow P V; a place of its own and one
//    score buffer for both tiles had every tile wait for the other's scores (547 us with an issuer warp for each, 470-480 with one).
//  - Rows by 16 and not 32 by half the keys: warps need nothing of one another, where they met at a barrier for every maximum.
//  - A part of the exponentials as polynomials on the FMA pipe (3 to 12 of 32 pairs) was slower every time: issue slots are short
//    as well (62 % in use).  Taking turns at the exponentials, which paid with 8 warps, did not with 16.
//  - (Pairs of CTAs sharing every MMA: 746 us against 555, their barrier arrivals cross the cluster twice per 128 keys.)
// The running maximum is only raised when a row's new maximum exceeds it by more than 8 (a factor e^8 of
// head-room in P); only then is the accumulator in TMEM rescaled, which for typical inputs happens once.
// Rounding follows the graph: the score is rounded to the operand type (the MatMul result), scaled (rounded
// again when the scale was applied in the operand type), softmax in fp32, P rounded to the operand type.
// Every mbarrier wait is bounded; on expiry a status word is set and the kernel runs to its end.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>

#include "chain.cuh"
#include "mm_launch.h"
#include "runtime.h"
#include "sm100_sync.cuh"
#include "vm_ops.cuh"

namespace dvmb {

__device__ WaitStatus g_attn_status = {0u, 0u};

namespace {

constexpr uint32_t kTileQ = 128, kTileKV = 128;
constexpr uint32_t kRingSlots = 4;
constexpr uint32_t kTileBytes = 128 * 128 * 2;      // one [128 x 128] 16-bit tile (two 64-column halves)
constexpr uint32_t kHalfBytes = 128 * 64 * 2;       // [128 rows x 64 elements], 128-byte swizzled rows
constexpr uint32_t kTileWarps = 8;                  // softmax warps of a row tile, 16 rows each
constexpr uint32_t kFirstSoftmaxWarp = 4;
constexpr uint32_t kThreads = 32 * (kFirstSoftmaxWarp + 2 * kTileWarps);
constexpr uint32_t kHeader = 1024;
constexpr uint32_t kStoreBytes = 16 * 64 * 2;       // [16 rows x 64 elements] of the result, 128-byte swizzled rows: a warp's
// shared memory: header | Q0 Q1 | result staging | ring[4]
constexpr uint32_t kOffQ = kHeader, kOffO = kOffQ + 2 * kTileBytes, kOffRing = kOffO + 2 * kTileWarps * kStoreBytes;
constexpr uint32_t kSmemBytes = kOffRing + kRingSlots * kTileBytes + 1024;
static_assert(kSmemBytes <= 227 * 1024, "shared memory of a CTA");
// Tensor memory columns, 512 in all: S0 S1, O0 O1, with d = 64 P0 P1 behind the narrower O; with d = 128 P lies in the columns of S.
constexpr uint32_t kTmemO = 256, kTmemP64 = 384, kTmemCols = 512;
constexpr float kRescaleThreshold = 8.0f;

struct AttnMaps {
  CUtensorMap q, k, v, o;
};

// barrier offsets inside the header
constexpr uint32_t kBarQ = 0, kBarQFree = 16, kBarKvFull = 32, kBarKvEmpty = 64, kBarSFull = 96, kBarPReady = 112,   // (P: [tile][half])
                   kBarPvDone = 144, kTmemSlot = 160;

// D[tmem] (+)= A[tmem] * B[smem]: a row of A is a lane, two neighbouring elements a column.
__device__ __forceinline__ void umma_f16_cta1_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
    "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
    "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
    : "memory");
}
// 16 rows (TMEM lanes) by 8 N columns of fp32.  Lane t of the warp holds, of every 8 columns, 2 (t % 4) and the next of row t / 4 in two
// registers and of row t / 4 + 8 in two more.  Waited for inside the statement: no copy of a register, nothing between.
__device__ __forceinline__ void tmem_ld_rows(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
    "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
    "tcgen05.wait::ld.sync.aligned;"
    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
    : "r"(taddr)
    : "memory");
}
__device__ __forceinline__ void tmem_ld_rows(uint32_t taddr, uint32_t (&r)[64]) {
  asm volatile(
    "tcgen05.ld.sync.aligned.16x256b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
    "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,"
    "%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47,"
    "%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%64];\n\t"
    "tcgen05.wait::ld.sync.aligned;"
    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
      "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
      "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
      "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
      "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]),
      "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]),
      "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
    : "r"(taddr)
    : "memory");
}
// The other way, fp32 again, and 16 rows by 4 N columns of packed pairs: column t % 4 of every 4, rows t / 4 and t / 4 + 8.
__device__ __forceinline__ void tmem_st_rows(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
               "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
               : "memory");
}
__device__ __forceinline__ void tmem_st_pairs(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
               "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
               "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Packed 2 x 16-bit arithmetic in the operand type: the product of two bf16 / fp16 values rounded once to that type
// is exactly "multiply in fp32, round to the type", the graph's scaled score.
template <uint32_t DT>
__device__ __forceinline__ uint32_t mul2(uint32_t a, uint32_t b) {
  uint32_t r;
  if (DT == T_BF16) {
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  } else {
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  }
  return r;
}
template <uint32_t DT>
__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) {
  uint32_t r;
  if (DT == T_BF16) {
    asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  } else {
    asm("max.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  }
  return r;
}
template <uint32_t DT>
__device__ __forceinline__ float2 unpack2(uint32_t p) {
  if (DT == T_BF16) return make_float2(__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u));
  return __half22float2(*reinterpret_cast<const __half2 *>(&p));
}

// Two neighbouring scores as one 64-bit register pair: one issue slot per packed operation, each half rounded on its own.
__device__ __forceinline__ uint64_t f2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 halves(uint64_t a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint32_t pack_pair(uint32_t dtype, float lo, float hi) {
  if (dtype == T_BF16) return pack_bf16x2(lo, hi);
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&h);
}

}  // namespace

namespace {
template <uint32_t DT>
__device__ __forceinline__ void attention_body(const AttnParam &P, const AttnMaps &maps, const LaunchTag epoch) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t *smem = smem_raw + (base - raw_addr);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t dhalves = P.d / 64;                  // 64-element halves of the head dimension (1 or 2)
  const uint32_t tiles = P.q_tiles;                   // row tiles per unit: 1 or 2
  const uint32_t unit_rows = kTileQ * tiles, qblocks = (P.sq + unit_rows - 1) / unit_rows;
  const uint32_t my_units = (P.units - blockIdx.x + gridDim.x - 1) / gridDim.x;   // units blockIdx.x, + gridDim.x, ...
  const uint32_t nkv = (P.skv + kTileKV - 1) / kTileKV;
  const uint32_t tile_bytes = dhalves * kHalfBytes;   // bytes of one staged Q / K / V tile
  constexpr uint64_t kTileStep = kTileBytes >> 4, kHalfStep = kHalfBytes >> 4;   // in address fields of descriptors
  constexpr uint32_t kFmt = DT == T_BF16 ? 1u : 0u;

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < kRingSlots; ++s) {
      mbar_init(base + kBarKvFull + 8 * s, 1);
      mbar_init(base + kBarKvEmpty + 8 * s, 1);
    }
    for (uint32_t g = 0; g < 2; ++g) {
      mbar_init(base + kBarQ + 8 * g, 1);
      mbar_init(base + kBarQFree + 8 * g, 1);
      mbar_init(base + kBarSFull + 8 * g, 1);
      for (uint32_t h = 0; h < 2; ++h) mbar_init(base + kBarPReady + 16 * g + 8 * h, kTileWarps);
      mbar_init(base + kBarPvDone + 8 * g, 1);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(base + kTmemSlot, kTmemCols);
    tmem_relinquish();
  }
  tcgen05_before_sync();
  __syncthreads();
  tcgen05_after_sync();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t *>(smem + kTmemSlot);
  chain_wait();
  chain_launch();

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    // (elect.sync, not `lane == 0`, here and in the MMA warp: see mm_tcgen05.cu)
    if (elect_one()) {
      uint32_t slot = 0, parity = 1;
      const uint32_t ntiles = 2 * nkv;
      for (uint32_t it = 0; it < my_units; ++it) {
        const uint32_t unit = blockIdx.x + it * gridDim.x, bz = unit / qblocks;
        // ring order = order of need: K0, then per key tile j: K(j+1) (its scores are issued early), V(j)
        for (uint32_t p = 0; p < ntiles; ++p) {
          // position p holds: K0 at 0; K(j) at 2j - 1; V(j) at 2j + 2, except the last V at 2 nkv - 1
          const bool is_v = p != 0 && ((p & 1u) == 0 || p == ntiles - 1);
          const uint32_t j = p == 0 ? 0u : (is_v ? (p == ntiles - 1 ? nkv - 1 : (p - 2) / 2) : (p + 1) / 2);
          const CUtensorMap *map = is_v ? &maps.v : &maps.k;
          mbar_wait(base + kBarKvEmpty + 8 * slot, parity, 1, &g_attn_status, epoch);
          mbar_expect_tx(base + kBarKvFull + 8 * slot, tile_bytes);
          for (uint32_t h = 0; h < dhalves; ++h)
            tma_load_3d(base + kOffRing + slot * kTileBytes + h * kHalfBytes, map, base + kBarKvFull + 8 * slot, (int)(h * 64),
                        (int)(j * kTileKV), (int)bz);
          if (++slot == kRingSlots) {
            slot = 0;
            parity ^= 1u;
          }
        }
      }
    }
  } else if (warp == 2) {
    // ------------------------------ Q producer ------------------------------
    if (elect_one()) {
      for (uint32_t it = 0; it < my_units; ++it) {
        const uint32_t unit = blockIdx.x + it * gridDim.x, bz = unit / qblocks, q_row0 = (unit - bz * qblocks) * unit_rows;
        for (uint32_t g = 0; g < tiles; ++g) {   // a tile's buffer is free once the unit before has all its scores
          if (it != 0) mbar_wait(base + kBarQFree + 8 * g, (it - 1) & 1u, 5, &g_attn_status, epoch);
          mbar_expect_tx(base + kBarQ + 8 * g, tile_bytes);
          for (uint32_t h = 0; h < dhalves; ++h)
            tma_load_3d(base + kOffQ + g * kTileBytes + h * kHalfBytes, &maps.q, base + kBarQ + 8 * g, (int)(h * 64), (int)(q_row0 + g * kTileQ), (int)bz);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    if (elect_one()) {
      // S = Q K^T: both operands have the head dimension innermost; M = 128, N = 128 keys
      const uint32_t idesc_s = (1u << 4) | (kFmt << 7) | (kFmt << 10) | ((kTileKV >> 3) << 17) | ((kTileQ >> 4) << 24);
      // O += P V: V is stored [key][d] (the contraction axis outermost); N = d
      const uint32_t idesc_o = (1u << 4) | (kFmt << 7) | (kFmt << 10) | (1u << 16) | ((P.d >> 3) << 17) | ((kTileQ >> 4) << 24);
      // descriptors of row tile 0 / ring slot 0; everything further is an addition to their address fields
      const uint64_t dq = make_smem_desc(base + kOffQ, 0, 1024);
      const uint64_t dk = make_smem_desc(base + kOffRing, 0, 1024), dv = make_smem_desc(base + kOffRing, kHalfBytes, 1024);
      const bool two_halves = P.d > 64;
      // ring position of K(j) / V(j) of a unit (see the producer), units one after the other -> slot and phase parity
      const uint32_t ntiles = 2 * nkv, total = my_units * nkv;
      auto k_pos = [&](uint32_t u, uint32_t j) { return u * ntiles + (j == 0 ? 0u : 2 * j - 1); };
      auto v_pos = [&](uint32_t u, uint32_t j) { return u * ntiles + (j + 1 < nkv ? 2 * j + 2 : ntiles - 1); };
      auto wait_kv = [&](uint32_t pos) { mbar_wait(base + kBarKvFull + 8 * (pos % kRingSlots), (pos / kRingSlots) & 1u, 6, &g_attn_status, epoch); };
      auto release = [&](uint32_t pos) { umma_commit_cta1(base + kBarKvEmpty + 8 * (pos % kRingSlots)); };
      // scores of row tile g and key tile j of unit u, into the columns sb
      auto issue_s = [&](uint32_t g, uint32_t sb, uint32_t u, uint32_t j) {
        const uint32_t pos = k_pos(u, j);
        if (j == 0) mbar_wait(base + kBarQ + 8 * g, u & 1u, 7, &g_attn_status, epoch);
        tcgen05_after_sync();
        const uint64_t a = dq + g * kTileStep, b = dk + (pos % kRingSlots) * kTileStep;
        const uint32_t d = tmem_base + sb * 128;
#pragma unroll
        for (uint32_t kk = 0; kk < 4; ++kk) umma_f16_cta1(d, a + kk * 2, b + kk * 2, idesc_s, kk != 0 ? 1u : 0u);
        if (two_halves) {
#pragma unroll
          for (uint32_t kk = 0; kk < 4; ++kk) umma_f16_cta1(d, a + kHalfStep + kk * 2, b + kHalfStep + kk * 2, idesc_s, 1u);
        }
        umma_commit_cta1(base + kBarSFull + 8 * sb);
        if (g + 1 == tiles) release(pos);
        if (j + 1 == nkv) umma_commit_cta1(base + kBarQFree + 8 * g);
      };
      // P V of row tile g, whose P belongs to the score columns sb: the first 64 keys while the exponentials of the others still run
      auto issue_pv = [&](uint32_t g, uint32_t sb, uint32_t phase, uint32_t pos, bool accumulate) {
        const uint64_t b = dv + (pos % kRingSlots) * kTileStep;
        const uint32_t d = tmem_base + kTmemO + g * P.d, a = tmem_base + (two_halves ? sb * 128 : kTmemP64 + sb * 64);
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
          mbar_wait(base + kBarPReady + 16 * sb + 8 * h, phase, 11, &g_attn_status, epoch);
          tcgen05_after_sync();
#pragma unroll
          for (uint32_t kk = 4 * h; kk < 4 * h + 4; ++kk)
            umma_f16_cta1_ts(d, a + kk * 8, b + kk * (2048 >> 4), idesc_o, (accumulate || kk != 0) ? 1u : 0u);
        }
        umma_commit_cta1(base + kBarPvDone + 8 * g);
        if (g + 1 == tiles) release(pos);
      };
      wait_kv(k_pos(0, 0));
      for (uint32_t g = 0; g < tiles; ++g) issue_s(g, g, 0, 0);
      uint32_t u = 0, j = 0;
      for (uint32_t n = 0; n < total; ++n) {   // key tile j of unit u, and the one behind it
        const bool more = n + 1 < total;
        const uint32_t u1 = j + 1 == nkv ? u + 1 : u, j1 = j + 1 == nkv ? 0u : j + 1;
        if (more) wait_kv(k_pos(u1, j1));
        wait_kv(v_pos(u, j));
        if (tiles == 2) {
          // The row tiles take turns: while the softmax of one runs, the tensor core has P V and the next scores of the other.
          // With d = 128 the scores overwrite P, which P V reads: the two MMAs run one after the other because one thread issues them
          // and they have the same shape and kind.  PTX promises that order for MMAs on one accumulator; that it holds for the tensor
          // core's queue as a whole is an assumption, one that published attention kernels with P over S make as well.
          for (uint32_t g = 0; g < 2; ++g) {
            issue_pv(g, g, n & 1u, v_pos(u, j), j != 0);
            if (more) issue_s(g, g, u1, j1);
          }
        } else {
          // One row tile has both score buffers: the next scores are there when its softmax comes to them.
          if (more) issue_s(0, (n + 1) & 1u, u1, j1);
          issue_pv(0, n & 1u, (n >> 1) & 1u, v_pos(u, j), j != 0);
        }
        u = u1;
        j = j1;
      }
    }
  } else if (warp >= kFirstSoftmaxWarp) {
    // ------------------------------ softmax warps ------------------------------
    const uint32_t g = (warp - kFirstSoftmaxWarp) / kTileWarps;     // row tile of this warp
    const uint32_t quarter = warp & 3u;                  // TMEM lane quarter this warp may access, and which 16 lanes of it it works on
    const uint32_t tile_row = quarter * 32 + ((warp >> 2) & 1u) * 16;
    const uint32_t lanes = tmem_base + (tile_row << 16), col = 2 * (lane & 3u);   // this lane's columns of every eight: col, col + 1
    const uint32_t t_o = lanes + kTmemO + g * P.d;
    const uint32_t staging = base + kOffO + (warp - kFirstSoftmaxWarp) * kStoreBytes;
    // A score is rounded to the operand type, multiplied by `factor` in that type, and taken to the log2 domain in fp32: a scale
    // applied in the operand type is the factor; one applied behind the cast to fp32 leaves its sign there (0 and NaN whole).
    constexpr float kLog2e = 1.4426950408889634f;
    const float scale = __uint_as_float(P.scale_bits);
    const float factor = P.scale_first ? scale : (scale > 0.0f ? 1.0f : (scale < 0.0f ? -1.0f : scale));
    const float to_log2 = (P.scale_first || scale == 0.0f ? 1.0f : fabsf(scale)) * kLog2e;
    const uint32_t factor2 = pack_pair(DT, factor, factor);
    uint32_t n = 0;                              // key tiles done, over all units
    for (uint32_t it = 0; it < my_units; ++it) {
      const uint32_t unit = blockIdx.x + it * gridDim.x, bz = unit / qblocks;
      const uint32_t warp_row0 = (unit - bz * qblocks) * unit_rows + g * kTileQ + tile_row;
      float m_used[2] = {-CUDART_INF_F, -CUDART_INF_F};   // of the lane's two rows, in the log2 domain
      float sum[2] = {0.0f, 0.0f};                        // ... their sums over the lane's columns
      // A key tile's exponentials are summed by themselves, even and odd columns: a running sum of all keys takes 16 times as many additions,
      // and like terms round in the same direction.  Added while the warp would wait for the next scores: behind the second half of P the
      // same additions cost [8, 32, 2048, 64] 425 us instead of 395.
      uint64_t part[2] = {0, 0};
      auto fold = [&]() {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float2 h = halves(part[i]);
          sum[i] += h.x + h.y;
          part[i] = 0;
        }
      };
      for (uint32_t j = 0; j < nkv; ++j, ++n) {
        const uint32_t sb = tiles == 2 ? g : n & 1u;
        const uint32_t t_s = lanes + sb * 128, t_p = P.d > 64 ? t_s : lanes + kTmemP64 + sb * 64;
        fold();
        mbar_wait(base + kBarSFull + 8 * sb, (tiles == 2 ? n : n >> 1) & 1u, 8, &g_attn_status, epoch);
        tcgen05_after_sync();
        // The scores, rounded to the operand type and (the graph's order) scaled in that type, two at a time: one conversion packs and
        // rounds, one packed multiply scales and rounds again.  Even registers are of the first row, odd ones of the second.
        uint32_t pk[32];
        {
          uint32_t raw[64];
          tmem_ld_rows(t_s, raw);
#pragma unroll
          for (int i = 0; i < 32; ++i) pk[i] = mul2<DT>(pack_pair(DT, u2f(raw[2 * i]), u2f(raw[2 * i + 1])), factor2);
        }
        const uint32_t kv_valid = P.skv - j * kTileKV;
        if (kv_valid < kTileKV) {   // the last key tile: mask what lies past the sequence
          constexpr uint32_t kNegInf2 = DT == T_BF16 ? 0xff80ff80u : 0xfc00fc00u;
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const uint32_t at = 8 * (i >> 1) + col;
            if (at + 1 >= kv_valid) pk[i] = (pk[i] & 0x0000ffffu) | (kNegInf2 & 0xffff0000u);
            if (at >= kv_valid) pk[i] = kNegInf2;
          }
        }
        // The rows' maxima: of the lane's columns two at a time, then both rows in one register over the four lanes that share them.
        uint32_t ma[2] = {pk[0], pk[2]}, mb[2] = {pk[1], pk[3]};
#pragma unroll
        for (int i = 4; i < 32; i += 4) {
          ma[0] = max2<DT>(ma[0], pk[i]);
          mb[0] = max2<DT>(mb[0], pk[i + 1]);
          ma[1] = max2<DT>(ma[1], pk[i + 2]);
          mb[1] = max2<DT>(mb[1], pk[i + 3]);
        }
        ma[0] = max2<DT>(ma[0], ma[1]);
        mb[0] = max2<DT>(mb[0], mb[1]);
        uint32_t both = max2<DT>(__byte_perm(ma[0], mb[0], 0x5410), __byte_perm(ma[0], mb[0], 0x7632));
        both = max2<DT>(both, __shfl_xor_sync(0xffffffffu, both, 1));
        both = max2<DT>(both, __shfl_xor_sync(0xffffffffu, both, 2));
        const float2 mm = unpack2<DT>(both);
        const float mx[2] = {mm.x * to_log2, mm.y * to_log2};
        bool raise[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) raise[i] = mx[i] > m_used[i] + kRescaleThreshold * kLog2e || m_used[i] == -CUDART_INF_F;
        if (__any_sync(0xffffffffu, raise[0] || raise[1])) {
          float alpha[2] = {1.0f, 1.0f};
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (raise[i]) {
              alpha[i] = m_used[i] == -CUDART_INF_F ? 0.0f : fast_exp2(m_used[i] - mx[i]);
              m_used[i] = mx[i];
              sum[i] *= alpha[i];
            }
          if (j != 0) {   // O, behind the P V before and in front of the next one
            mbar_wait(base + kBarPvDone + 8 * g, (n - 1) & 1u, 9, &g_attn_status, epoch);
            tcgen05_after_sync();
            for (uint32_t c = 0; c < P.d; c += 32) {
              uint32_t t[16];
              tmem_ld_rows(t_o + c, t);
#pragma unroll
              for (int i = 0; i < 16; ++i) t[i] = f2u(u2f(t[i]) * alpha[(i >> 1) & 1]);
              tmem_st_rows(t_o + c, t);
            }
          }
        }
        // (a maximum of -inf - every score so far - is not subtracted: -inf - -inf would be NaN, which the sums and O keep)
        const uint64_t c2 = f2(to_log2, to_log2);
        uint64_t mneg[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float from = m_used[i] == -CUDART_INF_F ? 0.0f : m_used[i];
          mneg[i] = f2(-from, -from);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {   // 64 keys each, so that P V begins while the second half is computed
          uint32_t p[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float2 v = unpack2<DT>(pk[16 * h + i]), t = halves(fma2(f2(v.x, v.y), c2, mneg[i & 1]));
            const float p0 = fast_exp2(t.x), p1 = fast_exp2(t.y);
            part[i & 1] = add2(part[i & 1], f2(p0, p1));
            p[i] = pack_pair(DT, p0, p1);
          }
          tmem_st_pairs(t_p + 32 * h, p);
          tmem_st_wait();
          tcgen05_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(base + kBarPReady + 16 * sb + 8 * h);
        }
      }
      fold();
      // ---- result: O / l, rounded to the operand type, 64 columns at a time through shared memory to a TMA store
      // (the next unit's first P V overwrites O; it waits for this warp's next P)
      mbar_wait(base + kBarPvDone + 8 * g, (n - 1) & 1u, 10, &g_attn_status, epoch);
      tcgen05_after_sync();
      float inv[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float l = sum[i];
        l += __shfl_xor_sync(0xffffffffu, l, 1);
        l += __shfl_xor_sync(0xffffffffu, l, 2);
        inv[i] = 1.0f / l;
      }
      for (uint32_t c = 0; c < P.d; c += 64) {
        if (lane == 0) tma_store_wait_read<0>();   // the store before has read the staging
        __syncwarp();
#pragma unroll
        for (uint32_t part = 0; part < 2; ++part) {
          uint32_t t[16];
          tmem_ld_rows(t_o + c + 32 * part, t);
#pragma unroll
          for (int i = 0; i < 8; ++i) {   // piece i / 2 of 16 bytes; first or second row
            const uint32_t o = pack_pair(DT, u2f(t[2 * i]) * inv[i & 1], u2f(t[2 * i + 1]) * inv[i & 1]);
            const uint32_t row = (lane >> 2) + 8 * (i & 1), addr = staging + row * 128 + (((4 * part + (i >> 1)) ^ (row & 7u)) << 4) + 2 * col;
            asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(o) : "memory");
          }
        }
        fence_async_shared();
        __syncwarp();
        if (lane == 0) {
          if (warp_row0 < P.sq)   // (rows past the last one are cut off by the tensor map)
            tma_store_3d(&maps.o, staging, (int)c, (int)warp_row0, (int)bz);
          tma_store_commit();
        }
      }
    }
    if (lane == 0) tma_store_wait_read<0>();   // shared memory stays until the last store has read it
  }
  __syncwarp();
  tcgen05_before_sync();
  __syncthreads();
  if (warp == 1) {
    tcgen05_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}
}  // namespace

#define DVMB_ATTN_KERNEL(NAME, DT)                                                                                  \
  __global__ void __launch_bounds__(kThreads, 1) NAME(const __grid_constant__ AttnParam P,                          \
                                                      const __grid_constant__ AttnMaps maps, const LaunchTag epoch) { \
    attention_body<DT>(P, maps, epoch);                                                                         \
  }
DVMB_ATTN_KERNEL(dvm_b200_attention_bf16, T_BF16)
DVMB_ATTN_KERNEL(dvm_b200_attention_f16, T_F16)
#undef DVMB_ATTN_KERNEL

namespace {

PFN_cuTensorMapEncodeTiled GetEncodeFn() {
  static PFN_cuTensorMapEncodeTiled fn = nullptr;
  if (fn == nullptr) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled>(p);
  }
  return fn;
}

// [batch, rows, d] row-major, box = [1, box_rows, 64 elements], 128-byte swizzle
int EncodeRows(CUtensorMap *map, uint64_t ptr, uint64_t d, uint64_t rows, uint64_t batch, uint32_t box_rows) {
  auto encode = GetEncodeFn();
  if (encode == nullptr) return -10;
  cuuint64_t dims[3] = {d, rows, batch};
  cuuint64_t strides[2] = {d * 2, d * rows * 2};
  cuuint32_t box[3] = {64, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, reinterpret_cast<void *>(ptr), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -100 - static_cast<int>(r);
}

}  // namespace

bool AttentionSupported(const AttnParam &p) {
  if (p.d != 64 && p.d != 128) return false;
  if (p.dtype != T_BF16 && p.dtype != T_F16) return false;
  if (p.sq == 0 || p.skv == 0 || p.batch == 0) return false;
  return true;
}

int LaunchAttention(const AttnParam &p_in, void *stream) {
  AttnParam p = p_in;
  if (!AttentionSupported(p)) return -1;
  if ((p.q_ptr | p.k_ptr | p.v_ptr | p.o_ptr) & 15u) return -2;
  if (p.sq <= kDecodeMaxRows) return LaunchAttentionDecode(p, stream);   // one MMA of 16 rows holds every query row
  int dev = 0;
  cudaGetDevice(&dev);
  using KernelFn = void (*)(const AttnParam, const AttnMaps, const LaunchTag);
  static const KernelFn kernels[2] = {dvm_b200_attention_bf16, dvm_b200_attention_f16};
  static bool attr_set[64] = {false};
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    for (auto fn : kernels) {
      cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
      if (e != cudaSuccess) return static_cast<int>(e);
    }
    attr_set[dev] = true;
  }
  const uint32_t sms = static_cast<uint32_t>(Runtime::Get().sm_count_or_default());
  const uint64_t blocks128 = static_cast<uint64_t>(p.batch) * ((p.sq + kTileQ - 1) / kTileQ);
  // one row tile per CTA while that leaves no CTA waiting for an SM: a tile alone takes little more than half the time of two
  p.q_tiles = blocks128 <= sms ? 1 : 2;
  const KernelFn kernel = kernels[p.dtype == T_BF16 ? 0 : 1];
  AttnMaps maps;
  int rc = EncodeRows(&maps.q, p.q_ptr, p.d, p.sq, p.batch, kTileQ);
  if (rc == 0) rc = EncodeRows(&maps.k, p.k_ptr, p.d, p.skv, p.batch, kTileKV);
  if (rc == 0) rc = EncodeRows(&maps.v, p.v_ptr, p.d, p.skv, p.batch, kTileKV);
  if (rc == 0) rc = EncodeRows(&maps.o, p.o_ptr, p.d, p.sq, p.batch, 16);   // what a warp stores at a time
  if (rc != 0) return rc;
  const uint32_t unit_rows = kTileQ * p.q_tiles;
  const uint64_t units = static_cast<uint64_t>(p.batch) * ((p.sq + unit_rows - 1) / unit_rows);
  if (units >= (1ull << 31) || units * ((p.skv + kTileKV - 1) / kTileKV) / sms >= (1ull << 30)) return -3;   // (32-bit counters)
  p.units = static_cast<uint32_t>(units);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3(p.units < sms ? p.units : sms, 1, 1);
  cfg.blockDim = dim3(32 * (kFirstSoftmaxWarp + kTileWarps * p.q_tiles), 1, 1);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = static_cast<cudaStream_t>(stream);
  ChainAttribute(&cfg, attr);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p, maps, NextLaunchEpoch());
  return e != cudaSuccess ? static_cast<int>(e) : static_cast<int>(cudaGetLastError());
}

unsigned int ReadAttentionStatus() {
  WaitStatus v = {0u, 0u};
  const unsigned int zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_attn_status, sizeof(v)) != cudaSuccess) return 0xffffffffu;
  if (v.first_error != 0) cudaMemcpyToSymbol(g_attn_status, &zero, sizeof(zero), offsetof(WaitStatus, first_error));
  return v.first_error;
}

}  // namespace dvmb
