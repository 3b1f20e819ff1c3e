// MatMul tiles for problems that do not fill the machine with 256 x 256 CTA pairs (mm_tcgen05.cu), or whose operands the
// copy engine cannot address: few rows (decode), few tiles, rows that do not start on 16 bytes.
//
// One CTA = one 128 x BN tile of C (BN = 64 or 128) over a slice of K; the S CTAs of a cluster share a tile and add their
// partial products through distributed shared memory, in rank order.
//   warp 0     TMA producer of the operands the copy engine can address
//   warp 1     MMA issuer: four tcgen05.mma (K = 16) per stage into one TMEM accumulator
//   warps 2-9  loaders of an operand the copy engine cannot address (16-byte loads from the aligned address below, shifted
//              into place in registers, written to shared memory in the 128-byte swizzled layout TMA would have written);
//              then TMEM -> shared memory
//   all warps  sum over the cluster, bias, rounding, post-fusion program; 16-bit results leave through shared memory (a CTA that
//              has its tile to itself drains TMEM by warps 2-9 instead, without the exchange)
//
// What bounds it: a [16, 8192] x [8192, 8192] product is the read of the weight (134 MB, 21 us at the measured copy
// bandwidth).  In 128 x 256 tiles that was 32 CTAs on 148 SMs; in tiles of 64 columns with K cut in two it is 256 CTAs
// with 2 x 80 KB of weight in flight per SM.  A product of [1024, 1001] and [1001, 5003] (rows of the second at any even
// address) took 6.4 ms on CUDA cores, element by element, 56 us with the work warps as loaders and 26 us with the operand
// repacked first (dvm_b200_mm_pack below); the loaders remain for what is not worth a copy and for launches without a workspace.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>

#include "chain.cuh"
#include "mm_epilogue.cuh"
#include "mm_launch.h"
#include "sm100_sync.cuh"

namespace dvmb {

__device__ WaitStatus g_mm_tile_status = {0u, 0u};

namespace {

constexpr uint32_t BM = 128, BK = 64;
constexpr uint32_t kWorkWarps = 8;
constexpr uint32_t kWorkThreads = 32 * kWorkWarps;
constexpr uint32_t kThreads = 64 + kWorkThreads;
constexpr uint32_t kHeader = 1024;           // barriers, TMEM address; the stages follow on a 1024-byte boundary
constexpr uint32_t kMaxStages = 16;
constexpr uint32_t kBarFull = 0, kBarEmpty = 128, kBarDone = 256, kTmemSlot = 264, kBiasOff = 512;   // (bias: up to 128 fp32)

struct TileMaps {
  CUtensorMap a, b;
  CUtensorMap o;   // the result (P.tma_out)
};

struct TileArgs {
  uint32_t a_rows;        // rows of A staged per k-block (a multiple of 8; below 128 when M is smaller)
  uint32_t stages, stage_bytes;
  uint32_t gather_a, gather_b;   // operand loaded by the work warps instead of TMA
  uint32_t out_off;       // byte offset (from the stage area) of the buffer 16-bit results leave through
};

// ---- operands at any even address ------------------------------------------------------------------------
struct Gather {
  const unsigned short *base;   // first element of the batch slice
  uint32_t inner, rows;         // extent of the contiguous axis (= row pitch) and of the other one
  bool kmajor;                  // contraction axis innermost
};

// One 16-byte piece of an operand box: piece i of a tile W wide along the non-contracted axis, at `mn0` along that axis and
// `k0` along the contraction.  K-major boxes are W rows of 64 k; the other form is 64-row boxes of [k][64].
struct Piece {
  uint4 lo, hi;
  uint32_t off, valid;
};
__device__ __forceinline__ void piece_at(const Gather &g, uint32_t i, uint32_t mn0, uint32_t k0, uint32_t &row, uint32_t &col) {
  if (g.kmajor) {
    row = mn0 + (i >> 3);
    col = k0 + (i & 7u) * 8u;
  } else {
    row = k0 + ((i >> 3) & 63u);
    col = mn0 + (i >> 9) * 64u + (i & 7u) * 8u;
  }
}
__device__ __forceinline__ void load_at(const Gather &g, uint32_t row, uint32_t col, Piece &p) {
  p.lo = p.hi = make_uint4(0, 0, 0, 0);
  p.off = 0;
  p.valid = 0;
  if (row >= g.rows || col >= g.inner) return;
  p.valid = min(8u, g.inner - col);
  const uint64_t s = reinterpret_cast<uint64_t>(g.base + ((uint64_t)row * g.inner + col));
  const uint64_t a = s & ~15ull;
  p.off = (uint32_t)(s & 15ull) >> 1;
  // (a 16-byte unit that holds at least one element of the row never leaves the row's memory page)
  p.lo = gload(reinterpret_cast<const uint4 *>(a));
  if (p.off + p.valid > 8u) p.hi = gload(reinterpret_cast<const uint4 *>(a) + 1);
}
__device__ __forceinline__ void load_piece(const Gather &g, uint32_t i, uint32_t mn0, uint32_t k0, Piece &p) {
  uint32_t row, col;
  piece_at(g, i, mn0, k0, row, col);
  load_at(g, row, col, p);
}
__device__ __forceinline__ uint4 elements_of(const Piece &p) {
  uint4 v = shift_in(p.lo, p.hi, p.off);
  if (p.valid < 8u) {   // what lies past the row (or outside the matrix) is zero
    uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) w[j] = 2 * j + 2 <= p.valid ? w[j] : (2 * j + 1 <= p.valid ? (w[j] & 0xffffu) : 0u);
    v = make_uint4(w[0], w[1], w[2], w[3]);
  }
  return v;
}
__device__ __forceinline__ void store_piece(const Gather &g, uint32_t i, uint32_t box, const Piece &p) {
  const uint4 v = elements_of(p);
  // both forms: rows of 128 bytes, 16-byte piece c of row r at c ^ (r & 7); boxes of the [k][64] form are 8 KB apart
  const uint32_t r = i >> 3, c = i & 7u;
  const uint32_t dst = box + r * 128u + ((c ^ (r & 7u)) << 4);
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

__device__ __forceinline__ float4 ld_cluster_v4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t cluster_nctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}

// Bytes per row of a partial product in shared memory; the 16 keep rows off each other's banks.
template <uint32_t BN>
constexpr uint32_t kPitch = BN * 4 + 16;

// The partial products of strips [i_begin, i_end) of a cluster's tile, added in rank order: 16 bytes per lane and side by side,
// every remote read of two rounds (one of eight CTAs) in flight before the first is used.  (Taken strip by strip, 64 bytes
// apart, one after the other, they were 12 us of the 37 us of a [128, 8192] x [8192, 8192] product.)  The sum replaces this
// CTA's own partial, which no one else reads, the four pieces of a strip at p ^ (strip / 2 & 3) so that the readers of
// whole strips do not meet on a bank.
template <uint32_t BN, uint32_t S>
__device__ __forceinline__ void sum_partials(uint32_t ring, uint32_t i_begin, uint32_t i_end) {
  constexpr uint32_t kRounds = S == 8 ? 1 : 2;
  for (uint32_t u0 = i_begin * 4u; u0 < i_end * 4u; u0 += kRounds * kThreads) {
    float4 v[kRounds][S];
    uint32_t to[kRounds];
#pragma unroll
    for (uint32_t h = 0; h < kRounds; ++h) {
      const uint32_t u = u0 + h * kThreads + threadIdx.x, row = u / (BN / 4), piece = u - row * (BN / 4);
      to[h] = 0;
      if (u < i_end * 4u) {
        const uint32_t at = ring + row * kPitch<BN>;
        to[h] = at + ((piece & ~3u) + ((piece & 3u) ^ ((piece >> 3) & 3u))) * 16u;
#pragma unroll
        for (uint32_t p = 0; p < S; ++p) v[h][p] = ld_cluster_v4(map_to_cta(at + piece * 16u, p));
      }
    }
    __syncwarp();   // (the pieces of a strip belong to lanes of one warp)
#pragma unroll
    for (uint32_t h = 0; h < kRounds; ++h) {
      if (to[h] == 0) continue;
      float4 w = v[h][0];
#pragma unroll
      for (uint32_t p = 1; p < S; ++p) {
        w.x += v[h][p].x;
        w.y += v[h][p].y;
        w.z += v[h][p].z;
        w.w += v[h][p].w;
      }
      asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(to[h]), "f"(w.x), "f"(w.y), "f"(w.z), "f"(w.w) : "memory");
    }
  }
}

template <uint32_t BN>
__device__ __forceinline__ void tile_body(const MmParam &P, const TileMaps &maps, const TileArgs &A, const LaunchTag epoch) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t *smem = smem_raw + (base - raw_addr);
  const uint32_t ring = base + kHeader;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t S = cluster_nctarank(), rank = cluster_ctarank();
  const uint32_t mblocks = (P.M + BM - 1) / BM, nblocks = (P.N + BN - 1) / BN, kblocks = (P.K + BK - 1) / BK;
  uint32_t bz, mb, nb;
  tile_coords(blockIdx.x / S, mblocks, nblocks, P.group_m, bz, mb, nb);
  const uint32_t b0 = bz / P.batch1, b1 = bz - b0 * P.batch1;
  const uint32_t za = b0 * P.a_mul0 + b1 * P.a_mul1, zb = b0 * P.b_mul0 + b1 * P.b_mul1;
  const uint32_t kb_begin = kblocks * rank / S, kb_end = kblocks * (rank + 1) / S;
  const uint32_t row0 = mb * BM, col0 = nb * BN;
  const bool gather = (A.gather_a | A.gather_b) != 0;

  if (mblocks == 1 && !A.gather_b && warp == 2 && elect_one()) {
    // A weight that each tile reads once comes from memory: its first stages are on their way to L2 while the kernel before
    // this one still runs (a prefetch reads nothing that could be stale, L2 holds whatever is written to it meanwhile;
    // [16, 8192] x [8192, 8192] 28.8 -> 27.6 us).  Where several rows of tiles share it, it mostly is in L2, and the
    // prefetches only delay the loads ([1000, 1000] x [1000, 1000] 9.2 -> 10.0).
    for (uint32_t kb = kb_begin; kb < min(kb_end, kb_begin + A.stages); ++kb) {
      const int k = (int)(kb * BK);
      if (P.b_kmajor) {
        tma_prefetch_3d(&maps.b, k, (int)col0, (int)zb);
      } else {
#pragma unroll
        for (uint32_t j = 0; j < BN / 64; ++j) tma_prefetch_3d(&maps.b, (int)(col0 + j * 64), k, (int)zb);
      }
    }
  }
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < A.stages; ++s) {
      mbar_init(base + kBarFull + 8 * s, gather ? 1u + kWorkWarps : 1u);
      mbar_init(base + kBarEmpty + 8 * s, 1);
    }
    mbar_init(base + kBarDone, 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(base + kTmemSlot, BN);
    tmem_relinquish();
  }
  tcgen05_before_sync();
  __syncthreads();
  tcgen05_after_sync();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t *>(smem + kTmemSlot);
  chain_wait();
  chain_launch();

  // stage: B [BN x 64] first, then A (its MMA reads 128 rows; the rows past a_rows are whatever follows, and only feed rows
  // of the accumulator that are never read)
  if (warp == 0) {
    const uint32_t bytes = (A.gather_a ? 0u : A.a_rows * 128u) + (A.gather_b ? 0u : BN * 128u);
    const bool tma_a = A.gather_a == 0, tma_b = A.gather_b == 0, a_m = P.a_mmajor != 0, b_k = P.b_kmajor != 0, a_two = A.a_rows > 64u;
    if (elect_one()) {
      uint32_t stage = 0, parity = 1, sb = ring;
      int k = (int)(kb_begin * BK);
      for (uint32_t kb = kb_begin; kb < kb_end; ++kb, k += (int)BK) {
        mbar_wait(base + kBarEmpty + 8 * stage, parity, 1, &g_mm_tile_status, epoch);
        const uint32_t full = base + kBarFull + 8 * stage, sa = sb + BN * 128u;
        if (bytes != 0) {
          mbar_expect_tx(full, bytes);
        } else {
          mbar_arrive(full);
        }
        if (tma_b) {
          if (b_k) {
            tma_load_3d(sb, &maps.b, full, k, (int)col0, (int)zb);
          } else {
  #pragma unroll
            for (uint32_t j = 0; j < BN / 64; ++j) tma_load_3d(sb + j * 8192u, &maps.b, full, (int)(col0 + j * 64), k, (int)zb);
          }
        }
        if (tma_a) {
          if (!a_m) {
            tma_load_3d(sa, &maps.a, full, k, (int)row0, (int)za);
          } else {
            tma_load_3d(sa, &maps.a, full, (int)row0, k, (int)za);
            if (a_two) tma_load_3d(sa + 8192u, &maps.a, full, (int)(row0 + 64), k, (int)za);
          }
        }
        sb += A.stage_bytes;
        if (++stage == A.stages) {
          stage = 0;
          parity ^= 1u;
          sb = ring;
        }
      }
    }
  } else if (warp == 1) {
    // instruction descriptor: see mm_tcgen05.cu
    const uint32_t fmt = P.in_dtype == T_BF16 ? 1u : 0u;
    const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((P.a_mmajor ? 1u : 0u) << 15) |
                           ((P.b_kmajor ? 0u : 1u) << 16) | ((BN >> 3) << 17) | ((BM >> 4) << 24);
    // (descriptor of stage 0; a stage or a K = 16 step further is an addition to its address field)
    const uint64_t da0 = P.a_mmajor ? make_smem_desc(ring + BN * 128u, 8192, 1024) : make_smem_desc(ring + BN * 128u, 0, 1024);
    const uint64_t db0 = P.b_kmajor ? make_smem_desc(ring, 0, 1024) : make_smem_desc(ring, 8192, 1024);
    const uint64_t step_a = P.a_mmajor ? 2048 >> 4 : 32 >> 4, step_b = P.b_kmajor ? 32 >> 4 : 2048 >> 4;
    const uint64_t step_stage = A.stage_bytes >> 4;
    if (elect_one()) {
      uint32_t stage = 0, parity = 0;
      uint64_t da = da0, db = db0;
      for (uint32_t kb = kb_begin; kb < kb_end; ++kb) {
        mbar_wait(base + kBarFull + 8 * stage, parity, 3, &g_mm_tile_status, epoch);
#pragma unroll
        for (uint32_t kk = 0; kk < BK / 16; ++kk)
          umma_f16_cta1(tmem_base, da + kk * step_a, db + kk * step_b, idesc, (kb != kb_begin || kk != 0) ? 1u : 0u);
        umma_commit_cta1(base + kBarEmpty + 8 * stage);
        da += step_stage;
        db += step_stage;
        if (++stage == A.stages) {
          stage = 0;
          parity ^= 1u;
          da = da0;
          db = db0;
        }
      }
      umma_commit_cta1(base + kBarDone);
    }
  } else if (gather) {
    const uint32_t wt = threadIdx.x - 64u;
    const Gather ga{reinterpret_cast<const unsigned short *>(P.a_ptr) + (uint64_t)za * P.M * P.K, P.a_mmajor ? P.M : P.K,
                    P.a_mmajor ? P.K : P.M, P.a_mmajor == 0};
    const Gather gb{reinterpret_cast<const unsigned short *>(P.b_ptr) + (uint64_t)zb * P.N * P.K, P.b_kmajor ? P.K : P.N,
                    P.b_kmajor ? P.N : P.K, P.b_kmajor != 0};
    constexpr uint32_t NA = BM * 8 / kWorkThreads, NB = BN * 8 / kWorkThreads;
    uint32_t stage = 0, parity = 1;
    for (uint32_t kb = kb_begin; kb < kb_end; ++kb) {
      const uint32_t sb = ring + stage * A.stage_bytes, sa = sb + BN * 128u;
      Piece pa[NA], pb[NB];
      // every load of the k-block is in flight before the first one is used
      if (A.gather_b) {
#pragma unroll
        for (uint32_t j = 0; j < NB; ++j) load_piece(gb, wt + j * kWorkThreads, col0, kb * BK, pb[j]);
      }
      if (A.gather_a) {
#pragma unroll
        for (uint32_t j = 0; j < NA; ++j)
          if (wt + j * kWorkThreads < A.a_rows * 8u) load_piece(ga, wt + j * kWorkThreads, row0, kb * BK, pa[j]);
      }
      mbar_wait(base + kBarEmpty + 8 * stage, parity, 1, &g_mm_tile_status, epoch);
      if (A.gather_b) {
#pragma unroll
        for (uint32_t j = 0; j < NB; ++j) store_piece(gb, wt + j * kWorkThreads, sb, pb[j]);
      }
      if (A.gather_a) {
#pragma unroll
        for (uint32_t j = 0; j < NA; ++j)
          if (wt + j * kWorkThreads < A.a_rows * 8u) store_piece(ga, wt + j * kWorkThreads, sa, pa[j]);
      }
      fence_async_shared();   // the MMA reads what the stores above wrote
      __syncwarp();
      if (lane == 0) mbar_arrive(base + kBarFull + 8 * stage);
      if (++stage == A.stages) {
        stage = 0;
        parity ^= 1u;
      }
    }
  }
  __syncwarp();

  // ---- the product of a CTA alone: TMEM -> result ----
  const uint32_t rows = min(BM, P.M - row0);
  if (S == 1) {
    if (warp >= 2) {
      const uint32_t wt = threadIdx.x - 64u;
      if (wt < BN && P.bias_ptr != 0) reinterpret_cast<float *>(smem + kBiasOff)[wt] = bias_at(P, col0 + wt);
      asm volatile("bar.sync 1, %0;" ::"n"(kWorkThreads) : "memory");
      if (kblocks != 0) mbar_wait(base + kBarDone, 0, 4, &g_mm_tile_status, epoch);
      tcgen05_after_sync();
      const uint32_t quarter = warp & 3u, half = (warp - 2) >> 2;
      if (quarter * 32u < rows) {
        EpiPos pos;
        pos.b0 = b0;
        pos.b1 = b1;
        with_mode(P, [&](auto mode) {
          drain<decltype(mode)::mode, decltype(mode)::dtype, BN / 2>(
            P, maps.o, tmem_base + ((quarter * 32u) << 16) + half * (BN / 2), kblocks == 0, pos, row0 + quarter * 32u, col0 + half * (BN / 2),
            base + kBiasOff + half * (BN / 2) * 4u, ring + (warp - 2) * kDrainBytes<BN / 2>, lane);   // (the stages are free)
        });
        if (elect_one()) tma_store_wait_read<0>();   // shared memory stays until the last store has read it
      }
    }
    __syncwarp();
    tcgen05_before_sync();
    __syncthreads();
    if (warp == 1) {
      tcgen05_after_sync();
      tmem_dealloc(tmem_base, BN);
    }
    return;
  }

  // ---- a partial product: TMEM -> shared memory (the stages are free: every MMA has completed) ----
  if (warp >= 2) {
    const uint32_t wt = threadIdx.x - 64u;
    if (wt < BN && P.bias_ptr != 0) reinterpret_cast<float *>(smem + kBiasOff)[wt] = bias_at(P, col0 + wt);
    mbar_wait(base + kBarDone, 0, 4, &g_mm_tile_status, epoch);
    tcgen05_after_sync();
    const uint32_t quarter = warp & 3u, half = (warp - 2) >> 2;
    if (quarter * 32u < rows) {
      const uint32_t taddr = tmem_base + ((quarter * 32u) << 16) + half * (BN / 2);
      uint32_t r[BN / 2];
#pragma unroll
      for (uint32_t c = 0; c < BN / 2; c += 32) tmem_ld_32x32b_x32_nowait(taddr + c, &r[c]);
      tmem_ld_wait();
      const uint32_t row = quarter * 32u + lane;
      const uint32_t dst = ring + row * kPitch<BN> + half * (BN / 2) * 4u;
      if (row < rows) {   // (the buffer holds the rows the matrix has)
#pragma unroll
        for (uint32_t c = 0; c < BN / 2; c += 4)
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst + c * 4u), "r"(r[c]), "r"(r[c + 1]), "r"(r[c + 2]), "r"(r[c + 3])
                       : "memory");
      }
    }
  }
  __syncwarp();
  tcgen05_before_sync();
  cluster_sync_all();
  if (warp == 1) {
    tcgen05_after_sync();
    tmem_dealloc(tmem_base, BN);
  }

  // ---- sum over the cluster and finish: this CTA's share of the tile's 16-column strips, row by row ----
  constexpr uint32_t kSpr = BN / 16;   // strips per row
  const uint32_t strips = rows * kSpr;
  const uint32_t i_begin = strips * rank / S, i_end = strips * (rank + 1) / S;
  if (S == 2) {
    sum_partials<BN, 2>(ring, i_begin, i_end);
  } else if (S == 4) {
    sum_partials<BN, 4>(ring, i_begin, i_end);
  } else {
    sum_partials<BN, 8>(ring, i_begin, i_end);
  }
  __syncthreads();
  with_mode(P, [&](auto mode) {
    for (uint32_t i = i_begin + threadIdx.x; i < i_end; i += kThreads) {
      const uint32_t row = i / kSpr, strip = i - row * kSpr;
      EpiPos pos;
      pos.b0 = b0;
      pos.b1 = b1;
      pos.row = row0 + row;
      pos.col = col0 + strip * 16u;
      if (pos.col >= P.N) continue;
      pos.valid = min(16u, P.N - pos.col);
      const uint32_t at = ring + row * kPitch<BN> + strip * 64u;
      uint32_t r[16], pk[8];
#pragma unroll
      for (uint32_t g = 0; g < 4; ++g)
        asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[4 * g]), "=r"(r[4 * g + 1]), "=r"(r[4 * g + 2]), "=r"(r[4 * g + 3])
                     : "r"(at + ((g ^ ((strip >> 1) & 3u)) << 4)));
      if (P.bias_ptr != 0) add_bias_staged(base + kBiasOff + strip * 64u, r);
      finish_strip<decltype(mode)::mode, decltype(mode)::dtype>(P, pos, r, pk);
      if (decltype(mode)::mode != EPI_PROGRAM) {
        const uint32_t dst = ring + A.out_off + (i - i_begin) * 32u;
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(pk[0]), "r"(pk[1]), "r"(pk[2]), "r"(pk[3]) : "memory");
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst + 16u), "r"(pk[4]), "r"(pk[5]), "r"(pk[6]), "r"(pk[7]) : "memory");
      }
    }
  });
  if (P.epi_mode >= EPI_STORE) {
    __syncthreads();
    const EpiTensor &t = P.tensor[P.out_slot];
    unsigned short *out = reinterpret_cast<unsigned short *>(t.ptr) + ((int64_t)b0 * t.sb0 + (int64_t)b1 * t.sb1);
    const uint8_t *staged = smem + kHeader + A.out_off;
    const bool vec = (reinterpret_cast<uint64_t>(out) & 15u) == 0 && (t.sm & 7) == 0;
    if (vec) {
      for (uint32_t j = threadIdx.x; j < 2u * (i_end - i_begin); j += kThreads) {
        const uint32_t i = i_begin + (j >> 1), row = i / kSpr, col = col0 + (i - row * kSpr) * 16u + (j & 1u) * 8u;
        if (col >= P.N) continue;
        unsigned short *dst = out + (int64_t)(row0 + row) * t.sm + col;
        const uint4 q = *reinterpret_cast<const uint4 *>(staged + 16u * j);
        if (col + 8u <= P.N) {
          *reinterpret_cast<uint4 *>(dst) = q;
        } else {
          const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
          for (uint32_t e = 0; e < 8; ++e)
            if (col + e < P.N) dst[e] = (unsigned short)(w[e >> 1] >> (16u * (e & 1u)));
        }
      }
    } else {
      // rows at any even address, or strips that start inside one
      const uint32_t r_begin = i_begin / kSpr, r_count = i_end > i_begin ? (i_end - 1) / kSpr + 1 - r_begin : 0u;
      constexpr uint32_t kUnits = 2 * kSpr - 1;
      auto row_of = [&](uint32_t r, unsigned short *&dst, uint32_t &col, uint32_t &run, uint32_t &from) {
        const uint32_t first = max(i_begin, r * kSpr), last = min(i_end, (r + 1) * kSpr);
        col = col0 + (first - r * kSpr) * 16u;
        run = (last - first) * 16u;
        from = (first - i_begin) * 32u;
        dst = out + (int64_t)(row0 + r) * t.sm + col;
      };
      unsigned short *dst;
      uint32_t col, run, from;
      for (uint32_t j = threadIdx.x; j < r_count * kUnits; j += kThreads) {
        const uint32_t r = j / kUnits, u = j - r * kUnits;
        row_of(r_begin + r, dst, col, run, from);
        const uint32_t ahead = elements_ahead(dst), at = ahead + 8u * u;
        if (at + 8u > run || col + at >= P.N) continue;
        const uint4 *piece = reinterpret_cast<const uint4 *>(staged + from) + (at >> 3);
        const uint4 lo = piece[0], hi = (ahead & 7u) != 0 ? piece[1] : lo;
        store_unit(dst + at, shift_in(lo, hi, ahead & 7u), P.N - (col + at));
      }
      for (uint32_t j = threadIdx.x; j < r_count * 8u; j += kThreads) {
        row_of(r_begin + (j >> 3), dst, col, run, from);
        const uint32_t at = single_at(j & 7u, elements_ahead(dst), run);
        if (col + at < P.N) dst[at] = *reinterpret_cast<const unsigned short *>(staged + from + 2u * at);
      }
    }
  }
  __syncwarp();
  cluster_sync_all();   // no CTA leaves while a peer may still read its partial product
}

}  // namespace

// (two CTAs per SM: one's loads and MMAs run beside the other's epilogue)
__global__ void __launch_bounds__(kThreads, 2) dvm_b200_mm_tile_n64(const __grid_constant__ MmParam P, const __grid_constant__ TileMaps maps,
                                                                    const __grid_constant__ TileArgs A, const LaunchTag epoch) {
  tile_body<64>(P, maps, A, epoch);
}
__global__ void __launch_bounds__(kThreads, 2) dvm_b200_mm_tile_n128(const __grid_constant__ MmParam P, const __grid_constant__ TileMaps maps,
                                                                     const __grid_constant__ TileArgs A, const LaunchTag epoch) {
  tile_body<128>(P, maps, A, epoch);
}

// Operands of unaligned rows, copied to rows of whole 16-byte units for the copy engine.  Loading them by the work warps of
// every tile costs 1700 cycles per k-block, seven times its MMAs, and each tile does it again.
// Bound by memory: one pass, four independent pieces per thread.  [4096, 4095] x [4001, 4095]^T: 886 -> 123 us in all,
// [2000, 2001] x [2001, 2001] 144 -> 34, [180, 511] x [565, 511]^T 12.7 -> 8.9.
struct PackJob {
  const unsigned short *src;
  uint4 *dst;
  uint32_t inner, rows;      // rows of all batch slices
  uint32_t units, blocks;    // 16-byte units per row of the copy; thread blocks of this job
};
constexpr uint32_t kPackThreads = 256, kPackPieces = 4;

__global__ void __launch_bounds__(kPackThreads) dvm_b200_mm_pack(const PackJob ja, const PackJob jb) {
  chain_wait();
  chain_launch();
  const bool second = blockIdx.x >= ja.blocks;
  const PackJob &j = second ? jb : ja;
  const Gather g{j.src, j.inner, j.rows, true};
  const uint32_t first = (blockIdx.x - (second ? ja.blocks : 0u)) * (kPackThreads * kPackPieces) + threadIdx.x;
  Piece p[kPackPieces];
#pragma unroll
  for (uint32_t i = 0; i < kPackPieces; ++i) {
    const uint32_t at = first + i * kPackThreads, row = at / j.units;
    load_at(g, row, (at - row * j.units) * 8u, p[i]);   // (nothing past the last row)
  }
#pragma unroll
  for (uint32_t i = 0; i < kPackPieces; ++i)
    if (p[i].valid != 0) j.dst[first + i * kPackThreads] = elements_of(p[i]);
}

int LaunchMmPack(MmParam *p, void *stream) {
  PackJob job[2];
  memset(job, 0, sizeof(job));
  auto fill = [](PackJob *j, uint64_t *ptr, uint32_t *pitch, uint64_t to, uint32_t inner, uint64_t rows) {
    j->src = reinterpret_cast<const unsigned short *>(*ptr);
    j->dst = reinterpret_cast<uint4 *>(to);
    j->inner = inner;
    j->rows = static_cast<uint32_t>(rows);
    j->units = (inner + 7) / 8;
    j->blocks = static_cast<uint32_t>((rows * j->units + kPackThreads * kPackPieces - 1) / (kPackThreads * kPackPieces));
    *ptr = to;
    *pitch = j->units * 8;
  };
  if (p->a_pack != 0 && MmGatherA(*p)) fill(&job[0], &p->a_ptr, &p->a_pitch, p->a_pack, MmInnerA(*p), static_cast<uint64_t>(MmRowsA(*p)) * p->a_batches);
  if (p->b_pack != 0 && MmGatherB(*p)) fill(&job[1], &p->b_ptr, &p->b_pitch, p->b_pack, MmInnerB(*p), static_cast<uint64_t>(MmRowsB(*p)) * p->b_batches);
  if (job[0].blocks + job[1].blocks == 0) return 0;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3(job[0].blocks + job[1].blocks, 1, 1);
  cfg.blockDim = dim3(kPackThreads, 1, 1);
  cfg.stream = static_cast<cudaStream_t>(stream);
  ChainAttribute(&cfg, attr);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, dvm_b200_mm_pack, job[0], job[1]);
  return e != cudaSuccess ? static_cast<int>(e) : static_cast<int>(cudaGetLastError());
}

int LaunchMmTile(const MmParam &p_in, uint32_t bn, uint32_t split, void *stream) {
  MmParam p = p_in;
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  constexpr uint32_t kBudget = 112 * 1024;   // two CTAs per SM
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(dvm_b200_mm_tile_n64, cudaFuncAttributeMaxDynamicSharedMemorySize, kBudget);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(dvm_b200_mm_tile_n128, cudaFuncAttributeMaxDynamicSharedMemorySize, kBudget);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set[dev] = true;
  }
  TileArgs a;
  memset(&a, 0, sizeof(a));
  a.gather_a = MmGatherA(p) ? 1u : 0u;
  a.gather_b = MmGatherB(p) ? 1u : 0u;
  // rows of A a tile really has, in whole swizzle groups (whole 64-row boxes when A is stored [k][m])
  const uint32_t m_rows = p.M < BM ? p.M : BM;
  a.a_rows = p.a_mmajor ? (m_rows + 63u) / 64u * 64u : (m_rows + 7u) / 8u * 8u;
  const uint32_t b_bytes = bn * 128u, a_bytes = a.a_rows * 128u, over = BM * 128u - a_bytes;
  a.stage_bytes = a_bytes + b_bytes;
  const uint32_t kblocks = (p.K + BK - 1) / BK, per_cta = (kblocks + split - 1) / split;
  uint32_t stages = (kBudget - kHeader - 1024u - over) / a.stage_bytes;
  if (stages > kMaxStages) stages = kMaxStages;
  if (stages > per_cta) stages = per_cta < 1u ? 1u : per_cta;
  a.stages = stages;
  a.out_off = BM * (bn * 4u + 16u);
  if (p.M < BM) a.out_off = (p.M * (bn * 4u + 16u) + 127u) & ~127u;
  const uint32_t strips = m_rows * (bn / 16u), share = (strips + split - 1) / split + 1;
  const uint32_t ring_bytes = stages * a.stage_bytes + over, out_bytes = a.out_off + share * 32u;
  const uint32_t drained = kWorkWarps * (bn == 64 ? kDrainBytes<32> : kDrainBytes<64>), after = split == 1 ? drained : out_bytes;
  const uint32_t smem = kHeader + 1024u + (ring_bytes > after ? ring_bytes : after);
  if (smem > kBudget) return -5;
  TileMaps maps;
  memset(&maps, 0, sizeof(maps));
  int rc = 0;
  if (!a.gather_a && kblocks != 0)
    rc = EncodeMmOperand(&maps.a, p.a_ptr, MmInnerA(p), MmPitchA(p), MmRowsA(p), p.a_batches, p.a_mmajor ? 64 : a.a_rows);
  if (rc == 0 && !a.gather_b && kblocks != 0)
    rc = EncodeMmOperand(&maps.b, p.b_ptr, MmInnerB(p), MmPitchB(p), MmRowsB(p), p.b_batches, p.b_kmajor ? bn : 64);
  if (rc != 0) return rc;
  p.tma_out = split == 1 && p.epi_mode >= EPI_STORE && EncodeMmResult(&maps.o, p) ? 1u : 0u;
  const uint64_t tiles = static_cast<uint64_t>((p.M + BM - 1) / BM) * ((p.N + bn - 1) / bn) * p.batch0 * p.batch1;
  if (tiles * split >= (1ull << 31)) return -6;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(static_cast<uint32_t>(tiles * split), 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  ChainAttribute(&cfg, attr);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, bn == 64 ? dvm_b200_mm_tile_n64 : dvm_b200_mm_tile_n128, p, maps, a, NextLaunchEpoch());
  return e != cudaSuccess ? static_cast<int>(e) : static_cast<int>(cudaGetLastError());
}

unsigned int ReadMmTileStatus() {
  WaitStatus v = {0u, 0u};
  const unsigned int zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_mm_tile_status, sizeof(v)) != cudaSuccess) return 0xffffffffu;
  if (v.first_error != 0) cudaMemcpyToSymbol(g_mm_tile_status, &zero, sizeof(zero), offsetof(WaitStatus, first_error));
  return v.first_error;
}

}  // namespace dvmb
