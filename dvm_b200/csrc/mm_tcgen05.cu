// MatMul (+ bias, + fused post-ops) on the sm_100a tensor cores: tcgen05.mma with the accumulator in tensor
// memory, operands staged by TMA into a shared-memory ring, post-fusion ops applied to the accumulator as it is
// drained from TMEM.
//
// Stands in for the reference's cube path, which exists only for Ascend (CubeOp src/ops_m.cc:271-696, the mix
// kernel that shards post-fusion ops per C tile src/xkernel.cc:157-361); the reference's CUDA backend has no
// MatMul at all (src/system.cc:290-294).  Semantics kept: fp16/bf16 operands, fp32 accumulation, optional bias
// added in fp32, result rounded to the operand dtype, then the fused vector ops.
//
// Two CTAs of a cluster = one 256 x 256 tile of C at a time (persistent over tiles, grouped along M for L2 reuse):
//   warp 0     TMA producer: A [128 x 64] and half of B [128 x 64] per stage (64 x 64 boxes when the operand is stored
//              with the contraction axis outermost)
//   warp 1     MMA issuer: four tcgen05.mma (K = 16) per stage into one of two TMEM accumulators
//   warps 2-9  epilogue: tcgen05.ld 16 columns at a time, bias, rounding, post-fusion program; 16-bit results leave as
//              runs of 128 bytes per row through shared memory
// Every mbarrier wait is bounded; on expiry a status word is set and the kernel runs to its end.
//
// Problems that do not fill the machine with such tiles, and problems the copy engine cannot address (row pitch or base
// not 16-byte aligned), run as smaller tiles (mm_tile.cu).
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <cstring>

#include "chain.cuh"
#include "mm_epilogue.cuh"
#include "mm_launch.h"
#include "runtime.h"
#include "sm100_sync.cuh"

namespace dvmb {

__device__ WaitStatus g_mm_status = {0u, 0u};

namespace {

// Tile geometry.  The two CTAs of a cluster share one MMA of 256 x 256: each stages its own 128 rows of A and one half
// (128 columns) of B, i.e. 32 KB per k-block.
constexpr uint32_t BM = 128, BN = 256, BK = 64;
constexpr uint32_t kABytes = BM * BK * 2;   // 16 KB
constexpr uint32_t kEpiWarps = 8;
constexpr uint32_t kEpiCols = BN / (kEpiWarps / 4);   // columns of the tile a warp drains
constexpr uint32_t kThreads = 64 + 32 * kEpiWarps;
constexpr uint32_t kTmemCols = 512;   // two 256-column fp32 accumulators
// shared memory: [0, 1024) barriers + tmem pointer, the bias of each epilogue warp's columns as fp32, then the stages
// (1024-byte aligned for the 128B swizzle)
constexpr uint32_t kBiasOff = 1024;
constexpr uint32_t kSmemHeader = kBiasOff + kEpiWarps * kEpiCols * 4;
constexpr uint32_t kBBytes = (BN / 2) * BK * 2;
constexpr uint32_t kStageBytes = kABytes + kBBytes;
constexpr uint32_t kStages = 5;
// Results of 64 columns at a time, per epilogue warp: 32 rows of 128 bytes.  Stored from the registers of the thread that owns
// the row, every 16-byte store was a write request of its own, and a tile's epilogue took 14 600 cycles against 5 100 for
// ten k-blocks of MMAs; worth more than the sixth operand stage that the 32 KB would hold.
constexpr uint32_t kOutBytes = kDrainBytes<kEpiCols>;
constexpr uint32_t kSmemBytes = kSmemHeader + kStages * kStageBytes + kEpiWarps * kOutBytes + 1024;

struct MmMaps {
  CUtensorMap a, b, b_half;   // b_half: the boxes of a half tile (an operand with the contraction axis innermost)
  CUtensorMap o;   // the result, boxes of 32 rows of 32 columns, 64-byte swizzle (P.tma_out)
};

// First tile that is worked on in halves: the tiles behind the last complete wave, if as halves they fit one wave.  A wave
// of six tiles cost a [1024, 1008] x [1008, 5008] product (80 tiles on 74 pairs) 4.7 us of 15.5.
__host__ __device__ inline uint32_t SplitFrom(uint32_t tiles, uint32_t units) {
  const uint32_t rest = tiles % units;
  return rest != 0 && rest * 2 <= units ? tiles - rest : tiles;
}

// HALVES: there are such tiles.  (A form of its own: the larger one cost a [16384, 512] x [512, 8192] product, which has none, 2 %.)
template <bool HALVES>
__device__ __forceinline__ void pair_body(const MmParam &P, const MmMaps &maps, const LaunchTag epoch) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // 1024-byte alignment of the stage area (required by the 128-byte swizzle pattern)
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t *smem = smem_raw + (base - raw_addr);
  const uint32_t bar_full = base, bar_empty = base + 64, bar_tfull = base + 128, bar_tempty = base + 160;
  volatile uint32_t *tmem_slot = reinterpret_cast<volatile uint32_t *>(smem + 192);
  const uint32_t stages = base + kSmemHeader;

  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t rank = cluster_ctarank();   // position inside the CTA pair
  const uint32_t unit = blockIdx.x / 2, num_units = gridDim.x / 2;
  const uint32_t mblocks = (P.M + BM * 2 - 1) / (BM * 2), nblocks = (P.N + BN - 1) / BN;
  const uint32_t batch = P.batch0 * P.batch1;
  // Work items: tiles, the tiles of an incomplete last wave (from item split_from on) as halves of 128 columns.
  const uint32_t tiles = mblocks * nblocks * batch, split_from = HALVES ? SplitFrom(tiles, num_units) : tiles;
  const uint32_t num_items = 2 * tiles - split_from;
  auto half_of = [&](uint32_t t) { return HALVES && t >= split_from; };
  auto tile_of = [&](uint32_t t) { return half_of(t) ? split_from + ((t - split_from) >> 1) : t; };
  auto side_of = [&](uint32_t t) { return half_of(t) ? ((t - split_from) & 1u) * (BN / 2) : 0u; };   // its first column in the tile
  const uint32_t kblocks = (P.K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < kStages; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (uint32_t a = 0; a < 2; ++a) {
      mbar_init(bar_tfull + 8 * a, 1);
      mbar_init(bar_tempty + 8 * a, kEpiWarps * 2);   // one arrival per epilogue warp of the pair
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(base + 192, kTmemCols);
    tmem_relinquish_pair();
  }
  tcgen05_before_sync();
  cluster_sync_all();   // the peer's barriers are initialised before anything signals them
  tcgen05_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  chain_wait();
  chain_launch();

  // (The two issuing loops run under elect.sync: inside a plain `lane == 0` branch every MMA took about 100 cycles to
  // issue and every TMA load 150-280 - operands moved to uniform registers one by one - and a k-block 560-630 cycles
  // whatever the tile, against 512 of tensor work.)
  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (elect_one()) {
      const bool a_m = P.a_mmajor != 0, b_k = P.b_kmajor != 0;
      uint32_t stage = 0, parity = 1;
      for (uint32_t t = unit; t < num_items; t += num_units) {
        uint32_t bz, mb, nb;
        tile_coords(tile_of(t), mblocks, nblocks, P.group_m, bz, mb, nb);
        const bool half = half_of(t);
        const uint32_t b0 = bz / P.batch1, b1 = bz - b0 * P.batch1;
        const int za = (int)(b0 * P.a_mul0 + b1 * P.a_mul1), zb = (int)(b0 * P.b_mul0 + b1 * P.b_mul1);
        const int row0 = (int)((mb * 2 + rank) * BM);
        const int col0 = (int)(nb * BN + side_of(t) + rank * (half ? BN / 4 : BN / 2));
        int k = 0;
        for (uint32_t kb = 0; kb < kblocks; ++kb, k += (int)BK) {
          mbar_wait(bar_empty + 8 * stage, parity, 1, &g_mm_status, epoch);
          const uint32_t sa = stages + stage * kStageBytes, sb = sa + kABytes;
          // the pair's first CTA counts the bytes of both CTAs on its barrier
          if (rank == 0) mbar_expect_tx(bar_full + 8 * stage, 2 * (kABytes + (half ? kBBytes / 2 : kBBytes)));
          const uint32_t full = map_to_cta(bar_full + 8 * stage, 0);
          if (!a_m) {
            tma_load_3d_pair(sa, &maps.a, full, k, row0, za);
          } else {
#pragma unroll
            for (uint32_t j = 0; j < BM / 64; ++j) tma_load_3d_pair(sa + j * (64 * BK * 2), &maps.a, full, row0 + (int)(j * 64), k, za);
          }
          if (b_k) {
            tma_load_3d_pair(sb, half ? &maps.b_half : &maps.b, full, k, col0, zb);
          } else {
#pragma unroll
            for (uint32_t j = 0; j < BN / 2 / 64; ++j)
              if (j == 0 || !half) tma_load_3d_pair(sb + j * (64 * BK * 2), &maps.b, full, col0 + (int)(j * 64), k, zb);
          }
          if (++stage == kStages) {
            stage = 0;
            parity ^= 1u;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (the pair's first CTA only) ------------------------------
    if (rank == 0 && elect_one()) {
      // instruction descriptor: D fp32 (bit 4), A/B format (bits 7, 10: 1 = bf16), A / B stored with the
      // contraction axis outermost (bits 15 / 16), N >> 3 at bit 17, M >> 4 at bit 24
      const uint32_t fmt = P.in_dtype == T_BF16 ? 1u : 0u;
      const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((P.a_mmajor ? 1u : 0u) << 15) |
                             ((P.b_kmajor ? 0u : 1u) << 16) | ((BN >> 3) << 17) | (((BM * 2) >> 4) << 24);
      const uint32_t idesc_half = idesc - ((BN / 2 >> 3) << 17);
      // (descriptors of stage 0; a stage or a K = 16 step further is an addition to their address fields)
      const uint64_t da0 = P.a_mmajor ? make_smem_desc(stages, 64 * BK * 2, 1024) : make_smem_desc(stages, 0, 1024);
      const uint64_t db0 = P.b_kmajor ? make_smem_desc(stages + kABytes, 0, 1024) : make_smem_desc(stages + kABytes, 64 * BK * 2, 1024);
      const uint64_t step_a = P.a_mmajor ? 2048 >> 4 : 32 >> 4, step_b = P.b_kmajor ? 32 >> 4 : 2048 >> 4;
      uint32_t stage = 0, parity = 0, acc = 0, acc_parity = 1;
      for (uint32_t t = unit; t < num_items; t += num_units) {
        mbar_wait(bar_tempty + 8 * acc, acc_parity, 2, &g_mm_status, epoch);
        tcgen05_after_sync();
        const uint32_t d_tmem = tmem_base + acc * BN, desc = half_of(t) ? idesc_half : idesc;
        for (uint32_t kb = 0; kb < kblocks; ++kb) {
          mbar_wait(bar_full + 8 * stage, parity, 3, &g_mm_status, epoch);
          const uint64_t da = da0 + stage * (kStageBytes >> 4), db = db0 + stage * (kStageBytes >> 4);
#pragma unroll
          for (uint32_t kk = 0; kk < BK / 16; ++kk)
            umma_f16_pair(d_tmem, da + kk * step_a, db + kk * step_b, desc, (kb | kk) != 0 ? 1u : 0u);
          umma_commit_pair(bar_empty + 8 * stage, 3);   // the stage is free (in both CTAs) once these MMAs have read it
          if (++stage == kStages) {
            stage = 0;
            parity ^= 1u;
          }
        }
        umma_commit_pair(bar_tfull + 8 * acc, 3);   // accumulator complete
        if (++acc == 2) {
          acc = 0;
          acc_parity ^= 1u;
        }
      }
    }
  } else {
    // ------------------------------ epilogue warps ------------------------------
    const uint32_t ew = warp - 2;
    const uint32_t quarter = warp & 3u;          // TMEM lane quarter this warp may read
    auto cols_of = [&](uint32_t t) { return half_of(t) ? kEpiCols / 2 : kEpiCols; };   // the columns this warp drains
    auto col0_of = [&](uint32_t t) { return (ew >> 2) * cols_of(t); };                  // ... and their first in the item
    const uint32_t out_saddr = stages + kStages * kStageBytes + ew * kOutBytes;
    const uint32_t bias_saddr = base + kBiasOff + ew * (kEpiCols * 4u);
    uint32_t acc = 0, acc_parity = 0;
    // Coordinates and bias of a tile are on their way while the tile before is drained: one after the other, in front of each
    // tile, they took 2000 cycles of a [4096, 1024] x [1024, 4096] product's 13 000 per tile.
    uint32_t bz, mb, nb;
    uint32_t bias[kEpiCols / 32];
    auto look_up = [&](uint32_t t) {
      tile_coords(tile_of(t), mblocks, nblocks, P.group_m, bz, mb, nb);
      if (P.bias_ptr == 0) return;
      // (columns past the last one are not stored: any bias will do.  No value is selected or converted here, that would wait)
      const uint32_t col = nb * BN + side_of(t) + col0_of(t) + lane;
      if (P.bias_dtype == T_F32) {
#pragma unroll
        for (uint32_t i = 0; i < kEpiCols / 32; ++i) bias[i] = gload(reinterpret_cast<const uint32_t *>(P.bias_ptr) + min(col + i * 32, P.N - 1));
      } else {
#pragma unroll
        for (uint32_t i = 0; i < kEpiCols / 32; ++i) bias[i] = gload(reinterpret_cast<const unsigned short *>(P.bias_ptr) + min(col + i * 32, P.N - 1));
      }
    };
    if (unit < num_items) look_up(unit);
    with_mode(P, [&](auto mode) {
      constexpr uint32_t MODE = decltype(mode)::mode, DT = decltype(mode)::dtype;
      for (uint32_t t = unit; t < num_items; t += num_units) {
        if (P.bias_ptr != 0) {
          __syncwarp();   // (the warp has read the previous tile's)
#pragma unroll
          for (uint32_t i = 0; i < kEpiCols / 32; ++i)
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(bias_saddr + 4u * (i * 32 + lane)), "f"(bias_value(P, bias[i])) : "memory");
          __syncwarp();
        }
        EpiPos pos;
        pos.b0 = bz / P.batch1;
        pos.b1 = bz - pos.b0 * P.batch1;
        const uint32_t first_row = (mb * 2 + rank) * BM + quarter * 32u, first_col = nb * BN + side_of(t) + col0_of(t);
        pos.row = first_row + lane;
        if (t + num_units < num_items) look_up(t + num_units);
        mbar_wait(bar_tfull + 8 * acc, acc_parity, 4, &g_mm_status, epoch);
        tcgen05_after_sync();
        const uint32_t taddr = tmem_base + ((quarter * 32u) << 16) + acc * BN + col0_of(t);
        if (half_of(t))   // (columns as a template argument: as a variable they cost every whole tile 6 %)
          drain<MODE, DT, kEpiCols / 2>(P, maps.o, taddr, false, pos, first_row, first_col, bias_saddr, out_saddr, lane);
        else
          drain<MODE, DT, kEpiCols>(P, maps.o, taddr, false, pos, first_row, first_col, bias_saddr, out_saddr, lane);
        tcgen05_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(map_to_cta(bar_tempty + 8 * acc, 0));
        if (++acc == 2) {
          acc = 0;
          acc_parity ^= 1u;
        }
      }
    });
    if (elect_one()) tma_store_wait_read<0>();   // shared memory stays until the last store has read it
  }
  __syncwarp();
  tcgen05_before_sync();
  cluster_sync_all();   // neither CTA leaves while the other may still read its shared memory or signal it
  if (warp == 1) {
    tcgen05_after_sync();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

}  // namespace

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
  dvm_b200_mm_tcgen05_pair(const __grid_constant__ MmParam P, const __grid_constant__ MmMaps maps, const LaunchTag epoch) {
  pair_body<false>(P, maps, epoch);
}
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
  dvm_b200_mm_tcgen05_pair_halves(const __grid_constant__ MmParam P, const __grid_constant__ MmMaps maps, const LaunchTag epoch) {
  pair_body<true>(P, maps, epoch);
}

namespace {

PFN_cuTensorMapEncodeTiled GetEncode() {
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

}  // namespace

// 3-d map over a [batches, rows, inner] row-major operand: box = [1, box_rows, 64 elements], 128-byte swizzle
// The result as [batch0, batch1, M, N] for the copy engine, if it can address it.
bool EncodeMmResult(CUtensorMap *map, const MmParam &p) {
  const EpiTensor &t = p.tensor[p.out_slot];
  auto encode = GetEncode();
  const int64_t row = t.sm * 2, b1 = p.batch1 > 1 ? t.sb1 * 2 : row * p.M, b0 = p.batch0 > 1 ? t.sb0 * 2 : b1 * p.batch1;
  if (encode == nullptr || ((t.ptr | row | b1 | b0) & 15) != 0 || row <= 0 || b1 <= 0 || b0 <= 0 || b0 >= (1ll << 40)) return false;
  cuuint64_t dims[4] = {p.N, p.M, p.batch1, p.batch0};
  cuuint64_t strides[3] = {static_cast<cuuint64_t>(row), static_cast<cuuint64_t>(b1), static_cast<cuuint64_t>(b0)};
  cuuint32_t box[4] = {32, 32, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, reinterpret_cast<void *>(t.ptr), dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int EncodeMmOperand(CUtensorMap *map, uint64_t ptr, uint64_t inner, uint64_t pitch, uint64_t rows, uint64_t batches, uint32_t box_rows) {
  auto encode = GetEncode();
  if (encode == nullptr) return -10;
  cuuint64_t dims[3] = {inner, rows, batches ? batches : 1};
  cuuint64_t strides[2] = {pitch * 2, pitch * rows * 2};
  cuuint32_t box[3] = {64, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, reinterpret_cast<void *>(ptr), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -100 - static_cast<int>(r);
}

bool MmOperandNeedsGather(uint64_t ptr, uint64_t pitch, uint64_t slice, uint32_t batches) {
  // the copy engine needs 16-byte aligned bases and row pitches (and slices, for batched operands)
  return (ptr & 15u) != 0 || (pitch & 7u) != 0 || (batches > 1 && (slice & 7u) != 0);
}

namespace {

struct MmPlan {
  uint32_t bn, split;   // bn 0: 256 x 256 tiles of CTA pairs; else 128 x bn tiles, K cut into `split` parts
};

// Estimated clock cycles (1850 per us) of a tiling.  The constants are a fit to 42 problem shapes (1 to 16384 rows) timed in
// every tiling; the tiling with the lowest estimate was on average 0.5 % slower than the fastest one of its shape.
//  - A k-block takes max(210 + 2.9 bn, bytes / 154) on a CTA alone on its SM, and max(that, 2 bytes / 79) two of them
//    together: the MMAs of a k-block and what L2 delivers to an SM.
//  - Loads by the work warps (operands at any even address) cost 1700 per k-block, and hardly overlap between two CTAs.
//  - Draining a column of 128 rows takes 30, with the gated form or a program 52; the sum over a cluster moves all of a tile but
//    its own share through distributed shared memory.
//  - A 256 x 256 tile of a pair takes 620 per k-block, or its epilogue, whichever is longer, a half tile 0.6 of that; the last
//    epilogue is exposed.
double TileCost(const MmParam &p, uint32_t bn, uint32_t split, int sms, bool gather) {
  const uint32_t kb = (p.K + BK - 1) / BK;
  const uint64_t batch = static_cast<uint64_t>(p.batch0) * p.batch1, mb = (p.M + BM - 1) / BM;
  const bool light = p.epi_mode == EPI_STORE || p.epi_mode == EPI_WIDEN;
  if (bn == 0) {
    const uint64_t tiles = (mb + 1) / 2 * ((p.N + BN - 1) / BN) * batch, pairs = sms / 2;
    const double whole = std::max(kb * 620.0, light ? 5800.0 : 9000.0), rest = static_cast<double>(tiles % pairs);
    const double waves = static_cast<double>(tiles / pairs) + (rest == 0 ? 0.0 : rest * 2 <= pairs && tiles > pairs ? 0.6 : 1.0);
    return (light ? 10400.0 : 14200.0) + waves * whole;
  }
  const double part = (p.M < BM ? p.M : BM) / static_cast<double>(BM), bytes = (part * BM + bn) * 128.0;
  const uint64_t ctas = mb * ((p.N + bn - 1) / bn) * batch * split;
  const uint32_t share = (kb + split - 1) / split;
  double one = std::max(210.0 + 2.9 * bn, bytes / 154.0), two = std::max(one, 2.0 * bytes / 79.0);
  if (gather) {
    one = 1700.0;
    two = 1.8 * one;
  }
  const double column = light ? 30.0 : 52.0;
  double finish = column * bn * part / split;
  if (split > 1) finish += 2940.0 + 36.0 * bn * part * (split - 1) / split + 144.0 * split;
  const uint64_t full = ctas / (2 * sms), rest = ctas % (2 * sms);   // two CTAs per SM
  double t = 4550.0 + static_cast<double>(full) * (share * two + 1.8 * finish);
  if (rest > static_cast<uint64_t>(sms)) {
    t += share * two + 1.8 * finish;
  } else if (rest > 0) {
    t += share * one + finish;
  }
  return t;
}

MmPlan ChoosePlan(const MmParam &p, int sms, bool gather, double *cost = nullptr) {
  const uint32_t kb = (p.K + BK - 1) / BK;
  MmPlan best{64, 1};
  double best_t = TileCost(p, 64, 1, sms, gather);
  if (cost != nullptr) *cost = best_t;
  auto consider = [&](uint32_t bn, uint32_t split) {
    const double t = TileCost(p, bn, split, sms, gather);
    if (t < best_t) {
      best_t = t;
      best = {bn, split};
      if (cost != nullptr) *cost = t;
    }
  };
  for (uint32_t split = 2; split <= 8 && split <= kb; split *= 2) consider(64, split);
  if (gather) return best;   // (64 columns measured faster than 128 at every size: the loads bound it, not the tile)
  for (uint32_t split = 1; split <= 8 && (split == 1 || split <= kb); split *= 2) consider(128, split);
  if (p.M > BM && kb != 0) consider(0, 1);
  return best;
}

}  // namespace

// A copy of an operand in rows of whole 16-byte units pays where the tiles read it often: it costs a launch (of which about
// 700 cycles show beside the product) and a cycle for 2700 bytes read or written; the estimates above say what it saves.
void MmPackBytes(const MmParam &p, uint64_t *a_bytes, uint64_t *b_bytes) {
  *a_bytes = *b_bytes = 0;
  if (p.M == 0 || p.N == 0 || p.K == 0 || p.batch0 * p.batch1 == 0) return;
  MmParam q = p;   // (addresses are not known yet: what the shapes alone make unaligned)
  q.a_ptr = q.b_ptr = 0;
  auto bytes = [](uint64_t inner, uint64_t rows, uint64_t batches) {
    const uint64_t pieces = (inner + 7) / 8 * rows * batches;
    return pieces < (1ull << 31) ? pieces * 16 : ~0ull;
  };
  const uint64_t a = MmGatherA(q) ? bytes(MmInnerA(p), MmRowsA(p), p.a_batches) : 0;
  const uint64_t b = MmGatherB(q) ? bytes(MmInnerB(p), MmRowsB(p), p.b_batches) : 0;
  if ((a | b) == 0 || a == ~0ull || b == ~0ull) return;
  int sms = Runtime::Get().sm_count_or_default();
  if (p.leave_sms != 0 && static_cast<int>(p.leave_sms) + 32 <= sms) sms -= static_cast<int>(p.leave_sms);
  double gathered = 0.0, packed = 0.0;
  ChoosePlan(p, sms, true, &gathered);
  ChoosePlan(p, sms, false, &packed);
  if (packed + 700.0 + 2.0 * static_cast<double>(a + b) / 2700.0 >= gathered) return;
  *a_bytes = a;
  *b_bytes = b;
}

int LaunchMatMul(const MmParam &p_in, void *stream) {
  MmParam p = p_in;
  static const int group_env = getenv("DVM_B200_MM_GROUP_M") ? atoi(getenv("DVM_B200_MM_GROUP_M")) : 0;
  p.group_m = group_env > 0 ? static_cast<uint32_t>(group_env) : 8u;
  // "copy acc, product; store tensor s; end" with a dense row layout: the kernel stores the product directly
  p.epi_mode = EPI_PROGRAM;
  p.out_slot = 0;
  {
    const uint64_t w0 = p.epilogue[0], w1 = p.epilogue[1], w2 = p.epilogue[2];
    if (DVMB_OPC(w0) == OP_COPY && DVMB_OKIND(w0) == K_TENSOR && DVMB_OIDX(w0) == p.mma_slot && DVMB_OPC(w1) == OP_ST &&
        DVMB_OPC(w2) == OP_END && DVMB_SUB(w1) < p.n_tensors) {
      const EpiTensor &t = p.tensor[DVMB_SUB(w1)];
      if (t.sn == 1 && (t.dtype == p.in_dtype || t.dtype == T_F32)) {
        p.epi_mode = t.dtype == p.in_dtype ? EPI_STORE : EPI_WIDEN;
        p.out_slot = DVMB_SUB(w1);
      }
    }
  }
  // the gated form x / (c2 + exp(c1 * (x + c0 * x^3))) of the product, rounded to the operand type and stored
  {
    static const bool off = getenv("DVM_B200_NO_FUSE") != nullptr;
    const uint64_t *w = p.epilogue;
    auto is = [&](int i, uint32_t opc, uint32_t sub, uint32_t okind) {
      return DVMB_OPC(w[i]) == opc && DVMB_SUB(w[i]) == sub && DVMB_OKIND(w[i]) == okind && DVMB_RND(w[i]) == RN_NONE &&
             (okind != K_TENSOR || DVMB_OIDX(w[i]) == p.mma_slot);
    };
    const uint32_t rnd_out = p.in_dtype == T_BF16 ? RN_BF16 : RN_F16;
    if (!off && DVMB_OPC(w[0]) == OP_COPY && DVMB_OKIND(w[0]) == K_TENSOR && DVMB_OIDX(w[0]) == p.mma_slot &&
        is(1, OP_BIN, B_MUL, K_ACC) && is(2, OP_BIN, B_MUL, K_TENSOR) && is(3, OP_BIN, B_MUL, K_IMM) && is(4, OP_BIN, B_ADD, K_TENSOR) &&
        is(5, OP_BIN, B_MUL, K_IMM) && DVMB_OPC(w[6]) == OP_UN && DVMB_SUB(w[6]) == U_EXP_FAST && DVMB_RND(w[6]) == RN_NONE &&
        is(7, OP_BIN, B_ADD, K_IMM) && is(8, OP_BIN, B_RDIV_FAST, K_TENSOR) && DVMB_OPC(w[9]) == OP_CVT && DVMB_SUB(w[9]) == V_RND &&
        DVMB_RND(w[9]) == rnd_out && DVMB_OPC(w[10]) == OP_ST && DVMB_OPC(w[11]) == OP_END && DVMB_SUB(w[10]) < p.n_tensors) {
      const EpiTensor &t = p.tensor[DVMB_SUB(w[10])];
      if (t.sn == 1 && t.dtype == p.in_dtype) {
        p.epi_mode = EPI_GATE;
        p.out_slot = DVMB_SUB(w[10]);
        p.gate_c[0] = DVMB_IMM(w[3]);
        p.gate_c[1] = DVMB_IMM(w[5]);
        p.gate_c[2] = DVMB_IMM(w[7]);
      }
    }
  }
  if (p.M == 0 || p.N == 0 || p.batch0 * p.batch1 == 0) return 0;
  if (p.in_dtype != T_BF16 && p.in_dtype != T_F16) return -3;
  int dev = 0;
  cudaGetDevice(&dev);
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (p.leave_sms != 0 && static_cast<int>(p.leave_sms) + 32 <= sms) sms -= static_cast<int>(p.leave_sms);
  if (MmNeedsGather(p) && (p.a_pack | p.b_pack) != 0) {
    const int rc = LaunchMmPack(&p, stream);
    if (rc != 0) return rc;
  }
  const bool gather = MmNeedsGather(p);
  MmPlan plan = ChoosePlan(p, sms, gather);
  static const char *const force = getenv("DVM_B200_MM_PLAN");   // "columns,split" (columns 0: CTA pairs)
  if (force != nullptr) {
    const uint32_t bn = static_cast<uint32_t>(atoi(force)), split = strchr(force, ',') ? static_cast<uint32_t>(atoi(strchr(force, ',') + 1)) : 1u;
    const bool pair_ok = bn == 0 && !gather && p.K != 0;
    if (pair_ok || ((bn == 64 || bn == 128) && (split == 1 || ((split == 2 || split == 4 || split == 8) && split * BK <= p.K)))) plan = {bn, split};
  }
  if (plan.bn != 0) return LaunchMmTile(p, plan.bn, plan.split, stream);
  static bool attr_set[64] = {false};
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    for (auto fn : {dvm_b200_mm_tcgen05_pair, dvm_b200_mm_tcgen05_pair_halves}) {
      cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
      if (e != cudaSuccess) return static_cast<int>(e);
    }
    attr_set[dev] = true;
  }
  MmMaps maps;
  memset(&maps.o, 0, sizeof(maps.o));
  // fp16 and bf16 are both 2-byte types for the copy engine; the MMA descriptor carries the real format
  int rc = EncodeMmOperand(&maps.a, p.a_ptr, MmInnerA(p), MmPitchA(p), MmRowsA(p), p.a_batches, p.a_mmajor ? 64 : BM);
  if (rc != 0) return rc;
  rc = EncodeMmOperand(&maps.b, p.b_ptr, MmInnerB(p), MmPitchB(p), MmRowsB(p), p.b_batches, p.b_kmajor ? BN / 2 : 64);
  if (rc != 0) return rc;
  maps.b_half = maps.b;
  if (p.b_kmajor) rc = EncodeMmOperand(&maps.b_half, p.b_ptr, MmInnerB(p), MmPitchB(p), MmRowsB(p), p.b_batches, BN / 4);
  if (rc != 0) return rc;
  p.tma_out = p.epi_mode >= EPI_STORE && EncodeMmResult(&maps.o, p) ? 1u : 0u;
  const uint32_t tiles = ((p.M + 2 * BM - 1) / (2 * BM)) * ((p.N + BN - 1) / BN) * p.batch0 * p.batch1;
  const uint32_t pairs = static_cast<uint32_t>(sms / 2);
  const uint32_t units = 2 * tiles <= pairs ? 2 * tiles : (tiles < pairs ? tiles : pairs);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3(units * 2, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = static_cast<cudaStream_t>(stream);
  ChainAttribute(&cfg, attr);
  const auto kernel = SplitFrom(tiles, units) < tiles ? dvm_b200_mm_tcgen05_pair_halves : dvm_b200_mm_tcgen05_pair;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p, maps, NextLaunchEpoch());
  return e != cudaSuccess ? static_cast<int>(e) : static_cast<int>(cudaGetLastError());
}

unsigned int ReadMatMulStatus() {
  WaitStatus v = {0u, 0u};
  const unsigned int zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_mm_status, sizeof(v)) != cudaSuccess) return 0xffffffffu;
  if (v.first_error != 0) cudaMemcpyToSymbol(g_mm_status, &zero, sizeof(zero), offsetof(WaitStatus, first_error));
  const unsigned int tile = ReadMmTileStatus();
  return v.first_error != 0 ? v.first_error : tile;
}

}  // namespace dvmb
