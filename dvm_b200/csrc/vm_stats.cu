// Statistics kernel: mean and variance of a group, then an affine map of it (row_match.cc), as a straight-line kernel:
// dvm_b200_stats_affine.
//
// A group - for a batch norm all planes of a channel - lies in the shared memory of the 1 to 8 CTAs of a cluster from its one read
// to its one write.  A thread copies the 16-byte units it works on itself (cp.async, which only it waits for), so that the tile needs
// no barrier; the sums of the warps cross the cluster once.  A run is the units that hold at least one of its elements: x and y lie
// alike relative to 16 bytes, lanes outside a run are masked, so a plane may start anywhere.  Units that are an end of a run go
// through a loop of their own behind the whole ones, which then need neither masks nor branches.
//
// What bounds it: [64, 256, 56, 56] fp16, 206 MB, 45 us (65 in the interpreter, which reads x twice; 31.8 at copy bandwidth).  74 groups are
// on the chip at a time, so the 256 take 3.5 turns of load, sums, store; HBM idles about 2.5 us in each while the CTAs of an SM, more or
// less in step, sum and meet.  Fewer instructions (107 a unit instead of 131) did not change it, nor did CTAs that stay and load the next
// group into the units they have just stored (43-45 us).  [32, 200, 27, 27]: 7.1 us (129 in the interpreter, element by element): one turn,
// a chain of launch, load, sums, store.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "chain.cuh"
#include "runtime.h"
#include "units.cuh"
#include "vm_stats.h"

namespace dvmb {

namespace {

constexpr uint32_t kMaxThreads = 1024, kMaxCluster = 8, kMaxPerThread = 16;

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void copy_unit(uint32_t to, const uint8_t *from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from) : "memory");
}

// kWhole: every run starts and ends on 16 bytes, so that every unit belongs to its run with all lanes.  J: units per thread at most;
// a thread keeps their offsets in registers.
template <uint32_t DT, bool kWhole, int J>
__device__ __forceinline__ void stats_affine_body(const StatsParam &P) {
  extern __shared__ __align__(128) uint8_t smem[];
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, T = blockDim.x, warps = T >> 5;
  const uint32_t CL = P.cluster, rank = CL > 1 ? cluster_rank() : 0u, senders = CL * warps;
  if (CL > 1) cluster_arrive();   // (every CTA of the cluster runs before a peer writes to it: waited for in front of the sums)
  const uint32_t sums = (uint32_t)__cvta_generic_to_shared(smem);   // float2 [senders], then the tile
  const uint32_t tile_at = ((8u * senders + 127u) & ~127u) + 16u * tid;   // the thread's first unit
  const uint32_t upr = P.units_per_run, total = P.runs * upr, u_first = rank * P.per_cta + tid, u_end = min(total, (rank + 1u) * P.per_cta);
  const uint32_t run_bytes = P.run_len << 1, run_step = P.run_stride << 1;
  uint32_t k[kMaxKept];
  group_coords(P.kept_size, blockIdx.x / CL, k);
  const uint64_t g_off = (uint64_t)group_offset(P.kstride, k) << 1;
  const uint32_t mis0 = kWhole ? 0u : (uint32_t)(P.x + g_off) & 15u;   // of x and of y
  const uint8_t *const x0 = reinterpret_cast<const uint8_t *>(P.x + g_off) - mis0;
  uint8_t *const y0 = reinterpret_cast<uint8_t *>(P.y + g_off) - mis0;

  // The thread's units u_first, + T, ...: their offsets, and which of them are (bit j) whole or an end of a run
  uint32_t off[J], inner = 0, ends = 0;
  {
    const uint32_t r = u_first / upr;
    uint32_t c = u_first - r * upr, run = r * run_step;
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const bool live = u_first + j * T < u_end;
      if (kWhole) {
        off[j] = run + 16u * c;
        inner |= live ? 1u << j : 0u;
      } else {
        const uint32_t at = mis0 + run, mis = at & 15u;
        off[j] = at - mis + 16u * c;
        const int32_t left = (int32_t)(mis + run_bytes) - (int32_t)(16u * c);   // bytes from the unit's start to the run's end
        const bool end = (c == 0 && mis != 0) || left < 16;
        inner |= live && !end ? 1u << j : 0u;
        ends |= live && end && left > 0 ? 1u << j : 0u;
      }
      run += P.step_runs * run_step;
      c += P.step_units;
      if (c >= upr) {
        c -= upr;
        run += run_step;
      }
    }
  }
  chain_wait();
  chain_launch();

#pragma unroll
  for (int j = 0; j < J; ++j)
    if ((inner | ends) >> j & 1u) copy_unit(sums + tile_at + 16u * j * T, x0 + off[j]);
  auto scalar_in = [&](const StatsScalar &s) { return u2f(load_elem(s.dtype, reinterpret_cast<const uint8_t *>(s.ptr), group_offset(s.kstride, k))); };
  const float shift = scalar_in(P.shift), gamma = P.have_gamma ? scalar_in(P.gamma) : 1.0f, beta = P.have_beta ? scalar_in(P.beta) : -0.0f;
  // fn(which unit of the thread, offset, first lane, lane behind the last) for the units that are an end of a run
  auto each_end = [&](auto &&fn) {
    for (uint32_t left_units = ends; left_units != 0; left_units &= left_units - 1u) {
      const uint32_t j = __ffs(left_units) - 1u, u = u_first + j * T, r = u / upr, c = u - r * upr, at = mis0 + r * run_step, mis = at & 15u;
      fn(j, at - mis + 16u * c, c == 0 ? mis >> 1 : 0u, min(kE, (mis + run_bytes - 16u * c) >> 1));
    }
  };
  asm volatile("cp.async.wait_all;" ::: "memory");

  // sums of d and d d, eight of each per thread
  F2 s1[kE / 2], s2[kE / 2];
#pragma unroll
  for (uint32_t i = 0; i < kE / 2; ++i) s1[i] = s2[i] = f2(0.0f, 0.0f);
  const F2 minus_shift = f2(-shift, -shift);
  const uint8_t *const tile = smem + tile_at;
  auto unit = [&](uint32_t j) { return *reinterpret_cast<const uint4 *>(tile + 16u * j * T); };
  auto deviations = [&](const uint4 &v, F2 (&d)[kE / 2]) {
    unpack_pairs<DT>(v, d);
#pragma unroll
    for (uint32_t i = 0; i < kE / 2; ++i) d[i] = add2(d[i], minus_shift);
  };
  auto accumulate = [&](const F2 (&d)[kE / 2]) {
#pragma unroll
    for (uint32_t i = 0; i < kE / 2; ++i) {
      s1[i] = add2(s1[i], d[i]);
      s2[i] = fma2(d[i], d[i], s2[i]);
    }
  };
  // fn(unit j, its elements) for the thread's whole units, four reads at a time where every lane has all four
  auto each_inner = [&](auto &&fn) {
#pragma unroll
    for (int b = 0; b < J; b += 4) {
      if (kWhole && __all_sync(0xffffffffu, (inner >> b & 15u) == 15u)) {
        uint4 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = unit(b + j);
#pragma unroll
        for (int j = 0; j < 4; ++j) fn(b + j, v[j]);
      } else {
#pragma unroll
        for (int j = b; j < b + 4; ++j)
          if (inner >> j & 1u) fn(j, unit(j));
      }
    }
  };
  each_inner([&](int, const uint4 &v) {
    F2 d[kE / 2];
    deviations(v, d);
    accumulate(d);
  });
  if (!kWhole)
    each_end([&](uint32_t j, uint32_t, uint32_t lo, uint32_t hi) {
      F2 d[kE / 2];
      deviations(unit(j), d);
      mask_pairs(d, lo, hi);
      accumulate(d);
    });
#pragma unroll
  for (uint32_t h = kE / 4; h > 0; h >>= 1)
#pragma unroll
    for (uint32_t i = 0; i < h; ++i) {
      s1[i] = add2(s1[i], s1[i + h]);
      s2[i] = add2(s2[i], s2[i + h]);
    }
  const float2 h1 = halves(s1[0]), h2 = halves(s2[0]);
  float2 t = make_float2(warp_sum(h1.x + h1.y), warp_sum(h2.x + h2.y));
  // every warp sends its sums to every CTA of the cluster, then each warp adds all of them in the same order
  const uint32_t mine = sums + 8u * (rank * warps + warp);
  if (CL > 1) {
    cluster_wait();
    if (lane < CL) {
      uint32_t to;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(mine), "r"(lane));
      asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(to), "f"(t.x), "f"(t.y) : "memory");
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();
  } else {
    if (lane == 0) asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(mine), "f"(t.x), "f"(t.y) : "memory");
    __syncthreads();
  }
  t = make_float2(0.0f, 0.0f);
  for (uint32_t i = lane; i < senders; i += 32u) {
    float2 q;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(q.x), "=f"(q.y) : "r"(sums + 8u * i) : "memory");
    t.x += q.x;
    t.y += q.y;
  }
  t = make_float2(warp_sum(t.x), warp_sum(t.y));
  const float tn = __fmul_rn(t.x, P.rec), mean = __fadd_rn(tn, shift), var = __fmul_rn(__fsub_rn(t.y, __fmul_rn(t.x, tn)), P.rec2);
  const float std = sqrtf(__fadd_rn(var, P.eps)), rstd = fast_div(1.0f, std);
  if (rank == 0 && tid < P.stores) {
    const StatsScalar &s = P.store[tid];
    const float v = s.value == SV_MEAN ? mean : (s.value == SV_VAR ? var : std);
    store_elem(s.dtype, reinterpret_cast<uint8_t *>(s.ptr), group_offset(s.kstride, k), f2u(v));
  }
  const F2 m0 = f2(-mean, -mean), m1 = f2(rstd, rstd), m2 = f2(gamma, gamma), m3 = f2(beta, beta);
  auto mapped = [&](const uint4 &v) {
    F2 d[kE / 2];
    unpack_pairs<DT>(v, d);
#pragma unroll
    for (uint32_t i = 0; i < kE / 2; ++i) d[i] = fma2(mul2(add2(d[i], m0), m1), m2, m3);
    return pack_pairs<DT>(d);
  };
  each_inner([&](int j, const uint4 &v) { *reinterpret_cast<uint4 *>(y0 + off[j]) = mapped(v); });
  if (!kWhole) each_end([&](uint32_t j, uint32_t o, uint32_t lo, uint32_t hi) { store_lanes(y0 + o, mapped(unit(j)), lo, hi); });
}

}  // namespace

#define DVMB_STATS(NAME, DT, WHOLE, J) \
  __global__ void __launch_bounds__(kMaxThreads, 1) NAME(const __grid_constant__ StatsParam P) { stats_affine_body<DT, WHOLE, J>(P); }
DVMB_STATS(dvm_b200_stats_affine_f16_4, T_F16, false, 4)
DVMB_STATS(dvm_b200_stats_affine_f16_8, T_F16, false, 8)
DVMB_STATS(dvm_b200_stats_affine_f16_16, T_F16, false, 16)
DVMB_STATS(dvm_b200_stats_affine_f16_whole_4, T_F16, true, 4)
DVMB_STATS(dvm_b200_stats_affine_f16_whole_8, T_F16, true, 8)
DVMB_STATS(dvm_b200_stats_affine_f16_whole_16, T_F16, true, 16)
DVMB_STATS(dvm_b200_stats_affine_bf16_4, T_BF16, false, 4)
DVMB_STATS(dvm_b200_stats_affine_bf16_8, T_BF16, false, 8)
DVMB_STATS(dvm_b200_stats_affine_bf16_16, T_BF16, false, 16)
DVMB_STATS(dvm_b200_stats_affine_bf16_whole_4, T_BF16, true, 4)
DVMB_STATS(dvm_b200_stats_affine_bf16_whole_8, T_BF16, true, 8)
DVMB_STATS(dvm_b200_stats_affine_bf16_whole_16, T_BF16, true, 16)
#undef DVMB_STATS

namespace {

// Every run of every group starts and ends on 16 bytes.
bool RunsWhole(const StatsParam &p) {
  uint64_t m = p.x | (static_cast<uint64_t>(p.run_len) << 1);
  if (p.runs > 1) m |= static_cast<uint64_t>(p.run_stride) << 1;
  for (int j = 0; j < kMaxKept; ++j)
    if (p.kept_size[j] != 1) m |= static_cast<uint64_t>(p.kstride[j]) << 1;
  return (m & 15u) == 0;
}
// 16-byte units a run touches at most: one more where runs may start inside a unit
uint32_t UnitsPerRun(const StatsParam &p) {
  const uint64_t bytes = static_cast<uint64_t>(p.run_len) << 1;
  return static_cast<uint32_t>(RunsWhole(p) ? bytes / 16 : (bytes + 15 + 14) / 16);
}

// A CTA's tile where four CTAs of 256 threads of 64 registers share an SM: a quarter of its shared memory, less the KB that every CTA takes
// and the header below
constexpr uint32_t kTileUnits = (228u * 1024u / 4u - 1024u - 8u * kMaxCluster * (256u / 32u)) / 16u;
constexpr uint32_t kTilePerThread = (kTileUnits + 255u) / 256u;
constexpr uint32_t kMaxTileUnits = 200u * 1024u / 16u;   // of a CTA: with the header below what an SM has

}  // namespace

bool StatsPays(const StatsParam &p) {
  if (!p.on || p.x == 0 || p.y == 0) return false;
  if (((p.x ^ p.y) & 15u) != 0 || ((p.x | p.y) & 1u) != 0) return false;
  if (static_cast<uint64_t>(p.runs) * p.run_stride + p.run_len >= (1ull << 30)) return false;   // (32-bit offsets inside a group)
  const uint64_t units = static_cast<uint64_t>(UnitsPerRun(p)) * p.runs;
  if (units > static_cast<uint64_t>(kMaxTileUnits) * kMaxCluster) return false;
  if (static_cast<uint64_t>(p.groups) * kMaxCluster >= (1ull << 31)) return false;   // (CTAs of a grid)
  // Many groups of at most 64 elements: a CTA each takes 1.05 ns, the interpreter, whose warps share them out, 0.15 (16 elements) to 0.6
  // (64) and 13 us for the launch; groups of 256 are faster here in any number.  In us, here | there: [100000, 16] 106 | 27,
  // [4096, 16] 6.2 | 13.3, [65536, 64] 70 | 54, [20000, 64] 23 | 26, [50000, 256] 54 | 145.
  double padded = 16.0;
  while (padded < static_cast<double>(p.run_len) * p.runs) padded *= 2.0;
  return 2.0 + 1.05e-3 * p.groups <= 13.0 + 9.5e-6 * p.groups * padded;
}

int LaunchStats(const StatsParam &p_in, void *stream) {
  StatsParam p = p_in;
  const uint32_t sms = static_cast<uint32_t>(Runtime::Get().sm_count_or_default());
  const bool whole = RunsWhole(p);
  p.units_per_run = UnitsPerRun(p);
  const uint32_t units = p.units_per_run * p.runs;
  // How a group is cut, from launches with 1 to 8 CTAs per group and 1 to 16 units per thread:
  //  - tiles of which four fit an SM (55 KB): while some wait for their sums others move data ([64, 256, 56, 56] in tiles of 49, 98, 196 KB: 45,
  //    49, 55 us; with a limit of 49 instead of 55 KB [9, 800, 56, 56] 18.9 instead of 14.9, [18, 800, 56, 56] 42.5 and 37.9, [38, 440, 27, 27] 13.0
  //    and 12.1, but [38, 300, 27, 27] 11.1 and 12.0); smaller ones where the groups alone leave SMs idle ([16, 48, 55, 55] on 1, 2, 4, 8 CTAs:
  //    8.6, 5.7, 5.3, 5.2);
  //  - 8 units per thread: more threads each pay the setup, fewer leave too few warps ([32, 200, 27, 27] with 4, 8, 16: 8.9, 7.0, 8.1;
  //    [64, 1024, 14, 14] with 6, 8, 14: 15.4, 12.9, 14.1); 4 while every CTA has an SM of its own ([16, 128, 28, 28] with 4, 8: 3.4, 3.6);
  //    14 where large tiles queue for SMs, for four of them to fit the registers ([64, 256, 56, 56] with 8 and 14: 51, 45);
  //  - 320 threads where three of them are what an SM gets at most: three fill the registers ([6, 440, 56, 56] 6.6 us, with 14 units per thread 9.3,
  //    [8, 300, 56, 56] 8.3 and 9.3, [24, 300, 27, 27] 7.9 and 8.3; with 12 units, where that makes 352 threads and two CTAs, up to a third slower).
  uint32_t cluster = 1;
  while (cluster < kMaxCluster && (units > cluster * kTileUnits || (units > cluster * 2048u && static_cast<uint64_t>(p.groups) * cluster < sms))) cluster *= 2;
  p.cluster = cluster;
  p.per_cta = (units + cluster - 1) / cluster;
  const uint64_t ctas = static_cast<uint64_t>(p.groups) * cluster;
  const uint32_t most = ctas <= sms ? 4u : (p.per_cta <= 2048u || ctas <= 2u * sms ? 8u : kTilePerThread);   // units per thread
  uint32_t threads = (p.per_cta + most - 1) / most;
  if (p.per_cta > 2048u && p.per_cta <= kTileUnits && ctas > 2u * sms && ctas <= 3u * sms) threads = 320u;
  threads = std::min(kMaxThreads, std::max(64u, (threads + 31u) & ~31u));
  const uint32_t per_thread = (p.per_cta + threads - 1) / threads;
  if (per_thread > kMaxPerThread) return -1;
  p.step_runs = threads / p.units_per_run;
  p.step_units = threads % p.units_per_run;
  using Fn = void (*)(const StatsParam);
  static const Fn fns[12] = {dvm_b200_stats_affine_f16_4,  dvm_b200_stats_affine_f16_8,  dvm_b200_stats_affine_f16_16,
                             dvm_b200_stats_affine_f16_whole_4,  dvm_b200_stats_affine_f16_whole_8,  dvm_b200_stats_affine_f16_whole_16,
                             dvm_b200_stats_affine_bf16_4, dvm_b200_stats_affine_bf16_8, dvm_b200_stats_affine_bf16_16,
                             dvm_b200_stats_affine_bf16_whole_4, dvm_b200_stats_affine_bf16_whole_8, dvm_b200_stats_affine_bf16_whole_16};
  static bool attr_set[64] = {false};   // the attribute is per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    for (const Fn fn : fns) {
      const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kMaxTileUnits * 16u + 4096u));
      if (e != cudaSuccess) return static_cast<int>(e);
    }
    attr_set[dev] = true;
  }
  const uint32_t header = (8u * cluster * (threads / 32) + 127u) & ~127u;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cfg.gridDim = dim3(p.groups * cluster, 1, 1);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = header + 16u * p.per_cta;
  cfg.stream = static_cast<cudaStream_t>(stream);
  if (cluster > 1) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.numAttrs = 1;
  }
  ChainAttribute(&cfg, attr);
  const Fn fn = fns[(p.dtype == T_F16 ? 0 : 6) + (whole ? 3 : 0) + (per_thread <= 4u ? 0 : (per_thread <= 8u ? 1 : 2))];
  const cudaError_t e = cudaLaunchKernelEx(&cfg, fn, p);
  return e != cudaSuccess ? static_cast<int>(e) : static_cast<int>(cudaGetLastError());
}

}  // namespace dvmb
