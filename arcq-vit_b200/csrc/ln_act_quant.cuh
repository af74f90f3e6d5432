// Residual add + LayerNorm + activation quantizer in one kernel over fp16 rows: the glue in front of the first
// packed linear of a sub-block (norm1 -> qkv, norm2 -> fc1) merged with that linear's input quantizer.
//   s    = fp16(x + y)                                    (written out when y is given: the residual stream)
//   h    = fp16((s - mean(s)) * rsqrt(var(s) + eps) * gamma + beta)     (never written, unless asked for)
//   xhat = fp16(reconstruction of the ARCQ quantization of h in groups of 64)
// The separate kernels write h and read it back; here it goes through shared memory.
//
// Bound by HBM for large inputs: [201728, 768] 211 us, 1.24 GB at 5.9 TB/s of the 6.5 a copy reaches ([50432, 768] 57.5 us, [12608, 384]
// 10.5 us).  253, 67.3 and 11.2 us with rows read by ordinary loads, whose latency every pass of phase 1 waited for, and with scalar
// arithmetic (36 instructions a value instead of 26).
//
// Two phases per tile, each in the thread layout that suits it, and each with the arithmetic of the kernel it
// replaces, so that the results are bit-identical to arcq_add_layernorm followed by arcq_act_quant:
//   1. LayerNorm with the lane layout of add_layernorm_rows_kernel (LANES lanes per row, 16-byte accesses, the same
//      device function), writing h into padded group rows of shared memory;
//   2. the quantizer of group_quant.cuh: one thread per 64-group works on its row in place, and each warp sends its 32 rows
//      out by TMA.
// A tile is 128 consecutive groups (the quantizer's unit), whatever the row length: the LayerNorm phase computes
// every row the tile touches (a row shared with the neighbouring tile is normalised by both; 1 row in 22 at
// K = 384) and keeps the groups that are the tile's.  Rows are owned (s and h written) by the tile that holds
// their first group.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>
#include "ptx.cuh"
#include "act_quant.cuh"
#include "group_quant.cuh"
#include "codes.cuh"
#include "add_layernorm.cuh"

namespace arcq {

constexpr int kLnqThreads = 128;
constexpr int kStatusLnqTimeout = 0x411;

// Rows that a tile of 128 groups can touch, and the block's shared memory: h and then the reconstruction, one group per row with the
// 128-byte swizzle; the tables; the tile's rows of x and y.  57.5 KB at most with what the system takes of each block: four an SM.
__host__ __device__ constexpr int lnq_max_rows(int lanes) { return kLnqThreads / (lanes * 24 / 64) + 2; }
struct LnqSmem {
  uint32_t tables, bar, x, y, total;
};
__host__ __device__ constexpr LnqSmem lnq_smem_layout(int lanes, bool has_y) {
  LnqSmem s = {};
  const uint32_t rows = static_cast<uint32_t>(lnq_max_rows(lanes) * lanes * 48);
  s.tables = kLnqThreads * 128;
  s.bar = s.tables + kGroupQuantTableBytes;
  s.x = s.bar + 16;
  s.y = s.x + rows;
  s.total = s.y + (has_y ? rows : 0);
  return s;
}
static_assert(lnq_smem_layout(8, true).total <= 57344 && lnq_smem_layout(16, true).total <= 57344 && lnq_smem_layout(32, true).total <= 57344,
              "four blocks an SM");

template <int LANES, int BITS, bool HAS_Y>
__global__ void __launch_bounds__(kLnqThreads, 4)
    add_layernorm_act_quant_kernel(const __grid_constant__ CUtensorMap tm_out, const __half* __restrict__ x,
                                   const __half* __restrict__ y, const NormParams np, float eps, long long M,
                                   const float* __restrict__ thresholds, const float* __restrict__ codebook,
                                   __half* __restrict__ sum_out, __half* __restrict__ h_out, int one_fma, uint32_t poll_limit,
                                   int* status, const __grid_constant__ UnpackJobs jobs) {
  pdl_launch_dependents();   // the next kernel of the stream may start its set-up
  extern __shared__ __align__(1024) uint8_t lnq_smem[];
  if (static_cast<int>(blockIdx.x) < jobs.blocks) {
    unpack_jobs_run(jobs, static_cast<int>(blockIdx.x), reinterpret_cast<float*>(lnq_smem));
    return;
  }

  constexpr int L = 1 << BITS;
  constexpr int K = LANES * 24, G = K / 64, kRowsPerWarp = 32 / LANES, kRowsPerPass = 4 * kRowsPerWarp;
  constexpr int kPasses = (lnq_max_rows(LANES) + kRowsPerPass - 1) / kRowsPerPass;
  constexpr LnqSmem S = lnq_smem_layout(LANES, HAS_Y);
  GroupQuantTables* const tables = reinterpret_cast<GroupQuantTables*>(lnq_smem + S.tables);
  uint64_t* const bar = reinterpret_cast<uint64_t*>(lnq_smem + S.bar);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, l = lane % LANES, sub = lane / LANES;
  if (tid == 0) {
    mbar_init(bar, 1);
    mbar_fence_init();
    tma_prefetch_desc(&tm_out);
  }
  // reads only this layer's constants, so it runs before the wait below
  const GroupQuantParams gp = group_quant_tables<L, false>(tables, thresholds, codebook, tid, kLnqThreads,
                                                           [](bool b) { return __syncthreads_and(b) != 0; });

  const long long total_groups = M * G;
  const long long tiles = (total_groups + kLnqThreads - 1) / kLnqThreads;
  const long long stride = gridDim.x - jobs.blocks;
  // The rows of a tile, contiguous in x and in y, come by one bulk copy each: all of them are on their way at once, and the next
  // tile's while this one is quantised.  (A copy and a barrier for each pass, so that the first pass starts early: no better where a
  // block has one tile, [201728, 768] 222 us instead of 211.)
  auto load = [&](long long tile) {
    const long long gi0 = tile * kLnqThreads, r0 = gi0 / G, r1 = min(gi0 + kLnqThreads - 1, total_groups - 1) / G;
    const uint32_t bytes = static_cast<uint32_t>((r1 - r0 + 1) * (K * 2));
    mbar_arrive_expect_tx(bar, HAS_Y ? 2 * bytes : bytes);
    bulk_load_1d(lnq_smem + S.x, x + r0 * K, bytes, bar);
    if (HAS_Y) bulk_load_1d(lnq_smem + S.y, y + r0 * K, bytes, bar);
  };
  pdl_wait();                // x and y may be the previous kernels' outputs
  long long tile = static_cast<long long>(blockIdx.x) - jobs.blocks;
  if (tid == 0 && tile < tiles) load(tile);
  uint32_t ph = 0;
  bool ok = true;
  for (; tile < tiles; tile += stride, ph ^= 1) {
    const long long gi0 = tile * kLnqThreads;
    const int ngroups = static_cast<int>(min(static_cast<long long>(kLnqThreads), total_groups - gi0));
    const long long r_first = gi0 / G;
    // ---- phase 1: LayerNorm of every row the tile touches, LANES lanes per row
    LaneNorm norm;                          // read for each tile: the quantizer needs the registers
    layernorm_lane_params<LANES>(np, l, &norm);
    ok = mbar_wait_warp(bar, ph, poll_limit);
#pragma unroll 1
    for (int pass = 0; pass < kPasses && ok; ++pass) {
      const int lr = pass * kRowsPerPass + warp * kRowsPerWarp + sub;
      const long long row = r_first + lr;
      const long long lg0 = row * G - gi0;                       // tile-local index of the row's first group
      const bool in_tile = row < M && lg0 < ngroups;             // the row has groups in this tile
      const bool owned = in_tile && lg0 >= 0;                    // ... and its first group is one of them
      const int off = (in_tile ? lr : 0) * (K * 2) + l * 16;     // idle sub-warps shadow the first row
      uint4 a[3], b[3], h[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        a[i] = *reinterpret_cast<const uint4*>(lnq_smem + S.x + off + LANES * 16 * i);
        if (HAS_Y) b[i] = *reinterpret_cast<const uint4*>(lnq_smem + S.y + off + LANES * 16 * i);
      }
      layernorm_row_compute<LANES>(a, b, HAS_Y, row, owned, l, norm, eps, sum_out, h);
      if (in_tile) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const int ch = l + LANES * i;                          // 16-byte chunk of the row: group ch / 8, part ch % 8
          const int lg = static_cast<int>(lg0) + (ch >> 3);
          if (lg >= 0 && lg < ngroups)
            *reinterpret_cast<uint4*>(lnq_smem + lg * 128 + (((ch ^ lg) & 7) << 4)) = h[i];
          if (owned && h_out != nullptr) reinterpret_cast<uint4*>(h_out + row * K)[ch] = h[i];
        }
      }
    }
    ok = __syncthreads_and(ok) != 0;
    if (!ok) break;                         // some warp's wait ran out: nothing of this tile is quantised, no copy over rows that may still come
    if (tid == 0 && tile + stride < tiles) load(tile + stride);

    // ---- phase 2: the activation quantizer on h, one thread per group, in place; a warp sends its 32 rows out by TMA
    // (rows of the last tile beyond the matrix hold stale values; the store clips them)
    if (tid < ngroups) group_quantize_row<__half, BITS, false, 1>(smem_u32(lnq_smem) + tid * 128, lane & 7, tables, gp, one_fma != 0);
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      tma_store_2d(&tm_out, lnq_smem + warp * 4096, 0, static_cast<int>(gi0) + warp * 32);
      tma_store_commit();
      tma_store_wait_read();
    }
    __syncthreads();   // the rows are free for the next tile
  }
  if (lane == 0) tma_store_wait_all();
  if (!ok && tid == 0) {
    mbar_wait(bar, ph);                     // the copy that is still on its way lands before the block leaves
    atomicExch(status, kStatusLnqTimeout);
  }
}

// ---------------------------------------------------------------------------------------------------------
// The same operation for small inputs (a few hundred rows: batch 1-16 of a ViT), where the forward is a chain of
// short launches and one launch fewer counts for more than instruction counts.  Blocks of twelve warps, two phases per
// tile of 128 / LANES rows, through 6 KB of shared memory (the quantizer phase has three times as many lanes as the
// LayerNorm phase has, so that it is a single pass and the block's latency is one LayerNorm plus one quantizer step):
//   1. warps 0-3: residual add + LayerNorm with the lane layout and the arithmetic of add_layernorm_rows_kernel
//      (the same device function), so s and h are bit-identical to that kernel's;
//   2. all warps: the quantizer with the lane layout and the arithmetic of act_quant_kernel (eight lanes per group, IEEE
//      division, chain sums in the reference's order), reading h from shared memory.
// Its reconstruction therefore equals, bit for bit, what the two separate kernels produce, and a model may switch
// between the merged and the separate form by batch size without changing a single output bit.
constexpr int kLnqRowsThreads = 384;

template <int LANES, int BITS, bool HAS_Y>
__global__ void __launch_bounds__(kLnqRowsThreads, 1) add_layernorm_act_quant_rows_kernel(const __half* __restrict__ x,
                                                                          const __half* __restrict__ y,
                                                                          const NormParams np, float eps,
                                                                          long long M,
                                                                          const float* __restrict__ thresholds,
                                                                          const float* __restrict__ codebook,
                                                                          __half* __restrict__ sum_out,
                                                                          __half* __restrict__ h_out,
                                                                          __half* __restrict__ xhat, int one_fma,
                                                                          const __grid_constant__ UnpackJobs jobs) {
  pdl_launch_dependents();
  if (static_cast<int>(blockIdx.x) < jobs.blocks) {
    unpack_jobs_block(jobs);
    return;
  }
  constexpr int L = 1 << BITS;
  constexpr int K = LANES * 24, G = K / 64, kRowsPerWarp = 32 / LANES, kRows = 4 * kRowsPerWarp;   // rows per tile
  constexpr int kSlots = kRows * G * 8;            // (group, lane-of-eight) pairs per tile: 384 for every width
  static_assert(kSlots == kLnqRowsThreads, "the quantizer phase is one pass of the block");
  __shared__ __align__(16) __half s_hid[kRows * K];
  __shared__ float s_th[16];
  __shared__ float s_cb[16];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, l = lane % LANES, sub = lane / LANES;
  if (tid < 16) {
    s_th[tid] = (tid < L - 1) ? thresholds[tid] : __int_as_float(0x7f800000);
    s_cb[tid] = (tid < L) ? codebook[tid] : 0.0f;
  }
  LaneNorm norm = {};
  if (warp < 4) layernorm_lane_params<LANES>(np, l, &norm);
  __syncthreads();
  pdl_wait();                // everything above is the layer's constants; x and y may be the previous kernel's output

  const int l8 = lane & 7, octet_base = lane & ~7;
  for (long long row0 = static_cast<long long>(blockIdx.x - jobs.blocks) * kRows; row0 < M; row0 += static_cast<long long>(gridDim.x - jobs.blocks) * kRows) {
    // ---- phase 1 (warps 0-3): one row per LANES lanes
    if (warp < 4) {
      const int local = warp * kRowsPerWarp + sub;
      const long long row = row0 + local;
      const bool valid = row < M;
      const long long rs = valid ? row : M - 1;
      uint4 h[3];
      layernorm_row<LANES>(x, HAS_Y ? y : nullptr, rs, row, valid, l, norm, eps, sum_out, h);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        reinterpret_cast<uint4*>(s_hid + local * K)[l + LANES * i] = h[i];
        if (valid && h_out != nullptr) reinterpret_cast<uint4*>(h_out + row * K)[l + LANES * i] = h[i];
      }
    }
    __syncthreads();
    // ---- phase 2 (all warps): eight lanes per 64-group, lane l8 holds elements 8c + l8
    {
      const int grp = tid >> 3;                              // group of the tile
      const int local = grp / G, g = grp - local * G;
      const long long row = row0 + local;
      const bool valid = row < M;
      const __half* hg = s_hid + local * K + g * 64 + l8;
      float v[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) v[c] = __half2float(hg[8 * c]);
      float cv[8];
      uint32_t codes;
      const OctetStats st = octet_quantize<BITS>(v, s_th, s_cb, octet_base, cv, codes);
      const ReconTerms rt = recon_terms(st.mean, st.scale, st.code_sum, one_fma != 0);
      if (valid) {
        __half* og = xhat + row * K + g * 64 + l8;
#pragma unroll
        for (int c = 0; c < 8; ++c) og[8 * c] = __float2half_rn(recon_value(rt, st.scale, cv[c]));
      }
    }
    __syncthreads();   // the tile's rows in shared memory are free for the next tile
  }
}

}  // namespace arcq
