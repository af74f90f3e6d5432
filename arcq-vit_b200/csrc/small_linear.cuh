// A packed linear on few rows in one launch: quantizer, weight unpack and product.
//     y[M,N] = xhat . W16^T + bias,   xhat the ARCQ reconstruction of x (optionally of GELU(x)), W16 the fp16 weight rebuilt from codes
//
// For large inputs the two are kernels of their own, each result written once and read by many blocks.  On a few dozen rows the GPU
// works for less time than the host needs for a second launch and the scratch matrices (a module call 10.2 us, of which 3.1 a launch), so
// here every block makes what it needs itself: `R` rows of xhat and `bn` rows of W16 into shared memory (the same rows of x are
// quantised by all N / bn blocks), then one thread issues the products.
//
// Arithmetic and bits are those of act_quant_kernel, of the weight unpack and of the GEMM kernels (ascending 16-wide steps over k).
//
// The product's tile has 128 rows whatever R is: the rows beyond R are whatever shared memory holds behind a sub-tile (the next ones,
// or the tail that is allocated for that), and their results are not read.
//
// Tensor memory is allocated after the previous kernel has ended and before the next one may start, as in the attention kernel.
#pragma once
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include "ptx.cuh"
#include "act_quant.cuh"
#include "codes.cuh"

namespace arcq {

constexpr int kStatusSmallLinearTimeout = 0x601;
constexpr int kSmallLinearThreads = 768;      // 96 groups at a time, six warps a tensor-memory lane quarter

struct SmallLinearParams {
  int M, N, K, G;
  int R;             // rows of a block: a multiple of 8, at most 128
  int bn;            // columns of a block: a multiple of 16, divides N, at most 256
  const float* thresholds;
  const float* codebook;
  int one_fma;
  UnpackWeightJob weight;     // out is not used
  const float* bias;          // may be null
  void* y;
  int y_f32;
  uint32_t tmem_cols;         // power of two >= bn, at least 32
  uint32_t poll_limit;
  int* status;
};

struct SmallLinearSmem {
  uint32_t w, tables, total;
};
__host__ __device__ inline SmallLinearSmem small_linear_smem_layout(int R, int bn, int G) {
  SmallLinearSmem s;
  s.w = static_cast<uint32_t>(G - 1) * R * 128u + 128u * 128u;   // the last sub-tile is read to its 128th row
  s.tables = s.w + static_cast<uint32_t>(G) * bn * 128u;
  s.total = s.tables + 3 * 16 * 4 /* thresholds, levels, the weight's levels */ + 8 /* barrier */ + 8 /* tensor-memory address */;
  return s;
}

template <typename T, int BITS, int PRE>
__global__ void __launch_bounds__(kSmallLinearThreads, 1) small_linear_kernel(const T* __restrict__ x, const SmallLinearParams p) {
  extern __shared__ __align__(1024) uint8_t sl_smem[];
  constexpr int L = 1 << BITS;
  const SmallLinearSmem S = small_linear_smem_layout(p.R, p.bn, p.G);
  float* const s_th = reinterpret_cast<float*>(sl_smem + S.tables);
  float* const s_cb = s_th + 16;
  float* const s_wcb = s_cb + 16;
  uint64_t* const bar = reinterpret_cast<uint64_t*>(s_wcb + 16);
  uint32_t* const s_tmem = reinterpret_cast<uint32_t*>(bar + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_slabs = p.N / p.bn, slab = static_cast<int>(blockIdx.x) % n_slabs;
  const int n0 = slab * p.bn, row0 = static_cast<int>(blockIdx.x) / n_slabs * p.R;
  const int rows = min(p.R, p.M - row0);
  const bool fp32_weight = p.weight.fp32_form();
  if (tid < 16) {
    s_th[tid] = tid < L - 1 ? __ldg(p.thresholds + tid) : __int_as_float(0x7f800000);
    s_cb[tid] = tid < L ? __ldg(p.codebook + tid) : 0.0f;
    const float level = tid < L ? __ldg(p.weight.codebook + tid) : 0.0f;
    if (fp32_weight) s_wcb[tid] = level;
    else reinterpret_cast<__half*>(s_wcb)[tid] = __float2half_rn(level);
  }
  if (tid == 0) {
    mbar_init(bar, 1);
    mbar_fence_init();
  }
  pdl_wait();                // x may be the previous kernel's output, and tensor memory has to be free
  if (warp == 0) {
    tmem_alloc(s_tmem, p.tmem_cols);
    tmem_relinquish();
    tc_fence_before_sync();
  }
  __syncthreads();
  pdl_launch_dependents();
  tc_fence_after_sync();
  const uint32_t tmem = *s_tmem;

  // ---- xhat: eight lanes per group, lane l holds elements 8c + l.  The first values are on their way while the weight is unpacked.
  constexpr int kGroupsAtATime = kSmallLinearThreads / 8;
  const int l = lane & 7, octet_base = lane & ~7, groups = rows * p.G;
  float v[8];
  auto load = [&](int g0) {
    const int gi = min(g0 + (lane >> 3), groups - 1);            // idle octets repeat the last group
    const T* const xg = x + static_cast<long long>(row0) * p.K + static_cast<long long>(gi) * 64 + l;
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = load_f32<T>(xg + 8 * c);
  };
  if (warp * 4 < groups) load(warp * 4);

  // ---- W16: sub-tiles of 64 columns, bn rows of 128 bytes each, 128-byte swizzle
  {
    UnpackWeightJob j = p.weight;
    j.packed += static_cast<long long>(n0) * p.K * BITS / 8;
    j.mu += static_cast<long long>(n0) * p.G;
    j.sigma += static_cast<long long>(n0) * p.G;
    j.codesum += static_cast<long long>(n0) * p.G;
    j.rows = p.bn;
    auto store = [&](long long r, int ch, uint4 w) {
      *reinterpret_cast<uint4*>(sl_smem + S.w + ((ch >> 3) * p.bn + static_cast<int>(r)) * 128 + (((ch ^ static_cast<int>(r)) & 7) << 4)) = w;
    };
    if (BITS == 3 && fp32_weight) unpack_weight_chunks<BITS>(j, s_wcb, tid, kSmallLinearThreads, store);
    else unpack_weight_chunks<BITS>(j, reinterpret_cast<const __half*>(s_wcb), tid, kSmallLinearThreads, store);
  }

  for (int g0 = warp * 4; g0 < groups; g0 += kGroupsAtATime) {
    const int gi = min(g0 + (lane >> 3), groups - 1), r = gi / p.G, g = gi - r * p.G;
    float e[8], level[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) e[c] = pre_op<T, PRE>(v[c]);
    if (g0 + kGroupsAtATime < groups) load(g0 + kGroupsAtATime);
    uint32_t codes;
    const OctetStats st = octet_quantize<BITS>(e, s_th, s_cb, octet_base, level, codes);
    const ReconTerms rt = recon_terms(st.mean, st.scale, st.code_sum, p.one_fma != 0);
    uint8_t* const a = sl_smem + (g * p.R + r) * 128 + 2 * l;
#pragma unroll
    for (int c = 0; c < 8; ++c)
      *reinterpret_cast<__half*>(a + ((c ^ (r & 7)) << 4)) = __float2half_rn(recon_value(rt, st.scale, level[c]));
  }
  fence_proxy_async_smem();
  __syncthreads();

  if (tid == 0) {
    const uint32_t idesc = umma_idesc_f16(128, p.bn);
    uint32_t acc = 0;
    for (int g = 0; g < p.G; ++g) {
      const uint64_t da = umma_desc_sw128(smem_u32(sl_smem) + g * p.R * 128), dw = umma_desc_sw128(smem_u32(sl_smem) + S.w + g * p.bn * 128);
#pragma unroll
      for (int k = 0; k < 4; ++k, acc = 1) umma_f16(tmem, da + 2 * k, dw + 2 * k, idesc, acc);
    }
    umma_commit(bar);
  }
  __syncwarp();
  const bool ok = mbar_wait_warp(bar, 0, p.poll_limit);     // a warp whose wait ran out stores none of its rows, and says so
  tc_fence_after_sync();
  // ---- a thread per row, the warps of a tensor-memory lane quarter sixteen columns each
  const int quarter = warp & 3, r = quarter * 32 + lane;
  if (ok && quarter * 32 < rows) {
    for (int c0 = (warp >> 2) * 16; c0 < p.bn; c0 += kSmallLinearThreads / 128 * 16) {
      uint32_t a[16];
      tmem_ld_32x16(tmem + (static_cast<uint32_t>(quarter * 32) << 16) + c0, a);
      tmem_ld_wait();
      float v[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(a[i]) + (p.bias != nullptr ? __ldg(p.bias + n0 + c0 + i) : 0.0f);
      if (r < rows) {
        const long long at = static_cast<long long>(row0 + r) * p.N + n0 + c0;
        if (p.y_f32) {
          float4* const o = reinterpret_cast<float4*>(static_cast<float*>(p.y) + at);
#pragma unroll
          for (int i = 0; i < 4; ++i) o[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        } else {
          uint32_t w[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const __half2 h = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
            w[i] = *reinterpret_cast<const uint32_t*>(&h);
          }
          uint4* const o = reinterpret_cast<uint4*>(static_cast<__half*>(p.y) + at);
          o[0] = make_uint4(w[0], w[1], w[2], w[3]);
          o[1] = make_uint4(w[4], w[5], w[6], w[7]);
        }
      }
    }
  }
  if (!ok && lane == 0) atomicExch(p.status, kStatusSmallLinearTimeout);
  if (!ok && tid == 0) mbar_wait(bar, 0);                   // the products end before their memory is given back
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, p.tmem_cols);
  }
}

}  // namespace arcq
