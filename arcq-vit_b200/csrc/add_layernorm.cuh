// Residual add + LayerNorm in one pass over fp16 rows, ld values apart (the glue between the packed linears of a block):
//   s = fp16(x + y)   (written out when y is given: the updated residual stream)
//   h = fp16((s - mean(s)) * rsqrt(var(s) + eps) * gamma + beta)
// One warp per row, 16-byte loads/stores, statistics in fp32 with a two-pass (mean, then centred sum of
// squares) over values held in registers.  HBM-bound: reads x (and y), writes h (and s) once.
#pragma once
#include <cuda_fp16.h>
#include "ptx.cuh"
#include "f32x2.cuh"

namespace arcq {

// gamma and beta in the type the module holds them in, so that nobody has to keep converted copies: the ARCQ_DT_* numbers.
struct NormParams {
  const void* gamma;
  const void* beta;
  int dtype;          // 0 fp32, 1 fp16, 2 bf16
};
// values 8 * chunk .. 8 * chunk + 7 as fp32
__device__ __forceinline__ void load_norm_chunk(const void* p, int dtype, int chunk, float (&v)[8]) {
  if (dtype == 0) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p) + 2 * chunk), b = __ldg(reinterpret_cast<const float4*>(p) + 2 * chunk + 1);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(p) + chunk);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
      v[2 * j] = dtype == 1 ? f.x : __uint_as_float(w[j] << 16);
      v[2 * j + 1] = dtype == 1 ? f.y : __uint_as_float(w[j] & 0xFFFF0000u);
    }
  }
}

constexpr int kLnMaxChunks = 8;  // 16-byte chunks per lane: rows up to 32 * 8 * 8 = 2048 values

__global__ void __launch_bounds__(256) add_layernorm_kernel(const __half* __restrict__ x, const __half* __restrict__ y,
                                                            const NormParams np, float eps, long long M, int K,
                                                            long long ld, __half* __restrict__ sum_out,
                                                            __half* __restrict__ h_out) {
  pdl_launch_dependents();   // the next kernel of the stream may start its set-up
  pdl_wait();                // the input may be the previous kernel's output

  const int lane = threadIdx.x & 31;
  const long long warps = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  const int chunks = K >> 3;
  for (long long row = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); row < M; row += warps) {
    const uint4* xr = reinterpret_cast<const uint4*>(x + row * ld);
    const uint4* yr = (y != nullptr) ? reinterpret_cast<const uint4*>(y + row * ld) : nullptr;
    float v[kLnMaxChunks][8];
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < kLnMaxChunks; ++i) {
      const int c = lane + 32 * i;
      if (c < chunks) {
        const uint4 a = __ldg(xr + c);
        const __half2* ah = reinterpret_cast<const __half2*>(&a);
        if (yr != nullptr) {
          const uint4 b = __ldg(yr + c);
          const __half2* bh = reinterpret_cast<const __half2*>(&b);
          uint4 so;
          __half2* sh = reinterpret_cast<__half2*>(&so);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 fa = __half22float2(ah[j]), fb = __half22float2(bh[j]);
            sh[j] = __floats2half2_rn(fa.x + fb.x, fa.y + fb.y);   // the fp16 sum a separate add would store
            const float2 fs = __half22float2(sh[j]);
            v[i][2 * j] = fs.x;
            v[i][2 * j + 1] = fs.y;
          }
          if (sum_out != nullptr) reinterpret_cast<uint4*>(sum_out + row * K)[c] = so;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 fa = __half22float2(ah[j]);
            v[i][2 * j] = fa.x;
            v[i][2 * j + 1] = fa.y;
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) sum += v[i][j];
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float mean = sum / static_cast<float>(K);
    float sq = 0.0f;
#pragma unroll
    for (int i = 0; i < kLnMaxChunks; ++i) {
      if (lane + 32 * i < chunks) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float d = v[i][j] - mean;
          sq += d * d;
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    const float rstd = rsqrtf(sq / static_cast<float>(K) + eps);
#pragma unroll
    for (int i = 0; i < kLnMaxChunks; ++i) {
      const int c = lane + 32 * i;
      if (c < chunks) {
        float gg[8], bb[8];
        load_norm_chunk(np.gamma, np.dtype, c, gg);
        load_norm_chunk(np.beta, np.dtype, c, bb);
        uint4 o;
        __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          oh[j] = __floats2half2_rn((v[i][2 * j] - mean) * rstd * gg[2 * j] + bb[2 * j],
                                    (v[i][2 * j + 1] - mean) * rstd * gg[2 * j + 1] + bb[2 * j + 1]);
        reinterpret_cast<uint4*>(h_out + row * K)[c] = o;
      }
    }
  }
}

// One row of LANES * 24 values (192 / 384 / 768: the DeiT widths) on LANES lanes, three 16-byte chunks per lane:
// s = fp16(x + y) (stored when asked), statistics in two passes, h = fp16((s - mean) * rstd * gamma + beta) returned
// as the lane's three packed chunks.  `rs` is the row to read (idle sub-warps shadow the last row), `row` the row
// to store (only if `valid`).  Shared by the LayerNorm kernel below and by the small-batch LayerNorm + quantizer
// kernel (ln_act_quant.cuh), so that the two produce the same bits.
// The lane's three chunks of row `rs` of x (and of y, if given).
template <int LANES>
__device__ __forceinline__ void layernorm_row_load(const __half* __restrict__ x, const __half* __restrict__ y,
                                                   long long rs, int l, uint4 (&a)[3], uint4 (&b)[3]) {
  constexpr int K = LANES * 24;
  const uint4* xr = reinterpret_cast<const uint4*>(x + rs * K);
#pragma unroll
  for (int i = 0; i < 3; ++i) a[i] = __ldg(xr + l + LANES * i);
  if (y != nullptr) {
    const uint4* yr = reinterpret_cast<const uint4*>(y + rs * K);
#pragma unroll
    for (int i = 0; i < 3; ++i) b[i] = __ldg(yr + l + LANES * i);
  }
}

// gamma and beta of the lane's three chunks
struct LaneNorm {
  f32x2 g[3][4], b[3][4];
};
template <int LANES> __device__ __forceinline__ void layernorm_lane_params(const NormParams& np, int l, LaneNorm* n) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    float g[8], b[8];
    load_norm_chunk(np.gamma, np.dtype, l + LANES * i, g);
    load_norm_chunk(np.beta, np.dtype, l + LANES * i, b);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      n->g[i][j] = pack2(g[2 * j], g[2 * j + 1]);
      n->b[i][j] = pack2(b[2 * j], b[2 * j + 1]);
    }
  }
}

// The sum of a chunk's eight values (SQUARES: of their squares).  A row's sum is taken chunk by chunk, then over the lane's chunks,
// then over the lanes, so that a kernel that holds the row in another layout can add in the same order.
template <bool SQUARES> __device__ __forceinline__ float layernorm_chunk_sum(const f32x2 (&v)[4]) {
  float lo, hi;
  if (SQUARES) unpack2(fma2(v[3], v[3], fma2(v[2], v[2], fma2(v[1], v[1], mul2(v[0], v[0])))), lo, hi);
  else unpack2(add2(add2(v[0], v[1]), add2(v[2], v[3])), lo, hi);
  return lo + hi;
}
__device__ __forceinline__ float layernorm_rstd(float squares, float k_inv, float eps) { return rsqrtf(squares * k_inv + eps); }

// The arithmetic of one row on chunks already loaded (`has_y`: b holds the residual branch).  Two values per instruction; the sum of
// two fp16 values rounded once is what the fp32 sum rounds to (their bits span less than fp32 holds wherever that could tie).
// About 10 instructions a value, loads and stores included; with scalar arithmetic on converted values it was 20.
template <int LANES>
__device__ __forceinline__ void layernorm_row_compute(const uint4 (&a)[3], const uint4 (&b)[3], bool has_y,
                                                      long long row, bool valid, int l, const LaneNorm& n, float eps,
                                                      __half* __restrict__ sum_out, uint4 (&h)[3]) {
  constexpr int K = LANES * 24;
  constexpr float kInv = 1.0f / static_cast<float>(K);
  f32x2 v[3][4];
  float sum = 0.0f;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    uint32_t s[4] = {a[i].x, a[i].y, a[i].z, a[i].w};
    if (has_y) {
      const uint32_t t[4] = {b[i].x, b[i].y, b[i].z, b[i].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const __half2 r = __hadd2(*reinterpret_cast<const __half2*>(&s[j]), *reinterpret_cast<const __half2*>(&t[j]));
        s[j] = *reinterpret_cast<const uint32_t*>(&r);
      }
      if (valid && sum_out != nullptr) reinterpret_cast<uint4*>(sum_out + row * K)[l + LANES * i] = make_uint4(s[0], s[1], s[2], s[3]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) v[i][j] = sixteen_to_pair<__half>(s[j]);
    const float c = layernorm_chunk_sum<false>(v[i]);
    sum = i == 0 ? c : sum + c;
  }
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  const float nm = -(sum * kInv);
  const f32x2 nm2 = pack2(nm, nm);
  float sq = 0.0f;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[i][j] = add2(v[i][j], nm2);
    const float c = layernorm_chunk_sum<true>(v[i]);
    sq = i == 0 ? c : sq + c;
  }
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
  const float rstd = layernorm_rstd(sq, kInv, eps);
  const f32x2 rstd2 = pack2(rstd, rstd);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = pair_to_sixteen<__half>(fma2(mul2(v[i][j], rstd2), n.g[i][j], n.b[i][j]));
    h[i] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

template <int LANES>
__device__ __forceinline__ void layernorm_row(const __half* __restrict__ x, const __half* __restrict__ y, long long rs,
                                              long long row, bool valid, int l, const LaneNorm& n, float eps,
                                              __half* __restrict__ sum_out, uint4 (&h)[3]) {
  uint4 a[3], b[3];
  layernorm_row_load<LANES>(x, y, rs, l, a, b);
  layernorm_row_compute<LANES>(a, b, y != nullptr, row, valid, l, n, eps, sum_out, h);
}

// Residual add + LayerNorm for rows of LANES * 24 values: LANES lanes per row, so every lane carries the same load
// and a warp works on 32 / LANES rows at once; gamma and beta stay in registers for all the rows a lane visits.
template <int LANES>
__global__ void __launch_bounds__(256) add_layernorm_rows_kernel(const __half* __restrict__ x,
                                                                 const __half* __restrict__ y,
                                                                 const NormParams np, float eps,
                                                                 long long M, long long ld,
                                                                 __half* __restrict__ sum_out,
                                                                 __half* __restrict__ h_out) {
  pdl_launch_dependents();   // the next kernel of the stream may start its set-up

  constexpr int K = LANES * 24, kRowsPerWarp = 32 / LANES;
  const int lane = threadIdx.x & 31, l = lane % LANES, sub = lane / LANES;
  LaneNorm n;
  layernorm_lane_params<LANES>(np, l, &n);
  pdl_wait();                // gamma and beta are the layer's constants; x and y may be the previous kernel's output
  const long long warps = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  const long long first = (static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kRowsPerWarp;
  for (long long row0 = first; row0 < M; row0 += warps * kRowsPerWarp) {
    const long long row = row0 + sub;
    const bool valid = row < M;
    const long long rs = valid ? row : M - 1;          // idle sub-warps shadow the last row, store nothing
    uint4 h[3];
    const long long skip = rs * (ld - K);              // input rows are ld values apart
    layernorm_row<LANES>(x + skip, y != nullptr ? y + skip : nullptr, rs, row, valid, l, n, eps, sum_out, h);
    if (valid) {
#pragma unroll
      for (int i = 0; i < 3; ++i) reinterpret_cast<uint4*>(h_out + row * K)[l + LANES * i] = h[i];
    }
  }
}

}  // namespace arcq
