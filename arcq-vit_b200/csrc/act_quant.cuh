// Activation quantizer kernel (group size 64): packed codes + per-group mean / scale / code sum,
// and optionally the reconstruction.  HBM-bound: every input element is read once, every output
// byte written once.
//
// Bit-exactness contract.  Codes must equal the reference CPU quantizer's, which computes in fp32
// with torch's reduction order: the 64 values of a group are seen as 8 chunks of 8 lanes; chunk c
// is added lane-wise to accumulator c % 4, the four accumulators are then added 0+1, +2, +3, and
// the 8 lanes of the result are added one after the other.  The mapping below gives lane l of an
// 8-lane "octet" exactly the elements {8c + l}, so the lane-wise part is local arithmetic in the
// same order and the final 8-term sum is a sequential shuffle chain.  All arithmetic uses the
// round-to-nearest intrinsics so that nothing is contracted into fused multiply-adds, and division
// and square root are the IEEE ones.
#pragma once
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include "ptx.cuh"
#include "element_types.cuh"
#include "codes.cuh"

namespace arcq {

// Optional element-wise op applied to the input before it is quantised (fused from the preceding layer).
// PRE = 1: exact (erf) GELU in fp32, then rounded to the input's element type -- the value a separate GELU kernel would have
// stored -- so the quantizer sees the same numbers as unfused.
template <typename T> __device__ __forceinline__ float round_to(float v);
template <> __device__ __forceinline__ float round_to<float>(float v) { return v; }
template <> __device__ __forceinline__ float round_to<__half>(float v) { return __half2float(__float2half_rn(v)); }
template <> __device__ __forceinline__ float round_to<__nv_bfloat16>(float v) {
  return __bfloat162float(__float2bfloat16_rn(v));
}
// GELU of an fp16 value in fp32, in all kernels the same to the bit: x * (0.5 + x * R(x^2)) for |x| < 2, with
// x * R(x^2) = erf(x / sqrt 2) / 2 and R of degree 7, fitted on Chebyshev nodes; erff beyond.  Rounded to fp16 it is, for each
// of the 65 536 inputs, what 0.5 x (1 + erff(x / sqrt 2)) in fp32 rounds to: the coefficient of degree 3 is three units in the
// last place off the fit, because with the fit itself x = -1.4853515625 came out one unit off.
constexpr float kGeluLimit = 2.0f;
__device__ __forceinline__ float gelu_r(int k) {       // k is a constant wherever this is used
  const float c[8] = {0.398942292f,    -0.0664903149f,  0.00997320935f, -0.00118661555f,
                      0.000114711416f, -9.03896398e-06f, 5.35578579e-07f, -1.75760011e-08f};
  return c[k];
}
__device__ __forceinline__ float gelu_large(float x) { return x * 0.5f * (1.0f + erff(x * 0.70710678118654752440f)); }
__device__ __forceinline__ float gelu(float x) {
  if (!(fabsf(x) < kGeluLimit)) return gelu_large(x);
  const float s = __fmul_rn(x, x);
  float r = gelu_r(7);
#pragma unroll
  for (int k = 6; k >= 0; --k) r = fmaf(r, s, gelu_r(k));
  return __fmul_rn(x, fmaf(x, r, 0.5f));
}
template <typename T, int PRE> __device__ __forceinline__ float pre_op(float x) {
  return PRE == 1 ? round_to<T>(gelu(x)) : x;
}

// The reconstruction of a level as c + (scale * (level + a) + b), in either of the two forms the GEMMs were built for:
//   three steps   mean + scale * (level - code_sum / 64), each rounded, as the reference's fp32 tensor operations;
//   one_fma       fma(scale, level, mean - scale * code_sum / 64), what arcq_packed_gemm rebuilds from packed codes.
// The other two operations add -0, which changes nothing.
struct ReconTerms {
  float a, b, c;
};
__device__ __forceinline__ ReconTerms recon_terms(float mean, float scale, float code_sum, bool one_fma) {
  const float vm = __fmul_rn(code_sum, 0.015625f);           // / 64: exact
  if (one_fma) return {-0.0f, __fmaf_rn(-scale, vm, mean), -0.0f};
  return {-vm, -0.0f, mean};
}
__device__ __forceinline__ float recon_value(const ReconTerms& t, float scale, float level) {
  return __fadd_rn(t.c, __fmaf_rn(scale, __fadd_rn(level, t.a), t.b));
}

// Sum of the value held by the 8 lanes of an octet, lane 0 first, as a chain of fp32 additions.
__device__ __forceinline__ float octet_chain_sum(float p, int octet_base) {
  float s = __shfl_sync(0xffffffffu, p, octet_base);
#pragma unroll
  for (int i = 1; i < 8; ++i) s = __fadd_rn(s, __shfl_sync(0xffffffffu, p, octet_base + i));
  return s;
}

// The quantizer of one group by an octet.  In: v[c] = element 8c + l in lane l.  Out: the levels of those elements' codes, the codes
// one per nibble, and the group's statistics.
struct OctetStats {
  float mean, scale, code_sum;
};
template <int BITS>
__device__ __forceinline__ OctetStats octet_quantize(const float (&v)[8], const float* s_th, const float* s_cb, int octet_base,
                                                     float (&level)[8], uint32_t& codes) {
  auto sum = [&](const float (&e)[8]) {
    const float a0 = __fadd_rn(e[0], e[4]), a1 = __fadd_rn(e[1], e[5]), a2 = __fadd_rn(e[2], e[6]), a3 = __fadd_rn(e[3], e[7]);
    return octet_chain_sum(__fadd_rn(__fadd_rn(__fadd_rn(a0, a1), a2), a3), octet_base);
  };
  OctetStats st;
  st.mean = __fdiv_rn(sum(v), 64.0f);
  float r[8], q[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    r[c] = __fsub_rn(v[c], st.mean);
    q[c] = __fmul_rn(r[c], r[c]);
  }
  st.scale = __fsqrt_rn(__fadd_rn(__fdiv_rn(sum(q), 64.0f), 1.0e-6f));      // sqrt(mean(r^2) + 1e-6)
  // codes: number of thresholds strictly below t (binary search in the sorted table)
  codes = 0;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const float t = __fdiv_rn(r[c], st.scale);
    int code = 0;
    if (BITS >= 4) code = (t > s_th[7]) ? 8 : 0;
    if (BITS >= 3) code += (t > s_th[code + 3]) ? 4 : 0;
    code += (t > s_th[code + 1]) ? 2 : 0;
    code += (t > s_th[code]) ? 1 : 0;
    codes |= static_cast<uint32_t>(code) << (4 * c);
    level[c] = s_cb[code];
  }
  st.code_sum = sum(level);
  return st;
}

// In: lane l of an octet holds, in nibble c, the code of element 8c + l.
// Out: lane l holds, in nibble j, the code of element 8l + j (an 8x8 nibble transpose over lanes).
__device__ __forceinline__ uint32_t octet_transpose_nibbles(uint32_t w, int l) {
  uint32_t p = __shfl_xor_sync(0xffffffffu, w, 4);
  w = (l & 4) ? ((w & 0xFFFF0000u) | (p >> 16)) : ((w & 0x0000FFFFu) | (p << 16));
  p = __shfl_xor_sync(0xffffffffu, w, 2);
  w = (l & 2) ? ((w & 0xFF00FF00u) | ((p >> 8) & 0x00FF00FFu)) : ((w & 0x00FF00FFu) | ((p << 8) & 0xFF00FF00u));
  p = __shfl_xor_sync(0xffffffffu, w, 1);
  w = (l & 1) ? ((w & 0xF0F0F0F0u) | ((p >> 4) & 0x0F0F0F0Fu)) : ((w & 0x0F0F0F0Fu) | ((p << 4) & 0xF0F0F0F0u));
  return w;
}

// 8 nibbles (each holding a 3-bit code) -> 24 contiguous bits; (2-bit codes) -> 16 contiguous bits.
__device__ __forceinline__ uint32_t squeeze_nibbles_3(uint32_t w) {
  uint32_t t = (w & 0x07070707u) | ((w & 0x70707070u) >> 1);
  uint32_t u = (t & 0x003F003Fu) | ((t & 0x3F003F00u) >> 2);
  return (u & 0xFFFu) | ((u >> 4) & 0xFFF000u);
}
__device__ __forceinline__ uint32_t squeeze_nibbles_2(uint32_t w) {
  uint32_t t = (w & 0x03030303u) | ((w & 0x30303030u) >> 2);
  uint32_t u = (t & 0x000F000Fu) | ((t & 0x0F000F00u) >> 4);
  return (u & 0xFFu) | ((u >> 8) & 0xFF00u);
}

// One warp handles 4 consecutive groups per step (8 lanes per group).  Groups are numbered
// row-major over [M, K/64]; with K a multiple of 64 the input, the packed output and the statistics
// are all contiguous in that numbering.
template <typename T, int BITS, typename XH, bool WRITE_XHAT, int PRE = 0>
__global__ void __launch_bounds__(256) act_quant_kernel(const T* __restrict__ x, long long total_groups,
                                                        const float* __restrict__ thresholds,
                                                        const float* __restrict__ codebook,
                                                        uint8_t* __restrict__ packed, float* __restrict__ mu_out,
                                                        float* __restrict__ sigma_out,
                                                        float* __restrict__ codesum_out, XH* __restrict__ xhat,
                                                        int one_fma, const __grid_constant__ UnpackJobs jobs) {
  pdl_launch_dependents();   // the next kernel of the stream may start its set-up
  if (static_cast<int>(blockIdx.x) < jobs.blocks) {
    unpack_jobs_block(jobs);
    return;
  }

  constexpr int L = 1 << BITS;
  __shared__ float s_th[16];
  __shared__ float s_cb[16];
  if (threadIdx.x < 16) {
    const int t = threadIdx.x;
    s_th[t] = (t < L - 1) ? thresholds[t] : __int_as_float(0x7f800000);
    s_cb[t] = (t < L) ? codebook[t] : 0.0f;
  }
  __syncthreads();
  pdl_wait();                // the tables above are the layer's constants; x may be the previous kernel's output

  const int lane = threadIdx.x & 31;
  const int l = lane & 7;
  const int octet_base = lane & ~7;
  const long long warps_total = static_cast<long long>(gridDim.x - jobs.blocks) * (blockDim.x >> 5);
  const long long tasks = (total_groups + 3) >> 2;

  for (long long task = static_cast<long long>(blockIdx.x - jobs.blocks) * (blockDim.x >> 5) + (threadIdx.x >> 5); task < tasks;
       task += warps_total) {
    const long long gi = task * 4 + (lane >> 3);
    const bool valid = gi < total_groups;
    const long long gs = valid ? gi : total_groups - 1;  // idle octets shadow the last group, store nothing
    const T* xg = x + gs * 64 + l;

    float v[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = pre_op<T, PRE>(load_f32<T>(xg + 8 * c));

    uint32_t w;
    float cv[8];
    const OctetStats st = octet_quantize<BITS>(v, s_th, s_cb, octet_base, cv, w);
    const float mean = st.mean, scale = st.scale, code_sum = st.code_sum;

    if (WRITE_XHAT) {
      const ReconTerms rt = recon_terms(mean, scale, code_sum, one_fma != 0);
      if (valid) {
        XH* og = xhat + gi * 64 + l;
#pragma unroll
        for (int c = 0; c < 8; ++c)
          store_from_f32<XH>(og + 8 * c, recon_value(rt, scale, cv[c]));
      }
    }

    if (packed != nullptr) {
      w = octet_transpose_nibbles(w, l);  // lane l now holds codes of elements 8l .. 8l+7
      if (BITS == 4) {
        if (valid) reinterpret_cast<uint32_t*>(packed)[gi * 8 + l] = w;
      } else if (BITS == 3) {
        const uint32_t v24 = squeeze_nibbles_3(w);
        // 8 lanes x 3 bytes -> 6 words; word j starts at byte 4j = chunk q, byte r of it
        const int q = (4 * l) / 3, rr = (4 * l) % 3;
        const uint32_t lo = __shfl_sync(0xffffffffu, v24, octet_base + (q & 7));
        const uint32_t hi = __shfl_sync(0xffffffffu, v24, octet_base + ((q + 1) & 7));
        const uint32_t word = (lo >> (8 * rr)) | (hi << (24 - 8 * rr));
        if (valid && l < 6) reinterpret_cast<uint32_t*>(packed)[gi * 6 + l] = word;
      } else {
        const uint32_t v16 = squeeze_nibbles_2(w);
        const uint32_t lo = __shfl_sync(0xffffffffu, v16, octet_base + ((2 * l) & 7));
        const uint32_t hi = __shfl_sync(0xffffffffu, v16, octet_base + ((2 * l + 1) & 7));
        if (valid && l < 4) reinterpret_cast<uint32_t*>(packed)[gi * 4 + l] = lo | (hi << 16);
      }
    }
    if (valid && mu_out != nullptr) {
      if (l == 0) mu_out[gi] = mean;
      if (l == 1) sigma_out[gi] = scale;
      if (l == 2 && codesum_out != nullptr) codesum_out[gi] = code_sum;
    }
  }
}

}  // namespace arcq
