// Bit-stream helpers and the small format kernels (unpack, pack, reconstruct).
// Layout: code j of a row occupies bits [j*bits, (j+1)*bits) of the row's little-endian bit stream.
#pragma once
#include <cuda_fp16.h>
#include "ptx.cuh"
#include "element_types.cuh"

namespace arcq {

// Inverse of squeeze_nibbles_3/2: spread 8 packed codes into one nibble each.
__device__ __forceinline__ uint32_t spread_3_to_nibbles(uint32_t v24) {
  uint32_t u = (v24 & 0xFFFu) | ((v24 & 0xFFF000u) << 4);
  uint32_t t = (u & 0x003F003Fu) | ((u & 0x0FC00FC0u) << 2);
  return (t & 0x07070707u) | ((t & 0x38383838u) << 1);
}
__device__ __forceinline__ uint32_t spread_2_to_nibbles(uint32_t v16) {
  uint32_t u = (v16 & 0xFFu) | ((v16 & 0xFF00u) << 8);
  uint32_t t = (u & 0x000F000Fu) | ((u & 0x00F000F0u) << 4);
  return (t & 0x03030303u) | ((t & 0x0C0C0C0Cu) << 2);
}

// The 8 codes of chunk `chunk` (elements 8*chunk .. 8*chunk+7) of a packed row, one per nibble.
// Reads exactly the bytes that hold those codes, never past the row.
template <int BITS>
__device__ __forceinline__ uint32_t load_codes8(const uint8_t* __restrict__ row, int chunk) {
  if (BITS == 4) {
    return __ldg(reinterpret_cast<const uint32_t*>(row) + chunk);
  } else if (BITS == 3) {
    const uint8_t* p = row + 3 * chunk;
    const uint32_t v = static_cast<uint32_t>(__ldg(p)) | (static_cast<uint32_t>(__ldg(p + 1)) << 8) |
                       (static_cast<uint32_t>(__ldg(p + 2)) << 16);
    return spread_3_to_nibbles(v);
  } else {
    return spread_2_to_nibbles(__ldg(reinterpret_cast<const uint16_t*>(row) + chunk));
  }
}

__global__ void unpack_codes_kernel(const uint8_t* __restrict__ packed, long long rows, long long length,
                                    long long packed_cols, int bits, uint8_t* __restrict__ out) {
  const long long total = rows * length;
  const unsigned mask = (1u << bits) - 1u;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / length, j = i - r * length;
    const long long bit = j * bits;
    const uint8_t* p = packed + r * packed_cols + (bit >> 3);
    const int sh = static_cast<int>(bit & 7);
    unsigned v = static_cast<unsigned>(p[0]) >> sh;
    if (sh + bits > 8) v |= static_cast<unsigned>(p[1]) << (8 - sh);
    out[i] = static_cast<uint8_t>(v & mask);
  }
}

// One thread per output byte: gathers the (at most 5) codes that overlap it.
__global__ void pack_codes_kernel(const uint8_t* __restrict__ codes, long long rows, long long length,
                                  long long packed_cols, int bits, uint8_t* __restrict__ out) {
  const long long total = rows * packed_cols;
  const unsigned mask = (1u << bits) - 1u;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / packed_cols, b = i - r * packed_cols;
    const long long bit0 = b * 8;
    long long j = bit0 / bits;
    unsigned acc = 0;
    for (; j < length && j * bits < bit0 + 8; ++j) {
      const long long cb = j * bits;  // first bit of code j
      const unsigned c = static_cast<unsigned>(codes[r * length + j]) & mask;
      acc |= (cb >= bit0) ? (c << (cb - bit0)) : (c >> (bit0 - cb));
    }
    out[i] = static_cast<uint8_t>(acc & 0xffu);
  }
}

// out[r, k] = mu + sigma * (cb[c] - codesum/gs); one thread per chunk of 8 codes.  Any group size, any alignment of the output.
template <int BITS, typename OUT>
__global__ void dequant_kernel(const uint8_t* __restrict__ packed, const float* __restrict__ mu,
                               const float* __restrict__ sigma, const float* __restrict__ codesum,
                               const float* __restrict__ codebook, long long rows, int K, int gs,
                               OUT* __restrict__ out) {
  __shared__ float s_cb[16];
  if (threadIdx.x < 16) s_cb[threadIdx.x] = (threadIdx.x < (1 << BITS)) ? codebook[threadIdx.x] : 0.0f;
  __syncthreads();
  const int chunks = K / 8;
  const int G = K / gs;
  const long long pc = static_cast<long long>(K) * BITS / 8;
  const long long total = rows * chunks;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / chunks;
    const int ch = static_cast<int>(i - r * chunks);
    const int g = (ch * 8) / gs;
    const uint32_t w = load_codes8<BITS>(packed + r * pc, ch);
    const float m = mu[r * G + g], s = sigma[r * G + g];
    const float vm = __fdiv_rn(codesum[r * G + g], static_cast<float>(gs));
    OUT* o = out + r * K + ch * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float v = __fadd_rn(m, __fmul_rn(s, __fsub_rn(s_cb[(w >> (4 * j)) & 15u], vm)));
      store_from_f32<OUT>(o + j, v);
    }
  }
}

// The same for groups of 64, with 16-byte stores: chunks, groups and outputs are contiguous in the same order, so a chunk's group is its
// number / 8 and nothing is divided.  Two chunks a thread, their loads issued together.  From 4-bit codes to fp16 [12608, 384] 3.6 us, [25216,
// 3072] 45 us (4.8 TB/s); 11.4 and 170 us when every chunk was found by a 64-bit division and stored a value at a time.
template <int BITS, typename OUT>
__global__ void __launch_bounds__(256) dequant64_kernel(const uint8_t* __restrict__ packed, const float* __restrict__ mu,
                                                        const float* __restrict__ sigma, const float* __restrict__ codesum,
                                                        const float* __restrict__ codebook, long long total, OUT* __restrict__ out) {
  pdl_launch_dependents();
  __shared__ float s_cb[16];
  pdl_wait();                // codes, statistics and levels are a call's arguments: any of them may be the previous kernel's output
  if (threadIdx.x < 16) s_cb[threadIdx.x] = (threadIdx.x < (1 << BITS)) ? __ldg(codebook + threadIdx.x) : 0.0f;
  __syncthreads();
  const long long stride = static_cast<long long>(gridDim.x) * 256;
  for (long long i0 = blockIdx.x * 256ll + threadIdx.x; i0 < total; i0 += 2 * stride) {
    uint32_t w[2];
    float m[2], s[2], vm[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const long long i = min(i0 + u * stride, total - 1), g = i >> 3;
      w[u] = load_codes8<BITS>(packed + g * (8 * BITS), static_cast<int>(i & 7));
      m[u] = __ldg(mu + g);
      s[u] = __ldg(sigma + g);
      vm[u] = __fmul_rn(__ldg(codesum + g), 0.015625f);          // / 64: rounds as the division does
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const long long i = i0 + u * stride;
      if (i >= total) break;
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = __fadd_rn(m[u], __fmul_rn(s[u], __fsub_rn(s_cb[(w[u] >> (4 * j)) & 15u], vm[u])));
      if constexpr (sizeof(OUT) == 4) {
        float4* const o = reinterpret_cast<float4*>(out + i * 8);
        o[0] = make_float4(v[0], v[1], v[2], v[3]);
        o[1] = make_float4(v[4], v[5], v[6], v[7]);
      } else {
        uint32_t h[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const __half2 p = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
          h[j] = *reinterpret_cast<const uint32_t*>(&p);
        }
        *reinterpret_cast<uint4*>(out + i * 8) = make_uint4(h[0], h[1], h[2], h[3]);
      }
    }
  }
}

// out[r, k] = fp16(mu' + sigma16 * cb16[c]) with mu' = fp16(mu - sigma*codesum/64), sigma16 = fp16(sigma),
// cb16 = fp16(cb[c]) and one half-precision fused multiply-add: bit for bit the weight the packed-weight
// GEMM kernels rebuild in shared memory, written out so that a dense GEMM can read it by TMA.
// One thread per chunk of 8 codes (16 bytes of output); groups of 64.
// fp32_form(): fp16(sigma * cb[c] + mu') with everything in fp32 up to the one rounding, which is what arcq_packed_gemm rebuilds:
// the weight of layers whose packed rows are no multiple of 16 bytes (only 3-bit rows of an odd number of groups, so it is
// built for 3 bits), which the packed-weight kernels do not take.  (576 x 192, 3 bits: rms relative error of the rebuilt weight
// 2.1e-4 against 3.6e-4 in the fp16 form.)
struct UnpackWeightJob {
  const uint8_t* packed;     // null: nothing to do
  const float* mu;
  const float* sigma;
  const float* codesum;
  const float* codebook;
  __half* out;
  long long rows;
  int K;
  int bits;
  // see above; not a member, so that the launches that carry jobs keep their size
  __device__ __forceinline__ bool fp32_form() const { return bits == 3 && (K & 64) != 0; }
};

// Chunks first, first + stride, ... of the job; `s_cb` holds the 16 codebook values, of type CB: __half, or float for the
// fp32 form.  Four chunks per round, all their loads issued before the first result is used: a caller with few warps (the spare warps of a
// GEMM kernel) has nothing else to hide the load latency with.
// `store(row, chunk, value)` takes a result.
template <int BITS, typename CB, typename Store>
__device__ __forceinline__ void unpack_weight_chunks(const UnpackWeightJob& j, const CB* s_cb, long long first, long long stride, Store store) {
  const int chunks = j.K / 8;
  const int G = j.K / 64;
  const long long pc = static_cast<long long>(j.K) * BITS / 8;
  const long long total = j.rows * chunks;
  constexpr int U = 4;
  for (long long i0 = first; i0 < total; i0 += U * stride) {
    uint32_t w[U];
    float sg[U], cs[U], mu[U];
    long long row[U];
    int chunk[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = i0 + u * stride;
      const bool in = i < total;
      const long long ii = in ? i : first;
      const long long r = ii / chunks;
      const int ch = static_cast<int>(ii - r * chunks);
      const long long sgi = r * G + (ch >> 3);
      w[u] = load_codes8<BITS>(j.packed + r * pc, ch);
      sg[u] = __ldg(j.sigma + sgi);
      cs[u] = __ldg(j.codesum + sgi);
      mu[u] = __ldg(j.mu + sgi);
      row[u] = in ? r : -1;
      chunk[u] = ch;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (row[u] < 0) continue;
      const float m = fmaf(-sg[u], cs[u] * (1.0f / 64.0f), mu[u]);
      uint32_t h[4];
      if constexpr (sizeof(CB) == 4) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const __half2 r2 = __floats2half2_rn(fmaf(sg[u], s_cb[(w[u] >> (8 * q)) & 15u], m),
                                               fmaf(sg[u], s_cb[(w[u] >> (8 * q + 4)) & 15u], m));
          h[q] = *reinterpret_cast<const uint32_t*>(&r2);
        }
      } else {
        const __half2 f2 = __floats2half2_rn(sg[u], m);
        const __half2 s2 = __low2half2(f2), m2 = __high2half2(f2);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const __half2 v2 = __halves2half2(s_cb[(w[u] >> (8 * q)) & 15u], s_cb[(w[u] >> (8 * q + 4)) & 15u]);
          const __half2 r2 = __hfma2(s2, v2, m2);
          h[q] = *reinterpret_cast<const uint32_t*>(&r2);
        }
      }
      store(row[u], chunk[u], make_uint4(h[0], h[1], h[2], h[3]));
    }
  }
}

template <int BITS, typename CB>
__device__ __forceinline__ void unpack_weight_f16_chunks(const UnpackWeightJob& j, const CB* s_cb, long long first, long long stride) {
  unpack_weight_chunks<BITS>(j, s_cb, first, stride, [&](long long r, int ch, uint4 v) { *reinterpret_cast<uint4*>(j.out + r * j.K + ch * 8) = v; });
}

// Weights that a kernel of the activation path unpacks on the side: its first `blocks` blocks take the jobs (chunks split over
// their threads), the others do the kernel's own work.  The unpack then needs no launch and no second stream, and it runs
// beside the quantizer, on SMs that a small input leaves idle.
struct UnpackJobs {
  UnpackWeightJob job[2];
  int blocks;                // 0: none
};
// `block` of u.blocks; s_ucb: 32 words of shared memory, 16 for the levels of each job.
__device__ __forceinline__ void unpack_jobs_run(const UnpackJobs& u, int block, float* s_ucb) {
  const int tid = threadIdx.x;
  if (tid < 32) {
    const UnpackWeightJob& j = u.job[tid >> 4];
    const int i = tid & 15;
    const float level = j.packed != nullptr && i < (1 << j.bits) ? __ldg(j.codebook + i) : 0.0f;
    float* const cb = s_ucb + (tid & 16);
    if (j.fp32_form()) cb[i] = level;
    else reinterpret_cast<__half*>(cb)[i] = __float2half_rn(level);
  }
  __syncthreads();
  pdl_wait();                // the matrices written here may still be read by the kernel before this one
  const long long first = static_cast<long long>(block) * blockDim.x + tid, stride = static_cast<long long>(u.blocks) * blockDim.x;
#pragma unroll 1
  for (int k = 0; k < 2; ++k) {
    const UnpackWeightJob& j = u.job[k];
    if (j.packed == nullptr) break;
    const float* const cb = s_ucb + 16 * k;
    const __half* const cb16 = reinterpret_cast<const __half*>(cb);
    if (j.bits == 4) unpack_weight_f16_chunks<4>(j, cb16, first, stride);
    else if (j.fp32_form()) unpack_weight_f16_chunks<3>(j, cb, first, stride);
    else if (j.bits == 3) unpack_weight_f16_chunks<3>(j, cb16, first, stride);
    else unpack_weight_f16_chunks<2>(j, cb16, first, stride);
  }
}
__device__ __forceinline__ void unpack_jobs_block(const UnpackJobs& u) {
  __shared__ float s_ucb[32];
  unpack_jobs_run(u, static_cast<int>(blockIdx.x), s_ucb);
}

// The jobs on their own.
__global__ void __launch_bounds__(256) unpack_jobs_kernel(const __grid_constant__ UnpackJobs jobs) {
  pdl_launch_dependents();
  unpack_jobs_block(jobs);
}

template <int BITS>
__global__ void unpack_weight_f16_kernel(const uint8_t* __restrict__ packed, const float* __restrict__ mu,
                                         const float* __restrict__ sigma, const float* __restrict__ codesum,
                                         const float* __restrict__ codebook, long long rows, int K,
                                         __half* __restrict__ out) {
  __shared__ __half s_cb[16];
  if (threadIdx.x < 16) s_cb[threadIdx.x] = __float2half_rn((threadIdx.x < (1 << BITS)) ? codebook[threadIdx.x] : 0.0f);
  __syncthreads();
  const UnpackWeightJob j = {packed, mu, sigma, codesum, codebook, out, rows, K, BITS};
  unpack_weight_f16_chunks<BITS>(j, s_cb, blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x,
                                 static_cast<long long>(gridDim.x) * blockDim.x);
}

}  // namespace arcq
