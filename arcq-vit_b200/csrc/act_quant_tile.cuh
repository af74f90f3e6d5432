// Activation quantizer for large inputs: one thread per 64-value group (group_quant.cuh), a warp per 32 groups, each warp on
// its own: it brings its tile in by TMA (32 rows of one group, 128-byte swizzle, so that a thread reads its row without bank
// conflicts), quantises it in place and sends the reconstruction out by TMA, with the next tile's load and the previous
// tile's store in flight meanwhile.  No block-wide synchronisation after the table set-up.
//
// Bound by issue slots (15 to 16 instructions per value, 23 with the GELU), then by shared-memory reads (about four
// wavefronts per 32 values); memory is half idle.
#pragma once
#include <cuda.h>
#include "ptx.cuh"
#include "group_quant.cuh"

namespace arcq {

constexpr int kAqtWarps = 4, kAqtThreads = kAqtWarps * 32;
constexpr int kStatusActQuantTimeout = 0x401;

template <typename T> struct AqtTile {          // bytes of 32 group rows, and how many of them a warp cycles through
  static constexpr int kBytes = 32 * 64 * static_cast<int>(sizeof(T)), kBufs = sizeof(T) == 2 ? 3 : 2;
};
template <typename T> __host__ __device__ constexpr size_t aqt_smem_bytes() {
  return 1024 /* alignment */ + static_cast<size_t>(kAqtWarps) * AqtTile<T>::kBytes * AqtTile<T>::kBufs +
         sizeof(GroupQuantTables) + 16 + kAqtWarps * AqtTile<T>::kBufs * 8;
}

template <typename T> __device__ __forceinline__ f32x2 sixteen_to_pair(uint32_t w);
template <> __device__ __forceinline__ f32x2 sixteen_to_pair<__half>(uint32_t w) { return half2_to_pair(w); }
template <> __device__ __forceinline__ f32x2 sixteen_to_pair<__nv_bfloat16>(uint32_t w) {
  return pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
}
template <typename T> __device__ __forceinline__ uint32_t pair_to_sixteen(f32x2 v);
template <> __device__ __forceinline__ uint32_t pair_to_sixteen<__half>(f32x2 v) { return pair_to_half2(v); }
template <> __device__ __forceinline__ uint32_t pair_to_sixteen<__nv_bfloat16>(f32x2 v) {
  float a, b;
  unpack2(v, a, b);
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// XH: element type of the reconstruction: T, or fp16 for an fp32 input.  PRE = 1: GELU first (fp16 input).
template <typename T, int BITS, typename XH, bool WRITE_XHAT, int PRE, bool WRITE_PACKED>
__global__ void __launch_bounds__(kAqtThreads, 4)
    act_quant_tile_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_out,
                          long long total_groups, const float* __restrict__ thresholds, const float* __restrict__ codebook,
                          uint8_t* __restrict__ packed, float* __restrict__ mu_out, float* __restrict__ sigma_out,
                          float* __restrict__ codesum_out, int* status) {
  pdl_launch_dependents();   // the next kernel of the stream may start its set-up
  constexpr int kTile = AqtTile<T>::kBytes, kBufs = AqtTile<T>::kBufs, L = 1 << BITS;
  static_assert(PRE == 0 || sizeof(T) == 2, "the GELU takes fp16");
  extern __shared__ uint8_t aqt_smem_raw[];
  uint8_t* const smem = aqt_smem_raw + ((1024u - (smem_u32(aqt_smem_raw) & 1023u)) & 1023u);
  GroupQuantTables* const tables = reinterpret_cast<GroupQuantTables*>(smem + kAqtWarps * kBufs * kTile);
  uint64_t* const bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(tables) + (sizeof(GroupQuantTables) + 15) / 16 * 16);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint8_t* const bufs = smem + warp * kBufs * kTile;
  uint64_t* const full = bars + warp * kBufs;
  if (lane == 0) {
    for (int i = 0; i < kBufs; ++i) mbar_init(&full[i], 1);
    mbar_fence_init();
    tma_prefetch_desc(&tm_x);
    if (WRITE_XHAT) tma_prefetch_desc(&tm_out);
  }
  // reads only the layer's constants, which no kernel of this library writes: done while the previous kernel still runs
  const GroupQuantParams gp = group_quant_tables<L>(tables, thresholds, codebook, tid, kAqtThreads,
                                                    [](bool b) { return __syncthreads_and(b) != 0; });
  const long long tiles = (total_groups + 31) >> 5;
  const long long stride = static_cast<long long>(gridDim.x) * kAqtWarps;
  long long tile = static_cast<long long>(blockIdx.x) * kAqtWarps + warp;
  auto load = [&](long long t, int b) {
    mbar_arrive_expect_tx(&full[b], kTile);
    tma_load_2d(bufs + b * kTile, &tm_x, &full[b], 0, static_cast<int>(sizeof(T) == 2 ? t * 32 : t * 64));
  };
  pdl_wait();
  if (lane == 0 && tile < tiles) load(tile, 0);
  int buf = 0;
  uint32_t ph = 0;
  for (; tile < tiles; tile += stride) {
    const int next_buf = buf + 1 == kBufs ? 0 : buf + 1;
    if (lane == 0 && tile + stride < tiles) {
      if (WRITE_XHAT) tma_store_wait_read_n<kBufs - 2>();     // the store that last used that buffer has read it
      load(tile + stride, next_buf);
    }
    if (!mbar_wait(&full[buf], ph)) {
      if (lane == 0) atomicExch(status, kStatusActQuantTimeout);
      break;
    }
    const uint32_t row = smem_u32(bufs + buf * kTile);
    f32x2 v[32];
    if constexpr (sizeof(T) == 2) {
      const uint32_t r = row + lane * 128, x7 = lane & 7;
      uint4 ch[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) ch[c] = lds128(r + ((c ^ x7) << 4));
      if (PRE == 1) gelu_row(ch, r, x7);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        v[4 * c] = sixteen_to_pair<T>(ch[c].x);
        v[4 * c + 1] = sixteen_to_pair<T>(ch[c].y);
        v[4 * c + 2] = sixteen_to_pair<T>(ch[c].z);
        v[4 * c + 3] = sixteen_to_pair<T>(ch[c].w);
      }
    } else {
      // a group is two 128-byte rows of the tile
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const uint32_t rr = 2 * lane + (c >> 3);
        const uint4 u = lds128(row + rr * 128 + (((c & 7) ^ (rr & 7)) << 4));
        v[2 * c] = pack2(__uint_as_float(u.x), __uint_as_float(u.y));
        v[2 * c + 1] = pack2(__uint_as_float(u.z), __uint_as_float(u.w));
      }
    }
    uint32_t words[8];
    const GroupStats st = group_quantize<BITS, WRITE_PACKED>(v, tables, gp, words);
    const long long gi = tile * 32 + lane;
    if (gi < total_groups) {
      if (WRITE_PACKED) {
        if (BITS == 4) {
          uint4* o = reinterpret_cast<uint4*>(packed + gi * 32);
          o[0] = make_uint4(words[0], words[1], words[2], words[3]);
          o[1] = make_uint4(words[4], words[5], words[6], words[7]);
        } else if (BITS == 3) {
          uint32_t ow[6];
#pragma unroll
          for (int p2 = 0; p2 < 2; ++p2) {                               // 4 chunks (12 bytes) -> 3 words
            const uint32_t a = squeeze_nibbles_3(words[4 * p2]), b = squeeze_nibbles_3(words[4 * p2 + 1]);
            const uint32_t c2 = squeeze_nibbles_3(words[4 * p2 + 2]), d = squeeze_nibbles_3(words[4 * p2 + 3]);
            ow[3 * p2] = a | (b << 24);
            ow[3 * p2 + 1] = (b >> 8) | (c2 << 16);
            ow[3 * p2 + 2] = (c2 >> 16) | (d << 8);
          }
          uint2* o2 = reinterpret_cast<uint2*>(packed + gi * 24);        // 24 bytes per group: 8-byte aligned
          o2[0] = make_uint2(ow[0], ow[1]);
          o2[1] = make_uint2(ow[2], ow[3]);
          o2[2] = make_uint2(ow[4], ow[5]);
        } else {
          uint32_t ow[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) ow[c] = squeeze_nibbles_2(words[2 * c]) | (squeeze_nibbles_2(words[2 * c + 1]) << 16);
          *reinterpret_cast<uint4*>(packed + gi * 16) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
        }
      }
      if (mu_out != nullptr) {
        mu_out[gi] = st.mean;
        sigma_out[gi] = st.scale;
        if (codesum_out != nullptr) codesum_out[gi] = st.code_sum;
      }
    }
    if (WRITE_XHAT) {
      const GroupRecon g = group_recon(st, gp);
      if constexpr (sizeof(XH) == 2) {
        if (sizeof(T) == 4) __syncwarp();                    // the fp16 rows overlap other threads' fp32 rows
        const uint32_t r = row + lane * 128, x7 = lane & 7;
#pragma unroll
        for (int c = 0; c < 8; ++c)
          sts128(r + ((c ^ x7) << 4), pair_to_sixteen<XH>(group_recon_pair(g, v[4 * c])),
                 pair_to_sixteen<XH>(group_recon_pair(g, v[4 * c + 1])), pair_to_sixteen<XH>(group_recon_pair(g, v[4 * c + 2])),
                 pair_to_sixteen<XH>(group_recon_pair(g, v[4 * c + 3])));
      } else {
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          const uint32_t rr = 2 * lane + (c >> 3);
          float f0, f1, f2, f3;
          unpack2(group_recon_pair(g, v[2 * c]), f0, f1);
          unpack2(group_recon_pair(g, v[2 * c + 1]), f2, f3);
          sts128(row + rr * 128 + (((c & 7) ^ (rr & 7)) << 4), __float_as_uint(f0), __float_as_uint(f1), __float_as_uint(f2),
                 __float_as_uint(f3));
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_2d(&tm_out, bufs + buf * kTile, 0, static_cast<int>(sizeof(XH) == 2 ? tile * 32 : tile * 64));
        tma_store_commit();
      }
    } else {
      __syncwarp();                                           // every lane has read its row before the buffer is refilled
    }
    if (next_buf == 0) ph ^= 1;
    buf = next_buf;
  }
  if (WRITE_XHAT && lane == 0) tma_store_wait_all();
}

}  // namespace arcq
