// Activation quantizer for large inputs (group_quant.cuh): each warp works on its own tiles of 32 groups.  It brings
// a tile in by TMA (a row per group, 128-byte swizzle, so that lanes read their rows without bank conflicts), quantises it in place and sends the reconstruction out by TMA, with the next tile's load and the previous
// tile's store in flight meanwhile.  No block-wide synchronisation after the table set-up.
//
// Bound by issue slots (half of them used: fixed latencies and instruction fetches of the straight-line group routine), then by
// shared-memory reads (about three wavefronts per 32 values).  One lane a group, 16 warps an SM.  [12608, 384] 4.9 us, [50432,
// 768] 28.7 us (5.4 TB/s), with GELU [12608, 1536] 25.1 us; 6.3, 31.2 and 24.5 us when a level took three table reads and a value
// at a threshold sent its seven neighbours through the exact path too.  Groups whose values are all equal, those beyond the matrix in the
// last tile among them, take that path for every value if a threshold is 0 (group_quant.cuh): [3001, 3072] with such a codebook 24.6 us.
#pragma once
#include <cuda.h>
#include "ptx.cuh"
#include "group_quant.cuh"
#include "codes.cuh"

namespace arcq {

constexpr int kStatusActQuantTimeout = 0x401;

template <typename T, bool WRITE_PACKED> struct AqtShape {
  static constexpr int kLpg = 1;
  static constexpr int kWarps = 4, kThreads = kWarps * 32;
  static constexpr int kGroups = 32 / kLpg;                                   // per warp and tile
  static constexpr int kTile = kGroups * 64 * static_cast<int>(sizeof(T));    // bytes
  static constexpr int kBufs = sizeof(T) == 2 ? 3 : 2;                        // tiles a warp cycles through
  static constexpr int kTables = kWarps * kBufs * kTile;                      // a multiple of 1 KB
  static constexpr int kBars = kTables + (static_cast<int>(sizeof(GroupQuantTables)) + 15) / 16 * 16;
  static constexpr int kSmem = 1024 /* alignment */ + kBars + kWarps * kBufs * 8;
  static constexpr int kBlocksPerSm = sizeof(T) == 4 ? 3 : 4;
};

// XH: element type of the reconstruction: T or fp16.  PRE = 1: GELU first (fp16 input).
template <typename T, int BITS, typename XH, bool WRITE_XHAT, int PRE, bool WRITE_PACKED>
__global__ void __launch_bounds__(AqtShape<T, WRITE_PACKED>::kThreads, AqtShape<T, WRITE_PACKED>::kBlocksPerSm)
    act_quant_tile_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_out,
                          long long total_groups, const float* __restrict__ thresholds, const float* __restrict__ codebook,
                          uint8_t* __restrict__ packed, float* __restrict__ mu_out, float* __restrict__ sigma_out,
                          float* __restrict__ codesum_out, int one_fma, int* status, const __grid_constant__ UnpackJobs jobs) {
  pdl_launch_dependents();   // the next kernel of the stream may start its set-up
  if (static_cast<int>(blockIdx.x) < jobs.blocks) {
    unpack_jobs_block(jobs);
    return;
  }
  using S = AqtShape<T, WRITE_PACKED>;
  constexpr int L = 1 << BITS, LPG = S::kLpg, PJ = 4 / LPG, kTile = S::kTile, kBufs = S::kBufs, kGroups = S::kGroups;
  static_assert(PRE == 0 || sizeof(T) == 2, "the GELU takes fp16");
  extern __shared__ uint8_t aqt_smem_raw[];
  uint8_t* const smem = aqt_smem_raw + ((1024u - (smem_u32(aqt_smem_raw) & 1023u)) & 1023u);
  GroupQuantTables* const tables = reinterpret_cast<GroupQuantTables*>(smem + S::kTables);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int gl = lane / LPG, h = LPG == 2 ? lane & 1 : 0;            // group of the tile, lane of the group
  uint8_t* const bufs = smem + warp * kBufs * kTile;
  uint64_t* const full = reinterpret_cast<uint64_t*>(smem + S::kBars) + warp * kBufs;
  if (lane == 0) {
    for (int i = 0; i < kBufs; ++i) mbar_init(&full[i], 1);
    mbar_fence_init();
    tma_prefetch_desc(&tm_x);
    if (WRITE_XHAT) tma_prefetch_desc(&tm_out);
  }
  // reads only the layer's constants, which no kernel of this library writes: done while the previous kernel still runs
  const GroupQuantParams gp = group_quant_tables<L, WRITE_PACKED>(tables, thresholds, codebook, tid, S::kThreads,
                                                    [](bool b) { return __syncthreads_and(b) != 0; });
  const long long tiles = (total_groups + kGroups - 1) / kGroups;
  const long long stride = static_cast<long long>(gridDim.x - jobs.blocks) * S::kWarps;
  long long tile = static_cast<long long>(blockIdx.x - jobs.blocks) * S::kWarps + warp;
  constexpr int kRowsPerGroup = sizeof(T) == 2 ? 1 : 2;              // 128-byte rows
  auto load = [&](long long t, int b) {
    mbar_arrive_expect_tx(&full[b], kTile);
    tma_load_2d(bufs + b * kTile, &tm_x, &full[b], 0, static_cast<int>(t * (kGroups * kRowsPerGroup)));
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
    const uint32_t base = smem_u32(bufs + buf * kTile);
    const uint32_t row = base + gl * 128 + 8 * h, x7 = gl & 7;       // 16-bit rows: this lane's part
    // fp32 rows: value chunk c (four values) of the group sits in row 2 gl + c / 8
    auto chunk32 = [&](int c) { return base + (2 * gl + (c >> 3)) * 128 + (((c & 7) ^ ((2 * gl + (c >> 3)) & 7)) << 4); };
    f32x2 v[32 / LPG];
    if constexpr (sizeof(T) == 2) {
      uint32_t w[32 / LPG];
      row_load<LPG>(w, row, x7);
      if (PRE == 1) gelu_words<LPG>(w, row, x7);
#pragma unroll
      for (int i = 0; i < 32 / LPG; ++i) v[i] = sixteen_to_pair<T>(w[i]);
    } else {
#pragma unroll
      for (int c = 0; c < 16 / LPG; ++c) {
        const uint4 u = lds128(chunk32(LPG * c + h));
        v[2 * c] = pack2(__uint_as_float(u.x), __uint_as_float(u.y));
        v[2 * c + 1] = pack2(__uint_as_float(u.z), __uint_as_float(u.w));
      }
    }
    uint32_t words[8];
    const GroupStats st = group_quantize<BITS, WRITE_PACKED, LPG>(v, tables, gp, words);
    const long long gi = tile * kGroups + gl;
    if (gi < total_groups && h == 0) {
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
      const GroupRecon g = group_recon(st, gp, one_fma != 0);
      if constexpr (sizeof(XH) == 2) {
        if (sizeof(T) == 4) __syncwarp();                    // the fp16 rows overlap other lanes' fp32 rows
        uint32_t w[32 / LPG];
#pragma unroll
        for (int i = 0; i < 32 / LPG; ++i) w[i] = pair_to_sixteen<XH>(group_recon_pair(g, v[i]));
        row_store<LPG>(w, row, x7);
      } else {
#pragma unroll
        for (int c = 0; c < 16 / LPG; ++c) {
          float f0, f1, f2, f3;
          unpack2(group_recon_pair(g, v[2 * c]), f0, f1);
          unpack2(group_recon_pair(g, v[2 * c + 1]), f2, f3);
          sts128(chunk32(LPG * c + h), __float_as_uint(f0), __float_as_uint(f1), __float_as_uint(f2), __float_as_uint(f3));
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_2d(&tm_out, bufs + buf * kTile, 0, static_cast<int>(tile * (kGroups * (sizeof(XH) == 2 ? 1 : 2))));
        tma_store_commit();
      }
    } else {
      if (PRE == 1) fence_proxy_async_smem();                 // the GELU may have written to it
      __syncwarp();                                           // every lane has read its row before the buffer is refilled
    }
    if (next_buf == 0) ph ^= 1;
    buf = next_buf;
  }
  if (WRITE_XHAT && lane == 0) tma_store_wait_all();
}

}  // namespace arcq
