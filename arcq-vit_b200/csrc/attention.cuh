// Multi-head self-attention for short sequences (ViT: 197 tokens, head width 64) on the fifth-generation tensor cores,
// optionally with the activation quantizer of the projection that consumes its output.
//   qkv  [B*T, 3*H*64] fp16: the output of the packed qkv linear (q | k | v, each H heads of 64)
//   out  [B*T, H*64] fp16:   softmax(q k^T / 8) v, heads side by side (the layout timm's Attention feeds to proj)
//   or   xhat [B*T, H*64] fp16: the ARCQ reconstruction of that matrix in groups of 64.  A head's 64 outputs of a
//        token are exactly one quantizer group, and one thread holds them.
//
// A work item is 128 queries of one (image, head); a block walks consecutive items, so that the second tile of a head finds
// its keys and values in shared memory.  The whole score row of a query (T <= 256 keys) fits tensor memory, so there is no
// online softmax and no rescaling: per item
//   S = Q K^T       128 x tk fp32 in tensor memory (tk: T rounded up to 16; the TMA fills the rows beyond T with zeros)
//   P = exp2(...)   a thread owns a query row: maximum, exponentials, sum; P as fp16 over the columns of S already read
//   O = P V         P from tensor memory, V from shared memory as it lies (keys outside, no transposition)
//   out             O / sum rounded to fp16, the quantizer of group_quant.cuh, 32 rows per warp to a TMA store
// Warps: 0-3 softmax and 4-7 output and quantizer (one tensor-memory lane quarter each), 8 TMA loads, 9 products.  Two blocks an
// SM, 256 tensor-memory columns each.  The next item's scores are computed, and its softmax runs, while this one's rows are
// quantised; the product with the upper half of the keys runs while the lower half's exponentials are computed.
//
// Tensor memory is allocated after the previous kernel has ended and before the next one may start: a GEMM that holds all of
// it while it waits for this kernel's result can then never be in the way.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>
#include "ptx.cuh"
#include "gemm_pair.cuh"
#include "act_quant.cuh"
#include "group_quant.cuh"

namespace arcq {

constexpr int kStatusAttentionTimeout = 0x501;
constexpr int kAttnRowWarps = 4;                  // softmax warps, and as many output warps
constexpr int kAttnThreads = 3 * 128;             // the third warp group: TMA and products
// Registers a thread, moved between the warp groups once they are running; the sum is that of the launch (80 each)
constexpr int kAttnLaunchRegs = 80, kAttnSoftmaxRegs = 72, kAttnOutputRegs = 120, kAttnIssueRegs = 48;
static_assert(kAttnSoftmaxRegs + kAttnOutputRegs + kAttnIssueRegs <= 3 * kAttnLaunchRegs, "registers beyond the launch's never come");
constexpr int kAttnMaxT = 256;
constexpr int kAttnQueries = 128;                 // per work item
// Tensor memory of an item: S in columns 0 .. tk-1.  P takes the first half of the columns of the part of S that it was made
// from: keys below attn_split(tk) at column 0, the others from column attn_split(tk) on.  O at 192, where S and P have ended
// once the upper part has been read.
constexpr uint32_t kAttnTmemCols = 256, kAttnOutCol = 192;
__host__ __device__ constexpr int attn_split(int tk) { return tk < 32 ? tk : (tk / 2 + 31) / 32 * 32; }

struct AttnParams {
  int T, H;
  int tk;                      // T rounded up to 16: keys of the products
  int qtiles;                  // work items of a head
  int items;                   // of all heads of all images
  const float* thresholds;     // quantizer form only
  const float* codebook;
  int one_fma;
  uint32_t poll_limit;         // waits of one warp for another give up after this many polls
  int* status;
};

struct AttnSmem {
  uint32_t q, k, v, stage, tables, sums, bars, total;
};
__host__ __device__ inline AttnSmem attn_smem_layout(int tk) {
  AttnSmem s;
  s.q = 0;
  s.k = s.q + kAttnQueries * 128;
  s.v = s.k + static_cast<uint32_t>(tk) * 128;              // tk * 128 is a multiple of 2 KB
  s.stage = s.v + static_cast<uint32_t>(tk) * 128;
  s.tables = s.stage + kAttnRowWarps * 4096;
  s.sums = s.tables + (static_cast<uint32_t>(sizeof(GroupQuantTables)) + 15) / 16 * 16;
  s.bars = s.sums + kAttnQueries * 4;
  s.total = s.bars + 16 * 8 + 16 + 1024 /* alignment */;
  return s;
}

__device__ __forceinline__ void tma_load_3d(void* smem_dst, const void* tmap, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tma_store_3d(const void* tmap, const void* smem_src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(tmap)),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z)
               : "memory");
}
// D[tmem] (+)= A[tmem, fp16 pairs] * B[smem]; issued by one thread
__device__ __forceinline__ void umma_f16_tmem_a(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float exp2_approx(float x) {
  float d;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(d) : "f"(x));
  return d;
}

template <bool QUANT, int BITS>
__global__ void __launch_bounds__(kAttnThreads, 2)
    attention_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_kv,
                     const __grid_constant__ CUtensorMap tm_out, const AttnParams p) {
  extern __shared__ uint8_t attn_smem_raw[];
  uint8_t* const smem = attn_smem_raw + ((1024u - (smem_u32(attn_smem_raw) & 1023u)) & 1023u);
  const AttnSmem L = attn_smem_layout(p.tk);
  uint64_t* const bars = reinterpret_cast<uint64_t*>(smem + L.bars);
  uint64_t *const q_full = bars, *const q_free = bars + 1, *const k_full = bars + 2, *const k_free = bars + 3,
           *const v_full = bars + 4, *const v_free = bars + 5, *const s_full = bars + 6, *const o_full = bars + 7,
           *const p_upper = bars + 8, *const p_lower = bars + 9, *const o_read = bars + 10, *const stopped = bars + 11;
  uint32_t* const s_tmem = reinterpret_cast<uint32_t*>(bars + 16);
  float* const s_sums = reinterpret_cast<float*>(smem + L.sums);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int T = p.T, C = p.H * 64;
  const int grid = static_cast<int>(gridDim.x), block = static_cast<int>(blockIdx.x);
  const int first = static_cast<int>(1ll * p.items * block / grid), last = static_cast<int>(1ll * p.items * (block + 1) / grid);
  // head of an item (image, first column), first query
  auto place = [&](int it, int* b, int* x) {
    const int head = it / p.qtiles;
    *b = head / p.H;
    *x = (head - *b * p.H) * 64;
    return (it - head * p.qtiles) * kAttnQueries;
  };

  if (tid == 0) {
    for (int i = 0; i < 8; ++i) mbar_init(bars + i, 1);
    for (int i = 8; i < 11; ++i) mbar_init(bars + i, kAttnRowWarps);
    mbar_init(stopped, 1);
    mbar_fence_init();
  }
  __syncthreads();
  const uint32_t polls = p.poll_limit;
  bool ok = true;

  if (warp >= 8) {
    fewer_registers<kAttnIssueRegs>();
    if (warp == 8) {
      // ---------------------------------------------------------------- TMA loads
      if (lane == 0) {
        tma_prefetch_desc(&tm_q);
        tma_prefetch_desc(&tm_kv);
        tma_prefetch_desc(&tm_out);
      }
      pdl_wait();
      uint32_t heads = 0, q_loads = 0, k_loads = 0;
      auto loads = [&](int it) {
        const uint32_t i = static_cast<uint32_t>(it - first);
        int b, x;
        const int q0 = place(it, &b, &x);
        if (i > 0 && !mbar_wait(q_free, (i - 1) & 1, polls)) return false;
        mbar_arrive_expect_tx(q_full, kAttnQueries * 128);
        tma_load_3d(smem + L.q, &tm_q, q_full, x, q0, b);
        ++q_loads;
        if (i == 0 || q0 == 0) {
          if (heads > 0 && !mbar_wait(k_free, (heads - 1) & 1, polls)) return false;
          mbar_arrive_expect_tx(k_full, static_cast<uint32_t>(p.tk) * 128);
          tma_load_3d(smem + L.k, &tm_kv, k_full, C + x, 0, b);
          ++k_loads;
          if (heads > 0 && !mbar_wait(v_free, (heads - 1) & 1, polls)) return false;
          mbar_arrive_expect_tx(v_full, static_cast<uint32_t>(p.tk) * 128);
          tma_load_3d(smem + L.v, &tm_kv, v_full, 2 * C + x, 0, b);
          ++heads;
        }
        return true;
      };
      if (lane == 0) ok = loads(first);
      __syncwarp();
      __syncthreads();                    // tensor memory allocated
      pdl_launch_dependents();
      if (lane == 0) {
        for (int it = first + 1; it < last && ok; ++it) ok = loads(it);
        // No copy may land after the block has left, whichever warp has given up: the last one of each kind.
        ok &= mbar_wait(q_full, (q_loads - 1) & 1) && mbar_wait(k_full, (k_loads - 1) & 1) && mbar_wait(v_full, (heads - 1) & 1);
        if (!ok) atomicExch(p.status, kStatusAttentionTimeout);
      }
      __syncwarp();
    } else {
      // ---------------------------------------------------------------- products (warp 9); warps 10 and 11 only keep step
      if (warp == 9) {
        pdl_wait();
        tmem_alloc(s_tmem, kAttnTmemCols);
        tmem_relinquish();
        tc_fence_before_sync();
      }
      __syncthreads();
      pdl_launch_dependents();
      tc_fence_after_sync();
      if (warp == 9 && lane == 0) {
        const uint32_t tmem = *s_tmem;
        const uint32_t idesc_s = umma_idesc_f16(kAttnQueries, p.tk);
        const uint32_t idesc_o = umma_idesc_f16(kAttnQueries, 64) | (1u << 16);      // B with its rows (keys) along K
        const uint64_t dq = umma_desc_sw128(smem_u32(smem + L.q)), dk = umma_desc_sw128(smem_u32(smem + L.k)),
                       dv = umma_desc_sw128(smem_u32(smem + L.v));
        const int split = attn_split(p.tk);
        uint32_t heads = 0;
        for (int it = first; it < last; ++it) {
          const uint32_t i = static_cast<uint32_t>(it - first);
          const int q_tile = it % p.qtiles;
          const bool new_head = i == 0 || q_tile == 0, end_head = it + 1 == last || q_tile + 1 == p.qtiles;
          heads += new_head ? 1 : 0;
          ok = (!new_head || mbar_wait(k_full, (heads - 1) & 1, polls)) && mbar_wait(q_full, i & 1, polls) &&
               (i == 0 || mbar_wait(o_read, (i - 1) & 1, polls));
          if (!ok) break;
          tc_fence_after_sync();
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_f16(tmem, dq + 2 * k, dk + 2 * k, idesc_s, k > 0);
          umma_commit(s_full);
          umma_commit(q_free);
          if (end_head) umma_commit(k_free);
          ok = (!new_head || mbar_wait(v_full, (heads - 1) & 1, polls)) && mbar_wait(p_upper, i & 1, polls);
          if (!ok) break;
          tc_fence_after_sync();
          uint32_t acc = 0;
          for (int k = split; k < p.tk; k += 16, acc = 1)
            umma_f16_tmem_a(tmem + kAttnOutCol, tmem + split + (k - split) / 2, dv + 8 * k, idesc_o, acc);
          ok = mbar_wait(p_lower, i & 1, polls);
          if (!ok) break;
          tc_fence_after_sync();
          for (int k = 0; k < split; k += 16, acc = 1) umma_f16_tmem_a(tmem + kAttnOutCol, tmem + k / 2, dv + 8 * k, idesc_o, acc);
          umma_commit(o_full);
          if (end_head) umma_commit(v_free);
        }
        if (!ok) {
          // products that were issued end before their tensor memory is given back
          umma_commit(stopped);
          mbar_wait(stopped, 0);
          atomicExch(p.status, kStatusAttentionTimeout);
        }
      }
      __syncwarp();
    }
  } else if (warp < kAttnRowWarps) {
    // ------------------------------------------------------------------ softmax: a thread per query row
    fewer_registers<kAttnSoftmaxRegs>();
    __syncthreads();
    pdl_launch_dependents();
    tc_fence_after_sync();
    const uint32_t slot = *s_tmem + (static_cast<uint32_t>(warp * 32) << 16);
    constexpr float kScale = 0.125f * 1.44269504088896340736f;             // 1 / sqrt(64) and base 2
    const int split = attn_split(p.tk), tk = p.tk;
    const float ninf = __int_as_float(0xff800000);
    for (int it = first; it < last; ++it) {
      const uint32_t ph = static_cast<uint32_t>(it - first) & 1;
      const bool live = (it % p.qtiles) * kAttnQueries + warp * 32 < T;    // some of the warp's rows are queries
      if (!mbar_wait(s_full, ph, polls)) { ok = false; break; }
      tc_fence_after_sync();
      // Loops with one body each, not unrolled over the row: the softmax and output warps of two blocks share an instruction
      // cache, and unrolled passes stalled on it more than on anything else (DeiT-S batch 64, with the quantizer: 27.0 -> 24.1 us).
      // The wait loops are part of that: with a constant limit instead of poll_limit 24.3 us against 21.4, 256 images of 12 heads 146
      // against 113.
      float nm = 0.0f;
      if (live) {
        float m0 = ninf, m1 = ninf, m2 = ninf, m3 = ninf;
        uint32_t s[2][32];
        int c = 0;
#pragma unroll 1
        for (; c + 64 <= T; c += 64) {
          tmem_ld_32x32(slot + c, s[0]);
          tmem_ld_32x32(slot + c + 32, s[1]);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 64; j += 8) {
            m0 = max3(m0, __uint_as_float(s[j >> 5][j & 31]), __uint_as_float(s[j >> 5][(j & 31) + 1]));
            m1 = max3(m1, __uint_as_float(s[j >> 5][(j & 31) + 2]), __uint_as_float(s[j >> 5][(j & 31) + 3]));
            m2 = max3(m2, __uint_as_float(s[j >> 5][(j & 31) + 4]), __uint_as_float(s[j >> 5][(j & 31) + 5]));
            m3 = max3(m3, __uint_as_float(s[j >> 5][(j & 31) + 6]), __uint_as_float(s[j >> 5][(j & 31) + 7]));
          }
        }
#pragma unroll 1
        for (; c < T; c += 16) {
          uint32_t t[16];
          tmem_ld_32x16(slot + c, t);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; j += 2)
            m0 = max3(m0, c + j < T ? __uint_as_float(t[j]) : ninf, c + j + 1 < T ? __uint_as_float(t[j + 1]) : ninf);
        }
        nm = -kScale * fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
      }
      const f32x2 k2 = pack2(kScale, kScale), nm2 = pack2(nm, nm);
      f32x2 sum0 = pack2(0.0f, 0.0f), sum1 = sum0;
      // sixteen scores to fp16 probabilities
      auto exponentials = [&](const uint32_t* s, uint32_t* w) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float e0, e1;
          unpack2(fma2(pack2(__uint_as_float(s[2 * j]), __uint_as_float(s[2 * j + 1])), k2, nm2), e0, e1);
          const f32x2 e = pack2(exp2_approx(e0), exp2_approx(e1));
          if (j & 1) sum1 = add2(sum1, e); else sum0 = add2(sum0, e);
          w[j] = pair_to_sixteen<__half>(e);
        }
      };
#pragma unroll 1
      for (int part = 1; part >= 0; --part) {                              // upper keys first
        if (live) {
          int c = part ? split : 0, p_col = c;
          const int to = part ? tk : split;
#pragma unroll 1
          for (; c + 32 <= min(to, T); c += 32, p_col += 16) {
            uint32_t s[32], w[16];
            tmem_ld_32x32(slot + c, s);
            tmem_ld_wait();
            exponentials(s, w);
            exponentials(s + 16, w + 8);
            tmem_st_32x16(slot + p_col, w);                                // over columns of S that have been read
          }
#pragma unroll 1
          for (; c < to; c += 16, p_col += 8) {
            uint32_t s[16], w[8];
            tmem_ld_32x16(slot + c, s);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) s[j] = c + j < T ? s[j] : 0xff800000u;        // keys beyond T: minus infinity
            exponentials(s, w);
            tmem_st_32x8(slot + p_col, w);
          }
          if (part == 0) {
            float x0, x1;
            unpack2(add2(sum0, sum1), x0, x1);
            s_sums[warp * 32 + lane] = x0 + x1;
          }
          tmem_st_wait();
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(part ? p_upper : p_lower);
      }
    }
    if (!ok && lane == 0) atomicExch(p.status, kStatusAttentionTimeout);
  } else {
    // ------------------------------------------------------------------ output: a thread per query row
    more_registers<kAttnOutputRegs>();
    const int quarter = warp - kAttnRowWarps;
    GroupQuantTables* const tables = reinterpret_cast<GroupQuantTables*>(smem + L.tables);
    GroupQuantParams gp = {};
    // reads only the layer's constants: done while the previous kernel still runs
    if (QUANT)
      gp = group_quant_tables<1 << BITS, false>(tables, p.thresholds, p.codebook, tid - 128, kAttnRowWarps * 32, [](bool b) {
        asm volatile("bar.sync 1, %0;" ::"n"(kAttnRowWarps * 32) : "memory");
        return b;
      });
    __syncthreads();
    pdl_launch_dependents();
    tc_fence_after_sync();
    const uint32_t t_out = *s_tmem + (static_cast<uint32_t>(quarter * 32) << 16) + kAttnOutCol;
    uint8_t* const stage = smem + L.stage + quarter * 4096;
    const uint32_t row = smem_u32(stage) + lane * 128, x7 = lane & 7;
    for (int it = first; it < last; ++it) {
      const uint32_t ph = static_cast<uint32_t>(it - first) & 1;
      int b, x;
      const int t0 = place(it, &b, &x) + quarter * 32;
      const bool live = t0 < T;
      // p_lower: the sums are there
      if (!mbar_wait(p_lower, ph, polls) || !mbar_wait(o_full, ph, polls)) { ok = false; break; }
      tc_fence_after_sync();
      uint32_t w[32];
      if (live) {
        const float inv = __frcp_rn(s_sums[quarter * 32 + lane]);
        const f32x2 inv2 = pack2(inv, inv);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t o[32];
          tmem_ld_32x32(t_out + 32 * h, o);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j)
            w[16 * h + j] = pair_to_sixteen<__half>(mul2(pack2(__uint_as_float(o[2 * j]), __uint_as_float(o[2 * j + 1])), inv2));
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(o_read);
        tma_store_wait_read();                             // the store that last used the staging rows has read them
      }
      __syncwarp();
      if (live) {
        if (QUANT) {
          f32x2 v[32];
          uint32_t words[8];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = sixteen_to_pair<__half>(w[j]);
          const GroupStats st = group_quantize<BITS, false, 1>(v, tables, gp, words);
          const GroupRecon g = group_recon(st, gp, p.one_fma != 0);
#pragma unroll
          for (int j = 0; j < 32; ++j) w[j] = pair_to_sixteen<__half>(group_recon_pair(g, v[j]));
        }
        row_store<1>(w, row, x7);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_3d(&tm_out, stage, x, t0, b);          // tokens beyond T are clipped
          tma_store_commit();
        }
      }
    }
    if (lane == 0) tma_store_wait_all();
    if (!ok && lane == 0) atomicExch(p.status, kStatusAttentionTimeout);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after_sync();
    tmem_dealloc(*s_tmem, kAttnTmemCols);
  }
}

}  // namespace arcq
