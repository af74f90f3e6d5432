// Multi-head self-attention for short sequences (ViT: 197 tokens, head width 64) on the fifth-generation tensor cores,
// optionally with the activation quantizer of the projection that consumes its output.
//   qkv  [B*T, 3*H*64] fp16: the output of the packed qkv linear (q | k | v, each H heads of 64)
//   out  [B*T, H*64] fp16:   softmax(q k^T / 8) v, heads side by side (the layout timm's Attention feeds to proj)
//   or   xhat [B*T, H*64] fp16: the ARCQ reconstruction of that matrix in groups of 64.  A head's 64 outputs of a
//        token are exactly one quantizer group, and one thread holds them.
//
// A work item is 128 queries of one (image, head); a block (one an SM) walks consecutive items, so that the second tile of a head finds
// its keys and values in shared memory.  The whole score row of a query (T <= 256 keys) fits tensor memory, so there is no
// online softmax and no rescaling: per item
//   S = Q K^T       128 x tk fp32 in tensor memory (tk: T rounded up to 16; the TMA fills the rows beyond T with zeros)
//   P = exp2(...)   two threads share a query row, one the lower keys, one the upper: maximum (exchanged through shared memory),
//                   exponentials, sums; P as fp16 over the columns of S already read
//   O = P V         P from tensor memory, V from shared memory as it lies (keys outside, no transposition)
//   out             O / sum rounded to fp16, the quantizer of group_quant.cuh, 32 rows per warp to a TMA store
// Warps (a tensor-memory lane quarter each): 0-3 upper keys, 4-7 lower keys, 8-11 and 12-15 output and quantizer of the even and of the
// odd items, 16 TMA loads, 17 products.
//
// Tensor memory holds two items, 256 columns each: while the softmax warps work on one, the other's product runs, its output is read
// and the scores of the item after the next are computed, so that the softmax warps go from item to item without a wait: 3700 cycles
// an item (maximum 600, exponentials 2100 alone and 2700 beside the output warps).  What is left is the exponentials' pipe, 8 cycles a
// warp or 1664 an item, issue slots, about 2400 an item, and instruction fetches.  With quantizer, 197 tokens: 64 images of 6 heads
// 20.0 -> 18.1 us, 32 images 14.3 -> 11.5, 256 images of 12 heads 112 -> 102, one image 7.7 -> 7.3, against two blocks an SM with one item
// each and a thread per row, whose softmax warps waited for P V, for the read of O and for the next Q K^T.
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
constexpr int kAttnRowWarps = 4;                  // of a group: a warp a tensor-memory lane quarter
constexpr int kAttnThreads = 5 * 128;             // two softmax groups, two output groups; the last: TMA and products
// Registers a thread, moved between the warp groups once they are running; the sum is that of a launch with 80 each
constexpr int kAttnLaunchRegs = 80, kAttnSoftmaxRegs = 80, kAttnOutputRegs = 96, kAttnIssueRegs = 48;
static_assert(2 * kAttnSoftmaxRegs + 2 * kAttnOutputRegs + kAttnIssueRegs <= 5 * kAttnLaunchRegs, "registers beyond the launch's never come");
constexpr int kAttnMaxT = 256;
constexpr int kAttnQueries = 128;                 // per work item
// Tensor memory of an item: S in columns 0 .. tk-1.  P takes the first half of the columns of the part of S that it was made
// from: keys below attn_split(tk) at column 0, the others from column attn_split(tk) on.  O at 192, where S and P have ended
// once the upper part has been read.
constexpr uint32_t kAttnTmemCols = 512, kAttnItemCols = 256, kAttnOutCol = 192;
__host__ __device__ constexpr int attn_split(int tk) { return tk < 32 ? tk : tk < 64 ? (tk / 2 + 15) / 16 * 16 : tk / 64 * 32; }

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
  uint32_t q, k, v, stage, tables, max, sums, bars, total;
};
__host__ __device__ inline AttnSmem attn_smem_layout(int tk) {
  AttnSmem s;                                               // q, k, v, max and sums twice: even and odd items (k, v: heads)
  s.q = 0;
  s.k = s.q + 2 * kAttnQueries * 128;
  s.v = s.k + 2 * static_cast<uint32_t>(tk) * 128;          // tk * 128 is a multiple of 2 KB
  s.stage = s.v + 2 * static_cast<uint32_t>(tk) * 128;
  s.tables = s.stage + 2 * kAttnRowWarps * 4096;
  s.max = s.tables + kGroupQuantTableBytes;
  s.sums = s.max + 4 * kAttnQueries * 4;
  s.bars = s.sums + 4 * kAttnQueries * 4;
  s.total = s.bars + 24 * 8 + 16 + 1024 /* alignment */;
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
// D[tmem] (+)= A[tmem, fp16 pairs] * B[smem]; issued by one thread.  Operands in shared memory by the low words of their descriptors
// (gemm_pair.cuh).
__device__ __forceinline__ void umma_f16_tmem_a_lo(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
      "mov.b64 db, {%2, %5};\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(kDescHi)
      : "memory");
}
// D[tmem] = A . B^T over the four 16-wide K steps of one 64-wide sub-tile
__device__ __forceinline__ void umma_f16_x4(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .b32 al, bl;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %4};\n\t"
      "mov.b64 db, {%2, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, 0;\n\t"
      "add.u32 al, %1, 2;\n\tadd.u32 bl, %2, 2;\n\tmov.b64 da, {al, %4};\n\tmov.b64 db, {bl, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, 1;\n\t"
      "add.u32 al, %1, 4;\n\tadd.u32 bl, %2, 4;\n\tmov.b64 da, {al, %4};\n\tmov.b64 db, {bl, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, 1;\n\t"
      "add.u32 al, %1, 6;\n\tadd.u32 bl, %2, 6;\n\tmov.b64 da, {al, %4};\n\tmov.b64 db, {bl, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, 1;\n\t}" ::"r"(d_tmem),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(kDescHi)
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
__global__ void __launch_bounds__(kAttnThreads, 1)
    attention_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_kv,
                     const __grid_constant__ CUtensorMap tm_out, const AttnParams p) {
  extern __shared__ uint8_t attn_smem_raw[];
  uint8_t* const smem = attn_smem_raw + ((1024u - (smem_u32(attn_smem_raw) & 1023u)) & 1023u);
  const AttnSmem L = attn_smem_layout(p.tk);
  uint64_t* const bars = reinterpret_cast<uint64_t*>(smem + L.bars);
  // [2] each, by the parity of the item (k, v: of the head)
  uint64_t *const q_full = bars, *const q_free = bars + 2, *const k_full = bars + 4, *const k_free = bars + 6, *const v_full = bars + 8,
           *const v_free = bars + 10, *const s_full = bars + 12, *const o_full = bars + 14, *const p_upper = bars + 16,
           *const p_lower = bars + 18, *const o_read = bars + 20, *const stopped = bars + 22;
  uint32_t* const s_tmem = reinterpret_cast<uint32_t*>(bars + 24);
  float* const s_max = reinterpret_cast<float*>(smem + L.max);               // [parity][upper, lower][row]
  float* const s_sums = reinterpret_cast<float*>(smem + L.sums);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int T = p.T, C = p.H * 64;
  const int grid = static_cast<int>(gridDim.x), block = static_cast<int>(blockIdx.x);
  const int first = static_cast<int>(1ll * p.items * block / grid), last = static_cast<int>(1ll * p.items * (block + 1) / grid);
  const int n = last - first;
  // head of an item (image, first column), first query
  auto place = [&](int it, int* b, int* x) {
    const int head = it / p.qtiles;
    *b = head / p.H;
    *x = (head - *b * p.H) * 64;
    return (it - head * p.qtiles) * kAttnQueries;
  };

  if (tid == 0) {
    for (int i = 0; i < 16; ++i) mbar_init(bars + i, 1);
    for (int i = 16; i < 22; ++i) mbar_init(bars + i, kAttnRowWarps);
    mbar_init(stopped, 1);
    mbar_fence_init();
  }
  __syncthreads();
  const uint32_t polls = p.poll_limit;
  // A thread whose wait ran out does not wait again, and the products' warp issues no more, but all go on through their loops: the lanes
  // of a warp have to be together for the instructions that need all of them, and every lane counts its own polls.  (The softmax warps
  // have one answer a warp and leave their rows out.)  The results are then worthless, which the status word says.  With a vote
  // behind every wait of every warp 64 images of 6 heads took 19.0 us and 256 of 12 111; this way 18.0 and 102, unprotected 17.8 and 100.
  bool ok = true;

  if (warp >= 16) {
    fewer_registers<kAttnIssueRegs>();
    if (warp == 16) {
      // ---------------------------------------------------------------- TMA loads
      if (lane == 0) {
        tma_prefetch_desc(&tm_q);
        tma_prefetch_desc(&tm_kv);
        tma_prefetch_desc(&tm_out);
      }
      pdl_wait();
      int heads = 0, q_loads = 0, k_loads = 0;
      auto loads = [&](int i) {
        int b, x;
        const int q0 = place(first + i, &b, &x), qb = i & 1;
        if (i > 1 && !mbar_wait(q_free + qb, ((i >> 1) - 1) & 1, polls)) return false;
        mbar_arrive_expect_tx(q_full + qb, kAttnQueries * 128);
        tma_load_3d(smem + L.q + qb * kAttnQueries * 128, &tm_q, q_full + qb, x, q0, b);
        ++q_loads;
        if (i == 0 || q0 == 0) {
          const int hb = heads & 1, use = heads >> 1;
          const uint32_t bytes = static_cast<uint32_t>(p.tk) * 128;
          if (use > 0 && !mbar_wait(k_free + hb, (use - 1) & 1, polls)) return false;
          mbar_arrive_expect_tx(k_full + hb, bytes);
          tma_load_3d(smem + L.k + hb * bytes, &tm_kv, k_full + hb, C + x, 0, b);
          ++k_loads;
          if (use > 0 && !mbar_wait(v_free + hb, (use - 1) & 1, polls)) return false;
          mbar_arrive_expect_tx(v_full + hb, bytes);
          tma_load_3d(smem + L.v + hb * bytes, &tm_kv, v_full + hb, 2 * C + x, 0, b);
          ++heads;
        }
        return true;
      };
      if (lane == 0) ok = loads(0);
      __syncwarp();
      __syncthreads();                    // tensor memory allocated
      pdl_launch_dependents();
      if (lane == 0) {
        for (int i = 1; i < n && ok; ++i) ok = loads(i);
        // No copy may land after the block has left, whichever warp has given up: the last two of each kind.
        auto landed = [&](uint64_t* bar, int loads) {
          bool in = true;
          for (int k = max(loads - 2, 0); k < loads; ++k) in &= mbar_wait(bar + (k & 1), (k >> 1) & 1);
          return in;
        };
        ok = landed(q_full, q_loads) && ok;
        ok = landed(k_full, k_loads) && ok;
        ok = landed(v_full, heads) && ok;
      }
      __syncwarp();
    } else {
      // ---------------------------------------------------------------- products (warp 17); warps 18 and 19 only keep step
      if (warp == 17) {
        pdl_wait();
        tmem_alloc(s_tmem, kAttnTmemCols);
        tmem_relinquish();
        tc_fence_before_sync();
      }
      __syncthreads();
      pdl_launch_dependents();
      tc_fence_after_sync();
      if (warp == 17) {
        // The whole warp walks the loop, one elected lane issues, and there is one copy of each product: this warp's instructions are
        // fetched anew for every item, behind the quantizer's.
        const uint32_t tmem = *s_tmem;
        const uint32_t idesc_s = umma_idesc_f16(kAttnQueries, p.tk);
        const uint32_t idesc_o = umma_idesc_f16(kAttnQueries, 64) | (1u << 16);      // B with its rows (keys) along K
        auto desc_lo = [&](uint32_t off) { return ((smem_u32(smem + off) & 0x3FFFFu) >> 4) | (1u << 16); };
        const uint32_t q0 = desc_lo(L.q), k0 = desc_lo(L.k), v0 = desc_lo(L.v), kv_step = static_cast<uint32_t>(p.tk) * 128u >> 4;
        const int split = attn_split(p.tk), tk = p.tk;
        int s_head = -1, o_head = -1, s_tile = first % p.qtiles, o_tile = s_tile;    // heads and tiles of the scores and of the products with V
#pragma unroll 1
        for (int j = 0; j < n + 2; ++j) {
          const uint32_t b = j & 1, item = tmem + b * kAttnItemCols, ph = (j >> 1) & 1;
          if (j >= 2) {
            // ---- P V of item j - 2
            const bool new_head = j == 2 || o_tile == 0;
            o_head += new_head ? 1 : 0;
            if (++o_tile == p.qtiles) o_tile = 0;
            const uint32_t hb = o_head & 1;
            ok = ok && (!new_head || mbar_wait(v_full + hb, (o_head >> 1) & 1, polls)) && mbar_wait(p_upper + b, ph ^ 1, polls);
            tc_fence_after_sync();
            uint32_t acc = 0;
            if (elect_one() && ok) {
#pragma unroll 1
              for (int k = split; k < tk; k += 16, acc = 1)
                umma_f16_tmem_a_lo(item + kAttnOutCol, item + split + ((k - split) >> 1), v0 + hb * kv_step + 8 * k, idesc_o, acc);
            }
            __syncwarp();
            acc = split < tk ? 1 : 0;
            ok = ok && mbar_wait(p_lower + b, ph ^ 1, polls);
            tc_fence_after_sync();
            if (elect_one() && ok) {
#pragma unroll 1
              for (int k = 0; k < split; k += 16, acc = 1)
                umma_f16_tmem_a_lo(item + kAttnOutCol, item + (k >> 1), v0 + hb * kv_step + 8 * k, idesc_o, acc);
              umma_commit(o_full + b);
              if (j == n + 1 || o_tile == 0) umma_commit(v_free + hb);
            }
            __syncwarp();
          }
          if (j < n) {
            // ---- the scores of item j, over an item whose output has been read
            const bool new_head = j == 0 || s_tile == 0;
            s_head += new_head ? 1 : 0;
            if (++s_tile == p.qtiles) s_tile = 0;
            const uint32_t hb = s_head & 1;
            ok = ok && (!new_head || mbar_wait(k_full + hb, (s_head >> 1) & 1, polls)) && mbar_wait(q_full + b, ph, polls) &&
                 (j < 2 || mbar_wait(o_read + b, ph ^ 1, polls));
            tc_fence_after_sync();
            if (elect_one() && ok) {
              umma_f16_x4(item, q0 + b * (kAttnQueries * 128 >> 4), k0 + hb * kv_step, idesc_s);
              umma_commit(s_full + b);
              umma_commit(q_free + b);
              if (j + 1 == n || s_tile == 0) umma_commit(k_free + hb);
            }
            __syncwarp();
          }
        }
      }
      __syncwarp();
    }
  } else if (warp < 8) {
    // ------------------------------------------------------------------ softmax: a query row for two threads
    fewer_registers<kAttnSoftmaxRegs>();
    __syncthreads();
    pdl_launch_dependents();
    tc_fence_after_sync();
    const int lower = warp >> 2, quarter = warp & 3;
    const uint32_t slot0 = *s_tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    constexpr float kScale = 0.125f * 1.44269504088896340736f;             // 1 / sqrt(64) and base 2
    const int split = attn_split(p.tk);
    const int from = lower ? 0 : split, to = lower ? split : p.tk, full = min(to, T);      // keys of this thread; those that there are
    const float ninf = __int_as_float(0xff800000);
    const int row = quarter * 32 + lane;
    int q_tile = first % p.qtiles;
    for (int i = 0; i < n; ++i) {
      const int b = i & 1;
      const bool rows = q_tile * kAttnQueries + quarter * 32 < T;          // some of the warp's rows are queries
      if (++q_tile == p.qtiles) q_tile = 0;
      ok = ok && mbar_wait_warp(s_full + b, (i >> 1) & 1, polls);
      tc_fence_after_sync();
      const uint32_t slot = slot0 + b * kAttnItemCols;
      // Loops with one body each, not unrolled over the row: the warps of an SM share an instruction cache, and unrolled passes stalled
      // on it more than on anything else.
      float* const mx = s_max + b * 2 * kAttnQueries + row;
      if (rows && ok) {
        float m0 = ninf, m1 = ninf, m2 = ninf, m3 = ninf;
        int c = from;
        auto thirty_two = [&](const uint32_t (&s)[32]) {
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            m0 = max3(m0, __uint_as_float(s[j]), __uint_as_float(s[j + 1]));
            m1 = max3(m1, __uint_as_float(s[j + 2]), __uint_as_float(s[j + 3]));
            m2 = max3(m2, __uint_as_float(s[j + 4]), __uint_as_float(s[j + 5]));
            m3 = max3(m3, __uint_as_float(s[j + 6]), __uint_as_float(s[j + 7]));
          }
        };
#pragma unroll 1
        for (; c + 64 <= full; c += 64) {
          uint32_t s0[32], s1[32];
          tmem_ld_32x32(slot + c, s0);
          tmem_ld_32x32(slot + c + 32, s1);
          tmem_ld_wait();
          thirty_two(s0);
          thirty_two(s1);
        }
        if (c + 32 <= full) {
          uint32_t s[32];
          tmem_ld_32x32(slot + c, s);
          tmem_ld_wait();
          thirty_two(s);
          c += 32;
        }
#pragma unroll 1
        for (; c < full; c += 16) {
          uint32_t t[16];
          tmem_ld_32x16(slot + c, t);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; j += 2)
            m0 = max3(m0, c + j < T ? __uint_as_float(t[j]) : ninf, c + j + 1 < T ? __uint_as_float(t[j + 1]) : ninf);
        }
        mx[lower * kAttnQueries] = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3));
      }
      // the two warps of a lane quarter: each other's maximum is there (and the values of two items ago have been read)
      asm volatile("bar.sync %0, 64;" ::"r"(4 + quarter) : "memory");
      if (rows && ok) {
        const float nm = -kScale * fmaxf(mx[0], mx[kAttnQueries]);
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
        int c = from, p_col = from;
#pragma unroll 1
        for (; c + 32 <= full; c += 32, p_col += 16) {
          uint32_t s[32], w[16];
          tmem_ld_32x32(slot + c, s);
          tmem_ld_wait();
          exponentials(s, w);
          exponentials(s + 16, w + 8);
          tmem_st_32x16(slot + p_col, w);                                  // over columns of S that have been read
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
        float x0, x1;
        unpack2(add2(sum0, sum1), x0, x1);
        s_sums[(b * 2 + lower) * kAttnQueries + row] = x0 + x1;
        tmem_st_wait();
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive((lower ? p_lower : p_upper) + b);
    }
  } else {
    // ------------------------------------------------------------------ output: a thread per query row
    more_registers<kAttnOutputRegs>();
    const int quarter = warp & 3, parity = (warp - 8) >> 2;
    GroupQuantTables* const tables = reinterpret_cast<GroupQuantTables*>(smem + L.tables);
    GroupQuantParams gp = {};
    // reads only the layer's constants: done while the previous kernel still runs
    if (QUANT)
      gp = group_quant_tables<1 << BITS, false>(tables, p.thresholds, p.codebook, tid - 256, 2 * kAttnRowWarps * 32, [](bool b) {
        asm volatile("bar.sync 1, %0;" ::"n"(2 * kAttnRowWarps * 32) : "memory");
        return b;
      });
    __syncthreads();
    pdl_launch_dependents();
    tc_fence_after_sync();
    const uint32_t t_out = *s_tmem + (static_cast<uint32_t>(quarter * 32) << 16) + parity * kAttnItemCols + kAttnOutCol;
    const float* const sums = s_sums + parity * 2 * kAttnQueries + quarter * 32 + lane;
    uint8_t* const stage = smem + L.stage + (warp - 8) * 4096;
    const uint32_t row = smem_u32(stage) + lane * 128, x7 = lane & 7;
    for (int i = parity; i < n; i += 2) {
      const uint32_t ph = (i >> 1) & 1;
      int b, x;
      const int t0 = place(first + i, &b, &x) + quarter * 32;
      const bool live = t0 < T;
      ok = ok && mbar_wait(o_full + parity, ph, polls) && mbar_wait(p_upper + parity, ph, polls) && mbar_wait(p_lower + parity, ph, polls);
      tc_fence_after_sync();
      uint32_t w[32];
      if (live) {
        const float inv = __frcp_rn(sums[0] + sums[kAttnQueries]);
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
        mbar_arrive(o_read + parity);
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
  }
  tc_fence_before_sync();
  const bool gave_up = __syncthreads_or(!ok) != 0;
  if (warp == 17) {
    tc_fence_after_sync();
    if (gave_up) {                                // nobody may have waited for the last products: they end before their memory is given back
      if (elect_one()) {
        umma_commit(stopped);
        atomicExch(p.status, kStatusAttentionTimeout);
      }
      __syncwarp();
      mbar_wait(stopped, 0);
      __syncwarp();
    }
    tmem_dealloc(*s_tmem, kAttnTmemCols);
  }
}

}  // namespace arcq
