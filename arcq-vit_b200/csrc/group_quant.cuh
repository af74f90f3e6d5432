// The ARCQ quantizer of one 64-value group, held by LPG = 1 or 2 lanes: statistics, codes and reconstruction.  Shared by
// the kernels that quantise activations out of shared memory (act_quant_tile.cuh, ln_act_quant.cuh).
//
// Two lanes a group (lane h holds the reference's summation lanes l = 4h .. 4h+3, half of every 16-byte chunk) need 64
// registers instead of 128 and half the straight-line code: 32 warps an SM instead of 16, and fewer instruction-cache
// misses; measured slower all the same (GELU [12608, 1536] 28.1 against 24.1 us: 25 instructions a value instead of 17).
//
// What bounds it is issue slots: nothing here waits for memory once the row is in shared memory.  So the arithmetic is
// two values per instruction (add / mul / fma.f32x2; each half rounds like the scalar instruction, so the bits are those of
// scalar code), and a level costs two table reads and one compare:
//
//   * Bounded argument.  sum r^2 = 64 var, so |r| / s <= 8 for every element of a group: a grid over [-16, 16) needs no
//     clamp.  One fma, rounded down, turns r into 1.5 * 2^21 + cell with two fraction bits below the cell, i.e. the low
//     bits of the result are 4 * cell: the byte offset into the tables.
//   * cell -> (threshold, level below it, level above it).  Consecutive cells lie in consecutive banks and the values of a
//     group span some twenty cells, so the reads are conflict-free without copies of the tables.
//   * level = r > th * s ? above : below: the sign of d = fma(-th, s, r) picks the table that is read.  (Both levels read and one
//     selected: a third read, and [50432, 768] 31.2 instead of 29.3 us together with the next item.)
//
// Exactness.  The code is the number of thresholds with RN(r / s) > th.  With h half the gap from th to the next fp32
// number, RN(r / s) > th <=> r > (th + h) * s, while the sign of d (rounding to nearest keeps signs) tells r > th * s.
// The two differ only if 0 < r - th * s <= h * s, so a value with |d| <= s * max h goes through the IEEE quotient and a search
// over all thresholds: about one in a million (15 thresholds, +-1.5e-7 each, at a density of 0.3), i.e. a few of nearly every
// launch's warps, which the launch then waits for.  A codebook with two thresholds closer than 1.1 cells takes that path for every
// value, and a threshold of exactly 0 (symmetric codebooks, every 2-bit one that is fitted) sends every value of a group of equal values
// there: one such warp costs a launch 16 us ([3001, 3072] 24.6 us, 8.3 with the thresholds moved by 0.01).
#pragma once
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include "ptx.cuh"
#include "f32x2.cuh"
#include "act_quant.cuh"

namespace arcq {

// a + OFFSET where d > 0
template <uint32_t OFFSET> __device__ __forceinline__ uint32_t offset_if_positive(uint32_t a, float d) {
  asm("{\n\t.reg .pred p;\n\tsetp.gt.f32 p, %1, 0f00000000;\n\t@p add.u32 %0, %0, %2;\n\t}" : "+r"(a) : "f"(d), "n"(OFFSET));
  return a;
}

// ---------------------------------------------------------------- per-layer tables in shared memory
constexpr int kGqCells = 256;
struct GroupQuantTables {            // 3 KB + 144 bytes, 1 KB more with codes; placed on a 1 KB boundary, so that cell offset and base merge in one OR
  float cell_nth[kGqCells];          // minus the threshold that a value of the cell can be above or below
  float cell_lo[kGqCells];           // the level below that threshold ...
  float cell_hi[kGqCells];           // ... and above
  float th[16], cb[16];              // +inf padded thresholds, levels
  float nz;                          // -0
  float pad[3];
  uint32_t cell_code4[kGqCells];     // 4 * (code below the threshold); only kernels that also write codes have it
};
constexpr uint32_t kGroupQuantTableBytes = 3 * kGqCells * 4 + 144;        // without it
struct GroupQuantParams {            // the same in every thread of the block
  float cells_per_unit;              // 4 or 8
  float tie;                         // times s: the |d| up to which a chunk takes the exact path (inf: always)
  f32x2 nz;                          // two -0 (see mul2_rn)
};

// Fills the tables; `sync_and(bool)` is a barrier over exactly the `nthreads` calling threads (numbered `tid`) that
// returns the conjunction of its arguments.  Ends with a barrier: the tables are complete on return.
template <int L, bool CODES, typename SyncAnd>
__device__ __forceinline__ GroupQuantParams group_quant_tables(GroupQuantTables* t, const float* __restrict__ thresholds,
                                                               const float* __restrict__ codebook, int tid, int nthreads,
                                                               SyncAnd sync_and) {
  if (tid < 16) {
    t->th[tid] = tid < L - 1 ? __ldg(thresholds + tid) : __int_as_float(0x7f800000);
    t->cb[tid] = tid < L ? __ldg(codebook + tid) : 0.0f;
  }
  if (tid == 0) t->nz = -0.0f;
  sync_and(true);
  // smallest gap and largest half-gap, by every thread (broadcast reads)
  float gap = 1.0e30f, hmax = 0.0f, reach = 0.0f;
#pragma unroll
  for (int i = 0; i < L - 1; ++i) {
    const float a = t->th[i];
    reach = fmaxf(reach, fabsf(a));
    if (i + 1 < L - 1) gap = fminf(gap, t->th[i + 1] - a);
  }
  hmax = fmaxf(reach * 0x1p-24f, 0x1p-140f);              // half a unit in the last place of the largest threshold
  GroupQuantParams p;
  // a cell widened by 0.05 on both sides must hold at most one threshold; cells outside [-16, 16) do not exist
  const bool wide = gap * 4.0f > 1.1f;
  p.cells_per_unit = wide ? 4.0f : 8.0f;
  const bool fast = (wide || gap * 8.0f > 1.1f) && reach < 15.0f;
  p.tie = fast ? 1.01f * hmax : __int_as_float(0x7f800000);
  for (int k = tid; k < kGqCells; k += nthreads) {
    // cell k holds quotients t with floor(t * cells_per_unit) + 128 == k
    const float lim = static_cast<float>(k - 128) - 0.05f;
    int c = 0;
#pragma unroll
    for (int i = 0; i < L - 1; ++i) c += (t->th[i] * p.cells_per_unit < lim) ? 1 : 0;
    if (k == kGqCells - 1) c = 0;                            // no quotient of a group gets here but NaN: code 0
    t->cell_nth[k] = -t->th[c];                               // c == L - 1: -inf, nothing is above it
    t->cell_lo[k] = t->cb[c];
    t->cell_hi[k] = t->cb[c + 1 < L ? c + 1 : L - 1];
    if (CODES) t->cell_code4[k] = 4u * static_cast<uint32_t>(c);
  }
  p.nz = pack2(t->nz, t->nz);
  sync_and(true);
  return p;
}

// The exact code of one value: IEEE quotient, search in the sorted thresholds.
template <int L>
__device__ __forceinline__ int group_quant_exact_code(const GroupQuantTables* t, float r, float s) {
  const float q = __fdiv_rn(r, s);
  int code = 0;
  if (L == 16) code = (q > t->th[7]) ? 8 : 0;
  if (L >= 8) code += (q > t->th[code + 3]) ? 4 : 0;
  code += (q > t->th[code + 1]) ? 2 : 0;
  code += (q > t->th[code]) ? 1 : 0;
  return code;
}

// ---------------------------------------------------------------- the group
// The pairs of values of a lane: v[c * PJ + j], PJ = 4 / LPG, holds elements 8c + 4h + 2j and the next (h = 0 with one lane).
// The reference adds (torch's CPU order)
//   v[l] = ((x[l]+x[32+l]) + (x[8+l]+x[40+l])) + (x[16+l]+x[48+l])) + (x[24+l]+x[56+l]),  l = 0..7
//   sum  = ((((((v0+v1)+v2)+v3)+v4)+v5)+v6)+v7
// The first line is local to a lane; with two lanes the chain crosses to the partner once and its end comes back.
template <int LPG>
__device__ __forceinline__ float sum64_pairs(const f32x2 (&v)[32 / LPG]) {
  constexpr int PJ = 4 / LPG;
  float p[8 / LPG];
#pragma unroll
  for (int j = 0; j < PJ; ++j)
    unpack2(add2(add2(add2(add2(v[j], v[4 * PJ + j]), add2(v[PJ + j], v[5 * PJ + j])), add2(v[2 * PJ + j], v[6 * PJ + j])),
                 add2(v[3 * PJ + j], v[7 * PJ + j])),
            p[2 * j], p[2 * j + 1]);
  float s = p[0];
#pragma unroll
  for (int l = 1; l < 8 / LPG; ++l) s = __fadd_rn(s, p[l]);
  if (LPG == 2) {
    const int lane = threadIdx.x & 31;
    float t = __shfl_sync(0xffffffffu, s, lane & ~1);              // the h = 0 lane's four
#pragma unroll
    for (int l = 0; l < 4; ++l) t = __fadd_rn(t, p[l]);            // meaningful in the h = 1 lane
    s = __shfl_sync(0xffffffffu, t, lane | 1);
  }
  return s;
}

struct GroupStats {
  float mean, scale, code_sum;
};

// In: v = the lane's values.  Out: v = the levels of their codes, statistics; words[c] = the codes of elements
// 8c .. 8c+7, one per nibble (CODES, one lane a group).
template <int BITS, bool CODES, int LPG>
__device__ __forceinline__ GroupStats group_quantize(f32x2 (&v)[32 / LPG], const GroupQuantTables* t,
                                                     const GroupQuantParams& p, uint32_t (&words)[8]) {
  static_assert(!CODES || LPG == 1, "codes are assembled by one lane");
  constexpr int L = 1 << BITS, PJ = 4 / LPG, CH = 2 * PJ;          // pairs and values of a chunk
  GroupStats st;
  st.mean = __fmul_rn(sum64_pairs<LPG>(v), 0.015625f);           // / 64: exact
  {
    const f32x2 nm = pack2(-st.mean, -st.mean);
    f32x2 q[32 / LPG];
#pragma unroll
    for (int i = 0; i < 32 / LPG; ++i) {
      v[i] = add2(v[i], nm);
      q[i] = mul2_rn(v[i], v[i], p.nz);
    }
    st.scale = __fsqrt_rn(__fadd_rn(__fmul_rn(sum64_pairs<LPG>(q), 0.015625f), 1.0e-6f));
  }
  const float s = st.scale;
  const float a = __fdividef(p.cells_per_unit, s);           // an approximate quotient is enough for the cell
  const f32x2 a2 = pack2(a, a), s2 = pack2(s, s), magic = pack2(3145728.0f + 128.0f, 3145728.0f + 128.0f);
  const float tie = __fmul_rn(p.tie, s);
  const uint32_t tab = smem_u32(t);
  constexpr uint32_t kLo = kGqCells * 4, kHi = 2 * kGqCells * 4, kCode = kGroupQuantTableBytes, kCb = 3 * kGqCells * 4 + 64;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    float m = 1.0e38f, out[CH], d[CH];
    uint32_t w = 0;
#pragma unroll
    for (int j = 0; j < PJ; ++j) {
      float u0, u1;
      float &d0 = d[2 * j], &d1 = d[2 * j + 1];
      unpack2(fma2_down(v[c * PJ + j], a2, magic), u0, u1);
      const uint32_t o0 = (__float_as_uint(u0) & 0x3FCu) | tab, o1 = (__float_as_uint(u1) & 0x3FCu) | tab;
      unpack2(fma2(pack2(lds_const_f32(o0), lds_const_f32(o1)), s2, v[c * PJ + j]), d0, d1);
      m = min3_abs(m, d0, d1);
      if (CODES) {
        uint32_t c0 = lds_const_u32(o0 + kCode), c1 = lds_const_u32(o1 + kCode);
        c0 += d0 > 0.0f ? 4u : 0u;
        c1 += d1 > 0.0f ? 4u : 0u;
        out[2 * j] = lds_const_f32(tab + kCb + c0);
        out[2 * j + 1] = lds_const_f32(tab + kCb + c1);
        w |= (c0 | (c1 << 4)) << (8 * j);                    // four times the codes; shifted down once per word below
        if (j == PJ - 1) words[c] = (w >> 2) | ((c1 >> 4) << 30);
      } else {
        out[2 * j] = lds_const_f32(offset_if_positive<kHi - kLo>(o0, d0) + kLo);
        out[2 * j + 1] = lds_const_f32(offset_if_positive<kHi - kLo>(o1, d1) + kLo);
      }
    }
    if (__builtin_expect(m <= tie, 0)) {
      // rare: a value of the chunk is too close to a threshold for the sign of d alone.  One of a kernel's warps gets here in
      // most launches, and the others wait for it at the end, so it looks at the values in question only (through local memory,
      // so that the common path keeps its registers where they are): all eight values took 1.1 us.
      float r[CH], level[CH];
      uint32_t hits = 0;
#pragma unroll
      for (int j = 0; j < PJ; ++j) unpack2(v[c * PJ + j], r[2 * j], r[2 * j + 1]);
#pragma unroll
      for (int j = 0; j < CH; ++j) {
        level[j] = out[j];
        hits |= fabsf(d[j]) <= tie ? 1u << j : 0u;
      }
#pragma unroll 1
      while (hits != 0) {
        const int j = __ffs(hits) - 1;
        hits &= hits - 1;
        const int code = group_quant_exact_code<L>(t, r[j], s);
        level[j] = t->cb[code];
        if (CODES) words[c] = (words[c] & ~(15u << (4 * j))) | (static_cast<uint32_t>(code) << (4 * j));
      }
#pragma unroll
      for (int j = 0; j < CH; ++j) out[j] = level[j];
    }
#pragma unroll
    for (int j = 0; j < PJ; ++j) v[c * PJ + j] = pack2(out[2 * j], out[2 * j + 1]);
  }
  st.code_sum = sum64_pairs<LPG>(v);
  return st;
}

// recon_value (act_quant.cuh) of two levels
struct GroupRecon {
  f32x2 scale, a, b, c;
};
__device__ __forceinline__ GroupRecon group_recon(const GroupStats& st, const GroupQuantParams& p, bool one_fma = false) {
  const ReconTerms t = recon_terms(st.mean, st.scale, st.code_sum, one_fma);
  // p.nz, not the constant -0 of t.b: the product must not be contracted with the last addition (see mul2_rn)
  return {pack2(st.scale, st.scale), pack2(t.a, t.a), one_fma ? pack2(t.b, t.b) : p.nz, pack2(t.c, t.c)};
}
__device__ __forceinline__ f32x2 group_recon_pair(const GroupRecon& g, f32x2 level) {
  return add2(g.c, fma2(g.scale, add2(level, g.a), g.b));
}

// ---------------------------------------------------------------- rows in shared memory
// The lane's part of a group's 128-byte row, 16-byte chunk c at ((c ^ x7) << 4): w[c * PJ + j] = the 32-bit word of pair j.
// With two lanes `row` already includes 8 * h.
template <int LPG>
__device__ __forceinline__ void row_load(uint32_t (&w)[32 / LPG], uint32_t row, uint32_t x7) {
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const uint32_t a = row + ((static_cast<uint32_t>(c) ^ x7) << 4);
    if constexpr (LPG == 1) {
      const uint4 u = lds128(a);
      w[4 * c] = u.x; w[4 * c + 1] = u.y; w[4 * c + 2] = u.z; w[4 * c + 3] = u.w;
    } else {
      const uint2 u = lds64(a);
      w[2 * c] = u.x; w[2 * c + 1] = u.y;
    }
  }
}
template <int LPG>
__device__ __forceinline__ void row_store(const uint32_t (&w)[32 / LPG], uint32_t row, uint32_t x7) {
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const uint32_t a = row + ((static_cast<uint32_t>(c) ^ x7) << 4);
    if constexpr (LPG == 1) sts128(a, w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
    else sts64(a, w[2 * c], w[2 * c + 1]);
  }
}

// ---------------------------------------------------------------- GELU of a group's fp16 values
// The arithmetic of gelu (act_quant.cuh), two values per instruction.  Arguments of 2 and more keep the value of x, are
// marked in a bit mask, and go through erff one by one in a loop over the lane's part of the row in shared memory: few of
// them sit in a group, and the loop is one copy of erff in the code instead of 64.  Each costs its whole warp an iteration,
// which is why the polynomial reaches to 2 (up to 1.3125 degree 5 would do, one instruction a value less: [100864, 3072] with
// values of 0.55 rms takes 407 us instead of 647).  The row is used for that exchange only.  The result is rounded to fp16,
// the value a separate GELU kernel would store.
template <int LPG>
__device__ __forceinline__ void gelu_words(uint32_t (&w)[32 / LPG], uint32_t row, uint32_t x7) {
  constexpr int PJ = 4 / LPG;
  const f32x2 half = pack2(0.5f, 0.5f);
  const __half2 lim = __floats2half2_rn(kGeluLimit, kGeluLimit);
  uint32_t big[2] = {0u, 0u};
#pragma unroll
  for (int i = 0; i < 32 / LPG; ++i) {
    const __half2 xh = *reinterpret_cast<const __half2*>(&w[i]);
    const uint32_t m = __hgeu2_mask(__habs2(xh), lim);                  // 0xffff per half (unordered: NaN counts as large)
    const f32x2 x = sixteen_to_pair<__half>(w[i]);
    const f32x2 s = mul2(x, x);
    f32x2 r = pack2(gelu_r(7), gelu_r(7));
#pragma unroll
    for (int k = 6; k >= 0; --k) r = fma2(r, s, pack2(gelu_r(k), gelu_r(k)));
    const uint32_t g = pair_to_sixteen<__half>(mul2(x, fma2(x, r, half)));
    big[i >> 4] |= m & (0x00010001u << (i & 15));
    w[i] = (m & w[i]) | (~m & g);
  }
  if ((big[0] | big[1]) != 0u) {
    row_store<LPG>(w, row, x7);
#pragma unroll 1
    for (int hw = 0; hw < 2 / LPG; ++hw) {
      uint32_t b = hw ? big[1] : big[0];
#pragma unroll 1
      while (b != 0u) {
        const int k = __ffs(b) - 1;
        b &= b - 1u;
        const uint32_t i = 16u * hw + (k & 15);                          // the word, in chunk i / PJ
        const uint32_t a = row + (((i / PJ) ^ x7) << 4) + 4u * (i % PJ) + 2u * (k >> 4);
        const float x = __half2float(__ushort_as_half(static_cast<unsigned short>(lds16(a))));
        sts16(a, __half_as_ushort(__float2half_rn(gelu_large(x))));
      }
    }
    row_load<LPG>(w, row, x7);
  }
}

// The quantizer on a fp16 row in shared memory, in place: values in, reconstruction out.
template <typename T, int BITS, bool GELU, int LPG>
__device__ __forceinline__ void group_quantize_row(uint32_t row, uint32_t x7, const GroupQuantTables* t,
                                                   const GroupQuantParams& p, bool one_fma = false) {
  uint32_t w[32 / LPG], words[8];
  f32x2 v[32 / LPG];
  row_load<LPG>(w, row, x7);
  if (GELU) gelu_words<LPG>(w, row, x7);
#pragma unroll
  for (int i = 0; i < 32 / LPG; ++i) v[i] = sixteen_to_pair<T>(w[i]);
  const GroupStats st = group_quantize<BITS, false, LPG>(v, t, p, words);
  const GroupRecon g = group_recon(st, p, one_fma);
#pragma unroll
  for (int i = 0; i < 32 / LPG; ++i) w[i] = pair_to_sixteen<T>(group_recon_pair(g, v[i]));
  row_store<LPG>(w, row, x7);
}

}  // namespace arcq
