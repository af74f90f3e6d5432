// The ARCQ quantizer of one 64-value group, held by one thread: statistics, codes and reconstruction.  Shared by every
// kernel that quantises activations a group per thread (act_quant_tile.cuh, ln_act_quant.cuh, attention.cuh,
// gemm_pair_dense.cuh).
//
// What bounds it is issue slots: nothing here waits for memory once the row is in shared memory.  So the arithmetic is
// two values per instruction (add / mul / fma.f32x2; each half rounds like the scalar instruction, so the bits are those of
// scalar code), and a code costs three table reads and one compare:
//
//   * Bounded argument.  sum r^2 = 64 var, so |r| / s <= 8 for every element of a group: a grid over [-16, 16) needs no
//     clamp.  One fma, rounded down, turns r into 1.5 * 2^21 + cell with two fraction bits below the cell, i.e. the low
//     bits of the result are 4 * cell: the byte offset into the tables.
//   * cell -> (threshold, level below it, level above it).  Consecutive cells lie in consecutive banks and the values of a
//     group span some twenty cells, so the reads are conflict-free without copies of the tables.
//   * level = r > th * s ? above : below, the sign of d = fma(-th, s, r).
//
// Exactness.  The code is the number of thresholds with RN(r / s) > th.  With h half the gap from th to the next fp32
// number, RN(r / s) > th <=> r > (th + h) * s, while the sign of d (rounding to nearest keeps signs) tells r > th * s.
// The two differ only if 0 < r - th * s <= h * s, so a chunk of eight values with some |d| <= s * max h goes through the
// IEEE quotient and a search over all thresholds: about one value in a million.  A codebook with two thresholds
// closer than 1.1 cells takes that path for every value.
#pragma once
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include "ptx.cuh"
#include "act_quant.cuh"

namespace arcq {

// ---------------------------------------------------------------- two fp32 values per instruction
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// A packed mul whose result feeds a packed add is contracted into one fma by the assembler, .rn on both notwithstanding (one
// rounding instead of two: a scale came out one unit in the last place off).  Where that matters, mul2_rn adds a -0 that
// the compiler cannot see (GroupQuantParams::nz), which leaves every product as it is.
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 mul2_rn(f32x2 a, f32x2 b, f32x2 nz) { return fma2(a, b, nz); }
__device__ __forceinline__ f32x2 fma2_down(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rm.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ float min3_abs(float m, float a, float b) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(m), "f"(fabsf(a)), "f"(fabsf(b)));
  return d;
}

// ---------------------------------------------------------------- per-layer tables in shared memory
constexpr int kGqCells = 256;
struct GroupQuantTables {            // 4 KB + 132 bytes
  float cell_nth[kGqCells];          // minus the threshold that a value of the cell can be above or below
  float cell_lo[kGqCells];           // the level below that threshold ...
  float cell_hi[kGqCells];           // ... and above
  float th[16], cb[16];              // +inf padded thresholds, levels
  uint32_t cell_code4[kGqCells];     // 4 * (code below the threshold), for kernels that also write codes
  float nz;                          // -0
};
struct GroupQuantParams {            // the same in every thread of the block
  float cells_per_unit;              // 4 or 8
  float tie;                         // times s: the |d| up to which a chunk takes the exact path (inf: always)
  f32x2 nz;                          // two -0 (see mul2_rn)
};

// Fills the tables; `sync_and(bool)` is a barrier over exactly the `nthreads` calling threads (numbered `tid`) that
// returns the conjunction of its arguments.  Ends with a barrier: the tables are complete on return.
template <int L, typename SyncAnd>
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
    t->cell_nth[k] = -t->th[c];                              // c == L - 1: -inf, nothing is above it
    t->cell_lo[k] = t->cb[c];
    t->cell_hi[k] = t->cb[c + 1 < L ? c + 1 : L - 1];
    t->cell_code4[k] = 4u * static_cast<uint32_t>(c);
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
// Values as pairs: v[4 * c + j] holds elements 8c + 2j and 8c + 2j + 1.  The reference adds (torch's CPU order)
//   v[l] = ((x[l]+x[32+l]) + (x[8+l]+x[40+l])) + (x[16+l]+x[48+l])) + (x[24+l]+x[56+l]),  l = 0..7
//   sum  = ((((((v0+v1)+v2)+v3)+v4)+v5)+v6)+v7
__device__ __forceinline__ float sum64_pairs(const f32x2 (&v)[32]) {
  float s = 0.0f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const f32x2 a = add2(add2(add2(add2(v[j], v[16 + j]), add2(v[4 + j], v[20 + j])), add2(v[8 + j], v[24 + j])),
                         add2(v[12 + j], v[28 + j]));
    float e, o;
    unpack2(a, e, o);
    s = j == 0 ? __fadd_rn(e, o) : __fadd_rn(__fadd_rn(s, e), o);
  }
  return s;
}

struct GroupStats {
  float mean, scale, code_sum;
};

// In: v = the group's values.  Out: v = the levels of their codes, statistics; words[c] = the codes of elements
// 8c .. 8c+7, one per nibble (CODES only).
template <int BITS, bool CODES>
__device__ __forceinline__ GroupStats group_quantize(f32x2 (&v)[32], const GroupQuantTables* t, const GroupQuantParams& p,
                                                     uint32_t (&words)[8]) {
  constexpr int L = 1 << BITS;
  GroupStats st;
  st.mean = __fmul_rn(sum64_pairs(v), 0.015625f);           // / 64: exact
  {
    const f32x2 nm = pack2(-st.mean, -st.mean);
    f32x2 q[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      v[i] = add2(v[i], nm);
      q[i] = mul2_rn(v[i], v[i], p.nz);
    }
    st.scale = __fsqrt_rn(__fadd_rn(__fmul_rn(sum64_pairs(q), 0.015625f), 1.0e-6f));
  }
  const float s = st.scale;
  const float a = __fdividef(p.cells_per_unit, s);           // an approximate quotient is enough for the cell
  const f32x2 a2 = pack2(a, a), s2 = pack2(s, s), magic = pack2(3145728.0f + 128.0f, 3145728.0f + 128.0f);
  const float tie = __fmul_rn(p.tie, s);
  const uint32_t tab = smem_u32(t);
  constexpr uint32_t kLo = kGqCells * 4, kHi = 2 * kGqCells * 4, kCb = 3 * kGqCells * 4 + 64, kCode = 3 * kGqCells * 4 + 128;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    float m = 1.0e38f, out[8];
    uint32_t w = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float u0, u1, d0, d1;
      unpack2(fma2_down(v[4 * c + j], a2, magic), u0, u1);
      const uint32_t k0 = tab + (__float_as_uint(u0) & 0x3FCu), k1 = tab + (__float_as_uint(u1) & 0x3FCu);
      unpack2(fma2(pack2(lds_f32(k0), lds_f32(k1)), s2, v[4 * c + j]), d0, d1);
      m = min3_abs(m, d0, d1);
      if (CODES) {
        uint32_t o0 = lds32(k0 + kCode), o1 = lds32(k1 + kCode);
        o0 += d0 > 0.0f ? 4u : 0u;
        o1 += d1 > 0.0f ? 4u : 0u;
        out[2 * j] = lds_f32(tab + kCb + o0);
        out[2 * j + 1] = lds_f32(tab + kCb + o1);
        w |= (o0 | (o1 << 4)) << (8 * j);                    // four times the codes; shifted down once per word below
        if (j == 3) words[c] = (w >> 2) | ((o1 >> 4) << 30);
      } else {
        const float l0 = lds_f32(k0 + kLo), h0 = lds_f32(k0 + kHi);
        const float l1 = lds_f32(k1 + kLo), h1 = lds_f32(k1 + kHi);
        out[2 * j] = d0 > 0.0f ? h0 : l0;
        out[2 * j + 1] = d1 > 0.0f ? h1 : l1;
      }
    }
    if (m <= tie) {
      // rare: some value of the chunk is too close to a threshold for the sign of d alone
      float r[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) unpack2(v[4 * c + j], r[2 * j], r[2 * j + 1]);
      uint32_t we = 0;
#pragma unroll 1
      for (int j = 0; j < 8; ++j) {
        const int code = group_quant_exact_code<L>(t, r[0], s);
        const float lv = t->cb[code];
        we = (we >> 4) | (static_cast<uint32_t>(code) << 28);
        // rotate: registers cannot be indexed by a loop counter
#pragma unroll
        for (int i = 0; i < 7; ++i) {
          r[i] = r[i + 1];
          out[i] = out[i + 1];
        }
        out[7] = lv;
      }
      if (CODES) words[c] = we;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) v[4 * c + j] = pack2(out[2 * j], out[2 * j + 1]);
  }
  st.code_sum = sum64_pairs(v);
  return st;
}

// mean + scale * (level - code_sum / 64) in the reference's three rounded steps
struct GroupRecon {
  f32x2 mean, scale, nvm, nz;
};
__device__ __forceinline__ GroupRecon group_recon(const GroupStats& st, const GroupQuantParams& p) {
  const float vm = __fmul_rn(st.code_sum, 0.015625f);        // exact
  return {pack2(st.mean, st.mean), pack2(st.scale, st.scale), pack2(-vm, -vm), p.nz};
}
__device__ __forceinline__ f32x2 group_recon_pair(const GroupRecon& g, f32x2 level) {
  return add2(g.mean, mul2_rn(g.scale, add2(level, g.nvm), g.nz));
}

__device__ __forceinline__ f32x2 half2_to_pair(uint32_t h) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
  return pack2(f.x, f.y);
}
__device__ __forceinline__ uint32_t pair_to_half2(f32x2 v) {
  float a, b;
  unpack2(v, a, b);
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// ---------------------------------------------------------------- GELU of a group's fp16 values
// g = x * (0.5 + x * R(x^2)) for |x| < 1.3125, with x * R(x^2) = erf(x / sqrt 2) / 2: R of degree 5 in x^2, fitted on
// Chebyshev nodes (2e-8 relative before rounding).  Over every fp16 input of that range the fp16 result differs from the
// correctly rounded one for 3 inputs of 31 742 (0.5 x (1 + erff(x / sqrt 2)) in fp32: 2).  Larger arguments keep the value of
// x, are counted in a bit mask, and go through erff one by one in a loop over the group's row in shared memory: few
// of them sit in a group, and the loop is one copy of erff in the code instead of 64.
// `row`: the thread's own 128-byte row, 16-byte chunk c at ((c ^ x7) << 4), used for that exchange only.  The result is
// rounded to fp16, the value a separate GELU kernel would store; ch[c] holds chunk c before and after.
__device__ __forceinline__ void gelu_row(uint4 (&ch)[8], uint32_t row, uint32_t x7) {
  const f32x2 c5 = pack2(-6.607886916754069e-06f, -6.607886916754069e-06f), c4 = pack2(0.00011030046152882278f, 0.00011030046152882278f);
  const f32x2 c3 = pack2(-0.0011828974820673466f, -0.0011828974820673466f), c2 = pack2(0.009971804916858673f, 0.009971804916858673f);
  const f32x2 c1 = pack2(-0.06649012118577957f, -0.06649012118577957f), c0 = pack2(0.3989422619342804f, 0.3989422619342804f);
  const f32x2 half = pack2(0.5f, 0.5f);
  const __half2 lim = __floats2half2_rn(1.3125f, 1.3125f);
  uint32_t big[2] = {0u, 0u};
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    uint32_t* const w = reinterpret_cast<uint32_t*>(&ch[c]);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const __half2 xh = *reinterpret_cast<const __half2*>(&w[q]);
      const uint32_t m = __hgeu2_mask(__habs2(xh), lim);                  // 0xffff per half (unordered: NaN counts as large)
      const f32x2 x = half2_to_pair(w[q]);
      const f32x2 s = mul2(x, x);
      f32x2 r = fma2(c5, s, c4);
      r = fma2(r, s, c3);
      r = fma2(r, s, c2);
      r = fma2(r, s, c1);
      r = fma2(r, s, c0);
      const uint32_t g = pair_to_half2(mul2(x, fma2(x, r, half)));
      big[c >> 2] |= m & (0x00010001u << (4 * (c & 3) + q));
      w[q] = (m & w[q]) | (~m & g);
    }
  }
  if ((big[0] | big[1]) != 0u) {
#pragma unroll
    for (int c = 0; c < 8; ++c) sts128(row + ((static_cast<uint32_t>(c) ^ x7) << 4), ch[c].x, ch[c].y, ch[c].z, ch[c].w);
#pragma unroll 1
    for (int hw = 0; hw < 2; ++hw) {
      uint32_t b = hw ? big[1] : big[0];
#pragma unroll 1
      while (b != 0u) {
        const int i = __ffs(b) - 1;
        b &= b - 1u;
        const uint32_t e = 32u * hw + 2u * (i & 15) + (i >> 4);           // element of the group
        const uint32_t a = row + (((e >> 3) ^ x7) << 4) + 2u * (e & 7u);
        const float x = __half2float(__ushort_as_half(static_cast<unsigned short>(lds16(a))));
        const float g = x * 0.5f * (1.0f + erff(x * 0.70710678118654752440f));
        sts16(a, __half_as_ushort(__float2half_rn(g)));
      }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) ch[c] = lds128(row + ((static_cast<uint32_t>(c) ^ x7) << 4));
  }
}

// The quantizer on the thread's fp16 row in shared memory, in place: values in, reconstruction out.
template <int BITS, bool GELU>
__device__ __forceinline__ void group_quantize_row(uint32_t row, uint32_t x7, const GroupQuantTables* t,
                                                   const GroupQuantParams& p) {
  f32x2 v[32];
  {
    uint4 ch[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) ch[c] = lds128(row + ((static_cast<uint32_t>(c) ^ x7) << 4));
    if (GELU) gelu_row(ch, row, x7);
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      v[4 * c] = half2_to_pair(ch[c].x);
      v[4 * c + 1] = half2_to_pair(ch[c].y);
      v[4 * c + 2] = half2_to_pair(ch[c].z);
      v[4 * c + 3] = half2_to_pair(ch[c].w);
    }
  }
  uint32_t words[8];
  const GroupRecon g = group_recon(group_quantize<BITS, false>(v, t, p, words), p);
#pragma unroll
  for (int c = 0; c < 8; ++c)
    sts128(row + ((static_cast<uint32_t>(c) ^ x7) << 4), pair_to_half2(group_recon_pair(g, v[4 * c])),
           pair_to_half2(group_recon_pair(g, v[4 * c + 1])), pair_to_half2(group_recon_pair(g, v[4 * c + 2])),
           pair_to_half2(group_recon_pair(g, v[4 * c + 3])));
}

}  // namespace arcq
