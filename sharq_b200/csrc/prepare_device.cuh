// Device code shared by the activation prepare kernels (prepare.cu) and the tensor-parallel
// transition kernel (sp_transition.cu): bf16 packing helpers, the 32-element group (pair
// selection, sparse main path, dense residual), the tensor-scale division, and small utilities.
#pragma once

#include "common.cuh"

namespace sharq {
namespace prep {

__device__ __forceinline__ float lo_f(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi_f(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// two floats -> packed bf16x2 (a in the low half), round to nearest even
__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t *>(&v);
}

// Two floats in a 64-bit register pair and the packed operations on them: one instruction for both lanes, each lane
// rounded as the scalar operation rounds (the kernels are bound by instruction issue).
__device__ __forceinline__ uint64_t pair_f32(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpair_f32(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// both bf16 values of a word times the pair b
__device__ __forceinline__ float2 mul_word(uint32_t w, uint64_t b) { return unpair_f32(mul_f32x2(pair_f32(lo_f(w), hi_f(w)), b)); }

// ---------------------------------------------------------------------------
// The 32-element group: selection, sparse quantisation, residual quantisation.
// ---------------------------------------------------------------------------
struct ScaleTables {
  float value[128];  // ue4m3 code -> float
  float recip[128];  // IEEE 1.0f / value
};

struct GroupOut {
  uint32_t q_res[4];     // 16 B dense residual payload
  uint32_t a_comp[2];    // 8 B compressed sparse payload
  uint32_t q_sparse[4];  // 16 B dense sparse payload (debug output only)
  uint32_t meta;         // 2 B metadata (4 nibbles)
  uint32_t sf_sparse;    // 1 B
  uint32_t sf_res;       // 2 B (first 16-group in the low byte)
  uint32_t second_min;   // smallest (key - 4) of the second selected pair over the four chunks (see kTinyKey)
};

// four packed e2m1x2 bytes -> four half2 words (element 2i of byte i in the low half)
__device__ __forceinline__ void decode_e2m1x8(uint32_t word, uint32_t (&h)[4]) {
  asm("{\n\t"
      ".reg .b8 b0, b1, b2, b3;\n\t"
      "mov.b32 {b0, b1, b2, b3}, %4;\n\t"
      "cvt.rn.f16x2.e2m1x2 %0, b0;\n\t"
      "cvt.rn.f16x2.e2m1x2 %1, b1;\n\t"
      "cvt.rn.f16x2.e2m1x2 %2, b2;\n\t"
      "cvt.rn.f16x2.e2m1x2 %3, b3;\n\t"
      "}"
      : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3])
      : "r"(word));
}

// The group scale code of max / 6.  The product with float(1/6) stands in for the quotient: both give the same code
// for every float of at most 13 significant bits (an exact multiple of 6 by a short value is hit exactly, every other such
// float is further from a code boundary than the product's error), and the maximum is a bf16 value or
// a residual x - q * s of at most 11 bits (x and q * s are multiples of 2^-9 of the power of two of s where q != 0, and the
// residual is below 2 s; where q == 0 it is x).  A NaN stays one.
__device__ __forceinline__ uint32_t scale_code_from_max(float mx) {
  return float_to_ue4m3(clamp_val(__fmul_rn(mx, 1.0f / 6.0f), kScaleEps, kFp8Max));
}

// max of three in one instruction; NaN operands are dropped as fmaxf drops them
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

template <bool kDebug>
__device__ __forceinline__ void quantize_group32(const uint32_t (&xw)[16], const ScaleTables &tbl, GroupOut &o) {
  float x[32];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    x[2 * i] = lo_f(xw[i]);
    x[2 * i + 1] = hi_f(xw[i]);
  }

  // -- pair selection per 8-element chunk on integer keys; of the selected pairs what is kept is 3 - index (the low key bits)
  uint32_t near_pair[4], far_pair[4];  // 3 - index: the later pair has the smaller value
  uint32_t max_key = 0;
  uint32_t meta = 0;
  uint32_t second_min = 0xFFFFFFFFu;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t key[4];
#pragma unroll
    for (int p = 0; p < 4; ++p)
      key[p] = __float_as_uint(fmaxf(fabsf(x[8 * c + 2 * p]), fabsf(x[8 * c + 2 * p + 1]))) | (uint32_t)(3 - p);
    const uint32_t m01 = max(key[0], key[1]), n01 = min(key[0], key[1]);
    const uint32_t m23 = max(key[2], key[3]), n23 = min(key[2], key[3]);
    const uint32_t best = max(m01, m23);
    const uint32_t second = max(min(m01, m23), max(n01, n23));
    const uint32_t ib = best & 3u, is = second & 3u;
    near_pair[c] = max(ib, is);
    far_pair[c] = min(ib, is);
    meta |= (near_pair[c] | (far_pair[c] << 2)) << (4 * c);
    max_key = max(max_key, best);
    second_min = min(second_min, second - 4u);  // an all-zero pair (key < 4) wraps to a huge value
  }
  o.meta = meta ^ 0xFFFFu;  // index = 3 - kept value, in every two-bit field
  o.second_min = second_min;

  // -- sparse main path scale (one UE4M3 per 32 logical elements)
  const uint32_t s_code = scale_code_from_max(__uint_as_float(max_key & 0xFFFF0000u));
  const float s_q = tbl.value[s_code];
  const float s_r = tbl.recip[s_code];
  o.sf_sparse = s_code;

  // -- quantise every pair, mask to the selected ones, form the residual
  float r[32];
  const uint64_t s_r2 = pair_f32(s_r, s_r), neg_s2 = pair_f32(-s_q, -s_q);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint64_t xp[4];
    float2 t[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      xp[p] = pair_f32(x[8 * c + 2 * p], x[8 * c + 2 * p + 1]);
      t[p] = unpair_f32(mul_f32x2(xp[p], s_r2));
    }
    const uint32_t all4 = pack_e2m1x8(t[0].x, t[0].y, t[1].x, t[1].y, t[2].x, t[2].y, t[3].x, t[3].y);
    const uint32_t mask4 = (0xFF000000u >> (8 * near_pair[c])) | (0xFF000000u >> (8 * far_pair[c]));
    const uint32_t dense4 = all4 & mask4;  // dropped pairs become +0,+0: their residual is x itself
    if (kDebug) o.q_sparse[c] = dense4;
    uint32_t h[4];
    decode_e2m1x8(dense4, h);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const float2 q = __half22float2(*reinterpret_cast<__half2 *>(&h[p]));
      // q * s_q is exact (2-bit x 4-bit significands), so the FMA rounds once like x - (q*s)
      const float2 d = unpair_f32(fma_f32x2(pair_f32(q.x, q.y), neg_s2, xp[p]));
      r[8 * c + 2 * p] = d.x;
      r[8 * c + 2 * p + 1] = d.y;
    }
    // the two kept pair-bytes, ascending pair order
    const uint32_t two = __byte_perm(dense4, 0u, 0x4433u - near_pair[c] - (far_pair[c] << 4));
    if (c & 1)
      o.a_comp[c >> 1] |= two << 16;
    else
      o.a_comp[c >> 1] = two;
  }

  // -- dense residual, one scale per 16
  uint32_t sf_res = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float mx = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; i += 2) mx = max3(mx, fabsf(r[16 * h + i]), fabsf(r[16 * h + i + 1]));
    const uint32_t code = scale_code_from_max(mx);
    const uint64_t rr2 = pair_f32(tbl.recip[code], tbl.recip[code]);
    sf_res |= code << (8 * h);
#pragma unroll
    for (int wv = 0; wv < 2; ++wv) {
      const int i = 16 * h + 8 * wv;
      float2 t[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) t[p] = unpair_f32(mul_f32x2(pair_f32(r[i + 2 * p], r[i + 2 * p + 1]), rr2));
      o.q_res[2 * h + wv] = pack_e2m1x8(t[0].x, t[0].y, t[1].x, t[1].y, t[2].x, t[2].y, t[3].x, t[3].y);
    }
  }
  o.sf_res = sf_res;
}

// bf16(y / scale) of 2 * kWords elements (a 32-element group, or a lane's part of one), y already bf16-exact floats.
// q = y * recip is within 2 ulp of the true quotient; when q is more than 4 ulp away from
// every bf16 rounding boundary (low 16 bits == 0x8000) the IEEE quotient rounds to the same
// bf16 value.  The boundary test is done on packed halves: the low
// 16 bits of both products of a word go into one register (one byte permute), 0x8004 is added
// to each half (a carry out of the low half can only raise the high half by one, which the
// wider threshold absorbs), and a packed unsigned minimum over the group is compared once.
// Where any product lies within the window the words concerned are redone.
template <int kWords>
__device__ __forceinline__ void scale_words(uint32_t (&w)[kWords], float scale, float recip) {
  uint32_t out[kWords];
  uint32_t nearest = 0xFFFFFFFFu;
  const uint64_t recip2 = pair_f32(recip, recip);
#pragma unroll
  for (int i = 0; i < kWords; ++i) {
    const float2 q = mul_word(w[i], recip2);
    const uint32_t lows = __byte_perm(__float_as_uint(q.x), __float_as_uint(q.y), 0x5410);
    nearest = __vminu2(nearest, lows + 0x80048004u);
    out[i] = pack_bf16x2(q.x, q.y);
  }
  if ((nearest & 0xFFFFu) < 10u || (nearest >> 16) < 10u) {
    // Some product of this group is close to a rounding boundary (exact ties are common when
    // the tensor absmax has a short mantissa).  Redo the words concerned with the correctly
    // rounded quotient: two residual corrections q += (y - q*scale) * recip with fused
    // multiply-adds (the classic division refinement, exact because recip is the correctly
    // rounded reciprocal), or an IEEE division for tiny operands or a subnormal quotient.
#pragma unroll
    for (int i = 0; i < kWords; ++i) {
      const float ya = lo_f(w[i]), yb = hi_f(w[i]);
      float qa = __fmul_rn(ya, recip), qb = __fmul_rn(yb, recip);
      const uint32_t ta = (__float_as_uint(qa) + 0x8004u) & 0xFFFFu;
      const uint32_t tb = (__float_as_uint(qb) + 0x8004u) & 0xFFFFu;
      if (ta < 9u || tb < 9u) {
        // residuals are exact for |y| >= 2^-100, and the refinement theorem needs a normal quotient
        if (fminf(fabsf(ya), fabsf(yb)) < 7.8886090522101181e-31f || fminf(fabsf(qa), fabsf(qb)) < 2.3509887e-38f) {
          qa = __fdiv_rn(ya, scale);
          qb = __fdiv_rn(yb, scale);
        } else {
          qa = __fmaf_rn(__fmaf_rn(-qa, scale, ya), recip, qa);
          qb = __fmaf_rn(__fmaf_rn(-qb, scale, yb), recip, qb);
          qa = __fmaf_rn(__fmaf_rn(-qa, scale, ya), recip, qa);
          qb = __fmaf_rn(__fmaf_rn(-qb, scale, yb), recip, qb);
        }
        out[i] = pack_bf16x2(qa, qb);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kWords; ++i) w[i] = out[i];
}

// A selected pair whose score is non-zero but below 2^-118 (key = float bits | pair index).
constexpr uint32_t kTinyKey = 0x04800000u - 4u;

// RMSNorm of both bf16 values of a word: bf16((x * inv) * gamma)
__device__ __forceinline__ uint32_t normalise_word(uint32_t x, uint32_t gamma, uint64_t inv2) {
  const float2 y = unpair_f32(mul_f32x2(mul_f32x2(pair_f32(lo_f(x), hi_f(x)), inv2), pair_f32(lo_f(gamma), hi_f(gamma))));
  return pack_bf16x2(y.x, y.y);
}

// float(bf16(x)): the divisor of the non-RMSNorm path.  On a CUDA device `x / scale` with a bf16
// tensor x and a 0-dim float32 tensor scale (model/quantize.py:179-183 of the reference) casts
// the scale to the common dtype bf16 before dividing in float.
__device__ __forceinline__ float round_to_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// Tensor-scale division and quantisation of one group.
//   kMode 1: the divisor is the float32 scale (the reference's RMSNorm kernel divides by it with
//            __fdiv_rn): products with a boundary test, see scale_words.
//   kMode 2: the divisor has an 8-bit significand (see round_to_bf16), and so has y.  The exact
//            quotient of two such numbers is either representable in 8 bits or at least a
//            relative 2^-17 away from every value with a 9-bit significand, i.e. from every bf16
//            rounding boundary, while y * (1/div) is within 2^-22 of it: the product rounds to
//            the same bf16 as the IEEE quotient, no test needed.  The argument needs a normal
//            quotient; subnormal quotients only matter when such a value takes part in a pair
//            selection, which the keys show (second_min): that group is redone with divisions.
//            The retry reads the group again through `reload` instead of keeping a second copy
//            of it in registers across the quantisation.
template <int kMode, bool kDebug, typename Reload>
__device__ __forceinline__ void scale_quantize_group(uint32_t (&y)[16], float div, float recip, const ScaleTables &tbl,
                                                     GroupOut &o, Reload reload) {
  if (kMode == 1) {
    scale_words(y, div, recip);
    quantize_group32<kDebug>(y, tbl, o);
  } else if (kMode == 2) {
#pragma unroll 1
    for (int attempt = 0; attempt < 2; ++attempt) {
      if (attempt == 0) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float2 q = mul_word(y[i], pair_f32(recip, recip));
          y[i] = pack_bf16x2(q.x, q.y);
        }
      } else {
        reload(y);
#pragma unroll
        for (int i = 0; i < 16; ++i) y[i] = pack_bf16x2(__fdiv_rn(lo_f(y[i]), div), __fdiv_rn(hi_f(y[i]), div));
      }
      quantize_group32<kDebug>(y, tbl, o);
      if (o.second_min >= kTinyKey) break;
    }
  } else {
    quantize_group32<kDebug>(y, tbl, o);
  }
}

// An 8-element chunk of a group whose four chunks lie in four neighbouring lanes (lane & 3): the arithmetic of quantize_group32, a
// quarter of the serial chain per lane.
struct ChunkOut {
  uint32_t q_res;      // 4 B dense residual payload
  uint32_t a_comp;     // 2 B compressed sparse payload
  uint32_t meta;       // a nibble
  uint32_t sf_sparse;  // the group's scale code, in all four lanes
  uint32_t sf_res;     // the 16-group's scale code, in both of its lanes
};

struct ChunkPick {
  uint32_t near_pair, far_pair;  // 3 - index of the kept pairs
  uint32_t best, second;         // their keys
};

__device__ __forceinline__ ChunkPick pick_pairs(const uint32_t (&xw)[4]) {
  uint32_t key[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) key[p] = __float_as_uint(fmaxf(fabsf(lo_f(xw[p])), fabsf(hi_f(xw[p])))) | (uint32_t)(3 - p);
  const uint32_t m01 = max(key[0], key[1]), n01 = min(key[0], key[1]);
  const uint32_t m23 = max(key[2], key[3]), n23 = min(key[2], key[3]);
  ChunkPick c;
  c.best = max(m01, m23);
  c.second = max(min(m01, m23), max(n01, n23));
  c.near_pair = max(c.best & 3u, c.second & 3u);
  c.far_pair = min(c.best & 3u, c.second & 3u);
  return c;
}

__device__ __forceinline__ void quantize_chunk8(const uint32_t (&xw)[4], const ChunkPick &pick, const ScaleTables &tbl, ChunkOut &o) {
  o.meta = (pick.near_pair | (pick.far_pair << 2)) ^ 0xFu;
  uint32_t max_key = pick.best;
  max_key = max(max_key, __shfl_xor_sync(0xffffffffu, max_key, 1));
  max_key = max(max_key, __shfl_xor_sync(0xffffffffu, max_key, 2));
  o.sf_sparse = scale_code_from_max(__uint_as_float(max_key & 0xFFFF0000u));
  const float s_q = tbl.value[o.sf_sparse], s_r = tbl.recip[o.sf_sparse];
  const uint64_t s_r2 = pair_f32(s_r, s_r), neg_s2 = pair_f32(-s_q, -s_q);
  uint64_t xp[4];
  float2 t[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    xp[p] = pair_f32(lo_f(xw[p]), hi_f(xw[p]));
    t[p] = unpair_f32(mul_f32x2(xp[p], s_r2));
  }
  const uint32_t all4 = pack_e2m1x8(t[0].x, t[0].y, t[1].x, t[1].y, t[2].x, t[2].y, t[3].x, t[3].y);
  const uint32_t mask4 = (0xFF000000u >> (8 * pick.near_pair)) | (0xFF000000u >> (8 * pick.far_pair));
  const uint32_t dense4 = all4 & mask4;
  uint32_t h[4];
  decode_e2m1x8(dense4, h);
  float mx = 0.0f;
  uint64_t r[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const float2 q = __half22float2(*reinterpret_cast<__half2 *>(&h[p]));
    r[p] = fma_f32x2(pair_f32(q.x, q.y), neg_s2, xp[p]);
    const float2 d = unpair_f32(r[p]);
    mx = max3(mx, fabsf(d.x), fabsf(d.y));
  }
  o.a_comp = __byte_perm(dense4, 0u, 0x4433u - pick.near_pair - (pick.far_pair << 4));
  mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
  o.sf_res = scale_code_from_max(mx);
  const float rr = tbl.recip[o.sf_res];
#pragma unroll
  for (int p = 0; p < 4; ++p) t[p] = unpair_f32(mul_f32x2(r[p], pair_f32(rr, rr)));
  o.q_res = pack_e2m1x8(t[0].x, t[0].y, t[1].x, t[1].y, t[2].x, t[2].y, t[3].x, t[3].y);
}

__device__ __forceinline__ void zero_range(uint8_t *base, size_t begin, size_t end, int worker, int workers) {
  if (base == nullptr || begin >= end) return;
  // byte-wise head until 16-byte alignment, then 16-byte stores
  size_t a = (begin + 15) & ~(size_t)15;
  if (a > end) a = end;
  for (size_t i = begin + worker; i < a; i += workers) base[i] = 0;
  size_t n16 = (end - a) / 16;
  uint4 z = make_uint4(0, 0, 0, 0);
  for (size_t i = worker; i < n16; i += workers) reinterpret_cast<uint4 *>(base + a)[i] = z;
  for (size_t i = a + n16 * 16 + worker; i < end; i += workers) base[i] = 0;
}

// uint4 index of 16-byte piece j of group g inside a cached row: the pieces of a group are
// permuted so that a quarter-warp reading or writing neighbouring groups hits distinct banks
__device__ __forceinline__ int cache_slot(int g, int j) { return (g << 2) + (j ^ ((g >> 1) & 3)); }

__device__ __forceinline__ unsigned int ld_acquire_gpu(const unsigned int *p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

}  // namespace prep
}  // namespace sharq
