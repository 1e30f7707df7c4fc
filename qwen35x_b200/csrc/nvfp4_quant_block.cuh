// One 16-element NVFP4 block: amax -> UE4M3 scale byte -> sixteen E2M1 codes.  Shared by the stand-alone
// quantiser (act_quant.cu) and the GEMM epilogue that emits quantised activations (gemm_epilogue.cuh), so that
// both produce the same bits from the same values.
//
// Recipes (all fp32, IEEE division, no fused contraction that could change a rounding):
//   engine     t = amax_blk / 6; sb = min(UE4M3(max(t / g, 1e-8)), 0x7e); d = max(decode(sb), 1e-8) * g
//   reference  d = max(amax_blk / 6, 1e-8); sb = UE4M3(d)      (src/runtime/cuda_bench.cu:98-213)
//   code_i = E2M1(x_i / d), element 2j in the low nibble (or swapped for the reference's cuBLASLt order)
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

#include "nvfp4_codec.cuh"

namespace q35b {

enum Recipe { kEngine = 0, kReference = 1 };

// x / d rounded to nearest, for a divisor whose refined reciprocal r is at hand: quotient estimate, then two
// residual corrections, the last one delivering the rounded result.  The block's sixteen quotients share one
// divisor, so this replaces sixteen full divisions (each with its own reciprocal and range check) by one
// reciprocal and five dependent-free FMA-pipe instructions per element.  Used only when the block's divisor and
// amax are far from the exponent limits (see quantize_block); tests/test_quant_gpu.py feeds it values placed
// ulp by ulp around every rounding boundary of the E2M1 encoder and compares with IEEE division on the host.
__device__ __forceinline__ float div_by_shared(float x, float d, float r) {
  float q = __fmul_rn(x, r);
  float e = __fmaf_rn(-d, q, x);
  q = __fmaf_rn(e, r, q);
  e = __fmaf_rn(-d, q, x);
  return __fmaf_rn(e, r, q);
}

// encode_e2m1_bounded (nvfp4_codec.cuh) on 32-bit values throughout: no narrowing to a byte and back per element.
__device__ __forceinline__ uint32_t e2m1_code_bounded(float q) {
  const uint32_t au = __float_as_uint(q) & 0x7fffffffu;
  const float a = __uint_as_float(au);
  const uint32_t high = min((au + (0x1fffffu - 0x3f800000u + 0x800000u)) >> 22, 7u);  // 2 + half-exponent steps above 1.0
  const uint32_t low = (a > 0.25f ? 1u : 0u) + (a > 0.75f ? 1u : 0u);
  return ((a >= 1.0f) ? high : low) | ((q < 0.0f) ? 8u : 0u);
}

// Quantise one 16-block; returns the scale byte, writes 8 code bytes.
template <int RECIPE>
__device__ __forceinline__ uint32_t quantize_block(const float (&v)[16], float g, bool swap, uint2 & out) {
  // block amax that turns NaN if any element is NaN (max.NaN), so that such a block is recognised below; the
  // reference's fmaxf chain, which skips NaNs, is recomputed for those blocks only
  float amax = 0.0f;
#pragma unroll
  for (int i = 0; i < 16; ++i) asm("max.NaN.f32 %0, %0, %1;" : "+f"(amax) : "f"(fabsf(v[i])));
  const bool has_nan = amax != amax;
  if (has_nan) {
    amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(v[i]));
  }
  uint32_t sb;
  float d;
  if (RECIPE == kEngine) {
    const float t = __fdiv_rn(amax, 6.0f);
    sb = encode_ue4m3(fmaxf(__fdiv_rn(t, g), 1.0e-8f));
    sb = sb > 0x7eu ? 0x7eu : sb;
    d = __fmul_rn(fmaxf(decode_e4m3(static_cast<uint8_t>(sb)), 1.0e-8f), g);
  } else {
    d = fmaxf(__fdiv_rn(amax, 6.0f), 1.0e-8f);
    sb = encode_ue4m3(d);
  }
  // exponents of d and amax inside [2^-60, 2^60]: no intermediate of the shared-reciprocal quotients can overflow,
  // and a quotient small enough to lose bits is far below the first rounding boundary (0.25); amax < 2^19 d keeps
  // every quotient finite and far inside the converter's range
  const uint32_t de = (__float_as_uint(d) >> 23) & 0xffu, ae = (__float_as_uint(amax) >> 23) & 0xffu;
  uint32_t word[2] = {0u, 0u};
  if (!has_nan && de >= 67u && de <= 187u && ae <= 187u && amax < d * 524288.0f) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    r = __fmaf_rn(r, __fmaf_rn(-d, r, 1.0f), r);
    // Bracket every quotient: x * r lies within 2^-23 (relative) of x / d, so lo = x * r (1 - 2^-20) and
    // hi = x * r (1 + 2^-20) enclose the correctly rounded quotient strictly.  The code is a monotone function of
    // the quotient and the hardware converter agrees with the reference's nearest-with-ties-down encoder
    // everywhere except exactly on a rounding boundary, so where lo and hi convert to the same code the
    // reference's code is that code; a boundary inside the bracket shows up as two different codes, and only that
    // pair of elements is redone with correctly rounded quotients and the ties-down encoder.  A negative value that
    // rounds to zero keeps its sign bit in both encoders; the + 0.0f turns x = -0 into +0, as (value < 0) does.
    const float r_lo = __fmul_rn(r, 1.0f - 0x1p-20f), r_hi = __fmul_rn(r, 1.0f + 0x1p-20f);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float lo[8], hi[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        lo[i] = __fmaf_rn(v[8 * h + i], r_lo, 0.0f);
        hi[i] = __fmaf_rn(v[8 * h + i], r_hi, 0.0f);
      }
      const uint32_t w_lo = to_e2m1x8(lo), w_hi = to_e2m1x8(hi);
      uint32_t w = w_lo;
      const uint32_t diff = w_lo ^ w_hi;
      if (diff != 0u) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if ((diff >> (8 * j)) & 0xffu) {
            const uint32_t c0 = e2m1_code_bounded(div_by_shared(v[8 * h + 2 * j], d, r));
            const uint32_t c1 = e2m1_code_bounded(div_by_shared(v[8 * h + 2 * j + 1], d, r));
            w = (w & ~(0xffu << (8 * j))) | ((c0 | (c1 << 4)) << (8 * j));
          }
        }
      }
      word[h] = w;
    }
  } else {
    uint32_t code[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) code[i] = encode_e2m1(__fdiv_rn(v[i], d));
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int i = 7; i >= 0; --i) word[h] = word[h] * 16u + code[8 * h + i];
    }
  }
  // element 2j sits in the low nibble of byte j; the reference's cuBLASLt order swaps the two nibbles of every byte
  if (swap) {
#pragma unroll
    for (int h = 0; h < 2; ++h) word[h] = ((word[h] & 0x0f0f0f0fu) << 4) | ((word[h] >> 4) & 0x0f0f0f0fu);
  }
  out = make_uint2(word[0], word[1]);
  return sb;
}

// ---- sixteen BF16 values, engine recipe -------------------------------------------------------------------------
//
// A BF16 value has eight significant bits, so with one divisor d the BF16 values next to b * d for a rounding boundary b are
// 2^-8 of it apart: one of them at most lies closer than 2^-21, and whether its correctly rounded quotient is above b (or
// on it, a tie that goes down) can be worked out beforehand.  If no such value has to go up, one multiplication by a
// reciprocal that is a little too small (1 - 2^-22) puts every quotient on its side of every boundary; if none has to go
// down, one that is a little too large does.  The hardware converter then finishes the job: one conversion per pair where
// quantize_block needs two and a comparison.  The choice depends on the block's scale byte and the tensor's scale only, so
// there are 127 multipliers per tensor: bf16_block_multiplier gives one of them, or 0 for "use quantize_block", and a
// kernel that quantises many blocks per CTA keeps them in a table.  (Such close values are no rarity: under the scale of
// a tensor, amax / 2688, an eighth of the scale bytes have divisors that are thirds of BF16 values.)

// The multiplier for scale byte sb (0..0x7e) under per-tensor scale g.
__device__ __forceinline__ float bf16_block_multiplier(uint32_t sb, float g) {
  if (!(g >= 0x1p-60f && g <= 0x1p60f)) return 0.0f;
  const float d = __fmul_rn(fmaxf(decode_e4m3(static_cast<uint8_t>(sb)), 1.0e-8f), g);
  if (!(d <= 0x1p15f)) return 0.0f;  // beyond, a quotient may round to zero, which loses its sign
  // The boundaries are 1, 1.25, 1.5 and 1.75 times powers of two.  p: d times one of these, in quarters of d's last bit;
  // BF16 values are 2^18 of them apart in the binade of d, 2^19 in the next one.
  const uint32_t mant = (__float_as_uint(d) & 0x7fffffu) | 0x800000u;
  bool up = false, down = false;
#pragma unroll 1
  for (uint32_t n = 4; n < 8; ++n) {
    const uint32_t p = mant * n, spacing = p < (1u << 26) ? (1u << 18) : (1u << 19);
    const uint32_t near = (p + (spacing >> 1)) & ~(spacing - 1);
    if (static_cast<uint32_t>(abs(static_cast<int>(near - p))) <= (p >> 21) + 1u) {
      const bool above = __fdiv_rn(static_cast<float>(near) * 0.25f, static_cast<float>(mant)) > static_cast<float>(n) * 0.25f;
      up = up || above;
      down = down || !above;
    }
  }
  if (up && down) return 0.0f;
  // errors of the reciprocal, the product and the quotient's own rounding are 2^-24 each: the sum stays below 2^-22, and
  // 2^-22 and all of them below 2^-21
  return __fmul_rn(__frcp_rn(d), up ? 1.0f + 0x1p-22f : 1.0f - 0x1p-22f);
}

__device__ __forceinline__ uint32_t bf16x2_abs_max_nan(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.NaN.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// quantize_block for what the multipliers do not cover (NaN, infinities, extreme scales, boundaries of both kinds), out of
// line.
static __device__ __noinline__ uint3 quantize_block_bf16_general(uint4 a, uint4 b, float g) {
  const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  float v[16];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
  uint2 packed;
  const uint32_t sb = quantize_block<kEngine>(v, g, false, packed);
  return make_uint3(packed.x, packed.y, sb);
}

// Two BF16 values of a register times m as fp32 (+ 0: a negative zero becomes positive, as (value < 0) has it).
__device__ __forceinline__ void bf16x2_scaled(uint32_t w, float m, float & lo, float & hi) {
  asm("{\n\t.reg .b32 l, h;\n\t.reg .b64 v, mm, z;\n\t"
      "shl.b32 l, %2, 16;\n\tand.b32 h, %2, 0xffff0000;\n\t"
      "mov.b64 v, {l, h};\n\tmov.b64 mm, {%3, %3};\n\tmov.b64 z, {%4, %4};\n\t"
      "fma.rn.f32x2 v, v, mm, z;\n\tmov.b64 {%0, %1}, v;\n\t}"
      : "=f"(lo), "=f"(hi)
      : "r"(w), "f"(m), "f"(0.0f));
}

// The bytes of quantize_block<kEngine> for sixteen BF16 values, two per register.  rg = 1 / g correctly rounded;
// TABLE: `table` holds the multipliers of this tensor by scale byte; else the one needed is worked out here.
template <bool TABLE>
__device__ __forceinline__ uint32_t quantize_block_bf16(const uint4 a, const uint4 b, float g, float rg, const float * table, uint2 & out) {
  uint32_t am = bf16x2_abs_max_nan(bf16x2_abs_max_nan(bf16x2_abs_max_nan(a.x, a.y), bf16x2_abs_max_nan(a.z, a.w)),
                                   bf16x2_abs_max_nan(bf16x2_abs_max_nan(b.x, b.y), bf16x2_abs_max_nan(b.z, b.w)));
  am = max((am << 16) & 0x7fffffffu, am & 0x7fff0000u);
  // amax / 6 / g: with a correctly rounded reciprocal the second correction delivers the rounded quotient (Markstein 1990)
  const float t = div_by_shared(__uint_as_float(am), 6.0f, 1.0f / 6.0f);
  const float s = div_by_shared(t, g, rg);
  const uint32_t u = __float_as_uint(s);
  // encode_ue4m3 up to 2^24, without its branches
  const uint32_t normal = min(((u + 0x7ffffu) >> 20) - 960u, 0x7eu);
  const uint32_t small = static_cast<uint32_t>(max(__float2int_ru(fmaf(s, 512.0f, -0.5f)), 0));
  const uint32_t sb = u < 0x3c800000u ? small : normal;
  float m;
  if constexpr (TABLE) m = table[sb]; else m = bf16_block_multiplier(sb, g);
  const bool in_range = am - 0x21800000u <= 0x5d800000u - 0x21800000u || am == 0u;  // 2^-60 .. 2^60: no rounding above is off
  if (!in_range || u >= 0x4b800000u || m == 0.0f) {
    const uint3 r = quantize_block_bf16_general(a, b, g);
    out = make_uint2(r.x, r.y);
    return r.z;
  }
  float q[8];
  bf16x2_scaled(a.x, m, q[0], q[1]);
  bf16x2_scaled(a.y, m, q[2], q[3]);
  bf16x2_scaled(a.z, m, q[4], q[5]);
  bf16x2_scaled(a.w, m, q[6], q[7]);
  out.x = to_e2m1x8(q);
  bf16x2_scaled(b.x, m, q[0], q[1]);
  bf16x2_scaled(b.y, m, q[2], q[3]);
  bf16x2_scaled(b.z, m, q[4], q[5]);
  bf16x2_scaled(b.w, m, q[6], q[7]);
  out.y = to_e2m1x8(q);
  return sb;
}

// ---- as the kernels that quantise activations use them: values as they lie in memory ----------------------------

// |values| of 16 bytes into the running maximum; like fmaxf both skip NaNs.
template <typename T>
__device__ __forceinline__ float abs_max(const uint4 q, float best);
template <>
__device__ __forceinline__ float abs_max<float>(const uint4 q, float best) {
  return fmaxf(best, fmaxf(fmaxf(fabsf(__uint_as_float(q.x)), fabsf(__uint_as_float(q.y))),
                           fmaxf(fabsf(__uint_as_float(q.z)), fabsf(__uint_as_float(q.w)))));
}
__device__ __forceinline__ uint32_t bf16x2_abs_max(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
template <>
__device__ __forceinline__ float abs_max<__nv_bfloat16>(const uint4 q, float best) {
  // two values per instruction; a pair of NaNs leaves one, which the last step skips
  const uint32_t m = bf16x2_abs_max(bf16x2_abs_max(q.x, q.y), bf16x2_abs_max(q.z, q.w));
  return fmaxf(best, fmaxf(fabsf(__uint_as_float(m << 16)), fabsf(__uint_as_float(m & 0xffff0000u))));
}

// Codes and scale byte of one block.
template <typename T, bool TABLE>
__device__ __forceinline__ uint32_t quantize_raw(const uint4 (&r)[sizeof(T)], float g, float rg, const float * table, uint2 & out) {
  if constexpr (sizeof(T) == 2) {
    return quantize_block_bf16<TABLE>(r[0], r[1], g, rg, table, out);
  } else {
    float v[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[4 * i] = __uint_as_float(r[i].x);
      v[4 * i + 1] = __uint_as_float(r[i].y);
      v[4 * i + 2] = __uint_as_float(r[i].z);
      v[4 * i + 3] = __uint_as_float(r[i].w);
    }
    return quantize_block<kEngine>(v, g, false, out);
  }
}

}  // namespace q35b
