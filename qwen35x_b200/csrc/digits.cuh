// Octal digits of BF16 activations as NVFP4 operand rows, for W4A16 products on the tensor cores (gemm_wstream.cu,
// gemm_resident.cu).
//
// A block of sixteen values whose largest has exponent e is counted in units of 2^(e - 1), which makes every value less than 4:
// digit 0 is the nearest E2M1 number (up to 4 the grid is no coarser than 1, so at most half a unit is left over), digit 1 the
// nearest to eight times the rest, and so on; all of it is exact in fp32.  The unit goes into the block's scale byte, a power
// of two relative to the largest exponent of the token's values (down to 2^-17 of it, the range of E4M3), and 8^-j into the
// epilogue.  d digits leave at most 2^(e + 1 - 3 d), and nothing of a value whose last bit is not below 2^(e + 2 - 3 d).
// Eight digits hold all eight bits of a value down to about 2^-16 of its block's largest one; six more, the deep digits,
// multiples of 2^-40 of the block's largest binade.
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

#include "nvfp4_codec.cuh"

namespace q35b {

constexpr int kDeepDigits = 6;

// The two E2M1 codes of a byte (low nibble first) -> fp32.
__device__ __forceinline__ void from_e2m1x2(uint32_t byte, float & lo, float & hi) {
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t.reg .b32 h;\n\t.reg .b16 l, u;\n\t"
      "mov.b32 {b0, b1, b2, b3}, %2;\n\t"
      "cvt.rn.f16x2.e2m1x2 h, b0;\n\t"
      "mov.b32 {l, u}, h;\n\t"
      "cvt.f32.f16 %0, l;\n\t"
      "cvt.f32.f16 %1, u;\n\t}"
      : "=f"(lo), "=f"(hi)
      : "r"(byte));
}

// Largest of the magnitudes' bit patterns of eight BF16 values.
__device__ __forceinline__ uint32_t bf16x8_abs_max(const uint4 & q) {
  const uint32_t a = __vmaxu2(__vmaxu2(q.x & 0x7fff7fffu, q.y & 0x7fff7fffu), __vmaxu2(q.z & 0x7fff7fffu, q.w & 0x7fff7fffu));
  return max(a & 0xffffu, a >> 16);
}

// `top`: exponent field of the largest value the digits are counted against (at least 1).  The scale of such an expansion,
// 2^(top - 136): the unit of a block at that exponent is 2^(top - 128), and its scale byte stands for 2^8.
__device__ __forceinline__ float digits_scale(int top) {
  return __uint_as_float(top > 9 ? static_cast<uint32_t>(top - 9) << 23 : 1u << (top + 13));
}
// Exponent field that a block is counted at whose largest magnitude is `b`.
__device__ __forceinline__ int digits_exponent(uint32_t b, int top) { return max(max(static_cast<int>(b >> 7), top - 17), 1); }
// E4M3 byte of 2^(8 + e - top).
__device__ __forceinline__ uint32_t digits_scale_byte(int e, int top) {
  const int s = 8 + e - top;
  return s >= -6 ? static_cast<uint32_t>(s + 7) << 3 : 8u >> (-6 - s);
}
// Eight values of a block at exponent e in its units.
__device__ __forceinline__ void digits_begin(const uint4 & q, int e, float (&v)[8]) {
  const float scale = __uint_as_float(static_cast<uint32_t>(255 - e) << 23);  // 2^(128 - e)
  const uint32_t r[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(r[i] << 16) * scale;
    v[2 * i + 1] = __uint_as_float(r[i] & 0xffff0000u) * scale;
  }
}
// The next digit of eight values as E2M1 codes; v: eight times what is left.
__device__ __forceinline__ uint32_t digits_next(float (&v)[8]) {
  const uint32_t w = to_e2m1x8(v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float d0, d1;
    from_e2m1x2(w >> (8 * i), d0, d1);
    v[2 * i] = (v[2 * i] - d0) * 8.0f;
    v[2 * i + 1] = (v[2 * i + 1] - d1) * 8.0f;
  }
  return w;
}

// The outputs (one per lane, weight row `row` of `rows`) of columns k0 .. k1 (k0 a multiple of 256) of a token that has
// infinities but no NaN there.  Next to an infinity the finite activations do not matter, so a warp looks for the infinities,
// 1024 columns at a time, and takes only their products: an infinity, or a NaN where the weight is zero.  It stops as soon as
// every output is a NaN, which opposite signs bring about within a few infinities.  [28672, 9216] with an infinity in seven of eight
// tokens: 76 us, with 256 columns at a time, one load waited for after the other, 141, against 34 without infinities.  (A
// serial sum over all columns for each output took ten times as long.)
static __device__ __noinline__ float infinite_dot(const uint8_t * w_codes, const uint8_t * w_scales, const __nv_bfloat16 * x_row, int rows, int k, int k0,
                                                  int k1, int row, int lane) {
  const bool live = row < rows;
  const uint8_t * codes = w_codes + static_cast<size_t>(live ? row : 0) * (k >> 1);
  const uint4 * x = reinterpret_cast<const uint4 *>(x_row);
  float sum = 0.0f;
  constexpr int kAhead = 4;
#pragma unroll 1
  for (int base0 = k0; base0 < k1; base0 += 256 * kAhead) {
    uint32_t found[kAhead];  // bit i: this lane's value i is infinite; bit 8 + i: and negative
#pragma unroll
    for (int h = 0; h < kAhead; ++h) {
      const int at = (base0 >> 3) + 32 * h + lane;
      const uint4 q = 8 * at < k1 ? __ldcg(x + at) : make_uint4(0u, 0u, 0u, 0u);
      const uint32_t r[4] = {q.x, q.y, q.z, q.w};
      found[h] = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t v = r[i >> 1] >> (16 * (i & 1)) & 0xffffu;
        if ((v & 0x7fffu) == 0x7f80u) found[h] |= (v >> 15 != 0u ? 0x101u : 1u) << i;
      }
    }
#pragma unroll
    for (int h = 0; h < kAhead; ++h) {
      uint32_t lanes = __ballot_sync(0xffffffffu, found[h] != 0u);
      while (lanes != 0u) {
        const int src = __ffs(lanes) - 1;
        lanes &= lanes - 1;
        const uint32_t f = __shfl_sync(0xffffffffu, found[h], src);
        const int c = (base0 >> 3) + 32 * h + src;  // eight columns of one block
        const uint32_t word = *reinterpret_cast<const uint32_t *>(codes + c * 4);
        const float scale = live ? decode_e4m3(w_scales[tiled_scale_offset(row, c >> 1, round_up_int(k >> 4, 4))]) : 0.0f;
#pragma unroll 1
        for (int i = 0; i < 8; ++i) {
          if ((f >> i & 1u) == 0u) continue;
          const float inf = __uint_as_float((f >> (8 + i) & 1u) != 0u ? 0xff800000u : 0x7f800000u);
          sum = fmaf(decode_e2m1(static_cast<uint8_t>(word >> (4 * i) & 15u)) * inf, scale, sum);
        }
        if (__all_sync(0xffffffffu, sum != sum || !live)) return sum;
      }
    }
  }
  return sum;
}

}  // namespace q35b
