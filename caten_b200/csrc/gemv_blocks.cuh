// Per-format arithmetic of one 32-wide block of a weight row against 32 activations held in
// registers.
#pragma once
#include "common.cuh"

namespace cb {

// Two fp32 values in a register pair, the first in the low half, and arithmetic on both in one instruction (each rounded by itself).
// Of use to Q8_0 (GPT-2 XL, one sequence at 300 positions: 1371 -> 1349 us a step); the nibble formats and dense rows were slower
// with it (XL Q4_0 1200 -> 1263, XL bf16 1473 -> 1776).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 f2(float a, float b) { return (f32x2)__float_as_uint(a) | (f32x2)__float_as_uint(b) << 32; }
__device__ __forceinline__ f32x2 f2u(uint32_t a, uint32_t b) { return (f32x2)a | (f32x2)b << 32; }
__device__ __forceinline__ float f2_sum(f32x2 v) { return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// ---- per-format block arithmetic -------------------------------------------------------------
// A thread owns one 32-wide column block kb of x and walks down the rows of W.
//
// Q4_0.  A nibble masked in place inside its 32-bit word, `w & (0xF << p)`, reinterpreted as a
// float, is the (sub)normal number nibble * 2^(p-149): the binary32 encoding is linear in its
// integer bit pattern below 2^24.  So with x pre-multiplied by 2^(64-p) (a power of two: exact),
// one AND plus one FMA accumulates x*nibble*2^-85 exactly as an fp32 FMA of x and nibble would,
// with no shift, integer-to-float conversion or subtraction per weight.  The "-8" offset of
// Q4_0 is folded into the accumulator's start value -8*sum(x)*2^-85, and 2^85 into the block
// scale.  Nibbles of the top byte (bits 24..31 overlap the exponent field) are taken from
// w >> 8.  Valid for |x| < 2^62; FMA with subnormal operands runs at full rate.
//
// x is scaled on its way to shared memory (stage: four consecutive elements, the j-th such group of their block), once for all
// the threads that use it, and the sum of each block lies beside it.
struct BlkQ4 {
  static constexpr bool HAS_M = false, HAS_QH = false, SUMS = true;
  static constexpr int WORDS = 4;
  float xs[32];
  float c0;
  static __device__ __forceinline__ float4 stage(float4 v, int j) {
    // elements 0..15 are the low nibbles of bytes 0..15 (p = 0, 8, 16 and, of w >> 8, 16), 16..31 the high ones (p = 4, 12, 20, 20)
    const float up = j < 4 ? 0x1p64f : 0x1p60f;
    return make_float4(v.x * up, v.y * (up * 0x1p-8f), v.z * (up * 0x1p-16f), v.w * (up * 0x1p-16f));
  }
  __device__ __forceinline__ void prep(const float *xv, float sum) {
    c0 = sum * -0x1p-82f;  // -8 * 2^-85
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        xs[8 * i + 2 * e] = xv[4 * i + e];
        xs[8 * i + 2 * e + 1] = xv[16 + 4 * i + e];
      }
  }
  __device__ __forceinline__ float dot(const uint32_t *w, float scale) const {
    float a0 = c0, a1 = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t q = w[i], q8 = q >> 8;
      a0 = fmaf(xs[8 * i + 0], __uint_as_float(q & 0x0000000Fu), a0);
      a1 = fmaf(xs[8 * i + 1], __uint_as_float(q & 0x000000F0u), a1);
      a0 = fmaf(xs[8 * i + 2], __uint_as_float(q & 0x00000F00u), a0);
      a1 = fmaf(xs[8 * i + 3], __uint_as_float(q & 0x0000F000u), a1);
      a0 = fmaf(xs[8 * i + 4], __uint_as_float(q & 0x000F0000u), a0);
      a1 = fmaf(xs[8 * i + 5], __uint_as_float(q & 0x00F00000u), a1);
      a0 = fmaf(xs[8 * i + 6], __uint_as_float(q8 & 0x000F0000u), a0);
      a1 = fmaf(xs[8 * i + 7], __uint_as_float(q8 & 0x00F00000u), a1);
    }
    return (a0 + a1) * (scale * 0x1p85f);
  }
};

// An unsigned integer below 2^23 or-ed into the mantissa of 2^23 is the float 2^23 + it, from which the subtraction of
// 2^23 (and of the code's offset) is exact: full-rate instructions where the integer-to-float conversion runs at an
// eighth of the rate (GPT-2 XL Q8_0, one sequence: a step took 1981 us with the conversion, 1758 us so).
__device__ __forceinline__ float code_to_float(uint32_t magic, float offset) { return __uint_as_float(magic) - (8388608.0f + offset); }

// Q8_0: byte (biased by 128) -> float -> FMA; (float)q * scale is exact in fp32 (8 + 11 bits), so
// scaling the 32-term sum once per block only changes where the roundings of the sum fall.
struct BlkQ8 {
  static constexpr bool HAS_M = false, HAS_QH = false, SUMS = false;
  static constexpr int WORDS = 8;
  float xs[32];
  static __device__ __forceinline__ float4 stage(float4 v, int) { return v; }
  __device__ __forceinline__ void prep(const float *xv, float) {
#pragma unroll
    for (int j = 0; j < 32; ++j) xs[j] = xv[j];
  }
  __device__ __forceinline__ float dot(const uint32_t *w, float scale) const {
    f32x2 a = 0, b = 0;
    const f32x2 off = f2(-8388736.0f, -8388736.0f);   // 2^23 + 128
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t q = w[i] ^ 0x80808080u;
      a = fma2(f2(xs[4 * i + 0], xs[4 * i + 1]), add2(f2u(__byte_perm(q, 0x4B000000u, 0x7440), __byte_perm(q, 0x4B000000u, 0x7441)), off), a);
      b = fma2(f2(xs[4 * i + 2], xs[4 * i + 3]), add2(f2u(__byte_perm(q, 0x4B000000u, 0x7442), __byte_perm(q, 0x4B000000u, 0x7443)), off), b);
    }
    return f2_sum(add2(a, b)) * scale;
  }
};

// Q4_1: w = q * d + m.  The nibble arithmetic of BlkQ4 without the -8 offset; the minimum enters
// once per block as m * sum(x).
struct BlkQ41 {
  static constexpr bool HAS_M = true, HAS_QH = false, SUMS = true;
  static constexpr int WORDS = 4;
  BlkQ4 nib;
  float sumx;
  static __device__ __forceinline__ float4 stage(float4 v, int j) { return BlkQ4::stage(v, j); }
  __device__ __forceinline__ void prep(const float *xv, float sum) {
    nib.prep(xv, sum);
    nib.c0 = 0.0f;
    sumx = sum;
  }
  __device__ __forceinline__ float dotx(const uint32_t *w, float scale, float mn, uint32_t) const {
    return nib.dot(w, scale) + mn * sumx;
  }
};

// Q5_0 (w = (q - 16) * d) and Q5_1 (w = q * d + m): code = nibble | bit e of qh << 4, converted
// with an integer-to-float instruction per weight.
template <bool WITH_MIN>
struct BlkQ5 {
  static constexpr bool HAS_M = WITH_MIN, HAS_QH = true, SUMS = WITH_MIN;
  static constexpr int WORDS = 4;
  float xs[32];
  float sumx;
  static __device__ __forceinline__ float4 stage(float4 v, int) { return v; }
  __device__ __forceinline__ void prep(const float *xv, float sum) {
#pragma unroll
    for (int j = 0; j < 32; ++j) xs[j] = xv[j];
    sumx = sum;
  }
  __device__ __forceinline__ float dotx(const uint32_t *w, float scale, float mn, uint32_t qh) const {
    constexpr float OFF = WITH_MIN ? 0.0f : 16.0f;
    float a0 = 0.0f, a1 = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int j = 4 * i + b;  // byte j: elements j and j + 16
        const uint32_t lo = 0x4B000000u | ((w[i] >> (8 * b)) & 15u) | (((qh >> j) & 1u) << 4);
        const uint32_t hi = 0x4B000000u | ((w[i] >> (8 * b + 4)) & 15u) | (((qh >> (j + 16)) & 1u) << 4);
        a0 = fmaf(xs[j], code_to_float(lo, OFF), a0);
        a1 = fmaf(xs[j + 16], code_to_float(hi, OFF), a1);
      }
    }
    const float r = (a0 + a1) * scale;
    return WITH_MIN ? r + mn * sumx : r;
  }
};

}  // namespace cb
