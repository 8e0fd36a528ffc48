// FP64 products, squares and quotients on the integer pipes, rounded exactly
// as the FP64 unit rounds them (round to nearest, ties to even).
//
// GB300 issues FP64 instructions at 1/64 of its FP32 rate: one FP64
// instruction of a warp holds its scheduler partition's FP64 pipe for about
// 64 cycles, in which the integer and FMA pipes can issue some 40 to 60 other
// instructions.  A product of two 53-bit significands is four 32 x 32 -> 64
// bit multiply-adds plus a shift and a rounding step (about 22 instructions),
// a quotient about 48, against 64 and 500 cycles of the FP64 pipe; and they
// run beside the FP64 additions of the surrounding formula instead of before
// them.  Each routine states the operand range it is exact for; the callers
// check the range once per formula and take the FP64 unit outside it.
//
// The arithmetic is plain binary floating point by its definition (integer
// significand product / long division, then IEEE 754 rounding); the division
// takes its quotient digits from a 31-bit reciprocal, corrected by the exact
// integer remainder.
#pragma once

#include <stdint.h>
#include <string.h>

namespace lsmgpu {
namespace fpi {

#ifdef __CUDACC__
#define LSMGPU_FPI __host__ __device__ __forceinline__
#else
#define LSMGPU_FPI inline
#endif

// the two 32-bit words of a double
struct W2 {
  uint32_t hi, lo;
};
LSMGPU_FPI W2 words(double x) {
#ifdef __CUDA_ARCH__
  return {(uint32_t)__double2hiint(x), (uint32_t)__double2loint(x)};
#else
  uint64_t b;
  memcpy(&b, &x, 8);
  return {(uint32_t)(b >> 32), (uint32_t)b};
#endif
}
LSMGPU_FPI double from_words(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)hi, (int)lo);
#else
  const uint64_t b = ((uint64_t)hi << 32) | lo;
  double x;
  memcpy(&x, &b, 8);
  return x;
#endif
}
// (h:l << s) >> 32, 0 < s < 32
LSMGPU_FPI uint32_t funnel(uint32_t l, uint32_t h, uint32_t s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(l, h, s);
#else
  return (h << s) | (l >> (32 - s));
#endif
}
LSMGPU_FPI uint32_t mul_hi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }

// An unpacked operand: its significand words (implicit bit set), exponent
// field in place, sign bit, and a mask that is 0 where the value counts as
// zero (all ones otherwise).
struct Op {
  uint32_t m1, m0;   // significand = m1 * 2^32 + m0, 2^52 <= significand < 2^53
  uint32_t e;        // biased exponent << 20
  uint32_t sign;     // 0 or 0x80000000
  uint32_t keep;     // 0: the operand counts as zero
};
// Values with a biased exponent below `floor_e` count as zero.
LSMGPU_FPI Op unpack(double x, uint32_t floor_e) {
  const W2 w = words(x);
  Op o;
  o.m1 = (w.hi & 0x000fffffu) | 0x00100000u;
  o.m0 = w.lo;
  o.e = w.hi & 0x7ff00000u;
  o.sign = w.hi & 0x80000000u;
  o.keep = o.e < (floor_e << 20) ? 0u : 0xffffffffu;
  return o;
}

// a * b for operands that are normal numbers (or count as zero) whose
// product is a normal number.
LSMGPU_FPI double mul(const Op &a, const Op &b) {
  // 106-bit significand product in words w3..w0
  const uint64_t p00 = (uint64_t)a.m0 * b.m0;
  const uint64_t t = (uint64_t)a.m1 * b.m0 + (p00 >> 32);
  const uint64_t u = (uint64_t)a.m0 * b.m1 + (uint32_t)t;
  const uint64_t h = (uint64_t)a.m1 * b.m1 + (t >> 32) + (u >> 32);
  const uint32_t w3 = (uint32_t)(h >> 32), w2 = (uint32_t)h, w1 = (uint32_t)u, w0 = (uint32_t)p00;
  // leading bit at bit 8 or 9 of w3: shift it to bit 20
  const uint32_t norm = w3 >> 9;
  const uint32_t s = 12 - norm;
  const uint32_t rem = funnel(w0, w1, s) | (w0 != 0u ? 1u : 0u);  // round bit on top, sticky at the bottom
  const uint64_t q = ((uint64_t)funnel(w2, w3, s) << 32) | funnel(w1, w2, s);
  // ties to even: carry out of rem + 0x7fffffff + (last bit)
  const uint64_t up = ((uint64_t)rem + 0x7fffffffu + ((uint32_t)q & 1u)) >> 32;
  const uint64_t r = q + up;
  // r holds the implicit bit, so the exponent field is added less one
  const uint32_t e = a.e + b.e + (norm << 20) - (1024u << 20);
  const uint32_t hi = (uint32_t)(r >> 32) + e;
  return from_words((hi & (a.keep & b.keep)) | (a.sign ^ b.sign), (uint32_t)r & (a.keep & b.keep));
}

// x * x, same range
LSMGPU_FPI double sqr(const Op &a) {
  const uint64_t p00 = (uint64_t)a.m0 * a.m0;
  const uint64_t c = (uint64_t)a.m1 * a.m0;  // < 2^53
  const uint64_t u = (c << 1) + (p00 >> 32);
  const uint64_t h = (uint64_t)a.m1 * a.m1 + (u >> 32);
  const uint32_t w3 = (uint32_t)(h >> 32), w2 = (uint32_t)h, w1 = (uint32_t)u, w0 = (uint32_t)p00;
  const uint32_t norm = w3 >> 9;
  const uint32_t s = 12 - norm;
  const uint32_t rem = funnel(w0, w1, s) | (w0 != 0u ? 1u : 0u);
  const uint64_t q = ((uint64_t)funnel(w2, w3, s) << 32) | funnel(w1, w2, s);
  const uint64_t up = ((uint64_t)rem + 0x7fffffffu + ((uint32_t)q & 1u)) >> 32;
  const uint64_t r = q + up;
  const uint32_t e = 2 * a.e + (norm << 20) - (1024u << 20);
  return from_words(((uint32_t)(r >> 32) + e) & a.keep, (uint32_t)r & a.keep);
}

// n / d for positive normal numbers whose quotient is a normal number.  Each
// approximation errs downwards: x by at most 5 units, so the first 31 bits by
// at most 7 (r1 < 8 D), and the 54-bit quotient by less than 2 before its
// floor, which one exact remainder test settles.
LSMGPU_FPI double div_pos(double n, double d) {
  const W2 nw = words(n), dw = words(d);
  const uint32_t D1 = (dw.hi & 0x000fffffu) | 0x00100000u;
  const uint64_t D = ((uint64_t)D1 << 32) | dw.lo;  // 2^52 <= D < 2^53
  const uint64_t N = ((uint64_t)((nw.hi & 0x000fffffu) | 0x00100000u) << 32) | nw.lo;
  // top 32 bits of D, leading bit set
  const uint32_t d1 = funnel(dw.lo, D1, 11);
  // x <= 2^63 / (d1 + 1), to about 30 bits: FP32 reciprocal of the leading
  // 24 bits, lowered so that it stays below, and one Newton step
  uint32_t x;
  {
    const uint32_t fb = 0x3f800000u | ((d1 >> 8) & 0x007fffffu);
    float f, y;
#ifdef __CUDA_ARCH__
    f = __uint_as_float(fb);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
    const uint32_t yb = __float_as_uint(y);
#else
    memcpy(&f, &fb, 4);
    y = 1.0f / f;
    uint32_t yb;
    memcpy(&yb, &y, 4);
#endif
    // y in [0.5, 1]; less 4 units of 2^-24, as an integer of units 2^-32
    const uint32_t x0 = (yb - 0x3f000000u - 4u) * 256u + 0x80000000u;
    const uint64_t err = 0x8000000000000000ull - (uint64_t)x0 * ((uint64_t)d1 + 1u);  // >= 0, < 2^43
    x = x0 + (mul_hi(x0, (uint32_t)(err >> 11)) >> 20);
  }
  // quotient scaled into [1/2, 1): halve the numerator where N >= D
  const uint32_t ge = N >= D ? 1u : 0u;
  // 2^31 N / D (or half of it): first 31 bits
  const uint32_t n1 = (uint32_t)(N >> 21) >> ge;  // leading 32 (31) bits of N
  const uint32_t qa = mul_hi(n1, x);
  // exact remainder r1 = (N << (31 - ge)) - qa D, 0 <= r1 < 8 D, modulo 2^64
  const uint64_t r1 = (N << (31 - ge)) - (uint64_t)qa * D;
  // next 23 bits, at most one too small
  uint32_t qb = mul_hi((uint32_t)(r1 >> 24), x) >> 5;
  const uint64_t r2 = (r1 << 23) - (uint64_t)qb * D;
  if (r2 >= D) qb++;
  // 54 quotient bits; the remainder is not a tie (a quotient of two 53-bit
  // numbers is never half way between two), so adding one rounds
  const uint64_t q = ((((uint64_t)qa << 23) + qb) + 1u) >> 1;
  const uint32_t e = (nw.hi & 0x7ff00000u) - (dw.hi & 0x7ff00000u) + ((1021u + ge) << 20);
  return from_words((uint32_t)(q >> 32) + e, (uint32_t)q);
}

// the bits of |v|: they order magnitudes as integers
LSMGPU_FPI unsigned long long mag(double v) {
  const W2 w = words(v);
  return ((unsigned long long)(w.hi & 0x7fffffffu) << 32) | w.lo;
}

}  // namespace fpi
}  // namespace lsmgpu
