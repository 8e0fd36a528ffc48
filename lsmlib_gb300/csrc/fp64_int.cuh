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

#include <math.h>
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

// An unpacked operand: its significand words (implicit bit set), the rest of
// its high word (sign and biased exponent less one, in place; these parts of
// two operands add like the numbers multiply), and whether it counts as zero.
struct Op {
  uint32_t m1, m0;  // significand = m1 * 2^32 + m0, 2^52 <= significand < 2^53
  uint32_t x;
  bool zero;
};
// Values with a biased exponent below `floor_e` count as zero.
LSMGPU_FPI Op unpack(double v, uint32_t floor_e) {
  const W2 w = words(v);
  Op o;
  o.m1 = (w.hi & 0x000fffffu) | 0x00100000u;
  o.m0 = w.lo;
  o.x = w.hi - o.m1;
  o.zero = (w.hi & 0x7fffffffu) < (floor_e << 20);
  return o;
}
// one known to be a normal number
LSMGPU_FPI Op unpack_normal(double v) {
  Op o = unpack(v, 1);
  o.zero = false;
  return o;
}

// Rounds the 106-bit significand product w3:w2:w1:w0 (leading bit at bit 8 or
// 9 of w3) to 53 bits, ties to even, under the sign and exponent part x.  The
// left shift by 11 or 12 is a multiplication: it runs on the multiply-add
// pipe, which these routines load less than the logic pipe.
LSMGPU_FPI double round_product(uint32_t w3, uint32_t w2, uint32_t w1, uint32_t w0, uint32_t x, bool zero) {
  const uint32_t norm = w3 >> 9;
  const uint32_t f = 4096u - norm * 2048u;
  const uint64_t c1 = (uint64_t)w1 * f;
  const uint64_t c2 = (uint64_t)w2 * f + (c1 >> 32);
  const uint32_t lo = (uint32_t)c2, hi = w3 * f + (uint32_t)(c2 >> 32);
  // round bit on top, the bits of w0 only as a sticky bit
  const uint32_t rem = (uint32_t)c1 | (w0 < 1u ? w0 : 1u);
  // carry out of rem + 0x7fffffff + (last bit) rounds up
  const uint64_t up = ((uint64_t)rem + 0x7fffffffu + (lo & 1u)) >> 32;
  const uint64_t r = (((uint64_t)(hi + x + norm * 0x00100000u) << 32) | lo) + up;
  return zero ? 0.0 : from_words((uint32_t)(r >> 32), (uint32_t)r);
}

// a * b for operands that are normal numbers (or count as zero) whose
// product is a normal number.  (A zero result is +0.)
LSMGPU_FPI double mul(const Op &a, const Op &b) {
  const uint64_t p00 = (uint64_t)a.m0 * b.m0;
  const uint64_t t = (uint64_t)a.m1 * b.m0 + (p00 >> 32);  // < 2^54
  const uint64_t u = (uint64_t)a.m0 * b.m1 + t;            // < 2^55
  const uint64_t h = (uint64_t)a.m1 * b.m1 + (u >> 32);
  return round_product((uint32_t)(h >> 32), (uint32_t)h, (uint32_t)u, (uint32_t)p00, a.x + b.x - 0x3fe00000u,
                       a.zero || b.zero);
}

// x * x, same range
LSMGPU_FPI double sqr(const Op &a) {
  const uint64_t p00 = (uint64_t)a.m0 * a.m0;
  const uint64_t u = (uint64_t)(2u * a.m1) * a.m0 + (p00 >> 32);  // < 2^55
  const uint64_t h = (uint64_t)a.m1 * a.m1 + (u >> 32);
  return round_product((uint32_t)(h >> 32), (uint32_t)h, (uint32_t)u, (uint32_t)p00, 2u * a.x - 0x3fe00000u, a.zero);
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

// sqrt(x) for a positive normal number.  Each approximation errs downwards:
// y by less than 2^-29 of itself, so the first 31 bits by at most 5 units and
// the 54-bit root by less than 1.5, which one exact remainder test settles.
LSMGPU_FPI double sqrt_pos(double x) {
  const W2 w = words(x);
  const uint32_t odd = (w.hi >> 20) & 1u;  // biased exponent odd: an even power of two
  const uint64_t M = ((uint64_t)((w.hi & 0x000fffffu) | 0x00100000u) << 32) | w.lo;
  // v = significand / 4 (even power) or / 2 (odd power), in [1/4, 1), as V 2^-64
  const uint64_t V = M << (11 - odd);
  const uint32_t v1 = (uint32_t)(V >> 32);
  // y <= 1 / sqrt(v) in units of 2^-31, to about 28 bits: FP32 reciprocal
  // square root of the leading 24 bits, lowered, and one Newton step
  uint32_t y;
  {
    const uint32_t fb = ((126u - odd) << 23) | ((uint32_t)(M >> 29) & 0x007fffffu);
    float f, r;
    uint32_t rb;
#ifdef __CUDA_ARCH__
    f = __uint_as_float(fb);
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
    rb = __float_as_uint(r);
#else
    memcpy(&f, &fb, 4);
    r = 1.0f / __builtin_sqrtf(f);
    memcpy(&rb, &r, 4);
#endif
    // r in [1, 2]; less 6 units of 2^-23, in units of 2^-31
    const uint32_t y0 = (rb - 0x3f800000u - 6u) * 256u + 0x80000000u;
    // g = 1 - v y0^2 (>= 0, < 2^-18) in units of 2^-62, v taken as v1 + 1
    const uint64_t vy = ((uint64_t)y0 * ((uint64_t)v1 + 1u)) >> 32;         // v y0, units 2^-31
    const uint64_t g = 0x4000000000000000ull - (uint64_t)y0 * (vy + 1u);
    y = y0 + (mul_hi(y0, (uint32_t)(g >> 13)) >> 18);                       // + y0 g / 2
  }
  // first 31 bits of sqrt(v): v y, at most a few units too small
  const uint32_t sa = mul_hi(v1, y);  // units of 2^-31
  // exact remainder V 2^-64 - sa^2 2^-62 in units of 2^-64
  const uint64_t r1 = V - ((uint64_t)sa * sa << 2);
  // next 23 bits: r1 / (2 sa) = (r1 y) / 2, units of 2^-54
  uint32_t sb = mul_hi((uint32_t)(r1 >> 7), y) >> 3;
  // remainder modulo 2^64 in units of 2^-108: (r1 << 44) - 2^24 sa sb - sb^2
  const uint64_t r2 = (r1 << 44) - ((uint64_t)sa * sb << 24) - (uint64_t)sb * sb;
  uint64_t q = ((uint64_t)sa << 23) + sb;
  // q is at most one too small
  if ((int64_t)(r2 - (2 * q + 1)) >= 0) q++;
  q = (q + 1u) >> 1;  // 54 bits, rounded (a square root is never half way between)
  // (e + 1022 + odd) / 2 is the result's biased exponent; less one for the implicit bit
  const uint32_t e = (((w.hi >> 20) & 0x7ffu) + 1022u + odd) >> 1;
  return from_words((uint32_t)(q >> 32) + ((e - 1u) << 20), (uint32_t)q);
}

// ---------------------------------------------------------------------------
// any operands: the integer routines inside their range, the FP64 unit outside
// ---------------------------------------------------------------------------
#ifdef __CUDACC__
#define LSMGPU_FPI_COLD static __device__ __noinline__
#else
#define LSMGPU_FPI_COLD static inline
#endif
// (calls, so that the FP64 instruction is branched around, not predicated: a
// predicated one still takes its turn on the pipe)
LSMGPU_FPI_COLD double unit_mul(double a, double b) { return a * b; }
LSMGPU_FPI_COLD double unit_div(double a, double b) { return a / b; }
LSMGPU_FPI_COLD double unit_sqrt(double a) { return sqrt(a); }

#ifdef __CUDACC__
#define LSMGPU_FPI_DEV __device__ __forceinline__
#else
#define LSMGPU_FPI_DEV inline
#endif
LSMGPU_FPI_DEV bool is_zero(const W2 &w) { return ((w.hi & 0x7fffffffu) | w.lo) == 0u; }
// zero, or a magnitude in [2^-LO, 2^LO): products of two with LO = 511, and
// quotients with LO = 500, are normal numbers (or zero)
template <uint32_t LO>
LSMGPU_FPI_DEV bool plain(const W2 &w) {
  return ((w.hi & 0x7fffffffu) - ((1023u - LO) << 20)) < ((2u * LO) << 20) || is_zero(w);
}
LSMGPU_FPI_DEV double mul_any(double a, double b) {
  const W2 aw = words(a), bw = words(b);
  if (plain<511>(aw) && plain<511>(bw)) {
    const W2 r = words(mul(unpack(a, 1), unpack(b, 1)));
    return from_words(r.hi | ((aw.hi ^ bw.hi) & 0x80000000u), r.lo);  // a zero gets its sign
  }
  return unit_mul(a, b);
}
// the same, but a zero product of numbers in range is +0
LSMGPU_FPI_DEV double mul_any_z(double a, double b) {
  if (plain<511>(words(a)) && plain<511>(words(b))) return mul(unpack(a, 1), unpack(b, 1));
  return unit_mul(a, b);
}
LSMGPU_FPI_DEV double sqr_any(double a) {
  if (plain<511>(words(a))) return sqr(unpack(a, 1));
  return unit_mul(a, a);
}
LSMGPU_FPI_DEV double div_any(double a, double b) {
  const W2 aw = words(a), bw = words(b);
  if (plain<500>(aw) && plain<500>(bw) && !is_zero(bw)) {
    const W2 q = words(div_pos(a, b));
    const uint32_t keep = is_zero(aw) ? 0u : 0xffffffffu;
    return from_words((q.hi & keep) | ((aw.hi ^ bw.hi) & 0x80000000u), q.lo & keep);
  }
  return unit_div(a, b);
}
LSMGPU_FPI_DEV double sqrt_any(double a) {
  const W2 w = words(a);
  if (w.hi - 0x00100000u < 0x7fe00000u) return sqrt_pos(a);  // positive and normal
  if (is_zero(w)) return a;
  return unit_sqrt(a);
}
// y + x / 4 as two roundings give it: x / 4 is exact, so one fma does, unless it
// is below the normal numbers
LSMGPU_FPI_DEV double plus_quarter(double y, double x) {
  const W2 w = words(x);
  if ((w.hi & 0x7fffffffu) >= (3u << 20) || is_zero(w)) return fma(0.25, x, y);
  return y + unit_mul(0.25, x);
}
// |a| and a with its sign flipped where `flip`, on the high word (a standalone
// FP64 absolute value or negation is an instruction of the FP64 pipe)
LSMGPU_FPI_DEV double abs_bits(double a) {
  const W2 w = words(a);
  return from_words(w.hi & 0x7fffffffu, w.lo);
}
LSMGPU_FPI_DEV double flip_if(double a, bool flip) {
  const W2 w = words(a);
  return from_words(w.hi ^ (flip ? 0x80000000u : 0u), w.lo);
}
// Comparisons on the bit patterns, with the FP64 unit's results for NaN
// (every comparison with NaN is false).
constexpr unsigned long long kInfBits = 0x7ff0000000000000ULL;
LSMGPU_FPI_DEV bool is_positive(double v) {
  const W2 w = words(v);
  return !(w.hi & 0x80000000u) && mag(v) - 1ULL < kInfBits;
}
LSMGPU_FPI_DEV double positive_part(double v) { return is_positive(v) ? v : 0.0; }  // v > 0 ? v : 0
// a > b ? a : b of two values that are not negative; b where either is NaN
LSMGPU_FPI_DEV double max_nonneg(double a, double b) { return mag(a) > mag(b) && mag(a) <= kInfBits ? a : b; }
// a < b, |a| < b and |a| >= b for a constant b > 0
LSMGPU_FPI_DEV bool less_than(double a, double b) {
  const uint32_t neg = words(a).hi & 0x80000000u;
  return (neg && mag(a) <= kInfBits) || (!neg && mag(a) < mag(b));
}
LSMGPU_FPI_DEV bool below(double a, double b) { return mag(a) < mag(b); }
LSMGPU_FPI_DEV bool at_least(double a, double b) { return mag(a) >= mag(b) && mag(a) <= kInfBits; }

}  // namespace fpi
}  // namespace lsmgpu
