// WENO5-JS in FP64 in LSMLIB's operation order, bit for bit
// (spatial_derivatives3d.f.in:1286-1367), with its products and quotients on
// the integer pipes (fp64_int.cuh) and only its additions on the FP64 unit.
//
// Per reconstruction the formula as written (weno5_unit64) costs 43 FP64 products, 28 sums, 4 maxima
// and 4 divisions, about 107 instructions of the FP64 pipe, which bounds every
// FP64 stage kernel.  Here 28 remain:
//  * products by 2, 4 and 1/4 are exact, so they ride in the fma of the sum
//    that follows (one rounding either way);
//  * the maximum of the squares is the square of the maximum (rounding is
//    monotone), taken on the integer bit patterns;
//  * every other product, and the four divisions, run as integer arithmetic.
// The plus and the minus side of an axis share the six differences, their
// products with the candidate coefficients and the inner maximum.
//
// Range: the integer routines handle normal numbers and zero.  A cell whose
// differences are all zero or lie within about 2^-500 .. 2^100 of each other's
// scale (see Wide64) keeps every intermediate value normal; others (and
// infinities and NaN) take the FP64 unit.  Squares of values below 2^-423 are
// taken as zero: they only enter sums with epsilon >= 1e-36, whose rounding
// they cannot change.
#pragma once

#include "fp64_int.cuh"
#include "stencil_math.cuh"

namespace lsmgpu {

// The formula as written, all on the FP64 unit; `tiny` is the floor of
// epsilon (the dense routines' 1e-36, the list routines' 1e-35)
static __device__ __noinline__ double weno5_unit64(double v1, double v2, double v3, double v4, double v5,
                                                   double tiny) {
  const double c13 = 1.0 / 3.0, c76 = 7.0 / 6.0, c116 = 11.0 / 6.0, c16 = 1.0 / 6.0, c56 = 5.0 / 6.0;
  const double c1312 = 13.0 / 12.0, c14 = 0.25;
  double m = v1 * v1;
  m = rmax(m, v2 * v2);
  m = rmax(m, v3 * v3);
  m = rmax(m, v4 * v4);
  m = rmax(m, v5 * v5);
  const double eps = 1e-6 * m + tiny;
  const double p1 = c13 * v1 - c76 * v2 + c116 * v3;
  const double p2 = -(c16 * v2) + c56 * v3 + c13 * v4;
  const double p3 = c13 * v3 + c56 * v4 - c16 * v5;
  double t = v1 - 2.0 * v2 + v3, u = v1 - 4.0 * v2 + 3.0 * v3;
  const double S1 = c1312 * (t * t) + c14 * (u * u);
  t = v2 - 2.0 * v3 + v4;
  u = v2 - v4;
  const double S2 = c1312 * (t * t) + c14 * (u * u);
  t = v3 - 2.0 * v4 + v5;
  u = 3.0 * v3 - 4.0 * v4 + v5;
  const double S3 = c1312 * (t * t) + c14 * (u * u);
  double a1 = 0.1 / ((S1 + eps) * (S1 + eps));
  double a2 = 0.6 / ((S2 + eps) * (S2 + eps));
  double a3 = 0.3 / ((S3 + eps) * (S3 + eps));
  const double is = 1.0 / (a1 + a2 + a3);
  a1 = a1 * is;
  a2 = a2 * is;
  a3 = a3 * is;
  return a1 * p1 + a2 * p2 + a3 * p3;
}

// 1/dx of an axis, unpacked, and the range of undivided differences the
// integer form takes with it: a difference counts as zero below 2^-523 (one
// that is not zero there is out of range), and 1/dx within 2^-200 .. 2^200
// puts the divided ones at 2^-723 or more; `lim` keeps those below 2^99, so
// that epsilon-scaled quotients stay far from the ends of the exponent range.
struct Wide64 {
  double inv;
  fpi::Op op;
  uint32_t lim;  // high words of |difference| must lie below
};
constexpr uint32_t kDiffFloor = 500, kValueFloor = 300, kSquareFloor = 600;
__device__ __forceinline__ Wide64 wide64(double inv) {
  Wide64 w;
  w.inv = inv;
  w.op = fpi::unpack_normal(inv);
  const uint32_t hi = fpi::words(inv).hi, e = hi >> 20;  // a negative or non-finite one is out of range
  w.lim = (e >= 823 && e <= 1223) ? (2145u - e) << 20 : 0u;
  return w;
}

// a divided difference, its operand form and its magnitude's bits
struct Diff64 {
  double v;
  fpi::Op o;
};

// collects whether every difference is in range
struct Range64 {
  uint32_t top = 0, low = 0;
  __device__ __forceinline__ void add(double d) {
    const fpi::W2 w = fpi::words(d);
    const uint32_t h = w.hi & 0x7fffffffu;
    top = max(top, h);
    low |= h < (kDiffFloor << 20) ? (h | w.lo) : 0u;
  }
  __device__ __forceinline__ bool ok(const Wide64 &w) const { return top < w.lim && low == 0u; }
};

__device__ __forceinline__ Diff64 divided(double d, const Wide64 &w) {
  Diff64 r;
  r.v = fpi::mul(fpi::unpack(d, kDiffFloor), w.op);
  r.o = fpi::unpack(r.v, kValueFloor);
  return r;
}
__device__ __forceinline__ double times(const Diff64 &d, double c) { return fpi::mul(d.o, fpi::unpack_normal(c)); }
__device__ __forceinline__ double times(double v, double c) {
  return fpi::mul(fpi::unpack(v, kValueFloor), fpi::unpack_normal(c));
}
__device__ __forceinline__ void swap64(double &x, double &y) {
  const double t = x;
  x = y;
  y = t;
}
__device__ __forceinline__ double square64(double v) { return fpi::sqr(fpi::unpack(v, kSquareFloor)); }
// 13/12 t^2 + u^2 / 4
__device__ __forceinline__ double indicator64(double t, double u) {
  return fma(0.25, square64(u), fpi::mul(fpi::unpack(square64(t), 1), fpi::unpack_normal(13.0 / 12.0)));
}
// epsilon from the bits of the largest |v|.  Where 1e-6 v^2 is 2^55 tiny or
// more, adding tiny rounds to it again, and the addition (one of 28) is left
// out (a call, as the unit_ functions are: predicated off it would still take
// its turn on the pipe).
static __device__ __noinline__ double unit_add(double a, double b) { return a + b; }
__device__ __forceinline__ double epsilon64(unsigned long long m, double tiny) {
  const double mm = square64(__longlong_as_double((long long)m));
  const double e = fpi::mul(fpi::unpack(mm, 1), fpi::unpack_normal(1e-6));
  if (fpi::words(e).hi >= fpi::words(0x1p55 * tiny).hi) return e;
  return unit_add(e, tiny);
}
// the weighted sum of the three candidates
__device__ __forceinline__ double combine64(double S1, double S2, double S3, double eps, double p1, double p2,
                                            double p3) {
  auto part = [&](double d, double S) { return fpi::div_pos(d, fpi::sqr(fpi::unpack_normal(S + eps))); };
  const double a1 = part(0.1, S1), a2 = part(0.6, S2), a3 = part(0.3, S3);
  const fpi::Op is = fpi::unpack_normal(fpi::div_pos(1.0, a1 + a2 + a3));
  auto term = [&](double a, double p) {
    return fpi::mul(fpi::unpack_normal(fpi::mul(fpi::unpack_normal(a), is)), fpi::unpack(p, 1));
  };
  return term(a1, p1) + term(a2, p2) + term(a3, p3);
}

// One side on the undivided differences d[0..4] (v1 .. v5 once divided); with
// `flip` the negated value of the negated differences, which is the same number
// but for the sign of a zero: the reconstruction of zeros is +0 either way.
__device__ __forceinline__ double weno5_side64(const double d[5], const Wide64 &w, double tiny, bool flip = false) {
  Range64 rg;
#pragma unroll
  for (int q = 0; q < 5; q++) rg.add(d[q]);
  if (!rg.ok(w)) {
    const double inv = flip ? -w.inv : w.inv;
    return weno5_unit64(d[0] * inv, d[1] * inv, d[2] * inv, d[3] * inv, d[4] * inv, tiny);
  }
  Diff64 v[5];
#pragma unroll
  for (int q = 0; q < 5; q++) v[q] = divided(d[q], w);
  unsigned long long m = fpi::mag(v[0].v);
#pragma unroll
  for (int q = 1; q < 5; q++) m = max(m, fpi::mag(v[q].v));
  const double eps = epsilon64(m, tiny);
  const double c13 = 1.0 / 3.0, c76 = 7.0 / 6.0, c116 = 11.0 / 6.0, c16 = 1.0 / 6.0, c56 = 5.0 / 6.0;
  const double p1 = times(v[0], c13) - times(v[1], c76) + times(v[2], c116);
  const double p2 = -times(v[1], c16) + times(v[2], c56) + times(v[3], c13);
  const double p3 = times(v[2], c13) + times(v[3], c56) - times(v[4], c16);
  const double v3x3 = times(v[2], 3.0);
  const double S1 = indicator64(fma(-2.0, v[1].v, v[0].v) + v[2].v, fma(-4.0, v[1].v, v[0].v) + v3x3);
  const double S2 = indicator64(fma(-2.0, v[2].v, v[1].v) + v[3].v, v[1].v - v[3].v);
  const double S3 = indicator64(fma(-2.0, v[3].v, v[2].v) + v[4].v, fma(-4.0, v[3].v, v3x3) + v[4].v);
  const double r = combine64(S1, S2, S3, eps, p1, p2, p3);  // a zero is +0
  return fpi::flip_if(r, flip && !fpi::is_zero(fpi::words(r)));
}

// Both sides of an axis at a cell on the undivided differences
// d[0..5] = D1(c-2) .. D1(c+3): minus on d[0..4], plus on d[5..1].
__device__ __forceinline__ void weno5_pm64(const double d[6], const Wide64 &w, double tiny, double &gp, double &gm) {
  Range64 rg;
#pragma unroll
  for (int q = 0; q < 6; q++) rg.add(d[q]);
  if (!rg.ok(w)) {
    double v[6];
#pragma unroll
    for (int q = 0; q < 6; q++) v[q] = d[q] * w.inv;
    gp = weno5_unit64(v[5], v[4], v[3], v[2], v[1], tiny);
    gm = weno5_unit64(v[0], v[1], v[2], v[3], v[4], tiny);
    return;
  }
  Diff64 v[6];
#pragma unroll
  for (int q = 0; q < 6; q++) v[q] = divided(d[q], w);
  const double c13 = 1.0 / 3.0, c76 = 7.0 / 6.0, c116 = 11.0 / 6.0, c16 = 1.0 / 6.0, c56 = 5.0 / 6.0;
  unsigned long long m = fpi::mag(v[1].v);
#pragma unroll
  for (int q = 2; q < 5; q++) m = max(m, fpi::mag(v[q].v));
  // products both sides take
  double a1 = times(v[1], c16), a4 = times(v[4], c16);
  double b2 = times(v[2], c56), b3 = times(v[3], c56);
  double e2 = times(v[2], c13), e3 = times(v[3], c13);
  double x2 = times(v[2], 3.0), x3 = times(v[3], 3.0);
  // The plus side is the minus side of the reversed differences: a second pass
  // of the same code on swapped values.  (With both sides inlined the kernels
  // waited for instructions, 13% of a warp's time: reinitialization 121 x 118 x
  // 109, 5 steps 10.95 ms, rolled 10.27, with the registers that frees 9.95.)
  double s0 = v[0].v, s1 = v[1].v, s2 = v[2].v, s3 = v[3].v, s4 = v[4].v, s5 = v[5].v, out = 0.0;
#pragma unroll 1
  for (int side = 0; side < 2; side++) {
    gm = out;
    const double eps = epsilon64(max(m, fpi::mag(s0)), tiny);
    const double p1 = times(s0, c13) - times(s1, c76) + times(s2, c116);
    const double p2 = -a1 + b2 + e3;
    const double p3 = e2 + b3 - a4;
    const double S1 = indicator64(fma(-2.0, s1, s0) + s2, fma(-4.0, s1, s0) + x2);
    const double S2 = indicator64(fma(-2.0, s2, s1) + s3, s1 - s3);
    const double S3 = indicator64(fma(-2.0, s3, s2) + s4, fma(-4.0, s3, x2) + s4);
    out = combine64(S1, S2, S3, eps, p1, p2, p3);
    swap64(s0, s5), swap64(s1, s4), swap64(s2, s3);
    swap64(a1, a4), swap64(b2, b3), swap64(e2, e3), swap64(x2, x3);
  }
  gp = out;
}

}  // namespace lsmgpu
