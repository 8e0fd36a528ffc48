// Compares the integer-pipe FP64 routines (csrc/fp64_int.cuh) and the WENO5
// reconstruction built on them (csrc/weno64.cuh) with the host's FP64
// arithmetic, bit for bit, on seeded operands: random significands, few-bit
// and nearly full significands, significands next to powers of two, and for
// WENO5 smooth, flat, linear, kinked, tiny, huge and non-finite data.
// Prints the number of differences.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__
using std::fabs;
using std::fma;
using std::max;
static inline double __longlong_as_double(long long x) {
  double d;
  memcpy(&d, &x, 8);
  return d;
}
static inline long long __double_as_longlong(double d) {
  long long x;
  memcpy(&x, &d, 8);
  return x;
}
#include "weno64.cuh"

using namespace lsmgpu;

static std::mt19937_64 g;

static double operand(int elo, int ehi) {
  uint64_t m = g() & 0xfffffffffffffull;
  switch (g() % 7) {
    case 0: m &= 0xfffff80000000ull; break;
    case 1: m |= 0xfffffff000000ull; break;
    case 2: m = g() % 5; break;
    case 3: m = 0xfffffffffffffull - (g() % 5); break;
    case 4: m = (1ull << (g() % 52)) | (1ull << (g() % 52)); break;
    default: break;
  }
  const uint64_t b = (g() & 0x8000000000000000ull) | ((uint64_t)(elo + g() % (ehi - elo + 1)) << 52) | m;
  return __longlong_as_double((long long)b);
}

static bool same(double a, double b) { return a == b || (a != a && b != b); }

static long scalar_routines(long n) {
  long bad = 0;
  const double c[4] = {0.1, 0.6, 0.3, 1.0};
  for (long i = 0; i < n; i++) {
    const double a = operand(512, 1534), b = operand(512, 1534), d = fabs(operand(600, 1446));
    bad += fpi::mul(fpi::unpack(a, 1), fpi::unpack(b, 1)) != a * b;
    bad += fpi::mul(fpi::unpack(i & 1 ? 0.0 : -0.0, 1), fpi::unpack(b, 1)) != 0.0;
    bad += fpi::sqr(fpi::unpack(a, 1)) != a * a;
    bad += fpi::div_pos(c[i & 3], d) != c[i & 3] / d;
    const double num = fabs(operand(600, 1446));
    bad += fpi::div_pos(num, d) != num / d;
    const double r = fabs(operand(1, 2046)), sq = r > 1e-150 && r < 1e150 ? r * r : r;
    bad += fpi::sqrt_pos(r) != std::sqrt(r);
    bad += fpi::sqrt_pos(sq) != std::sqrt(sq);
  }
  return bad;
}

// the forms that take any operand, over the whole range and the special values
static long any_operands(long n) {
  long bad = 0;
  const double special[10] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 5e-324, 2.2250738585072014e-308,
                              1.7976931348623157e308, 1e-200, 1e200};
  for (long i = 0; i < n; i++) {
    const double a = g() % 8 ? operand(0, 2046) : special[g() % 10], b = g() % 8 ? operand(0, 2046) : special[g() % 10];
    bad += !same(fpi::mul_any(a, b), a * b) || !same(fpi::sqr_any(a), a * a);
    bad += !same(fpi::div_any(a, b), a / b) || !same(fpi::sqrt_any(a), std::sqrt(a));
    bad += !same(fpi::abs_bits(a), fabs(a)) || !same(fpi::flip_if(a, i & 1), (i & 1) ? -a : a);
    bad += fpi::is_positive(a) != (a > 0) || !same(fpi::positive_part(a), a > 0 ? a : 0.0);
    const double x = fabs(a), y = fabs(b), t = 1e-11;
    bad += !same(fpi::max_nonneg(x, y), x > y ? x : y);
    bad += fpi::less_than(a, t) != (a < t) || fpi::below(a, t) != (fabs(a) < t) || fpi::at_least(a, t) != (fabs(a) >= t);
  }
  return bad;
}

static long reconstructions(long n) {
  long bad = 0;
  std::normal_distribution<double> nd;
  for (long i = 0; i < n; i++) {
    const int mode = (int)(g() % 13);
    const double u = (double)(g() >> 11) * 0x1p-53 - 0.5;
    const double scale = std::exp(u * (mode == 9 ? 1400 : mode == 8 ? 400 : 20));
    const double a = nd(g), b = 0.1 * nd(g), c = 0.01 * nd(g);
    double phi[7], d[6], v[6];
    for (int k = 0; k < 7; k++) {
      const double x = k - 3;
      switch (mode) {
        case 0: phi[k] = a + b * x + c * x * x; break;
        case 1: phi[k] = a + 0.25 * x; break;
        case 2: phi[k] = a; break;
        case 3: phi[k] = (double)(g() % 7) - 3; break;
        case 4: phi[k] = a + b * x * (1 + 1e-12 * nd(g)); break;
        case 5: phi[k] = fabs(x * b + c) - a; break;
        case 6: phi[k] = k == 3 ? 1e-20 * a : 0; break;
        case 7: phi[k] = std::sqrt((0.1 * x + a) * (0.1 * x + a) + b * b); break;
        case 10: phi[k] = 1e-18 * a * (double)(g() % 4); break;
        case 11: phi[k] = g() % 8 ? a * k : (g() & 1 ? INFINITY : NAN); break;
        default: phi[k] = scale * nd(g); break;
      }
    }
    const double inv = (i & 1) ? 128.0 : 1.0 / std::exp(-8 * (u + 0.5));
    const double tiny = (i & 2) ? 1e-36 : 1e-35;
    for (int q = 0; q < 6; q++) {
      d[q] = phi[q + 1] - phi[q];
      v[q] = d[q] * inv;
    }
    const Wide64 w = wide64(inv);
    double gp, gm;
    weno5_pm64(d, w, tiny, gp, gm);
    bad += !same(gp, weno5_unit64(v[5], v[4], v[3], v[2], v[1], tiny));
    bad += !same(gm, weno5_unit64(v[0], v[1], v[2], v[3], v[4], tiny));
    bad += !same(gm, weno5_side64(d, w, tiny));
  }
  return bad;
}

int main(int argc, char **argv) {
  const long n = argc > 1 ? atol(argv[1]) : 1000000;
  g.seed(argc > 2 ? (uint64_t)atol(argv[2]) : 1);
  printf("%ld %ld %ld\n", scalar_routines(n), any_operands(n), reconstructions(n));
  return 0;
}
