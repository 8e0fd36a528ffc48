// Fused narrow-band curvature flow: phi_t + Vn |grad phi| = 0 with
// Vn = a_n - b_n * kappa, HJ WENO5 on a narrow band, TVD-RK3, the band rebuilt
// every `rebuild_every` steps.  It replaces the LSMLIB local call sequence
// per stage (on level-0 cells):
//   lsm3dCentralGradOrder2LOCAL -> lsm3dGradientMagnitudeLocal ->
//   lsm3dComputeMeanCurvatureOrder2Local -> Vn = a_n - b_n*kappa ->
//   HJ WENO5 LOCAL -> lsm3dZeroOut/AddNormalVelTermToLSERHSLOCAL ->
//   (stage 1: lsm3dComputeStableNormalVelDtLOCAL) ->
//   lsm3dMultiplyCutOffLSERHSLOCAL -> lsm3dTVDRK3StageNLOCAL
// with one gather kernel per stage (stage 1 is split at the dt reduction).
//
// The band.  Of LSMLIB's band the flow needs the level-0 cells, |phi| < gamma
// at a rebuild.  The first build finds them over the grid; since the flow
// writes phi at level-0 cells only, a later level 0 is the sub-sequence of the
// previous one that passes the test.  LSMLIB's neighbour levels 1..3 exist so
// that the stage fields hold phi^n where the stencils reach outside level 0;
// here the stage fields hold phi at every cell outside level 0 from the start
// (one copy of phi, then the cells that leave level 0 at a rebuild), so no
// neighbour level is built.  The list holds one offset per cell, in the
// reference's sweep order.
//
// LSMGPU_BANDFLOW_EXACT selects the FP64 parity arithmetic (this unit is
// compiled with -fmad=false); the FP32 form uses the fast WENO weights.
#pragma once
#include "band.cuh"
#include "fused_stage.cuh"
#include "stencil_math.cuh"
#include "../../include/lsmgpu.h"

namespace lsmgpu {
namespace bandflow {

template <class R>
struct BandArgs {
  View<const R> src;      // stage source (phi^n, u1, u2)
  View<const R> phin;     // phi^n (stages 2, 3)
  View<R> out;            // stage output
  const int *off0;        // offset of each level-0 cell in its array
  int n0;                 // level-0 entries (list elements 0..n0-1)
  R dx, a_n, b_n, beta, gamma, cfl;
  // per-call constants of the stencils, divided on the host in R exactly as
  // the per-cell expressions would: 0.5/dx, 1/dx/dx, 0.25/dx/dx, 1/dx
  R f_half, f_xx, f_xy, inv_dx;
  R *rhs;                 // stage 1: the RHS per level-0 entry (FP32 form: a
                          // (src, src, rhs, rhs) record per entry pair)
  const R *dt;            // device scalar
  unsigned long long *key;
  int stage;
};

__device__ __forceinline__ unsigned long long okey(double v) {
  unsigned long long u = (unsigned long long)__double_as_longlong(v);
  return (u & 0x8000000000000000ULL) ? ~u : (u | 0x8000000000000000ULL);
}
__device__ __forceinline__ double okey_inv(unsigned long long k) {
  unsigned long long u = (k & 0x8000000000000000ULL) ? (k & 0x7fffffffffffffffULL) : ~k;
  return __longlong_as_double((long long)u);
}

// running maximum of the dt keys: the key only grows, so a warp whose key
// does not exceed the value it reads cannot raise it and skips the atomic
// (a stale read only costs an atomic); keeps tens of thousands of warps from
// queueing on one address
__device__ __forceinline__ void raise_key(unsigned long long *key, unsigned long long k) {
  if (k > __ldcg(key)) atomicMax(key, k);
}

// normal speed Vn = a_n - b_n kappa at a level-0 cell: central gradient,
// |grad phi| with zero_tol clamps, mean curvature
// (spatial_derivatives3d_local.f.in:825-839, :1251-1272; curvature3d_local.f.in)
template <class R>
__device__ __forceinline__ R cell_vn(const BandArgs<R> &a, const R *c, const long long s[3]) {
  const R f = a.f_half;
  const R g0 = mul_z_(c[s[0]] - c[-s[0]], f), g1 = mul_z_(c[s[1]] - c[-s[1]], f), g2 = mul_z_(c[s[2]] - c[-s[2]], f);
  const R mag = grad_magnitude(g0, g1, g2, R(Consts<double>::zero_tol));
  const R kappa = mean_curvature2(c, s[0], s[1], s[2], g0, g1, g2, mag, a.f_xx, a.f_xx, a.f_xx, a.f_xy, a.f_xy, a.f_xy);
  return a.a_n - mul_(a.b_n, kappa);
}

// Godunov normal-velocity term (level_set_evolution3d_local.f.in:236-273) from
// the WENO5 plus/minus derivatives, and the cell's H/dx
// (math_utils3d_local.f.in:396-414)
template <class R>
__device__ __forceinline__ R godunov_rhs(const BandArgs<R> &a, R vn, const R gp[3], const R gm[3], R &h_over_dx) {
  const R tol = Consts<double>::zero_tol;
  const R sq = godunov_normal_sq<R>(is_pos_(vn), gp, gm);
  R rhs = R(0);
  if (at_least_(vn, tol)) rhs = rhs - mul_(vn, sqrt_(sq));
  const R dx = a.dx, inv = a.inv_dx;
  const R mx2 = dx * dx;
  const R cx = max_nonneg_(abs_(gp[0]), abs_(gm[0])), cy = max_nonneg_(abs_(gp[1]), abs_(gm[1]));
  const R cz = max_nonneg_(abs_(gp[2]), abs_(gm[2]));
  const R ng = sqrt_(sqr_(cx) + sqr_(cy) + sqr_(cz) + mx2);
  h_over_dx = (ng > tol) ? mul_z_(div_(abs_(vn), ng), mul_z_(cx, inv) + mul_z_(cy, inv) + mul_z_(cz, inv)) : R(-1.0);
  return rhs;
}

// the RHS of one level-0 cell, before the cut-off; also the cell's H/dx for dt
template <class R>
__device__ __forceinline__ R cell_rhs(const BandArgs<R> &a, long long o, R &h_over_dx) {
  const R *c = a.src.p + o;
  const long long s[3] = {1, a.src.s1, a.src.s2};
  const R vn = cell_vn<R>(a, c, s);
  // HJ WENO5 plus/minus from the band values of src, with the local routines'
  // epsilon floor (spatial_derivatives2d_local.f.in:892)
  R gp[3], gm[3];
#pragma unroll 1
  for (int d = 0; d < 3; d++) {
    R D[6];
#pragma unroll
    for (int q = -2; q <= 3; q++) D[q + 2] = c[q * s[d]] - c[(q - 1) * s[d]];
    weno5_pm64(D, wide64(a.inv_dx), 1.e-35, gp[d], gm[d]);
  }
  return godunov_rhs<R>(a, vn, gp, gm, h_over_dx);
}

// Two cells of a field by their byte offsets: the stencil's displacements are
// the same for all cells, so they are added to the field's address once per
// warp and a load takes that address and the cell's offset as they are (512^3,
// 100 steps: 30.9 ms with an address computed per load, 30.0 with this).  I:
// unsigned for fields below 4 GB, else 64 bits.
template <class I>
struct Pair {
  const char *p;
  I o0, o1;  // byte offsets
  __device__ __forceinline__ float2 at(long long e) const {
    const char *q = p + e * (long long)sizeof(float);
    return make_float2(*reinterpret_cast<const float *>(q + o0), *reinterpret_cast<const float *>(q + o1));
  }
};

// cell_vn on two cells in packed FP32x2: the central gradient, the second
// differences and the curvature numerator (summed as
// xx (y^2 + z^2) + yy (x^2 + z^2) + zz (x^2 + y^2) - 2 (xy x y + xz x z + yz y z))
// run on the pair; the zero_tol clamps, |grad phi| and the division per cell
template <class I>
static __device__ __forceinline__ float2 cell_vn_x2(const BandArgs<float> &a, const Pair<I> &c, const long long s[3]) {
  using fused::add2;
  using fused::fma2;
  using fused::mul2;
  using fused::sp;
  using fused::sub2;
  const auto at = [&](long long o) { return c.at(o); };
  const float2 cc = at(0);
  const float2 xp = at(s[0]), xm = at(-s[0]), yp = at(s[1]), ym = at(-s[1]), zp = at(s[2]), zm = at(-s[2]);
  const float2 f = sp(a.f_half);
  const float2 gx = mul2(sub2(xp, xm), f), gy = mul2(sub2(yp, ym), f), gz = mul2(sub2(zp, zm), f);
  const float tol = Consts<double>::zero_tol;
  const float2 sx = mul2(gx, gx), sy = mul2(gy, gy), sz = mul2(gz, gz);
  // |grad phi| with each square below zero_tol dropped
  const float2 q = add2(add2(make_float2(sx.x < tol ? 0.f : sx.x, sx.y < tol ? 0.f : sx.y),
                             make_float2(sy.x < tol ? 0.f : sy.x, sy.y < tol ? 0.f : sy.y)),
                        make_float2(sz.x < tol ? 0.f : sz.x, sz.y < tol ? 0.f : sz.y));
  float m0 = sqrtf(q.x), m1 = sqrtf(q.y);
  m0 = (m0 < tol) ? 0.f : m0;
  m1 = (m1 < tol) ? 0.f : m1;
  const float2 fxx = sp(a.f_xx), fxy = sp(a.f_xy), m2 = sp(-2.f);
  const float2 xx = mul2(add2(fma2(m2, cc, xp), xm), fxx);
  const float2 yy = mul2(add2(fma2(m2, cc, yp), ym), fxx);
  const float2 zz = mul2(add2(fma2(m2, cc, zp), zm), fxx);
  const float2 xy = mul2(add2(sub2(sub2(at(s[0] + s[1]), at(s[0] - s[1])), at(-s[0] + s[1])), at(-s[0] - s[1])), fxy);
  const float2 xz = mul2(add2(sub2(sub2(at(s[0] + s[2]), at(s[0] - s[2])), at(-s[0] + s[2])), at(-s[0] - s[2])), fxy);
  const float2 yz = mul2(add2(sub2(sub2(at(s[1] + s[2]), at(s[1] - s[2])), at(-s[1] + s[2])), at(-s[1] - s[2])), fxy);
  const float2 diag = fma2(xx, add2(sy, sz), fma2(yy, add2(sx, sz), mul2(zz, add2(sx, sy))));
  const float2 cross = fma2(mul2(xy, gx), gy, fma2(mul2(xz, gx), gz, mul2(mul2(yz, gy), gz)));
  const float2 num = fma2(m2, cross, diag);
  const float d0 = m0 * m0 * m0, d1 = m1 * m1 * m1;
  const float k0 = (d0 < tol) ? 0.f : num.x / d0, k1 = (d1 < tol) ? 0.f : num.y / d1;
  return make_float2(a.a_n - a.b_n * k0, a.a_n - a.b_n * k1);
}

// FP32 RHS of two level-0 cells (padded offsets o0, o1): the six WENO5
// reconstructions and the curvature run on the pair in Blackwell's packed
// FP32x2 arithmetic (WENO5: both sides of an axis together); the Godunov term
// per cell
template <class I>
static __device__ __forceinline__ float2 cell_rhs_x2(const BandArgs<float> &a, const Pair<I> &c, float2 &hd) {
  const long long s[3] = {1, a.src.s1, a.src.s2};
  const float2 vn = cell_vn_x2(a, c, s);
  const float vn0 = vn.x, vn1 = vn.y;
  const float2 inv = fused::sp(a.inv_dx);
  float gp0[3], gm0[3], gp1[3], gm1[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    float2 x[7], v[6];
#pragma unroll
    for (int q = 0; q < 7; q++) x[q] = c.at((q - 3) * s[d]);
#pragma unroll
    for (int q = 0; q < 6; q++) v[q] = fused::mul2(fused::sub2(x[q + 1], x[q]), inv);
    float2 p, m;
    fused::weno5_pm_x2(v, p, m);
    gp0[d] = p.x; gp1[d] = p.y;
    gm0[d] = m.x; gm1[d] = m.y;
  }
  float h0, h1;
  const float r0 = godunov_rhs<float>(a, vn0, gp0, gm0, h0);
  const float r1 = godunov_rhs<float>(a, vn1, gp1, gm1, h1);
  hd = make_float2(h0, h1);
  return make_float2(r0, r1);
}

// cubic cut-off between beta and gamma (localization3d.f:527-553)
template <class R>
__device__ __forceinline__ R cutoff(R rhs, R phi, R beta, R gamma) {
  const R av = fabs(phi);
  R co;
  if (av <= beta) {
    co = R(1);
  } else if (av <= gamma) {
    const R c1 = gamma - 3 * beta;
    R c2 = (gamma - beta);
    c2 = c2 * c2 * c2;
    const R tt = av - gamma;
    co = (tt * tt * (2 * av + c1)) / c2;
  } else {
    co = R(0);
  }
  return co * rhs;
}

template <class R>
__device__ __forceinline__ R rk_update(int stage, R un, R us, R dt, R rhs) {
  if (stage == 1) return un + dt * rhs;
  if (stage == 2) return R(0.75) * un + R(0.25) * (us + dt * rhs);
  return R(1.0 / 3.0) * un + R(2.0 / 3.0) * (us + dt * rhs);
}

// stage 1, pass 1: RHS (cut off) per entry and the dt maximum
template <class R>
__global__ void k_band_rhs(BandArgs<R> a) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  double h = -1.0e308;
  if (l < a.n0) {
    const long long o = a.off0[l];
    R hd;
    const R r = cell_rhs<R>(a, o, hd);
    h = (double)hd;
    a.rhs[l] = cutoff<R>(r, a.src.p[o], a.beta, a.gamma);
  }
  for (int o = 16; o > 0; o >>= 1) h = fmax(h, __shfl_xor_sync(0xffffffffu, h, o));
  if ((threadIdx.x & 31) == 0) raise_key(a.key, okey(h));
}

template <class R>
__global__ void k_band_dt(const unsigned long long *key, R *dt, R cfl, double *dt_log) {
  double m = okey_inv(*key);
  if (m < -1.0) m = -1.0;  // the reference's running maximum starts at -1
  const R d = cfl / ((R)m + (R)Consts<double>::tiny);
  *dt = d;
  if (dt_log) *dt_log = (double)d;
}

// stage 1, pass 2: the update
template <class R>
__global__ void k_band_update1(BandArgs<R> a) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= a.n0) return;
  const long long o = a.off0[l];
  a.out.p[o] = rk_update<R>(1, a.src.p[o], a.src.p[o], *a.dt, a.rhs[l]);
}

// stages 2 and 3: RHS, cut-off and update in one pass
template <class R>
__global__ void k_band_stage(BandArgs<R> a) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= a.n0) return;
  const long long o = a.off0[l];
  R hd;
  const R us = a.src.p[o];
  const R r = cutoff<R>(cell_rhs<R>(a, o, hd), us, a.beta, a.gamma);
  a.out.p[o] = rk_update<R>(a.stage, a.phin.p[o], us, *a.dt, r);
}

// FP32 forms of k_band_rhs and k_band_stage on pairs of consecutive list
// entries (the second of an odd tail repeats the first and is not written)
// offsets of the entry pair l0, l0 + 1 (the second repeats the first at an
// odd tail); off0 has an even number of elements, so the pair load is in bounds
template <class I>
static __device__ __forceinline__ Pair<I> entry_pair(const BandArgs<float> &a, const float *field, int l0, bool two) {
  const int2 p = *reinterpret_cast<const int2 *>(a.off0 + l0);
  const I o0 = (I)p.x * 4u, o1 = (I)p.y * 4u;
  return {reinterpret_cast<const char *>(field), o0, two ? o1 : o0};
}
template <class I>
static __device__ __forceinline__ void store_entries(const Pair<I> &c, float *field, bool two, float2 u) {
  char *q = reinterpret_cast<char *>(field);
  *reinterpret_cast<float *>(q + c.o0) = u.x;
  if (two) *reinterpret_cast<float *>(q + c.o1) = u.y;
}

// Stage 1 of the FP32 form stores, per entry pair p, the float4
// (src[l0], src[l1], rhs[l0], rhs[l1]) at a.rhs + 4p, so that the update
// after the dt reduction reads one contiguous record instead of gathering src.
// The dt maximum is taken in FP32 (a maximum is exact in either precision;
// the one conversion to FP64 per warp gives the same key) to keep the slow
// FP64 pipe out of the kernel.
template <class I>
__global__ void __launch_bounds__(128, 8) k_band_rhs_x2(BandArgs<float> a) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  const int l0 = 2 * p;
  float h = -INFINITY;
  if (l0 < a.n0) {
    const bool two = l0 + 1 < a.n0;
    const Pair<I> c = entry_pair<I>(a, a.src.p, l0, two);
    float2 hd;
    const float2 r = cell_rhs_x2(a, c, hd);
    h = two ? fmaxf(hd.x, hd.y) : hd.x;
    const float2 s = c.at(0);
    reinterpret_cast<float4 *>(a.rhs)[p] =
        make_float4(s.x, s.y, cutoff<float>(r.x, s.x, a.beta, a.gamma), cutoff<float>(r.y, s.y, a.beta, a.gamma));
  }
  for (int o = 16; o > 0; o >>= 1) h = fmaxf(h, __shfl_xor_sync(0xffffffffu, h, o));
  if ((threadIdx.x & 31) == 0) raise_key(a.key, okey((double)h));
}

// stage 1, pass 2 of the FP32 form: one entry pair per thread from its record
template <class I>
__global__ void k_band_update1_x2(BandArgs<float> a) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  const int l0 = 2 * p;
  if (l0 >= a.n0) return;
  const bool two = l0 + 1 < a.n0;
  const float4 v = reinterpret_cast<const float4 *>(a.rhs)[p];
  const float dt = *a.dt;
  store_entries(entry_pair<I>(a, a.src.p, l0, two), a.out.p, two,
                make_float2(rk_update<float>(1, v.x, v.x, dt, v.z), rk_update<float>(1, v.y, v.y, dt, v.w)));
}

template <class I>
__global__ void __launch_bounds__(128, 8) k_band_stage_x2(BandArgs<float> a) {
  const int l0 = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (l0 >= a.n0) return;
  const bool two = l0 + 1 < a.n0;
  const Pair<I> c = entry_pair<I>(a, a.src.p, l0, two);
  float2 hd;
  const float2 r = cell_rhs_x2(a, c, hd);
  const float dt = *a.dt;
  const float2 us = c.at(0);
  const float2 un = Pair<I>{reinterpret_cast<const char *>(a.phin.p), c.o0, c.o1}.at(0);
  store_entries(c, a.out.p, two,
                make_float2(rk_update<float>(a.stage, un.x, us.x, dt, cutoff<float>(r.x, us.x, a.beta, a.gamma)),
                            rk_update<float>(a.stage, un.y, us.y, dt, cutoff<float>(r.y, us.y, a.beta, a.gamma))));
}

// The level-0 test |phi| < width in FP64 whatever the field's precision: for
// a float a, (double)a < width is a <= the largest float below width.
template <class R>
struct Width {
  R lim;
  explicit Width(double w) {
    if constexpr (sizeof(R) == 4) {
      lim = (float)w;
      if ((double)lim >= w) lim = nextafterf(lim, -INFINITY);
    } else {
      lim = w > 0.0 ? w : 0.0;  // (below_ takes a width that is not negative)
    }
  }
  __device__ __forceinline__ bool in(R v) const {
    if constexpr (sizeof(R) == 4) return fabsf(v) <= lim;
    else return below_(v, lim);
  }
};

// Classifiers of the ordered compaction (band.cuh).  First build: every cell
// of the array in memory order, which is the reference's sweep order.
template <class R>
struct FlowGrid {
  const R *phi;
  Width<R> width;
  int *off;
  static constexpr bool kPrefetch = true;
  typedef R V;
  __device__ R load(long long e) const { return phi[e]; }
  __device__ int classify(R v, long long) const { return width.in(v) ? 1 : 0; }
  __device__ int flags(long long e) const { return classify(phi[e], e); }
  __device__ void counted(long long, int) const {}
  __device__ void emit(long long e, int, long long r0, long long, long long) const { off[r0] = (int)e; }
};

// Rebuild: the previous list; a cell that leaves level 0 gets phi in the
// stage fields (in the count pass, which sees each cell once).
template <class R>
struct FlowList {
  const R *phi;
  Width<R> width;
  const int *old;
  int *off;
  R *u1, *u2;
  static constexpr bool kPrefetch = true;
  typedef R V;
  __device__ R load(long long e) const { return phi[old[e]]; }
  __device__ int classify(R v, long long) const { return width.in(v) ? 1 : 0; }
  __device__ int flags(long long e) const { return classify(load(e), e); }
  __device__ void counted(long long e, int bits) const {
    if (bits) return;
    const int o = old[e];
    u1[o] = u2[o] = phi[o];
  }
  __device__ void emit(long long e, int, long long r0, long long, long long) const { off[r0] = old[e]; }
};

// phi -> u1, u2, the whole array
template <class R>
__global__ void __launch_bounds__(256) k_copy_fields(const R *__restrict__ phi, R *__restrict__ u1,
                                                     R *__restrict__ u2, long long n) {
  constexpr int kPer = 8;
  const long long base = (long long)blockIdx.x * (256 * kPer) + threadIdx.x;
  R v[kPer];
#pragma unroll
  for (int q = 0; q < kPer; q++)
    if (base + 256 * q < n) v[q] = phi[base + 256 * q];
#pragma unroll
  for (int q = 0; q < kPer; q++)
    if (base + 256 * q < n) u1[base + 256 * q] = u2[base + 256 * q] = v[q];
}

template <class R, bool EXACT>
int run(const char *name, R *phi_user, const Box &gb, const Box &fb, R dx, R a_n, R b_n, R cfl, R gamma, R beta,
        int n_steps, int rebuild_every, double *dt_log, long long *band_log) {
  Call call(name);
  if (!gb.contains(fb, 0, 0, 0)) call.fail("fill box outside the ghost box");
  if (rebuild_every <= 0) call.fail("rebuild_every must be positive");
  if (gb.size() >= (1LL << 31)) call.fail("ghost box of 2^31 cells or more");
  if (!call.ok()) return LSMGPU_ERR_BOUNDS;
  if (n_steps <= 0) return LSMGPU_OK;
  const long long n = gb.size();
  R *phi = call.inout(phi_user, n);
  R *u1 = call.temp<R>(n), *u2 = call.temp<R>(n);
  constexpr bool packed = !EXACT && sizeof(R) == 4;
  R *rhs = nullptr;  // per level-0 entry; sized at the first build
  int *off0 = nullptr, *off1 = nullptr;  // level-0 lists: this one, and the next rebuild's
  R *dt = call.temp<R>(1);
  unsigned long long *key = call.temp<unsigned long long>(1);
  double *dtl = dt_log ? call.temp<double>(n_steps) : nullptr;
  if (!call.ok()) return lsmgpu_get_last_error(nullptr, 0);
  cudaStream_t s = stream();
  if (dtl) cudaMemsetAsync(dtl, 0, sizeof(double) * n_steps, s);  // steps after the band has emptied
  const Width<R> width((double)gamma);
  int n0 = 0, nrebuild = 0;
  for (int step = 0; step < n_steps; step++) {
    if (step % rebuild_every == 0) {
      Compaction c;
      long long tot[3] = {0, 0, 0};
      if (nrebuild == 0) {
        FlowGrid<R> f{phi, width, nullptr};
        if (!c.count(call, f, n, tot)) return lsmgpu_get_last_error(nullptr, 0);
        if (tot[0] > 0) {
          // later lists are sub-sequences of this one; an even number of
          // elements for the pair loads, a 4-value record per entry pair in
          // the FP32 form
          off0 = call.temp<int>(tot[0] + 2);
          off1 = call.temp<int>(tot[0] + 2);
          rhs = call.temp<R>(packed ? 2 * tot[0] + 4 : tot[0]);
          if (!call.ok()) return lsmgpu_get_last_error(nullptr, 0);
          f.off = off0;
          c.emit(f);
          LSMGPU_LAUNCH(k_copy_fields<R>, (unsigned)((n + 2047) / 2048), 256, 0, phi, u1, u2, n);
        }
      } else if (n0 > 0) {
        const FlowList<R> f{phi, width, off0, off1, u1, u2};
        if (!c.count(call, f, n0, tot)) return lsmgpu_get_last_error(nullptr, 0);
        c.emit(f);
        int *t = off0;
        off0 = off1;
        off1 = t;
      }
      n0 = (int)tot[0];
      if (band_log) band_log[nrebuild] = tot[0];
      nrebuild++;
    }
    if (n0 == 0) continue;
    BandArgs<R> a{};
    a.off0 = off0;
    a.n0 = n0;
    a.dx = dx; a.a_n = a_n; a.b_n = b_n; a.beta = beta; a.gamma = gamma; a.cfl = cfl;
    a.f_half = R(0.5) / dx;
    a.f_xx = R(1.0) / dx / dx;
    a.f_xy = R(0.25) / dx / dx;
    a.inv_dx = R(1.0) / dx;
    a.rhs = rhs;
    a.dt = dt;
    a.key = key;
    const unsigned blocks = (unsigned)((n0 + 127) / 128);
    const bool small = n < (1LL << 30);  // byte offsets of the FP32 form in 32 bits
    const unsigned blocks2 = (unsigned)((n0 + 255) / 256);  // pairs of entries
    // stage 1
    a.src = view((const R *)phi, gb);
    a.phin = a.src;
    a.out = view(u1, gb);
    a.stage = 1;
    cudaMemsetAsync(key, 0, sizeof(unsigned long long), s);
    if constexpr (packed) LSMGPU_LAUNCH((small ? k_band_rhs_x2<unsigned> : k_band_rhs_x2<unsigned long long>), blocks2, 128, 0, a);
    else LSMGPU_LAUNCH(k_band_rhs<R>, blocks, 128, 0, a);
    LSMGPU_LAUNCH(k_band_dt<R>, 1, 1, 0, key, dt, cfl, dtl ? dtl + step : nullptr);
    if constexpr (packed) LSMGPU_LAUNCH((small ? k_band_update1_x2<unsigned> : k_band_update1_x2<unsigned long long>), blocks2, 128, 0, a);
    else LSMGPU_LAUNCH(k_band_update1<R>, blocks, 128, 0, a);
    // stage 2
    a.src = view((const R *)u1, gb);
    a.out = view(u2, gb);
    a.phin = view((const R *)phi, gb);
    a.stage = 2;
    if constexpr (packed) LSMGPU_LAUNCH((small ? k_band_stage_x2<unsigned> : k_band_stage_x2<unsigned long long>), blocks2, 128, 0, a);
    else LSMGPU_LAUNCH(k_band_stage<R>, blocks, 128, 0, a);
    // stage 3 (in place on phi: each cell reads only its own phi^n)
    a.src = view((const R *)u2, gb);
    a.out = view(phi, gb);
    a.stage = 3;
    if constexpr (packed) LSMGPU_LAUNCH((small ? k_band_stage_x2<unsigned> : k_band_stage_x2<unsigned long long>), blocks2, 128, 0, a);
    else LSMGPU_LAUNCH(k_band_stage<R>, blocks, 128, 0, a);
  }
  if (dt_log) cudaMemcpyAsync(dt_log, dtl, sizeof(double) * n_steps, cudaMemcpyDeviceToHost, s);
  call.finish();
  cudaStreamSynchronize(s);
  return lsmgpu_get_last_error(nullptr, 0);
}

}  // namespace bandflow
}  // namespace lsmgpu
