// Fused TVD Runge-Kutta stage kernels: one kernel per stage computes the
// HJ WENO5 derivatives, the level-set right-hand side (advection, or the
// reinitialization Hamiltonian) and the stage update in a single pass, with
// the periodic ghost images of the result written in the same pass.
//
// Work layout in HBM (one buffer per stage field): interior cells (0..nx-1,
// 0..ny-1, 0..nz-1) with GX = 4 ghost cells below x and 3 above, 3 ghost
// layers in y and z; rows padded to a multiple of 32 elements so each row
// starts on a 128-byte boundary.  A CTA stages its tile plus a 3-cell halo into
// shared memory with one 3D TMA load; the x origin of the box is the tile's
// row offset, a multiple of 16 cells, which satisfies TMA's 16-byte rule for
// both element sizes.
//
// Here: the FP64 stage (k_stage: LSMLIB's operation order, the including unit
// compiled with -fmad=false; 32 x 8 threads, each walking its z column of a
// 32 x 8 tile of 1 to 4 planes, 8 on grids of more than 262140), and the FP32
// arithmetic of the stages in adv_x2.cuh and reinit_x2.cuh, with FMA contraction
// and epsilon-scaled WENO weights that cannot under- or overflow in single
// precision (see weno5_fast).
#pragma once

#include <cmath>
#include <type_traits>

#include "lsmgpu_common.cuh"
#include "stencil_math.cuh"
#include "tma.cuh"
#include "weno64.cuh"

namespace lsmgpu {
namespace fused {

constexpr int GX = 4, GY = 3, GZ = 3;
constexpr int TX = 32, TY = 8, TZ = 8;
constexpr int SX = TX + 8, SY = TY + 6, SZ = TZ + 6;
constexpr uint32_t kMaxPolls = 1u << 22;

struct Layout {
  int nx, ny, nz;
  long long py, pz;  // element pitches of y and z
  __host__ __device__ long long idx(int i, int j, int k) const {
    return (long long)(i + GX) + py * (long long)(j + GY) + pz * (long long)(k + GZ);
  }
  __host__ long long elems() const { return pz * (long long)(nz + 2 * GZ); }
};

inline Layout make_layout(int nx, int ny, int nz) {
  Layout L;
  L.nx = nx; L.ny = ny; L.nz = nz;
  L.py = ((long long)nx + GX + 3 + 31) / 32 * 32;
  L.pz = L.py * (long long)(ny + 2 * GY);
  return L;
}

enum Mode { ADV_CONST = 0, ADV_FIELD = 1, REINIT = 2 };

template <class R>
struct StageArgs {
  Layout L;
  const R *phi_n;    // u^n at the cell (stages 2 and 3)
  const R *phi0;     // sign source of the phi0 reinitialization form
  const R *vel[3];   // velocity fields (ADV_FIELD)
  R *out;
  R vconst[3];       // constant velocity (ADV_CONST)
  R inv[3];          // 1/dx, 1/dy, 1/dz
  R floor4[3];       // FP32 ADV_CONST: eps_floor4 per axis
  R dt, dx_sq;
  int stage;         // 1, 2 or 3
  int use0;          // reinitialization sign from phi0
  int periodic;      // write periodic ghost images of the result
  int ghost;         // 0, or the LSMGPU_BC_* extrapolation whose face ghosts
                     // the kernel computes in shared memory from the tile
  int *err;
};

// The FP32 constant-velocity stages square undivided differences, so the grid
// spacing enters the range of the squares.  The copies into the work layout
// therefore multiply phi by this power of two (exact; divided out by the copies
// back), which keeps the spacings as the stages see them between 2^-9, where the
// floor of epsilon (eps_floor4) is still a normal number, and 2^24, where the
// squares and weight products of slopes up to 7e10 stay finite.  1 for every
// spacing already there.  (Axes more than 2^33 apart cannot both be: the widest
// decides; and with dx below 2^-9 a phi beyond 3.4e38 / scale becomes infinite.)
template <class R>
inline float spacing_scale(const R dx[3]) {
  int lo = 0, hi = 0;
  for (int d = 0; d < 3; d++) {
    const double h = std::fabs((double)dx[d]);
    if (!(h > 0.0) || !std::isfinite(h)) return 1.f;
    const int e = std::ilogb(h);  // 2^e <= h < 2^(e+1)
    lo = d == 0 || e < lo ? e : lo;
    hi = d == 0 || e > hi ? e : hi;
  }
  int p = lo < -9 ? -9 - lo : 0;
  if (hi + p > 23) p = 23 - hi;
  p = p > 126 ? 126 : (p < -126 ? -126 : p);  // 1 / scale is a normal number too
  return std::ldexp(1.f, p);
}
// The weights' common scale (window_q) and 4 (1e-36 dx^2) times it, dx scaled:
// LSMLIB's floor is in units of the divided differences.  (Kept a normal number
// where one axis' spacing is out of the range above.)
constexpr float kWeightScale = 1024.f;
constexpr float kFloor4 = 4e-36f * kWeightScale;  // dx = 1
inline float eps_floor4(double dx) {
  const double f = (double)kFloor4 * dx * dx;
  return f < 1.5e-38 ? 1.5e-38f : (f < 3e38 ? (float)f : 3e38f);
}

// One-axis extrapolation of LSMLIB's ghost-cell routines
// (boundary_conditions3d.f:46-462) at distance g from the edge value e, with
// n the value next inside: linear (slope e - n), signed linear (slope
// sign(e) |e - n|, :203-206) or copy (homogeneous Neumann).
template <class R>
__device__ __forceinline__ R extrap(R e, R n, int g, int kind) {
  if (kind == LSMGPU_BC_COPY) return e;
  const R s = (kind == LSMGPU_BC_SIGNED_LINEAR) ? copysign(R(1.0), e) * fabs(e - n) : e - n;
  return e + s * R(g);
}

// The ghost cells a stage's stencils read (face ghosts: one coordinate in
// the 3-cell layer, the other two interior) that lie in a staged tile,
// computed from the tile's interior cells with LSMLIB's extrapolation
// (boundary_conditions3d.f:46-462): identical values to a fill of the
// stored array, whose faces are written x, then y, then z, because a face
// ghost of an axis is written only by that axis' pass from interior cells.
// (Edge and corner ghosts are read by no axis-aligned stencil.)
// Only the lines that the tile's own cells read are filled (x ghosts of its
// rows, y and z ghosts of its columns), one per thread and pass of 256
// threads: on small grids the stage is the latency of an edge tile.  The faces
// write disjoint cells and read only interior ones, so they are filled in any
// order; a tile inside the domain on every axis has none (one uniform test).
// Not inlined, so the stage kernels' register allocation does not depend on it.
// us per reinitialization stage with the whole halo's lines filled face by face
// / with these: FP32 37 x 33 x 41 5.8 / 4.9, 128^3 21.2 / 19.8, 256^3 129 / 121;
// FP64 121 x 118 x 109 662 / 637.
template <class R, int W, int H>
__device__ __noinline__ void fill_face_ghosts(R *tile, int tzn, int x0, int y0, int z0, const Layout &L, int kind,
                                              int tid) {
  constexpr int sy = W + 8, sz = sy * (H + 6), T = 256;
  if (x0 >= 3 && x0 + W + 3 <= L.nx && y0 >= 3 && y0 + H + 3 <= L.ny && z0 >= 3 && z0 + tzn + 3 <= L.nz) return;
  R *const cells = tile + 4 + 3 * sy + 3 * sz;  // cell (x0, y0, z0)
  // ghost layers 1 .. n beyond the edge cell, away from the interior along `out`
  auto line = [&](R *edge, int out, int n) {
    const R e = edge[0], in = edge[-out];
#pragma unroll
    for (int g = 1; g <= 3; g++)
      if (g <= n) edge[g * out] = extrap(e, in, g, kind);
  };
  const int kx = min(W, L.nx - x0), ky = min(H, L.ny - y0), kz = min(tzn, L.nz - z0);  // own cells
  // layers below and above that the tile reads, and the edge cells' offsets
  const int bx = 3 - x0, by = 3 - y0, bz = 3 - z0;
  const int ax = x0 + W + 3 - L.nx, ay = y0 + H + 3 - L.ny, az = z0 + tzn + 3 - L.nz;
  if (bx > 0 || ax > 0)
    for (int e = tid; e < H * kz; e += T) {
      const int y = e % H, z = e / H;
      R *row = cells + y * sy + z * sz;
      if (y < ky) {
        if (bx > 0) line(row - x0, -1, bx);
        if (ax > 0) line(row + L.nx - 1 - x0, 1, ax);
      }
    }
  if (by > 0 || ay > 0)
    for (int e = tid; e < W * kz; e += T) {
      const int x = e % W, z = e / W;
      R *col = cells + x + z * sz;
      if (x < kx) {
        if (by > 0) line(col - y0 * sy, -sy, by);
        if (ay > 0) line(col + (L.ny - 1 - y0) * sy, sy, ay);
      }
    }
  if (bz > 0 || az > 0)
    for (int e = tid; e < W * ky; e += T) {
      const int x = e % W, y = e / W;
      R *col = cells + x + y * sy;
      if (x < kx) {
        if (bz > 0) line(col - z0 * sz, -sz, bz);
        if (az > 0) line(col + (L.nz - 1 - z0) * sz, sz, az);
      }
    }
}

// ---------------------------------------------------------------------------
// FP32 arithmetic
// ---------------------------------------------------------------------------
// WENO5-JS with the nonlinear weights rewritten as
//   w_k = d_k prod_{j != k} q_j / sum_i d_i prod_{j != i} q_j,
//   q_k = (S_k / eps + 1)^2,
// which equals d_k/(S_k+eps)^2 normalised.  S_k <= 64 max v^2 and
// eps >= 1e-6 max v^2, so 1 <= q_k <= 4.2e15 and every product stays below
// 2e31: no underflow to 0/0 on near-flat data (where the direct form's
// (S+eps)^2 underflows in FP32) and no overflow, with two reciprocals
// instead of four divisions.
__device__ __forceinline__ float weno5_fast(float v1, float v2, float v3, float v4, float v5) {
  const float c13 = 1.f / 3.f, c76 = 7.f / 6.f, c116 = 11.f / 6.f, c16 = 1.f / 6.f, c56 = 5.f / 6.f;
  const float c1312 = 13.f / 12.f;
  const float m = fmaxf(fmaxf(fmaxf(v1 * v1, v2 * v2), fmaxf(v3 * v3, v4 * v4)), v5 * v5);
  const float eps = fmaf(1e-6f, m, 1e-36f);
  const float p1 = fmaf(c13, v1, fmaf(-c76, v2, c116 * v3));
  const float p2 = fmaf(-c16, v2, fmaf(c56, v3, c13 * v4));
  const float p3 = fmaf(c13, v3, fmaf(c56, v4, -c16 * v5));
  float t = v1 - 2.f * v2 + v3, u = v1 - 4.f * v2 + 3.f * v3;
  const float S1 = fmaf(c1312 * t, t, 0.25f * u * u);
  t = v2 - 2.f * v3 + v4; u = v2 - v4;
  const float S2 = fmaf(c1312 * t, t, 0.25f * u * u);
  t = v3 - 2.f * v4 + v5; u = 3.f * v3 - 4.f * v4 + v5;
  const float S3 = fmaf(c1312 * t, t, 0.25f * u * u);
  const float r = __fdividef(1.f, eps);
  float q1 = fmaf(S1, r, 1.f), q2 = fmaf(S2, r, 1.f), q3 = fmaf(S3, r, 1.f);
  q1 *= q1; q2 *= q2; q3 *= q3;
  const float n1 = 0.1f * (q2 * q3), n2 = 0.6f * (q1 * q3), n3 = 0.3f * (q1 * q2);
  return __fdividef(fmaf(n1, p1, fmaf(n2, p2, n3 * p3)), n1 + n2 + n3);
}

// ---------------------------------------------------------------------------
// the stage kernel
// ---------------------------------------------------------------------------
// The FP64 stage.  Bound by its arithmetic (weno64.cuh: the FP64 pipe with the
// integer pipes close behind), so the tile only has to be there in time: tiles
// of `tz` planes (1 to 4, chosen by the launcher so that the last wave of
// tiles is a small part of the run), at 40 registers for six CTAs per SM
// (reinitialization 121 x 118 x 109, 5 steps: four 10.27 ms, five 10.04, six
// 9.95, seven 10.14; field advection 111 x 104 x 92: five 3.95, six 3.87,
// seven 3.93; both on tiles of one plane).  Tiles of one and two planes leave
// room for six, four planes (44.8 KB staged) for five.
template <class R, int MODE, bool EXACT>
__global__ void __launch_bounds__(TX * TY, 6) k_stage(const __grid_constant__ CUtensorMap tm, StageArgs<R> a, int tzn) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  R *tile = reinterpret_cast<R *>(smem_raw);
  __shared__ __align__(8) uint64_t bar;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int tid = tx + TX * ty;
  const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY, z0 = blockIdx.z * tzn;
  const int szn = tzn + 6;

  if (tid == 0) {
    prefetch_tmap(&tm);
    mbar_init(&bar, 1);
    fence_barrier_init();
  }
  __syncthreads();
  if (tid == 0) {
    mbar_arrive_expect_tx(&bar, (uint32_t)(SX * SY * szn * sizeof(R)));
    // padded coordinates of interior cell (x0 - 4, y0 - 3, z0 - 3)
    tma_load_3d(tile, &tm, x0 + GX - 4, y0 + GY - 3, z0 + GZ - 3, &bar);
  }
  if (!mbar_wait(&bar, 0, kMaxPolls)) {
    if (tid == 0) atomicExch(a.err, LSMGPU_ERR_TIMEOUT);
    mbar_wait(&bar, 0, kMaxPolls);  // let an in-flight copy land before exit
    return;
  }
  if (a.ghost) {
    fill_face_ghosts<R, TX, TY>(tile, tzn, x0, y0, z0, a.L, a.ghost, tid);
    __syncthreads();
  }

  const Layout &L = a.L;
  const int i = x0 + tx, j = y0 + ty;
  if (i >= L.nx || j >= L.ny) return;
  const int sx = tx + 4, sy = ty + 3;
  const int kmax = min(tzn, L.nz - z0);

  for (int tz = 0; tz < kmax; tz++) {
    const int k = z0 + tz;
    const int sz = tz + 3;
    const R *c = tile + (sz * SY + sy) * SX + sx;
    R rhs;
    if (MODE == REINIT) {
      const R pc = a.use0 ? a.phi0[L.idx(i, j, k)] : c[0];
      R n2 = R(0);
#pragma unroll 1
      for (int d = 0; d < 3; d++) {
        const int s = d == 0 ? 1 : (d == 1 ? SX : SX * SY);
        R D[6], gp, gm;  // D1(c-2 .. c+3)
#pragma unroll
        for (int f = -2; f <= 3; f++) D[f + 2] = c[f * s] - c[(f - 1) * s];
        weno5_pm64(D, wide64(a.inv[d]), Consts<R>::tiny, gp, gm);
        const R t = reinit_axis(pc, gp, gm);
        n2 = d == 0 ? sqr_(t) : n2 + sqr_(t);
      }
      rhs = reinit_from_sq<R>(pc, n2, a.dx_sq, a.use0 != 0);
    } else {
      R dot = R(0);
#pragma unroll 1
      for (int d = 0; d < 3; d++) {
        // spatial_derivatives3d.f.in:2756-2812: |v| < zero_tol gives 0, v > 0
        // takes the backward stencil, otherwise the forward one, which is
        // the backward one of the mirrored line, negated: v g = |v| g'
        const R u = (MODE == ADV_CONST) ? a.vconst[d] : a.vel[d][L.idx(i, j, k)];
        R g = R(0);
        if (!below_(u, R(Consts<double>::zero_tol))) {
          const int s0 = d == 0 ? 1 : (d == 1 ? SX : SX * SY), s = is_pos_(u) ? s0 : -s0;
          R D[5];
#pragma unroll
          for (int f = -2; f <= 2; f++) D[f + 2] = c[f * s] - c[(f - 1) * s];
          g = weno5_side64(D, wide64(a.inv[d]), Consts<R>::tiny);
        }
        const R t = mul_z_(abs_(u), g);
        dot = d == 0 ? t : dot + t;
      }
      // lsm3dZeroOutLevelSetEqnRHS then lsm3dAddAdvectionTermToLSERHS
      // (level_set_evolution3d.f.in:38, :113-116)
      rhs = R(0) - dot;
    }

    const long long cell = L.idx(i, j, k);
    R u = c[0] + mul_(a.dt, rhs);  // tvd_runge_kutta3d.f:78
    if (a.stage == 2) u = fpi::plus_quarter(mul_(R(0.75), a.phi_n[cell]), u);  // :403-404
    if (a.stage == 3) u = mul_(R(1.0 / 3.0), a.phi_n[cell]) + mul_(R(2.0 / 3.0), u);  // :490-492
    a.out[cell] = u;

    if (a.periodic) {
      // periodic images in the ghost layers (3 cells per side)
      int oi[2] = {0, 0}, oj[2] = {0, 0}, ok_[2] = {0, 0};
      int ni = 1, nj = 1, nk = 1;
      if (i < 3) oi[ni++] = L.nx; else if (i >= L.nx - 3) oi[ni++] = -L.nx;
      if (j < 3) oj[nj++] = L.ny; else if (j >= L.ny - 3) oj[nj++] = -L.ny;
      if (k < 3) ok_[nk++] = L.nz; else if (k >= L.nz - 3) ok_[nk++] = -L.nz;
      if (ni + nj + nk > 3) {
        for (int p = 0; p < ni; p++)
          for (int q = 0; q < nj; q++)
            for (int r = 0; r < nk; r++)
              if (p | q | r) a.out[L.idx(i + oi[p], j + oj[q], k + ok_[r])] = u;
      }
    }
  }
}

}  // namespace fused
}  // namespace lsmgpu

// ---------------------------------------------------------------------------
// FP32 arithmetic on cell pairs: two cells at a time, one per lane of
// Blackwell's packed FP32x2 instructions (FADD2 / FMUL2 / FFMA2), which halves
// the issued instructions of the WENO5 arithmetic.  Comparisons, selections and
// the reciprocals stay per lane.
// ---------------------------------------------------------------------------
namespace lsmgpu {
namespace fused {

__device__ __forceinline__ float2 sp(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return fma2(b, sp(-1.f), a); }
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float2 rcp2(float2 x) { return make_float2(rcp_approx(x.x), rcp_approx(x.y)); }
__device__ __forceinline__ float max3f(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float2 max5(float2 a, float2 b, float2 c, float2 d, float2 e) {
  return make_float2(max3f(max3f(a.x, b.x, c.x), d.x, e.x), max3f(max3f(a.y, b.y, c.y), d.y, e.y));
}

// 2^-floor(log2 x) for a positive normal float x, from the exponent bits (no
// reciprocal instruction).  x * pow2_recip(x) lies in [1, 2).
__device__ __forceinline__ float pow2_recip(float x) {
  return __int_as_float(0x7f000000 - (__float_as_int(x) & 0x7f800000));
}
__device__ __forceinline__ float2 pow2_recip2(float2 x) { return make_float2(pow2_recip(x.x), pow2_recip(x.y)); }

// num / den per lane for den a normal number below 2^126: the product with
// the approximate reciprocal, without the scaling a general quotient carries
__device__ __forceinline__ float2 quot2(float2 num, float2 den) { return mul2(num, rcp2(den)); }

// WENO5-JS on two cells at once, the epsilon-scaled weight form of
// weno5_fast with the common factors folded: only S/eps enters the weights,
// so the smoothness indicators are kept as 4 S and epsilon as 12 eps (the
// factor 3 goes into the scale), and the weights as 10 d_k prod q_j^2.
__device__ __forceinline__ float2 weno5_x2(float2 v1, float2 v2, float2 v3, float2 v4, float2 v5) {
  const float2 q1s = mul2(v1, v1), q2s = mul2(v2, v2), q3s = mul2(v3, v3), q4s = mul2(v4, v4), q5s = mul2(v5, v5);
  const float2 m = max5(q1s, q2s, q3s, q4s, q5s);
  const float2 eps = fma2(sp(12e-6f), m, sp(12e-36f));  // 12 eps
  const float c13 = 1.f / 3.f, c76 = 7.f / 6.f, c116 = 11.f / 6.f, c16 = 1.f / 6.f, c56 = 5.f / 6.f;
  const float2 P1 = fma2(sp(c13), v1, fma2(sp(-c76), v2, mul2(sp(c116), v3)));
  const float2 P2 = fma2(sp(-c16), v2, fma2(sp(c56), v3, mul2(sp(c13), v4)));
  const float2 P3 = fma2(sp(c13), v3, fma2(sp(c56), v4, mul2(sp(-c16), v5)));
  // 4 * smoothness indicators: 13/3 t^2 + u^2
  const float c133 = 13.f / 3.f;
  float2 t = fma2(sp(-2.f), v2, add2(v1, v3));
  float2 u = fma2(sp(-4.f), v2, fma2(sp(3.f), v3, v1));
  const float2 S1 = fma2(u, u, mul2(mul2(sp(c133), t), t));
  t = fma2(sp(-2.f), v3, add2(v2, v4));
  u = fma2(sp(-1.f), v4, v2);
  const float2 S2 = fma2(u, u, mul2(mul2(sp(c133), t), t));
  t = fma2(sp(-2.f), v4, add2(v3, v5));
  u = fma2(sp(-4.f), v4, fma2(sp(3.f), v3, v5));
  const float2 S3 = fma2(u, u, mul2(mul2(sp(c133), t), t));
  // q_k = (S_k + eps) 2^-e with 2^e <= eps < 2^(e+1): the weights only see
  // ratios of the q_k, so any common scale of S + eps gives the same weights
  // as (S_k / eps + 1); with eps 2^-e in [1, 2), 1 <= q_k < 7e7 and the
  // products below stay under 1e32
  const float2 r = pow2_recip2(eps);
  const float2 e = mul2(eps, r), r3 = mul2(sp(3.f), r);
  const float2 q1 = fma2(S1, r3, e), q2 = fma2(S2, r3, e), q3 = fma2(S3, r3, e);
  const float2 q23 = mul2(q2, q3), q13 = mul2(q1, q3), q12 = mul2(q1, q2);
  // 10 d_k prod_{j != k} q_j^2 (the common factor cancels)
  const float2 n1 = mul2(q23, q23);
  const float2 n2 = mul2(mul2(sp(6.f), q13), q13);
  const float2 n3 = mul2(mul2(sp(3.f), q12), q12);
  const float2 num = fma2(n1, P1, fma2(n2, P2, mul2(n3, P3)));
  const float2 den = add2(add2(n1, n2), n3);
  return quot2(num, den);
}

// A triple of consecutive differences (d0, d1, d2): its second difference t
// and the three smoothness-indicator forms it takes in a window, times 4:
//   first triple of a window:  13/3 t^2 + (d0 - 4 d1 + 3 d2)^2
//   middle triple:             13/3 t^2 + (d0 - d2)^2
//   last triple:               13/3 t^2 + (3 d0 - 4 d1 + d2)^2
// (spatial_derivatives3d.f.in:1306-1311), with d0 - 4 d1 + 3 d2 =
// 2 t + (d2 - d0) and 3 d0 - 4 d1 + d2 = 2 t - (d2 - d0).
struct Tri {
  float2 t, s1, s2, s3;
};
__device__ __forceinline__ Tri tri_forms(float2 d0, float2 d1, float2 d2) {
  Tri r;
  r.t = fma2(sp(-2.f), d1, add2(d0, d2));
  const float2 b = sub2(d2, d0);
  const float2 T = mul2(mul2(sp(13.f / 3.f), r.t), r.t);
  const float2 u = fma2(sp(2.f), r.t, b), w = fma2(sp(-2.f), r.t, b);
  r.s1 = fma2(u, u, T);
  r.s2 = fma2(b, b, T);
  r.s3 = fma2(w, w, T);
  return r;
}

// Weight products of a window from its three indicator forms (x4) and the
// maximum squared difference m: q_k = (4 S_k / (4 eps) + 1) / kWeightScale =
// (S_k + eps) / eps / kWeightScale, eps = 1e-6 m + 1e-36 (LSMLIB's,
// spatial_derivatives3d.f.in:1296, in units of the unscaled differences, or
// with the floor scaled to them; floor4 is 4 kWeightScale times it); only
// ratios of the q_k enter the weights.  2^-10 <= q_k < 4e4, so the squared
// products lie between 2^-40 and 3e18: their products with differences up to
// 1e18, whose squares are the next to overflow, are finite, and those with
// differences down to 1e-26 normal.
struct WQ {
  float2 q23, q13, q12;  // (q2 q3)^2, (q1 q3)^2, (q1 q2)^2
};
__device__ __forceinline__ WQ window_q(float2 s1, float2 s2, float2 s3, float2 m, float floor4 = kFloor4) {
  // 1 / (4 eps kWeightScale), finite: floor4 is a normal number
  const float2 s = rcp2(fma2(sp(4e-6f * kWeightScale), m, sp(floor4)));
  const float2 one = sp(1.f / kWeightScale);
  const float2 q1 = fma2(s1, s, one), q2 = fma2(s2, s, one), q3 = fma2(s3, s, one);
  const float2 a = mul2(q2, q3), b = mul2(q1, q3), c = mul2(q1, q2);
  return {mul2(a, a), mul2(b, b), mul2(c, c)};
}

// The sides are kept doubled (the factor goes into the 1/dx^2 of |grad phi|^2):
// with the central candidate 2 p2 = D(c) + D(c+1) - t(c-1) / 3 (minus) or
// D(c-1) + D(c) - t(c-1) / 3 (plus), A = q23, B = q12, C = q13,
//   2 minus(c)  = 2 p2 + (A TD(c-2) + 3/2 B TD(c-1)) / (3/2 A + 9 C + 9/2 B)
//   2 plus(c-1) = 2 p2 - (3/2 A TD(c-2) + B TD(c-1)) / (9/2 A + 9 C + 3/2 B)
// `a` is TD(c-2), `nb` is -TD(c-1).
__device__ __forceinline__ float2 side_minus(const WQ &w, float2 a, float2 nb, float2 p2) {
  const float2 num = fma2(sp(-1.5f), mul2(w.q12, nb), mul2(w.q23, a));
  const float2 den = fma2(sp(1.5f), w.q23, fma2(sp(4.5f), w.q12, mul2(sp(9.f), w.q13)));
  return fma2(num, rcp2(den), p2);
}
__device__ __forceinline__ void sides_both(const WQ &w, float2 a, float2 nb, float2 p2m, float2 p2p, float2 &minus,
                                           float2 &plus) {
  const float2 u = mul2(w.q23, a), v = mul2(w.q12, nb);
  const float2 g = mul2(sp(9.f), w.q13);
  const float2 den_m = fma2(sp(1.5f), w.q23, fma2(sp(4.5f), w.q12, g));
  const float2 den_p = fma2(sp(1.5f), w.q12, fma2(sp(4.5f), w.q23, g));
  minus = fma2(fma2(sp(-1.5f), v, u), rcp2(den_m), p2m);
  plus = fma2(fma2(sp(-1.5f), u, v), rcp2(den_p), p2p);
}

// 2 minus(c) of the window W(c) = D[0..4] = D(c-2 .. c+2), per lane
__device__ __forceinline__ float2 minus_of_window(const float2 D[5], float floor4 = kFloor4, Tri *mid = nullptr,
                                                  Tri *last = nullptr) {
  const Tri a0 = tri_forms(D[0], D[1], D[2]), a1 = tri_forms(D[1], D[2], D[3]), a2 = tri_forms(D[2], D[3], D[4]);
  float2 sq[5];
#pragma unroll
  for (int q = 0; q < 5; q++) sq[q] = mul2(D[q], D[q]);
  const WQ wq = window_q(a0.s1, a1.s2, a2.s3, max5(sq[0], sq[1], sq[2], sq[3], sq[4]), floor4);
  const float2 p2m = fma2(sp(-1.f / 3.f), a1.t, add2(D[2], D[3]));
  if (mid) *mid = a1;
  if (last) *last = a2;
  return side_minus(wq, sub2(a0.t, a1.t), sub2(a2.t, a1.t), p2m);
}

// Periodic images of a cell's new value in the 3 ghost layers along y and z
// (and their x images), for a cell within 3 of a y or z face; its image along
// x alone is written by the caller.  dx, dy, dz: the element offsets of the
// cell's image along each axis (0: none).  Not inlined: the stage loop then
// keeps none of its index arithmetic.
static __device__ __noinline__ void write_yz_images(float *c, int dx, long long dy, long long dz, float val) {
  if (dy) c[dy] = val;
  if (dz) c[dz] = val;
  if (dx && dy) c[dx + dy] = val;
  if (dx && dz) c[dx + dz] = val;
  if (dy && dz) c[dy + dz] = val;
  if (dx && dy && dz) c[dx + dy + dz] = val;
}
// index offset of the periodic image of index i of n (0: none)
__device__ __forceinline__ int image_of(int i, int n) { return i < 3 ? n : (i >= n - 3 ? -n : 0); }

// Stores the pair (u.x, u.y) of a row at out + cell (the second cell where
// `two`), with its periodic images: those along x are two predicated stores
// (px0, px1: image_of of both cells; every row of a tile column at an x face
// has such cells), the others concern whole rows and planes (j and k are the
// warp's).
__device__ __forceinline__ void store_pair(float *out, const Layout &L, long long cell, float2 u, bool two, int px0,
                                           int px1, int py, int pz) {
  float *c = out + cell;
  if (two) *reinterpret_cast<float2 *>(c) = u;
  else c[0] = u.x;
  if (px0) c[px0] = u.x;
  if (px1) c[1 + px1] = u.y;
  if ((py | pz) != 0) {
    const long long dy = L.py * py, dz = L.pz * pz;
    write_yz_images(c, px0, dy, dz, u.x);
    if (two) write_yz_images(c + 1, px1, dy, dz, u.y);
  }
}

// 2 minus(c) of two cells from phi(c-3 .. c+2), in units of phi (WENO5 is
// homogeneous of degree one: the caller scales by 1/(2 dx) once); 51 packed
// operations where weno5_x2 with its scaled differences takes 66.
__device__ __forceinline__ float2 weno5_backward_x2(const float2 x[6], float floor4) {
  float2 D[5];
#pragma unroll
  for (int q = 0; q < 5; q++) D[q] = sub2(x[q + 1], x[q]);
  return minus_of_window(D, floor4);
}

// Both one-sided WENO5 values of one axis for two cells: minus side on
// D(c-2 .. c+2), plus side on D(c+3 .. c-1), given D[0..5] = D(c-2 .. c+3).
// The two sides share two of their three candidate stencils (plus P2 = minus
// P3, plus P3 = minus P2), the second differences t of their middle and outer
// smoothness indicators (plus t2 = minus t3, plus t3 = minus t2), and four of
// the five squared differences of the epsilon maximum; each is computed once.
__device__ __forceinline__ void weno5_pm_x2(const float2 D[6], float2 &gp, float2 &gm) {
  float2 sq[6];
#pragma unroll
  for (int i = 0; i < 6; i++) sq[i] = mul2(D[i], D[i]);
  const float cx = max3f(sq[1].x, sq[2].x, sq[3].x), cy = max3f(sq[1].y, sq[2].y, sq[3].y);
  // 12 eps of each side, its power-of-two scale r and 12 eps r in [1, 2)
  const float2 em = fma2(sp(12e-6f), make_float2(max3f(cx, sq[4].x, sq[0].x), max3f(cy, sq[4].y, sq[0].y)), sp(12e-36f));
  const float2 ep = fma2(sp(12e-6f), make_float2(max3f(cx, sq[4].x, sq[5].x), max3f(cy, sq[4].y, sq[5].y)), sp(12e-36f));
  const float2 rm = pow2_recip2(em), rp = pow2_recip2(ep);
  const float2 emr = mul2(em, rm), epr = mul2(ep, rp);
  const float2 rm3 = mul2(sp(3.f), rm), rp3 = mul2(sp(3.f), rp);
  // candidate stencils
  const float c13 = 1.f / 3.f, c76 = 7.f / 6.f, c116 = 11.f / 6.f, c16 = 1.f / 6.f, c56 = 5.f / 6.f;
  const float2 P1m = fma2(sp(c13), D[0], fma2(sp(-c76), D[1], mul2(sp(c116), D[2])));
  const float2 A = fma2(sp(-c16), D[1], fma2(sp(c56), D[2], mul2(sp(c13), D[3])));  // minus p2, plus p3
  const float2 B = fma2(sp(c13), D[2], fma2(sp(c56), D[3], mul2(sp(-c16), D[4])));  // minus p3, plus p2
  const float2 P1p = fma2(sp(c13), D[5], fma2(sp(-c76), D[4], mul2(sp(c116), D[3])));
  // second differences t and the asymmetric parts u of the indicators
  const float2 t1m = fma2(sp(-2.f), D[1], add2(D[0], D[2]));
  const float2 t2 = fma2(sp(-2.f), D[2], add2(D[1], D[3]));  // minus t2, plus t3
  const float2 t3 = fma2(sp(-2.f), D[3], add2(D[2], D[4]));  // minus t3, plus t2
  const float2 t1p = fma2(sp(-2.f), D[4], add2(D[5], D[3]));
  const float2 u1m = fma2(sp(-4.f), D[1], fma2(sp(3.f), D[2], D[0]));
  const float2 u2m = fma2(sp(-1.f), D[3], D[1]);
  const float2 u3m = fma2(sp(-4.f), D[3], fma2(sp(3.f), D[2], D[4]));
  const float2 u1p = fma2(sp(-4.f), D[4], fma2(sp(3.f), D[3], D[5]));
  const float2 u2p = fma2(sp(-1.f), D[2], D[4]);
  const float2 u3p = fma2(sp(-4.f), D[2], fma2(sp(3.f), D[3], D[1]));
  // 4 * smoothness indicators, 13/3 t^2 + u^2 (times 3 r below gives 12 S r)
  const float c133 = 13.f / 3.f;
  const float2 T1m = mul2(mul2(sp(c133), t1m), t1m), T2 = mul2(mul2(sp(c133), t2), t2);
  const float2 T3 = mul2(mul2(sp(c133), t3), t3), T1p = mul2(mul2(sp(c133), t1p), t1p);
  const float2 q1m = fma2(fma2(u1m, u1m, T1m), rm3, emr);
  const float2 q2m = fma2(fma2(u2m, u2m, T2), rm3, emr);
  const float2 q3m = fma2(fma2(u3m, u3m, T3), rm3, emr);
  const float2 q1p = fma2(fma2(u1p, u1p, T1p), rp3, epr);
  const float2 q2p = fma2(fma2(u2p, u2p, T3), rp3, epr);
  const float2 q3p = fma2(fma2(u3p, u3p, T2), rp3, epr);
  // weights 10 d_k prod_{j != k} q_j^2 (the common factor cancels)
  auto combine = [](float2 q1, float2 q2, float2 q3, float2 p1, float2 p2, float2 p3) {
    const float2 q23 = mul2(q2, q3), q13 = mul2(q1, q3), q12 = mul2(q1, q2);
    const float2 n1 = mul2(q23, q23);
    const float2 n2 = mul2(mul2(sp(6.f), q13), q13);
    const float2 n3 = mul2(mul2(sp(3.f), q12), q12);
    const float2 num = fma2(n1, p1, fma2(n2, p2, mul2(n3, p3)));
    const float2 den = add2(add2(n1, n2), n3);  // <= 1e32 < 2^126
    return quot2(num, den);
  };
  gm = combine(q1m, q2m, q3m, P1m, A, B);
  gp = combine(q1p, q2p, q3p, P1p, B, A);
}

}  // namespace fused
}  // namespace lsmgpu
