// FP32 constant-velocity advection on the x cell pairs and the z march of
// reinit_x2.cuh: the stage kernel of single grids, and the tile routine that
// the batched kernel (batched.cu) shares with it.
//
// The velocity's sign is the same for every cell of a grid, and the forward
// value of a negative velocity is the backward one of the mirrored line,
// negated, so v g = |v| g'.  The callers therefore lay the grid out mirrored
// along each axis of negative velocity (flip bits of the copies into and out
// of the work layout) and these kernels know one direction: v >= 0, the minus
// side of one window per cell and axis.  Every rounding is symmetric, so the
// bits are those of the unmirrored formulas.  With nothing to hand between
// rows, the plane loop has no barrier:
//  * z: the thread marches along its column and carries the last two triples'
//    forms (one new triple per cell);
//  * x: a thread owns two x-neighbouring cells as the lanes of the packed
//    instructions and takes the forms of the two triples before its own from
//    the previous lane (the first lane of a row from a per-tile prologue);
//  * y: the row's three triples, evaluated in place.
// Bound by the issue of FP32 and data-movement instructions (62% and 38% of
// their pipes at 64% of the issue slots): about 130 packed operations per cell
// pair, where a cell-by-cell tile took 165 and as many again in loads,
// selection and set-up.  The differences are not divided by the spacing; phi
// comes in units in which that keeps their squares in range (spacing_scale).
// Measured us per periodic stage, the cell-by-cell tile
// / one kernel per sign triple on 64 x 8 tiles / this kernel: 37 x 33 x 41 4.5
// / 5.3 / 3.8, 128^3 21.2 / 18.3 / 15.7, 256^3 140 / 98.6 / 95.1, 32 x 256 x
// 256 21.6 / 21.6 / 17.3.  (Signed strides for the two axes that need no
// mirrored lanes: 128^3 18.7, 256^3 109.  Planes unrolled by 1 / 2 / 4 / 8: 37 x
// 33 x 41 3.9 / 3.8 / 3.95 / 4.0, 100^3 12.3 / 11.3 / 11.7 / 11.8, 256^3 - / 95.1
// / 92.8 / 95: a run of planes longer than the instruction cache holds costs
// the short tiles more than the moves it saves.)
#pragma once

#include "reinit_x2.cuh"

namespace lsmgpu {
namespace fused {

// the axes along which a grid of velocity v is laid out mirrored, bit d
template <class R>
inline int mirrored_axes(const R v[3]) { return (v[0] < 0 ? 1 : 0) | (v[1] < 0 ? 2 : 0) | (v[2] < 0 ? 4 : 0); }

// a tile's rows are W cells wide; T threads, two cells each, cover a plane of it
template <int W, int T>
struct AdvTile {
  static constexpr int LX = W / 2;        // threads of a row
  static constexpr int ROWS = T / LX;     // rows
  static constexpr int SXW = W + 8, SYW = ROWS + 6;  // staged plane
  // a thread's row; rows of 16 cells: a half-warp takes rows two apart, whose
  // staged words lie in different banks (48 words apart; adjacent rows are 24)
  __device__ static __forceinline__ int row(int tid) {
    return W == 16 ? ((tid >> 5) << 2) | ((tid >> 4) & 1) | ((tid >> 2) & 2) : tid / LX;
  }
  static constexpr size_t smem(int tz) { return (size_t)SXW * SYW * (tz + 6) * sizeof(float); }
};

// One tile of W x ROWS x tzn cells at (x0, y0, z0) whose haloed input is in
// `tile`; `xedge`: 5 x DEPTH x ROWS floats of shared memory.  All T threads call
// it (it has a barrier); tzn is even, at most DEPTH.
template <int W, int T, int DEPTH, int UNROLL>
__device__ __forceinline__ void adv_tile(const float *tile, float *xedge, const StageArgs<float> &a, int x0, int y0,
                                         int z0, int tzn, int tid) {
  using Q = AdvTile<W, T>;
  const Layout &L = a.L;
  constexpr int st_y = Q::SXW, st_z = Q::SXW * Q::SYW;
  const int lx = tid % Q::LX;
  const int w = Q::row(tid);
  constexpr int es = Q::ROWS * DEPTH;  // one quantity's part of xedge
  // ---- prologue: per (plane, row) s1 and t of triple x0-2, s1, s2 and t of
  // x0-1; two planes a thread
  for (int e = tid; e < Q::ROWS * tzn / 2; e += T) {
    const int pw = e % Q::ROWS, pz = 2 * (e / Q::ROWS);
    const float *r0 = tile + (pz + 3) * st_z + (pw + 3) * st_y, *r1 = r0 + st_z;
    float2 p[5], D[4];  // phi(x0-3 ..), D(x0-2 ..)
#pragma unroll
    for (int q = 0; q < 5; q++) p[q] = make_float2(r0[q + 1], r1[q + 1]);
#pragma unroll
    for (int q = 0; q < 4; q++) D[q] = sub2(p[q + 1], p[q]);
    const Tri t2 = tri_forms(D[0], D[1], D[2]), t1 = tri_forms(D[1], D[2], D[3]);
    const float2 v[5] = {t2.s1, t2.t, t1.s1, t1.s2, t1.t};
#pragma unroll
    for (int q = 0; q < 5; q++) {
      xedge[q * es + pz * Q::ROWS + pw] = v[q].x;
      xedge[q * es + (pz + 1) * Q::ROWS + pw] = v[q].y;
    }
  }
  __syncthreads();

  // Rows and lanes outside the grid compute on tile padding and store nothing
  // (whole warps of such rows leave).
  const int i = x0 + 2 * lx, j = y0 + w;
  if (!__any_sync(0xffffffffu, j < L.ny)) return;
  const bool live = i < L.nx && j < L.ny;
  const bool two = i + 1 < L.nx;
  // offsets of the periodic images of the pair's cells along x and y
  const int px0 = a.periodic ? image_of(i, L.nx) : 0, px1 = a.periodic && two ? image_of(i + 1, L.nx) : 0;
  const int py = a.periodic ? image_of(j, L.ny) : 0;
  const int kmax = min(tzn, L.nz - z0);
  const float *col = tile + 3 * st_z + (w + 3) * st_y + 2 * lx + 4;  // cell (i, j) of the first plane
  const float *edge = xedge + w;
  auto ld2 = [](const float *p) { return *reinterpret_cast<const float2 *>(p); };
  // |v| / (2 dx) per axis; 0 where |v| is below the reference's zero tolerance
  float wv[3];
#pragma unroll
  for (int d = 0; d < 3; d++) wv[d] = a.vconst[d] < 1e-11f ? 0.f : 0.5f * a.vconst[d] * a.inv[d];
  auto add_axis = [&](float2 dot, int d, float2 g) {
    const float2 r = fma2(sp(wv[d]), g, dot);
    return wv[d] != 0.f ? r : dot;
  };

  // ---- z march: the carried state for the window of the first cell c ----------
  float2 fl, d0, d1, s1a, s1b, s2b, ta, tb, pm2, pm1, sq0, sq1;
  {
    float2 p[5], D[4], sq[4];  // phi(c-3 .. c+1), D(c-2 .. c+1)
#pragma unroll
    for (int q = 0; q < 5; q++) p[q] = ld2(col + (q - 3) * st_z);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      D[q] = sub2(p[q + 1], p[q]);
      sq[q] = mul2(D[q], D[q]);
    }
    const Tri t2 = tri_forms(D[0], D[1], D[2]), t1 = tri_forms(D[1], D[2], D[3]);
    fl = p[4];
    d0 = D[2];
    d1 = D[3];
    s1a = t2.s1;
    ta = t2.t;
    s1b = t1.s1;
    s2b = t1.s2;
    tb = t1.t;
    pm2 = make_float2(fmaxf(sq[0].x, sq[1].x), fmaxf(sq[0].y, sq[1].y));  // max sq(c-2), sq(c-1)
    pm1 = make_float2(fmaxf(sq[1].x, sq[2].x), fmaxf(sq[1].y, sq[2].y));  // max sq(c-1), sq(c)
    sq0 = sq[2];
    sq1 = sq[3];
  }

  const float *un_src = a.stage == 1 ? nullptr : a.phi_n;
  long long cell = L.idx(live ? i : 0, live ? j : 0, z0);
  float2 un_next = un_src ? ld2(un_src + cell) : sp(0.f);

  // (unrolled: the carried quantities change names instead of registers)
#pragma unroll UNROLL
  for (int tz = 0; tz < kmax; tz++) {
    const float2 un = un_next;  // read one plane ahead of its use
    if (tz + 1 < kmax && un_src) un_next = ld2(un_src + cell + L.pz);
    const float2 u0 = ld2(col);  // phi(i), phi(i+1)
    float2 gx, gy, gz;
    // ---- x: windows W(i), W(i+1) ------------------------------------------------
    {
      const float2 e0 = ld2(col - 4), e1 = ld2(col - 2), e3 = ld2(col + 2);
      const float2 o0 = make_float2(e0.y, e1.x), o1 = make_float2(e1.y, u0.x), o2 = make_float2(u0.y, e3.x);
      // P_s = (D(s), D(s+1)) for s = i-2 .. i+2
      const float2 P0 = sub2(e1, o0), P2 = sub2(u0, o1), P3 = sub2(o2, u0), P4 = sub2(e3, o2);
      const Tri C = tri_forms(P2, P3, P4);  // (tri(i), tri(i+1))
      // (tri(i-2), tri(i-1)) are the previous lane's C
      float a_s1x = __shfl_up_sync(0xffffffffu, C.s1.x, 1), a_s1y = __shfl_up_sync(0xffffffffu, C.s1.y, 1);
      float a_s2y = __shfl_up_sync(0xffffffffu, C.s2.y, 1);
      float a_tx = __shfl_up_sync(0xffffffffu, C.t.x, 1), a_ty = __shfl_up_sync(0xffffffffu, C.t.y, 1);
      if (lx == 0) {
        a_s1x = edge[0];
        a_tx = edge[es];
        a_s1y = edge[2 * es];
        a_s2y = edge[3 * es];
        a_ty = edge[4 * es];
      }
      const float2 At = make_float2(a_tx, a_ty), Bt = make_float2(a_ty, C.t.x);
      const float2 q0 = mul2(P0, P0), q2 = mul2(P2, P2), q4 = mul2(P4, P4);  // sq(i-2 .. i+3)
      const float inner = fmaxf(max3f(q0.y, q2.x, q2.y), q4.x);
      const float2 m = make_float2(fmaxf(inner, q0.x), fmaxf(inner, q4.y));
      const WQ wq = window_q(make_float2(a_s1x, a_s1y), make_float2(a_s2y, C.s2.x), C.s3, m, a.floor4[0]);
      gx = side_minus(wq, sub2(At, Bt), sub2(C.t, Bt), fma2(sp(-1.f / 3.f), Bt, add2(P2, P3)));
    }
    // ---- y: window W(j) ---------------------------------------------------------
    {
      const float2 r[6] = {ld2(col - 3 * st_y), ld2(col - 2 * st_y), ld2(col - st_y), u0, ld2(col + st_y),
                           ld2(col + 2 * st_y)};
      gy = weno5_backward_x2(r, a.floor4[1]);
    }
    // ---- z: window W(k), c = k ----------------------------------------------------
    {
      const float2 f = ld2(col + 2 * st_z);  // phi(c+2)
      const float2 d2 = sub2(f, fl);
      const float2 sq2 = mul2(d2, d2);
      const Tri n = tri_forms(d0, d1, d2);  // tri(c)
      const float2 pmn = make_float2(fmaxf(sq0.x, sq1.x), fmaxf(sq0.y, sq1.y));
      const float2 m = make_float2(max3f(pm2.x, pmn.x, sq2.x), max3f(pm2.y, pmn.y, sq2.y));
      const WQ wq = window_q(s1a, s2b, n.s3, m, a.floor4[2]);
      gz = side_minus(wq, sub2(ta, tb), sub2(n.t, tb), fma2(sp(-1.f / 3.f), tb, add2(d0, d1)));
      fl = f;
      d0 = d1;
      d1 = d2;
      s1a = s1b;
      s1b = n.s1;
      s2b = n.s2;
      ta = tb;
      tb = n.t;
      pm2 = pm1;
      pm1 = pmn;
      sq0 = sq1;
      sq1 = sq2;
    }
    const float2 dot = add_axis(add_axis(add_axis(sp(0.f), 0, gx), 1, gy), 2, gz);
    const float2 rhs = make_float2(-dot.x, -dot.y);
    float2 u = fma2(sp(a.dt), rhs, u0);  // tvd_runge_kutta3d.f:78
    if (a.stage == 2) u = fma2(sp(0.75f), un, mul2(sp(0.25f), u));                  // :403-404
    else if (a.stage == 3) u = fma2(sp(1.f / 3.f), un, mul2(sp(2.f / 3.f), u));  // :490-492
    if (live) store_pair(a.out, L, cell, u, two, px0, px1, py, a.periodic ? image_of(z0 + tz, L.nz) : 0);
    col += st_z;
    edge += Q::ROWS;
    cell += L.pz;
  }
}

// ---------------------------------------------------------------------------
// advection by a velocity field
// ---------------------------------------------------------------------------
// One tile of a stage with a velocity per cell: the upwind side is chosen per
// cell (a lane), so every cell evaluates its own three windows, from the six
// scaled differences D1(c-2 .. c+3) of each axis.  A thread owns two
// x-neighbouring cells, as above, which makes the tile's loads, the velocity's
// and the result's 64 bits wide, and marches along z, carrying that axis'
// differences (one new one per cell); the next plane's velocity and phi^n are
// read a plane ahead.  Same bits as evaluating each cell on its own.  Bound by
// issue: the three windows are 220 packed operations per cell pair and their
// selection 60 moves.  us per stage, two z-neighbouring cells per thread of a
// 32 x 8 tile / this: 64^3 5.96 / 5.4, 100^3 19.3 / 14.4, 192^3 76 / 62, 256^3
// 167 / 133.  (Four CTAs per SM at 64 registers; three at 80: 192^3 65, 256^3
// 138; ten planes of 64 or 16 cells, 64.5 and 58.4 KB staged, leave room for
// three.  Planes unrolled by 1 / 4: 192^3 gradient 1% slower.)
template <int W, int T, int UNROLL>
__device__ __forceinline__ void adv_field_tile(const float *tile, const StageArgs<float> &a, int x0, int y0, int z0,
                                               int tzn, int tid) {
  using Q = AdvTile<W, T>;
  const Layout &L = a.L;
  constexpr int st_y = Q::SXW, st_z = Q::SXW * Q::SYW;
  const int lx = tid % Q::LX, w = Q::row(tid);
  const int i = x0 + 2 * lx, j = y0 + w;
  if (i >= L.nx || j >= L.ny) return;
  const bool two = i + 1 < L.nx;
  const int px0 = a.periodic ? image_of(i, L.nx) : 0, px1 = a.periodic && two ? image_of(i + 1, L.nx) : 0;
  const int py = a.periodic ? image_of(j, L.ny) : 0;
  const int kmax = min(tzn, L.nz - z0);
  const float *col = tile + 3 * st_z + (w + 3) * st_y + 2 * lx + 4;  // cell (i, j) of the first plane
  auto ld2 = [](const float *p) { return *reinterpret_cast<const float2 *>(p); };
  const float2 ix = sp(a.inv[0]), iy = sp(a.inv[1]), iz = sp(a.inv[2]);
  auto diff = [](float2 lo, float2 hi) { return fma2(sp(-1.f), lo, hi); };
  // the upwind value from the differences (spatial_derivatives3d.f.in:2756-2812):
  // D1(c-2 .. c+2) for v > 0, D1(c+3 .. c-1) otherwise, 0 where |v| < zero_tol
  auto upwind = [](const float2 D[6], float2 vel) {
    const bool b0 = vel.x > 0.f, b1 = vel.y > 0.f;
    float2 v[5];
#pragma unroll
    for (int q = 0; q < 5; q++) v[q] = make_float2(b0 ? D[q].x : D[5 - q].x, b1 ? D[q].y : D[5 - q].y);
    float2 g = weno5_x2(v[0], v[1], v[2], v[3], v[4]);
    if (fabsf(vel.x) < 1e-11f) g.x = 0.f;
    if (fabsf(vel.y) < 1e-11f) g.y = 0.f;
    return g;
  };

  // z march: D1(z0-2 .. z0+2) and the scaled phi(z0+2)
  float2 Dz[6], zl;
  {
    float2 p[6];
#pragma unroll
    for (int q = 0; q < 6; q++) p[q] = mul2(ld2(col + (q - 3) * st_z), iz);
#pragma unroll
    for (int q = 0; q < 5; q++) Dz[q + 1] = diff(p[q], p[q + 1]);
    zl = p[5];
  }
  const float *un_src = a.stage == 1 ? nullptr : a.phi_n;
  long long cell = L.idx(i, j, z0);
  float2 vn[3], un_next = un_src ? ld2(un_src + cell) : sp(0.f);
#pragma unroll
  for (int d = 0; d < 3; d++) vn[d] = ld2(a.vel[d] + cell);
#pragma unroll UNROLL
  for (int tz = 0; tz < kmax; tz++) {
    const float2 vx = vn[0], vy = vn[1], vz = vn[2], un = un_next;
    if (tz + 1 < kmax) {
#pragma unroll
      for (int d = 0; d < 3; d++) vn[d] = ld2(a.vel[d] + cell + L.pz);
      if (un_src) un_next = ld2(un_src + cell + L.pz);
    }
    const float2 u0 = ld2(col);  // phi(i), phi(i+1)
    float2 dot = sp(0.f), D[6];
    {
      const float2 e0 = mul2(ld2(col - 4), ix), e1 = mul2(ld2(col - 2), ix), e2 = mul2(u0, ix);
      const float2 e3 = mul2(ld2(col + 2), ix), e4 = mul2(ld2(col + 4), ix);
      // (phi(s), phi(s+1)) for s = i-3, i-1, i+1, i+3
      const float2 o0 = make_float2(e0.y, e1.x), o1 = make_float2(e1.y, e2.x), o2 = make_float2(e2.y, e3.x);
      const float2 o3 = make_float2(e3.y, e4.x);
      D[0] = diff(o0, e1); D[1] = diff(e1, o1); D[2] = diff(o1, e2);
      D[3] = diff(e2, o2); D[4] = diff(o2, e3); D[5] = diff(e3, o3);
      dot = fma2(vx, upwind(D, vx), dot);
    }
    {
      float2 p[7];
#pragma unroll
      for (int q = 0; q < 7; q++) p[q] = mul2(q == 3 ? u0 : ld2(col + (q - 3) * st_y), iy);
#pragma unroll
      for (int q = 0; q < 6; q++) D[q] = diff(p[q], p[q + 1]);
      dot = fma2(vy, upwind(D, vy), dot);
    }
    {
      const float2 p = mul2(ld2(col + 3 * st_z), iz);
#pragma unroll
      for (int q = 0; q < 5; q++) Dz[q] = Dz[q + 1];
      Dz[5] = diff(zl, p);
      zl = p;
      dot = fma2(vz, upwind(Dz, vz), dot);
    }
    const float2 rhs = make_float2(-dot.x, -dot.y);
    float2 u = fma2(sp(a.dt), rhs, u0);  // tvd_runge_kutta3d.f:78
    if (a.stage == 2) u = fma2(sp(0.75f), un, mul2(sp(0.25f), u));                  // :403-404
    else if (a.stage == 3) u = fma2(sp(1.f / 3.f), un, mul2(sp(2.f / 3.f), u));  // :490-492
    store_pair(a.out, L, cell, u, two, px0, px1, py, a.periodic ? image_of(z0 + tz, L.nz) : 0);
    col += st_z;
    cell += L.pz;
  }
}

// the stage kernel of a single grid: tiles of W x ROWS x tzn cells
constexpr int kAdvThreads = 256;
template <int W, bool FIELD>
static __global__ void __launch_bounds__(kAdvThreads, FIELD ? 4 : 3)
    k_adv_x2(const __grid_constant__ CUtensorMap tm, StageArgs<float> a, int tzn) {
  using Q = AdvTile<W, kAdvThreads>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float *tile = reinterpret_cast<float *>(smem_raw);
  __shared__ __align__(8) uint64_t bar;
  __shared__ float xedge[FIELD ? 1 : 5 * RZ_MAX * Q::ROWS];
  const int tid = threadIdx.x + 32 * threadIdx.y;
  const int x0 = blockIdx.x * W, y0 = blockIdx.y * Q::ROWS, z0 = blockIdx.z * tzn;
  if (tid == 0) {
    prefetch_tmap(&tm);
    mbar_init(&bar, 1);
    fence_barrier_init();
  }
  __syncthreads();
  if (tid == 0) {
    mbar_arrive_expect_tx(&bar, (uint32_t)Q::smem(tzn));
    tma_load_3d(tile, &tm, x0 + GX - 4, y0 + GY - 3, z0 + GZ - 3, &bar);
  }
  if (!mbar_wait(&bar, 0, kMaxPolls)) {
    if (tid == 0) atomicExch(a.err, LSMGPU_ERR_TIMEOUT);
    mbar_wait(&bar, 0, kMaxPolls);  // let an in-flight copy land before exit
    return;
  }
  if (a.ghost) {
    fill_face_ghosts<float, W, Q::ROWS>(tile, tzn, x0, y0, z0, a.L, a.ghost, tid);
    __syncthreads();
  }
  if constexpr (FIELD) adv_field_tile<W, kAdvThreads, 2>(tile, a, x0, y0, z0, tzn, tid);
  else adv_tile<W, kAdvThreads, RZ_MAX, 2>(tile, xedge, a, x0, y0, z0, tzn, tid);
}

// the instance for a row length
using StageX2 = void (*)(const CUtensorMap, StageArgs<float>, int);
template <bool FIELD>
inline StageX2 adv_x2_kernel(int w) {
  return w == 64 ? k_adv_x2<64, FIELD> : (w == 32 ? k_adv_x2<32, FIELD> : k_adv_x2<16, FIELD>);
}

}  // namespace fused
}  // namespace lsmgpu
