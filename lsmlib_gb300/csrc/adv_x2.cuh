// FP32 constant-velocity advection stage on the x cell pairs and the z march
// of reinit_x2.cuh.
//
// The velocity's sign is the same for every cell, so of each window only one
// side is needed: minus(c) of W(c) where the component is positive, plus(c) of
// W(c+1) where it is negative.  The kernel is instantiated for the eight sign
// triples (OX, OY, OZ: 1 where the component is negative, the window's offset
// from the cell).  With one window per cell and axis there is nothing to hand
// between rows, so the plane loop has no barrier:
//  * z: the thread marches up its column and carries the last two triples'
//    forms (one new triple per cell);
//  * x: a thread owns two x-neighbouring cells as the lanes of the packed
//    instructions and takes the forms of the two triples before its own from
//    the previous lane (the first lane from a per-tile prologue);
//  * y: the row's three triples, evaluated in place.
// Bound by FMA issue: about 130 packed operations per cell pair, where the
// cell-by-cell tile (adv tile of fused_stage.cuh) takes 165 and as many again
// in loads, selection and per-tile set-up.  The arithmetic is that tile's
// (minus_of_window, and its mirror image for the plus side), operation for
// operation, so both give the same bits.  Measured per stage, periodic, with
// this kernel and before it: 37 x 33 x 41 5.3 and 5.8 us, 128^3 18.3 and 23.0,
// 256^3 98.6 and 143.
#pragma once

#include "reinit_x2.cuh"

namespace lsmgpu {
namespace fused {

// 2 minus(c) (PLUS = 0) or 2 plus(c-1) (PLUS = 1) of window W(c): its weight
// products, TD(c-2), -TD(c-1), t(c-1) and D(c-1), D(c), D(c+1)
template <int PLUS>
__device__ __forceinline__ float2 one_side(const WQ &w, float2 a, float2 nb, float2 t, float2 dm, float2 d0,
                                           float2 dp) {
  if constexpr (PLUS == 0) {
    return side_minus(w, a, nb, fma2(sp(-1.f / 3.f), t, add2(d0, dp)));
  } else {
    const float2 num = fma2(sp(-1.5f), mul2(w.q23, a), mul2(w.q12, nb));
    const float2 den = fma2(sp(1.5f), w.q12, fma2(sp(4.5f), w.q23, mul2(sp(9.f), w.q13)));
    return fma2(num, rcp2(den), fma2(sp(-1.f / 3.f), t, add2(dm, d0)));
  }
}

template <int OX, int OY, int OZ>
static __global__ void __launch_bounds__(256, 3)
    k_adv_x2(const __grid_constant__ CUtensorMap tm, StageArgs<float> a, int tzn) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float *tile = reinterpret_cast<float *>(smem_raw);
  __shared__ __align__(8) uint64_t bar;
  // per (plane, row): s1 and t of triple x0-2+OX, s1, s2 and t of x0-1+OX
  __shared__ float xedge[5][RZ_MAX][RY];
  const int lane = threadIdx.x, w = threadIdx.y;
  const int tid = lane + 32 * w;
  const int x0 = blockIdx.x * RX, y0 = blockIdx.y * RY, z0 = blockIdx.z * tzn;
  const Layout &L = a.L;

  if (tid == 0) {
    prefetch_tmap(&tm);
    mbar_init(&bar, 1);
    fence_barrier_init();
  }
  __syncthreads();
  if (tid == 0) {
    mbar_arrive_expect_tx(&bar, (uint32_t)reinit_x2_smem(tzn));
    tma_load_3d(tile, &tm, x0 + GX - 4, y0 + GY - 3, z0 + GZ - 3, &bar);
  }
  if (!mbar_wait(&bar, 0, kMaxPolls)) {
    if (tid == 0) atomicExch(a.err, LSMGPU_ERR_TIMEOUT);
    mbar_wait(&bar, 0, kMaxPolls);  // let an in-flight copy land before exit
    return;
  }
  if (a.ghost) {
    fill_face_ghosts<float>(tile, RSX, RSY, tzn + 6, x0 - 4, y0 - 3, z0 - 3, L, a.ghost);
    __syncthreads();
  }

  const int st_y = RSX, st_z = RSX * RSY;
  // ---- prologue: the forms before the tile's first cell, two planes a thread --
  if (tid < RY * tzn / 2) {
    const int pw = tid % RY, pz = 2 * (tid / RY);
    const float *r0 = tile + ((pz + 3) * RSY + pw + 3) * RSX, *r1 = r0 + st_z;
    float2 p[5], D[4];  // phi(x0-3+OX ..), D(x0-2+OX ..)
#pragma unroll
    for (int q = 0; q < 5; q++) p[q] = make_float2(r0[q + 1 + OX], r1[q + 1 + OX]);
#pragma unroll
    for (int q = 0; q < 4; q++) D[q] = sub2(p[q + 1], p[q]);
    const Tri t2 = tri_forms(D[0], D[1], D[2]), t1 = tri_forms(D[1], D[2], D[3]);
    const float2 v[5] = {t2.s1, t2.t, t1.s1, t1.s2, t1.t};
#pragma unroll
    for (int q = 0; q < 5; q++) {
      xedge[q][pz][pw] = v[q].x;
      xedge[q][pz + 1][pw] = v[q].y;
    }
  }
  __syncthreads();

  // Rows and lanes outside the grid compute on tile padding and store nothing
  // (whole warps of such rows leave).
  const int i = x0 + 2 * lane, j = y0 + w;
  if (j >= L.ny) return;
  const bool two = i + 1 < L.nx;
  const bool live = i < L.nx;
  // offsets of the periodic images of the pair's cells along x and y
  const int px0 = a.periodic ? image_of(i, L.nx) : 0, px1 = a.periodic && two ? image_of(i + 1, L.nx) : 0;
  const int py = a.periodic ? image_of(j, L.ny) : 0;
  const int kmax = min(tzn, L.nz - z0);
  const float *col = tile + (w + 3) * st_y + 2 * lane + 4;  // (i, j) column, plane index sz
  auto ld2 = [&](int sz, int dx, int dy) {
    return *reinterpret_cast<const float2 *>(col + sz * st_z + dy * st_y + dx);
  };
  // |v| / (2 dx) per axis; 0 where |v| is below the reference's zero tolerance
  float wv[3];
#pragma unroll
  for (int d = 0; d < 3; d++) wv[d] = fabsf(a.vconst[d]) < 1e-11f ? 0.f : 0.5f * fabsf(a.vconst[d]) * a.inv[d];
  // the backward value of the line walked with the velocity's sign: -plus
  auto add_axis = [&](float2 dot, int d, int neg, float2 g) {
    const float2 r = fma2(sp(neg ? -wv[d] : wv[d]), g, dot);
    return wv[d] != 0.f ? r : dot;
  };

  // ---- z march: the carried state for the window of cell z0, c = z0 + OZ ------
  float2 fl, dm, d0, d1, s1a, s1b, s2b, ta, tb, pm2, pm1, sq0, sq1;
  {
    float2 p[5], D[4], sq[4];  // phi(c-3 .. c+1), D(c-2 .. c+1)
#pragma unroll
    for (int q = 0; q < 5; q++) p[q] = ld2(q + OZ, 0, 0);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      D[q] = sub2(p[q + 1], p[q]);
      sq[q] = mul2(D[q], D[q]);
    }
    const Tri t2 = tri_forms(D[0], D[1], D[2]), t1 = tri_forms(D[1], D[2], D[3]);
    fl = p[4];
    dm = D[1];
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
  const long long cell0 = L.idx(live ? i : 0, j, z0);
  float2 un_next = un_src ? *reinterpret_cast<const float2 *>(un_src + cell0) : sp(0.f);

  // (unrolled: the carried quantities change names instead of registers; 256^3,
  // 2 planes per pass 100.6 us per stage, 8 planes 98.6, 10 with two CTAs per SM
  // 105.4)
#pragma unroll 8
  for (int tz = 0; tz < kmax; tz++) {
    const int k = z0 + tz;
    const int sz = tz + 3;
    const long long cell = cell0 + (long long)tz * L.pz;
    const float2 un = un_next;  // read one plane ahead of its use
    if (tz + 1 < kmax && un_src) un_next = *reinterpret_cast<const float2 *>(un_src + cell + L.pz);
    const float2 u0 = ld2(sz, 0, 0);  // phi(i), phi(i+1)
    float2 gx, gy, gz;
    // ---- x: windows W(c), W(c+1), c = i + OX ------------------------------------
    {
      // P_s = (D(s), D(s+1)) for s = c-2 .. c+2
      float2 P0, P1, P2, P3, P4;
      if constexpr (OX == 1) {
        const float2 e0 = ld2(sz, -2, 0), e2 = ld2(sz, 2, 0), e3 = ld2(sz, 4, 0);
        const float2 o0 = make_float2(e0.y, u0.x), o1 = make_float2(u0.y, e2.x), o2 = make_float2(e2.y, e3.x);
        P0 = sub2(o0, e0); P1 = sub2(u0, o0); P2 = sub2(o1, u0); P3 = sub2(e2, o1); P4 = sub2(o2, e2);
      } else {
        const float2 e0 = ld2(sz, -4, 0), e1 = ld2(sz, -2, 0), e3 = ld2(sz, 2, 0);
        const float2 o0 = make_float2(e0.y, e1.x), o1 = make_float2(e1.y, u0.x), o2 = make_float2(u0.y, e3.x);
        P0 = sub2(e1, o0); P1 = sub2(o1, e1); P2 = sub2(u0, o1); P3 = sub2(o2, u0); P4 = sub2(e3, o2);
      }
      const Tri C = tri_forms(P2, P3, P4);  // (tri(c), tri(c+1))
      // (tri(c-2), tri(c-1)) are the previous lane's C
      float a_s1x = __shfl_up_sync(0xffffffffu, C.s1.x, 1), a_s1y = __shfl_up_sync(0xffffffffu, C.s1.y, 1);
      float a_s2y = __shfl_up_sync(0xffffffffu, C.s2.y, 1);
      float a_tx = __shfl_up_sync(0xffffffffu, C.t.x, 1), a_ty = __shfl_up_sync(0xffffffffu, C.t.y, 1);
      if (lane == 0) {
        a_s1x = xedge[0][tz][w];
        a_tx = xedge[1][tz][w];
        a_s1y = xedge[2][tz][w];
        a_s2y = xedge[3][tz][w];
        a_ty = xedge[4][tz][w];
      }
      const float2 At = make_float2(a_tx, a_ty), Bt = make_float2(a_ty, C.t.x);
      const float2 q0 = mul2(P0, P0), q2 = mul2(P2, P2), q4 = mul2(P4, P4);  // sq(c-2 .. c+3)
      const float inner = fmaxf(max3f(q0.y, q2.x, q2.y), q4.x);
      const float2 m = make_float2(fmaxf(inner, q0.x), fmaxf(inner, q4.y));
      const WQ wq = window_q(make_float2(a_s1x, a_s1y), make_float2(a_s2y, C.s2.x), C.s3, m, a.floor4[0]);
      gx = one_side<OX>(wq, sub2(At, Bt), sub2(C.t, Bt), Bt, P1, P2, P3);
    }
    // ---- y: window W(c), c = j + OY ---------------------------------------------
    {
      float2 r[6], D[5];  // phi(c-3 .. c+2)
#pragma unroll
      for (int q = 0; q < 6; q++) r[q] = (q + OY == 3) ? u0 : ld2(sz, 0, q - 3 + OY);
#pragma unroll
      for (int q = 0; q < 5; q++) D[q] = sub2(r[q + 1], r[q]);
      const Tri t2 = tri_forms(D[0], D[1], D[2]), t1 = tri_forms(D[1], D[2], D[3]), t0 = tri_forms(D[2], D[3], D[4]);
      float2 sq[5];
#pragma unroll
      for (int q = 0; q < 5; q++) sq[q] = mul2(D[q], D[q]);
      const WQ wq = window_q(t2.s1, t1.s2, t0.s3, max5(sq[0], sq[1], sq[2], sq[3], sq[4]), a.floor4[1]);
      gy = one_side<OY>(wq, sub2(t2.t, t1.t), sub2(t0.t, t1.t), t1.t, D[1], D[2], D[3]);
    }
    // ---- z: window W(c), c = k + OZ ----------------------------------------------
    {
      const float2 f = ld2(sz + 2 + OZ, 0, 0);  // phi(c+2)
      const float2 d2 = sub2(f, fl);
      const float2 sq2 = mul2(d2, d2);
      const Tri n = tri_forms(d0, d1, d2);  // tri(c)
      const float2 pmn = make_float2(fmaxf(sq0.x, sq1.x), fmaxf(sq0.y, sq1.y));
      const float2 m = make_float2(max3f(pm2.x, pmn.x, sq2.x), max3f(pm2.y, pmn.y, sq2.y));
      const WQ wq = window_q(s1a, s2b, n.s3, m, a.floor4[2]);
      gz = one_side<OZ>(wq, sub2(ta, tb), sub2(n.t, tb), tb, dm, d0, d1);
      fl = f;
      dm = d0;
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
    const float2 dot = add_axis(add_axis(add_axis(sp(0.f), 0, OX, gx), 1, OY, gy), 2, OZ, gz);
    const float2 rhs = make_float2(-dot.x, -dot.y);
    float2 u = fma2(sp(a.dt), rhs, u0);  // tvd_runge_kutta3d.f:78
    if (a.stage == 2) u = fma2(sp(0.75f), un, mul2(sp(0.25f), u));                  // :403-404
    else if (a.stage == 3) u = fma2(sp(1.f / 3.f), un, mul2(sp(2.f / 3.f), u));  // :490-492
    if (live) store_pair(a.out, L, cell, u, two, px0, px1, py, a.periodic ? image_of(k, L.nz) : 0);
  }
}

// the instance for a velocity's signs
using StageX2 = void (*)(const CUtensorMap, StageArgs<float>, int);
inline StageX2 adv_x2_kernel(const float v[3]) {
  static const StageX2 k[8] = {k_adv_x2<0, 0, 0>, k_adv_x2<1, 0, 0>, k_adv_x2<0, 1, 0>, k_adv_x2<1, 1, 0>,
                             k_adv_x2<0, 0, 1>, k_adv_x2<1, 0, 1>, k_adv_x2<0, 1, 1>, k_adv_x2<1, 1, 1>};
  return k[(v[0] < 0.f ? 1 : 0) | (v[1] < 0.f ? 2 : 0) | (v[2] < 0.f ? 4 : 0)];
}

}  // namespace fused
}  // namespace lsmgpu
