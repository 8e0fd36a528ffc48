// Batched WENO5 / TVD-RK3 advection of many independent, unevenly sized grids.
//
// All grids live in one set of work buffers (the padded layout of the fused
// steppers, one region per grid).  Each RK stage is ONE launch over the tiles
// of all grids, so small and large grids share the machine; a table of (grid,
// tile position) per CTA, built on the host, replaces any search or division
// in the kernel, and the tiles come by TMA through per-grid tensor maps kept
// in global memory.  The n_steps x 3 stage launches of a call are one CUDA
// graph, kept for later calls with the same buffers and launch parameters.
//
// A tile is adv_tile (adv_x2.cuh) on 128 threads: 32 x 8 or 16 x 16 cells of a
// plane, whichever covers fewer cells of the grid's, and up to kDepth planes,
// the grid's planes split evenly.  Six CTAs per SM hide one another's loads
// (memory is at 27%: the arithmetic bounds it, as in adv_x2.cuh); the plane
// loop is unrolled by two, since the bodies of CTAs in flight share the
// instruction cache.  512 grids of 16 to 96 cells a side, 10 steps, whole call
// in ms: cell-by-cell tiles on persistent, autotuned CTAs 27.6; this 19.5; five
// CTAs 20.5; unrolled by 1 / 4 / 8 planes 20.4 / 21.1 / 25.1; 6- / 10-plane
// tiles 23.4 / 20.0 (the latter with five CTAs).
// The table lists the grids by tile shape, so that the CTAs in flight mostly
// run one of the kernel's two bodies.
//
// For comparison the same batch can run as a loop of single-grid launches
// (one stage kernel per grid per stage), which is what calling the
// single-grid stepper grid by grid amounts to.
#include <algorithm>
#include <vector>

#include "adv_x2.cuh"
#include "lsmgpu_common.cuh"
#include "../../include/lsmgpu.h"

namespace lsmgpu {
namespace batch {

using fused::AdvTile;
using fused::GX;
using fused::GY;
using fused::GZ;
using fused::Layout;
using fused::StageArgs;

struct GridDesc {
  Layout L;
  long long off;  // element offset of this grid's region in each work buffer
  float vconst[3], inv[3], floor4[3], dt;  // |velocity|
  float scale;    // of phi in the work layout (spacing_scale)
  int flip;       // axes of negative velocity: mirrored in the work layout
  int wide;       // 1: 32 x 8 tiles, 0: 16 x 16 tiles
  int tz;         // tile depth, even
  int ntx, nty, ntz;
};

constexpr int kThreads = 128;
constexpr int kDepth = 8;  // planes of the deepest tile
using Wide = AdvTile<32, kThreads>;
using Narrow = AdvTile<16, kThreads>;
// the launch loop's tiles, of the single-grid kernel
constexpr int kLoopW = 32, kLoopRows = AdvTile<kLoopW, fused::kAdvThreads>::ROWS;
constexpr int kRowsMax = Narrow::ROWS;
constexpr size_t kSmem = Wide::smem(kDepth) > Narrow::smem(kDepth) ? Wide::smem(kDepth) : Narrow::smem(kDepth);

// one tile: its grid, position (tiles per axis < 2^16 per grid), shape and depth
struct TileRef {
  int g;
  unsigned short bx, by, bz;
  unsigned char wide, tz;
};

__global__ void __launch_bounds__(kThreads, 6) k_batch_stage(const GridDesc *__restrict__ gd,
                                                             const CUtensorMap *__restrict__ tmaps,
                                                             const TileRef *__restrict__ tiles, int stage, float *A,
                                                             float *B, float *C, int *err) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float *const tile = reinterpret_cast<float *>(smem_raw);
  __shared__ __align__(8) uint64_t bar;
  __shared__ float xedge[5 * kDepth * kRowsMax];
  const int tid = threadIdx.x;
  const TileRef r = tiles[blockIdx.x];
  const int tw = r.wide ? 32 : 16, th = r.wide ? Wide::ROWS : Narrow::ROWS;
  const int x0 = r.bx * tw, y0 = r.by * th, z0 = r.bz * r.tz;
  if (tid == 0) {
    mbar_init(&bar, 1);
    fence_barrier_init();
    const CUtensorMap *m = tmaps + 3 * r.g + (stage - 1);  // of A, B, C
    // the maps live in global memory and are rewritten between calls
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"((uint64_t)m) : "memory");
    mbar_arrive_expect_tx(&bar, (uint32_t)(r.wide ? Wide::smem(r.tz) : Narrow::smem(r.tz)));
    tma_load_3d(tile, m, x0 + GX - 4, y0 + GY - 3, z0 + GZ - 3, &bar);
  }
  const GridDesc &G = gd[r.g];
  StageArgs<float> a{};
  a.L = G.L;
  a.phi_n = A + G.off;
  a.out = (stage == 1 ? B : (stage == 2 ? C : A)) + G.off;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    a.vconst[d] = G.vconst[d];
    a.inv[d] = G.inv[d];
    a.floor4[d] = G.floor4[d];
  }
  a.dt = G.dt;
  a.stage = stage;
  a.periodic = 1;
  __syncthreads();  // the barrier is initialised
  if (!mbar_wait(&bar, 0, fused::kMaxPolls)) {
    if (tid == 0) atomicExch(err, LSMGPU_ERR_TIMEOUT);
    mbar_wait(&bar, 0, fused::kMaxPolls);  // let an in-flight copy land before exit
    return;
  }
  if (r.wide) fused::adv_tile<32, kThreads, kDepth, 2>(tile, xedge, a, x0, y0, z0, r.tz, tid);
  else fused::adv_tile<16, kThreads, kDepth, 2>(tile, xedge, a, x0, y0, z0, r.tz, tid);
}

// copies between the caller's packed LSMLIB arrays (3 ghost cells per side)
// and the padded work regions, phi scaled and divided out again (a power of
// two); blockIdx.y is the grid, a warp takes x rows (an index division per row,
// not per cell)
__global__ void __launch_bounds__(256) k_batch_pack(float *work, float *user, const GridDesc *gd,
                                                    const long long *uoff, int unpack) {
  const GridDesc &G = gd[blockIdx.y];
  const Layout L = G.L;
  const int ux = L.nx + 6, uy = L.ny + 6;
  const long long rows = (long long)uy * (L.nz + 6);
  const float scale = unpack ? fused::pow2_recip(G.scale) : G.scale;
  float *const w0 = work + G.off;
  float *const u0 = user + uoff[blockIdx.y];
  for (long long r = blockIdx.x * 8 + threadIdx.x / 32; r < rows; r += gridDim.x * 8) {
    const int k = (int)(r / uy), j = (int)(r - (long long)k * uy);
    const int wj = G.flip & 2 ? uy - 1 - j : j, wk = G.flip & 4 ? L.nz + 5 - k : k;
    float *const w = w0 + L.idx(G.flip & 1 ? L.nx + 2 : -3, wj - 3, wk - 3);
    const int step = G.flip & 1 ? -1 : 1;
    float *const u = u0 + r * ux;
    if (unpack) {
      for (int i = threadIdx.x % 32; i < ux; i += 32) u[i] = w[step * i] * scale;
    } else {
      for (int i = threadIdx.x % 32; i < ux; i += 32) w[step * i] = u[i] * scale;
    }
  }
}

}  // namespace batch
}  // namespace lsmgpu

using namespace lsmgpu;
using namespace lsmgpu::batch;

extern "C" int lsmgpu_advect_batch_weno5_tvdrk3_f32(float *phi, const long long *offsets, const int *dims,
                                                   int n_grids, const float *vel, const float *spacing,
                                                   const float *dt, int n_steps, int bc, int flags) {
  const char *name = "lsmgpu_advect_batch_weno5_tvdrk3_f32";
  Call call(name);
  if (!phi || !offsets || !dims || !vel || !spacing || !dt || n_grids <= 0) {
    set_error(LSMGPU_ERR_ARGUMENT, "%s: null argument or no grids", name);
    return LSMGPU_ERR_ARGUMENT;
  }
  if (bc != LSMGPU_BC_PERIODIC) {
    set_error(LSMGPU_ERR_ARGUMENT, "%s: only periodic boundaries are supported for batches", name);
    return LSMGPU_ERR_ARGUMENT;
  }
  std::vector<GridDesc> desc(n_grids);
  long long user_total = 0;
  std::vector<long long> uoff(n_grids);
  for (int g = 0; g < n_grids; g++) {
    const int nx = dims[3 * g], ny = dims[3 * g + 1], nz = dims[3 * g + 2];
    if (nx < 6 || ny < 6 || nz < 6) {
      set_error(LSMGPU_ERR_BOUNDS, "%s: grid %d is smaller than 6 cells on an axis", name, g);
      return LSMGPU_ERR_BOUNDS;
    }
    // tile positions are 16-bit (16-cell tiles at the finest)
    if (nx > 65535 * 16 || ny > 65535 * 8 || nz > 65535 * 4) {
      set_error(LSMGPU_ERR_BOUNDS, "%s: grid %d has more than 65535 tiles along an axis", name, g);
      return LSMGPU_ERR_BOUNDS;
    }
    desc[g].scale = fused::spacing_scale(spacing + 3 * g);
    uoff[g] = offsets[g];
    user_total = std::max(user_total, offsets[g] + (long long)(nx + 6) * (ny + 6) * (nz + 6));
  }
  const int want_loop = flags & LSMGPU_BATCH_LOOP;
  const int use_graph = !(flags & LSMGPU_BATCH_NO_GRAPH);
  const int forced_tz = (flags >> 8) & 0xff;  // 0: by the batch

  float *user = call.inout(phi, user_total);
  long long *uoff_d = call.temp<long long>(n_grids);
  if (!call.ok()) return lsmgpu_get_last_error(nullptr, 0);
  cudaStream_t s = stream();

  int nsm = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);

  // layouts and tiles of `depth` planes at most (the scales are there)
  long long total = 0, ntiles = 0;
  auto build_desc = [&](int depth) {
    total = ntiles = 0;
    for (int g = 0; g < n_grids; g++) {
      GridDesc &G = desc[g];
      G.L = fused::make_layout(dims[3 * g], dims[3 * g + 1], dims[3 * g + 2]);
      G.off = total;
      total += (G.L.elems() + 31) / 32 * 32;
      for (int d = 0; d < 3; d++) {
        G.vconst[d] = vel[3 * g + d] < 0.f ? -vel[3 * g + d] : vel[3 * g + d];
        G.inv[d] = 1.0f / spacing[3 * g + d];
        G.floor4[d] = fused::eps_floor4((double)spacing[3 * g + d] * G.scale);
      }
      G.dt = dt[g];
      G.flip = fused::mirrored_axes(vel + 3 * g);
      auto cover = [&](int w, int h) { return (long long)((G.L.nx + w - 1) / w) * ((G.L.ny + h - 1) / h); };
      // (the launch loop runs the single-grid kernel's 32 x 16 tiles)
      G.wide = want_loop || cover(32, Wide::ROWS) <= cover(16, Narrow::ROWS) ? 1 : 0;
      const int tw = G.wide ? 32 : 16, th = want_loop ? kLoopRows : (G.wide ? Wide::ROWS : Narrow::ROWS);
      const int deep = G.L.nz > 65535 * depth ? kDepth : depth;  // tile positions are 16-bit
      G.ntz = (G.L.nz + deep - 1) / deep;
      G.tz = ((G.L.nz + G.ntz - 1) / G.ntz + 1) / 2 * 2;
      G.ntz = (G.L.nz + G.tz - 1) / G.tz;
      G.ntx = (G.L.nx + tw - 1) / tw;
      G.nty = (G.L.ny + th - 1) / th;
      ntiles += (long long)G.ntx * G.nty * G.ntz;
    }
  };
  if (forced_tz) {
    build_desc(std::min(std::max(forced_tz / 2 * 2, 2), kDepth));
  } else {
    // shallower tiles where deep ones leave SMs idle (8 grids of 16 to 30
    // cells, 10 steps: 229 us; thresholds of one and four tiles per SM 219
    // and 234, within the noise)
    for (int depth = kDepth; depth >= 2; depth /= 2) {
      build_desc(depth);
      if (ntiles >= 2 * nsm) break;
    }
  }
  if (ntiles > 0x7fffffffLL) {
    set_error(LSMGPU_ERR_CAPACITY, "%s: more than 2^31 tiles", name);
    return LSMGPU_ERR_CAPACITY;
  }
  std::vector<TileRef> tref;
  if (!want_loop) {
    tref.reserve((size_t)ntiles);
    for (int wide = 0; wide < 2; wide++)
      for (int g = 0; g < n_grids; g++) {
        const GridDesc &G = desc[g];
        if (G.wide != wide) continue;
        for (int bz = 0; bz < G.ntz; bz++)
          for (int by = 0; by < G.nty; by++)
            for (int bx = 0; bx < G.ntx; bx++)
              tref.push_back(TileRef{g, (unsigned short)bx, (unsigned short)by, (unsigned short)bz,
                                     (unsigned char)G.wide, (unsigned char)G.tz});
      }
  }
  float *A = call.temp<float>(total), *B = call.temp<float>(total), *C = call.temp<float>(total);
  GridDesc *gd = call.temp<GridDesc>(n_grids);
  TileRef *trd = call.temp<TileRef>(std::max(ntiles, 1LL));
  CUtensorMap *tm = (CUtensorMap *)call.temp<unsigned char>((long long)sizeof(CUtensorMap) * 3 * n_grids);
  int *err = call.temp<int>(1);
  if (!call.ok()) return lsmgpu_get_last_error(nullptr, 0);
  cudaMemcpyAsync(uoff_d, uoff.data(), sizeof(long long) * n_grids, cudaMemcpyHostToDevice, s);
  cudaMemsetAsync(err, 0, sizeof(int), s);
  // B and C need no initial values: a stage writes every interior cell of its
  // output and the periodic images that the next stage reads

  std::vector<CUtensorMap> tmh(3 * (size_t)n_grids);
  {
    float *bufs[3] = {A, B, C};
    for (int g = 0; g < n_grids; g++) {
      const GridDesc &G = desc[g];
      const int sx = want_loop ? kLoopW + 8 : (G.wide ? Wide::SXW : Narrow::SXW);
      const int sy = want_loop ? kLoopRows + 6 : (G.wide ? Wide::SYW : Narrow::SYW);
      for (int q = 0; q < 3; q++)
        if (!encode_tmap_3d(&tmh[3 * g + q], bufs[q] + G.off, 4, (long long)G.L.nx + GX + 3, (long long)G.L.ny + 2 * GY,
                            (long long)G.L.nz + 2 * GZ, G.L.py, G.L.pz, sx, sy, G.tz + 6)) {
          call.fail("tensor map encoding failed");
          return LSMGPU_ERR_CUDA;
        }
    }
  }
  cudaMemcpyAsync(gd, desc.data(), sizeof(GridDesc) * n_grids, cudaMemcpyHostToDevice, s);
  {
    dim3 grd(64, n_grids);
    LSMGPU_LAUNCH(k_batch_pack, grd, 256, 0, A, user, gd, uoff_d, 0);
  }

  if (want_loop) {
    // comparison mode: one single-grid stage launch per grid per stage
    const auto kern = fused::adv_x2_kernel<false>(kLoopW);
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)AdvTile<kLoopW, fused::kAdvThreads>::smem(kDepth));
    for (int step = 0; step < n_steps; step++)
      for (int stage = 1; stage <= 3; stage++)
        for (int g = 0; g < n_grids; g++) {
          const GridDesc &G = desc[g];
          StageArgs<float> a{};
          a.L = G.L;
          a.phi_n = A + G.off;
          a.out = (stage == 1 ? B : (stage == 2 ? C : A)) + G.off;
          for (int d = 0; d < 3; d++) { a.vconst[d] = G.vconst[d]; a.inv[d] = G.inv[d]; a.floor4[d] = G.floor4[d]; }
          a.dt = G.dt;
          a.stage = stage;
          a.periodic = 1;
          a.err = err;
          kern<<<dim3(G.ntx, G.nty, G.ntz), dim3(32, 8), AdvTile<kLoopW, fused::kAdvThreads>::smem(G.tz), s>>>(
              tmh[3 * g + stage - 1], a, G.tz);
          note_launch();
        }
  } else {
    cudaMemcpyAsync(tm, tmh.data(), sizeof(CUtensorMap) * tmh.size(), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(trd, tref.data(), sizeof(TileRef) * tref.size(), cudaMemcpyHostToDevice, s);
    cudaFuncSetAttribute(k_batch_stage, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    // all stages of the call, replayed as one CUDA graph when the same buffers
    // and launch parameters come again (the grids' sizes, velocities and
    // tensor maps are read from device memory)
    auto stages = [&]() {
      for (int step = 0; step < n_steps; step++)
        for (int stage = 1; stage <= 3; stage++)
          LSMGPU_LAUNCH(k_batch_stage, (unsigned)ntiles, kThreads, kSmem, gd, tm, trd, stage, A, B, C, err);
    };
    if (n_steps > 0) {
      GraphKey gk;
      gk.add((int)0x62617463);  // this call's kind among the cached graphs
      gk.add(n_steps); gk.add(ntiles);
      gk.add(gd); gk.add(tm); gk.add(trd); gk.add(A); gk.add(B); gk.add(C); gk.add(err);
      if (!use_graph || !graph_replay(gk, stages)) stages();
    }
  }
  {
    dim3 grd(64, n_grids);
    LSMGPU_LAUNCH(k_batch_pack, grd, 256, 0, A, user, gd, uoff_d, 1);
  }
  int herr = 0;
  cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s);
  call.finish();
  cudaStreamSynchronize(s);
  if (herr) {
    set_error(herr, "%s: a bounded device wait gave up (TMA tile load)", name);
    return herr;
  }
  return lsmgpu_get_last_error(nullptr, 0);
}
