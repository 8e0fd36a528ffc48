// FP32 form of the fused steppers (FMA contraction, fast reciprocals).
#define LSMGPU_FUSED_R float
#define LSMGPU_FUSED_EXACT false
#define LSMGPU_FUSED_SUFFIX f32
#include "fused_entry.cuh"

extern "C" int lsmgpu_stage_tile_f32(int mode, int nx, int ny, int nz, int *tile) {
  using namespace lsmgpu::fused;
  if (!tile || nx < 1 || ny < 1 || nz < 1 || mode < ADV_CONST || mode > REINIT) return LSMGPU_ERR_ARGUMENT;
  const Layout L = make_layout(nx, ny, nz);
  const TileX2 t = mode == REINIT ? reinit_tile(L) : adv_tile_of(L, mode == ADV_FIELD);
  tile[0] = t.w;
  tile[1] = t.h;
  tile[2] = t.tz;
  return LSMGPU_OK;
}
