"""The tiles of the FP32 stage kernels (csrc/fused_driver.cuh): which the
steppers choose, and that every shape and depth computes the same.

The choice depends on the SM count; the cases below are for 152 SMs, which the
library also assumes where there is no GPU."""
import numpy as np
import pytest

import lsmlib_gb300 as L


@pytest.mark.parametrize("mode", ["advect_const", "advect"])
@pytest.mark.parametrize("n,width", [((6, 6, 20000), 16), ((8, 8, 5000), 16), ((16, 16, 3000), 16), ((30, 10, 2000), 32),
                                     ((20, 8, 500), 32), ((64, 8, 5000), 64), ((128, 128, 128), 64),
                                     ((256, 256, 256), 64)])
def test_narrow_grids_run_narrow_rows(mode, n, width):
    """A grid narrower than a row leaves lanes of it idle, so of tiles equal in
    number and depth the narrower ones run (6 x 6 x 20000 took 63 us per stage
    on 64-cell rows, 43 on 16-cell ones)."""
    w, h, tz = L.stage_tile(mode, n)
    assert (w, h) == (width, 512 // width) and tz in (2, 4, 6, 8, 10)


def test_invalid_grids_are_refused():
    with pytest.raises(ValueError):
        L.stage_tile("advect", (0, 6, 6))
    with pytest.raises(ValueError):
        L.stage_tile("upwind", (6, 6, 6))


# a grid for every tile the rules can choose, ragged on every axis
TILES = {
    "advect_const": {(64, 2): (69, 19, 43), (64, 4): (97, 9, 230), (64, 6): (193, 33, 90), (64, 8): (203, 17, 303),
                     (64, 10): (50, 125, 189), (32, 2): (17, 6, 7), (32, 4): (17, 33, 311), (32, 6): (17, 97, 349),
                     (32, 8): (18, 195, 279), (32, 10): (17, 189, 379), (16, 2): (7, 60, 101), (16, 4): (6, 66, 307),
                     (16, 6): (6, 162, 409), (16, 8): (35, 98, 303), (16, 10): (231, 125, 49)},
    "advect": {(64, 2): (69, 19, 43), (64, 4): (97, 9, 389), (64, 6): (36, 41, 409), (64, 8): (130, 34, 375),
               (64, 10): (194, 21, 379), (32, 2): (17, 6, 7), (32, 4): (17, 50, 391), (32, 6): (17, 97, 349),
               (32, 8): (17, 226, 367), (32, 10): (17, 189, 379), (16, 2): (7, 60, 101), (16, 4): (6, 98, 387),
               (16, 6): (6, 162, 409), (16, 8): (34, 130, 369), (16, 10): (35, 108, 379)},
    "reinit": {(64, 2): (37, 33, 41), (64, 4): (6, 9, 303), (64, 6): (6, 25, 383), (64, 8): (6, 25, 299),
               (64, 10): (6, 17, 403)},
}
CASES = [(mode, tile, n) for mode, tiles in TILES.items() for tile, n in tiles.items()]


@pytest.mark.parametrize("mode,tile,n", CASES)
def test_each_grid_runs_its_tile(mode, tile, n):
    w, h, tz = L.stage_tile(mode, n)
    assert (w, tz) == tile and w * h == 512


@pytest.mark.gpu
@pytest.mark.parametrize("bc", [L.BC_PERIODIC, L.BC_LINEAR])
@pytest.mark.parametrize("mode,tile,n", CASES)
def test_every_tile_against_fp64(mode, tile, n, bc, gpu_lib):
    """Two steps on each tile against the FP64 form (which equals the oracle bit
    for bit), interior cells, to the FP32 tests' 1e-5 on a field of order one."""
    import torch
    assert (L.stage_tile(mode, n)[0], L.stage_tile(mode, n)[2]) == tile
    fb = tuple(v for m in n for v in (0, m - 1))
    gb = tuple(v for m in n for v in (-3, m + 2))
    x, y, z = [(2 * np.pi * (np.arange(-3, m + 3) + 0.5) / m).reshape([-1 if a == q else 1 for a in range(3)])
               for q, m in enumerate(n)]
    dx = 2.0 / max(n)
    ty = np.float32
    if mode == "reinit":
        phi = np.sin(x + 0.2) * np.cos(y) * 0.3 + 0.2 * np.cos(z)
    else:
        phi = np.sin(x) * np.cos(y) + 0.4 * np.cos(2 * z + 0.3) * np.sin(y)
    to_gpu = lambda a: torch.from_numpy(np.ascontiguousarray(np.broadcast_to(a, phi.shape).T.astype(ty))).cuda()
    t32 = to_gpu(phi)
    t64 = t32.double()
    vel = [to_gpu(np.where(np.abs(v) < 0.05, 0.0, v)) for v in
           (0.5 * np.sin(y + 0.2) * np.cos(z), -0.4 * np.cos(x) * np.sin(z + 0.1), 0.3 * np.sin(x + y))]
    for t, precision, cast in ((t32, "f32", lambda v: v), (t64, "f64", lambda v: v.double())):
        if mode == "reinit":
            L.reinit_weno5_tvdrk3(t, gb, fb, dx, 0.5 * dx, 2, use_phi0_for_sgn=int(bc == L.BC_LINEAR), bc=bc,
                                  precision=precision)
        elif mode == "advect":
            L.advect_weno5_tvdrk3(t, gb, fb, dx, 0.5 * dx, 2, vel=[cast(v) for v in vel], vel_gb=gb, bc=bc,
                                  precision=precision)
        else:
            L.advect_weno5_tvdrk3(t, gb, fb, dx, 0.5 * dx, 2, vel_const=(0.4, -0.5, -0.3), bc=bc, precision=precision)
    L.check()
    inner = (slice(3, -3),) * 3
    assert float((t64[inner] - to_gpu(phi).double()[inner]).abs().max()) > 1e-3 * dx
    assert float((t32.double() - t64)[inner].abs().max()) <= 1e-5
