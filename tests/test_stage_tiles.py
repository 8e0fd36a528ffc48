"""The tiles of the FP32 stage kernels (csrc/fused_driver.cuh): which the
steppers choose, and that every shape and depth computes the same.

The choice depends on the SM count; the cases below are for 152 SMs, which the
library also assumes where there is no GPU."""
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
