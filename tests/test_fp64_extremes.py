"""FP64 at the ends of the exponent range: the drop-ins and the fused steppers
return the oracle's numbers where products become subnormal."""
import numpy as np
import pytest

import lsmlib_gb300 as L
from tests import harness as H
from tests import oracle_runs as O

GB, FB = (-3, 20, -3, 18, -3, 16), (0, 17, 0, 15, 0, 13)
# integer multiples of the smallest subnormal, and values around the smallest
# normal number
KINDS = {"subnormal": lambda rng, n: rng.integers(-4000, 4000, size=n) * 5e-324,
         "smallest normals": lambda rng, n: rng.standard_normal(n) * 1e-307}


@pytest.mark.gpu
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_rk_stage_2_dropin(kind, gpu_lib):
    sym = "lsm3dtvdrk3stage2_"
    vals = H.dense_case(sym, seed=4)
    rng = np.random.default_rng(2)
    for name, a in vals.items():
        if isinstance(a, np.ndarray):
            vals[name] = np.asfortranarray(KINDS[kind](rng, a.shape))
    want, _ = H.run(H.oracle(), sym, vals)
    got, _ = H.run(gpu_lib, sym, vals)
    L.check()
    assert H.same(want["u_stage2"], got["u_stage2"])


@pytest.mark.gpu
@pytest.mark.parametrize("bc", [L.BC_PERIODIC, L.BC_LINEAR])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_fused_advection(kind, bc, gpu_lib):
    phi = np.asfortranarray(KINDS[kind](np.random.default_rng(3), H.shape_of(GB)))
    dx, dt, v = 2.0 / 24, 0.03, (0.3, -0.4, 0.5)
    vel = [np.full(H.shape_of(GB), q, order="F") for q in v]
    if bc == L.BC_PERIODIC:
        O.periodic_fill(phi, GB, FB)
    want = O.tvdrk3_run(H.oracle(), "advect", phi, GB, FB, dx, dt, 2, bc, vel=vel)
    for kw in ({"vel_const": v}, {"vel": vel, "vel_gb": GB}):
        got = phi.copy(order="F")
        L.advect_weno5_tvdrk3(got, GB, FB, dx, dt, 2, bc=bc, **kw)
        assert H.same(want, got)
