"""FP32 constant-velocity advection, single grids and batches, on any spacing.

WENO5's weights depend on the differences divided by the spacing (their floor
of epsilon is 1e-36 in those units), so phi and the spacing may come in any
units.  Against the FP64 stepper (equal to the oracle bit for bit) on the same
FP32 input; the tolerance is the other FP32 tests' 1e-5 of the field's
amplitude."""
import numpy as np
import pytest

import lsmlib_gb300 as L

N = 24
GB, FB = (-3, N + 2) * 3, (0, N - 1) * 3
VEL = (0.3, -0.5, 0.4)
# of a distance-like field (1), and with 1e-6 v^2 about at the floor and below it
AMPLITUDES = [1.0, 1e-14, 1e-17]
SPACINGS = [1e-30, 1e-25, 1e-19, 1e-10, 1e-3, 2.0 ** -9, 1 / 64, 0.06, 1.0, 1e6, 2.0 ** 24, 1e9, 1e12, 1e18, 1e20, 1e30]


def field(amplitude):
    """Smooth with kinks (|.|), so that the nonlinear weights matter."""
    x, y, z = np.meshgrid(*[2 * np.pi * (np.arange(-3, N + 3) + 0.5) / N] * 3, indexing="ij")
    f = np.abs(np.sin(x) * np.cos(y) + 0.4 * np.cos(2 * z + 0.3) * np.sin(y)) - 0.3
    return np.asfortranarray((f * amplitude).astype(np.float32))


def fp64_run(phi, spacing, dt, steps, bc):
    import torch
    t = torch.from_numpy(np.ascontiguousarray(phi.astype(np.float64).T)).cuda()
    L.advect_weno5_tvdrk3(t, GB, FB, spacing[0], dt, steps, vel_const=VEL, bc=bc, dy=spacing[1], dz=spacing[2])
    return t.cpu().numpy().T


def cases():
    for h in SPACINGS:
        for a in AMPLITUDES:
            amp = a * h * N / 6  # slopes of about `a`
            if 1e-34 < amp < 1e34:
                yield (h, h, h), amp
    for hs in [(1e-3, 1.0, 1e3), (1e6, 1e-6, 1.0), (1e-9, 1e-9, 1e3)]:
        yield hs, 1.0 * min(hs)


CASES = list(cases())


@pytest.mark.gpu
@pytest.mark.parametrize("bc", [L.BC_PERIODIC, L.BC_SIGNED_LINEAR])
@pytest.mark.parametrize("spacing,amp", CASES)
def test_single_grid(spacing, amp, bc, gpu_lib):
    import torch
    phi = field(amp)
    dt = 0.5 * float(np.float32(min(spacing)))
    want = fp64_run(phi, spacing, dt, 2, bc)
    t = torch.from_numpy(np.ascontiguousarray(phi.T)).cuda()
    L.advect_weno5_tvdrk3(t, GB, FB, spacing[0], dt, 2, vel_const=VEL, bc=bc, precision="f32", dy=spacing[1],
                          dz=spacing[2])
    L.check()
    got = t.cpu().numpy().T.astype(np.float64)
    assert np.max(np.abs(want - phi)) > 0.01 * amp
    assert np.max(np.abs(got - want)[3:-3, 3:-3, 3:-3]) <= 1e-5 * amp


@pytest.mark.gpu
@pytest.mark.parametrize("flags", [0, L.BATCH_LOOP])
def test_batch(flags, gpu_lib):
    """All of them in one batch."""
    n = len(CASES)
    spacing = np.array([c[0] for c in CASES], dtype=np.float32)
    dt = 0.5 * spacing.min(axis=1)
    phis = [field(amp) for _, amp in CASES]
    size = phis[0].size
    buf = np.concatenate([p.ravel(order="F") for p in phis])
    L.advect_batch_weno5_tvdrk3(buf, np.arange(n) * size, np.full((n, 3), N), np.array([VEL] * n), spacing, dt, 2,
                                flags=flags)
    L.check()
    for g, (_, amp) in enumerate(CASES):
        want = fp64_run(phis[g], tuple(map(float, spacing[g])), float(dt[g]), 2, L.BC_PERIODIC)
        got = buf[g * size:(g + 1) * size].reshape(phis[g].shape, order="F").astype(np.float64)
        assert np.max(np.abs(got - want)[3:-3, 3:-3, 3:-3]) <= 1e-5 * amp, CASES[g]


@pytest.mark.gpu
@pytest.mark.parametrize("spacing", [1e-3, 1.0, 1e20])
def test_ghosts_and_zero_steps_keep_their_bits(spacing, gpu_lib):
    """Still fields come back as they went in, in every value."""
    rng = np.random.default_rng(9)
    phi = np.asfortranarray(rng.standard_normal((N + 6,) * 3).astype(np.float32) * np.float32(spacing))
    got = phi.copy(order="F")
    inner = (slice(3, -3),) * 3
    L.advect_weno5_tvdrk3(got, GB, FB, spacing, 0.1 * spacing, 2, vel_const=(0.0, 0.0, 0.0), bc=L.BC_PERIODIC,
                          precision="f32")
    # 3/4 phi + 1/4 phi and 1/3 phi + 2/3 phi round
    assert np.max(np.abs(got[inner] - phi[inner])) <= 4e-7 * np.max(np.abs(phi))
    buf = phi.ravel(order="F").copy()
    L.advect_batch_weno5_tvdrk3(buf, np.array([0]), np.array([(N, N, N)]), np.array([VEL]), np.full((1, 3), spacing),
                                np.array([0.1 * spacing]), 0)
    L.check()
    assert np.array_equal(buf, phi.ravel(order="F"))
