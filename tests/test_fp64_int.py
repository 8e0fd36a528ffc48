"""FP64 arithmetic on the integer pipes (csrc/fp64_int.cuh) and the WENO5
reconstruction on it (csrc/weno64.cuh): the same bits as FP64 hardware.

On the host the routines are compiled with the system compiler and compared
with the host's FP64 operations; on the GPU the drop-in WENO5 routines are
compared with the oracle on fields that take both of their paths."""
import os
import subprocess

import numpy as np
import pytest

import lsmlib_gb300 as L
from tests import harness as H

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("seed", [1, 2])
def test_host_arithmetic_equals_hardware(seed, tmp_path):
    exe = str(tmp_path / "fp64_int")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "lsmlib_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "fp64_int_driver.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe, "300000", str(seed)], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["0", "0", "0"]


def field(kind, gb):
    """Fields on which the integer path, the FP64-unit path or a mix of both
    runs, cell by cell."""
    rng = np.random.default_rng(17)
    f = H.rough_field(rng, gb)
    if kind == "flat":
        f[...] = 0.75
    elif kind == "dyadic":
        f = np.round(f * 4) / 4
    elif kind == "tiny":
        f *= 1e-170
    elif kind == "mixed":
        f *= 10.0 ** rng.integers(-200, 120, size=f.shape)
    elif kind == "nonfinite":
        f[rng.random(f.shape) < 0.01] = np.inf
        f[rng.random(f.shape) < 0.01] = np.nan
    return np.asfortranarray(f)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["rough", "flat", "dyadic", "tiny", "mixed", "nonfinite"])
@pytest.mark.parametrize("sym", ["lsm3dhjweno5_", "lsm3dupwindhjweno5_"])
def test_dropin_weno5_on_all_scales(sym, kind, gpu_lib):
    vals = H.dense_case(sym, seed=3)
    vals["phi"] = field(kind, H.GB)
    with np.errstate(all="ignore"):
        want, _ = H.run(H.oracle(), sym, vals)
        got, _ = H.run(gpu_lib, sym, vals)
    L.check()
    for name in H.written_names(sym):
        if name in got and not name.startswith("d"):
            assert H.same(want[name], got[name]), name


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["rough", "flat", "dyadic", "tiny", "mixed", "nonfinite"])
@pytest.mark.parametrize("sym", ["lsm3dgradientmagnitude_", "lsm3dcomputemeancurvatureorder2_",
                                 "lsm3dcomputereinitializationeqnrhs_", "lsm3daddnormalveltermtolserhs_",
                                 "lsm3daddconstcurvtermtolserhs_", "lsm3daddadvectiontermtolserhs_",
                                 "lsm3dtvdrk3stage2_", "lsm3dtvdrk3stage3_", "lsm3dcomputestableadvectiondt_",
                                 "lsm3dcomputestablenormalveldt_", "lsm3dmaxnormdiff_"])
def test_dropin_elementwise_on_all_scales(sym, kind, gpu_lib):
    """The FP64 drop-ins whose products, quotients and roots run on the
    integer pipes, with one input array of each of these kinds at a time."""
    base = H.dense_case(sym, seed=4)
    written = set(H.written_names(sym))
    for name in [k for k, v in base.items() if isinstance(v, np.ndarray) and k not in written]:
        vals = dict(base)
        vals[name] = field(kind, H.GB)
        if kind == "nonfinite" and sym.endswith(("dt_", "normdiff_")):
            vals[name][np.isnan(vals[name])] = 0.5  # a maximum over NaN depends on the order of the comparisons
        with np.errstate(all="ignore"):
            want, wsc = H.run(H.oracle(), sym, vals)
            got, gsc = H.run(gpu_lib, sym, vals)
        L.check()
        for k in want:
            assert H.same(want[k], got[k]), (name, k)
        for k in wsc:
            assert wsc[k] == gsc[k] or (wsc[k] != wsc[k] and gsc[k] != gsc[k]), (name, k)


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1e-6, 1e-9, 1e-11, 1e-13, 1e-15, 1e-18, 1e-30])
@pytest.mark.parametrize("sym", ["lsm3dhjweno5_", "lsm3dupwindhjweno5_"])
def test_dropin_weno5_around_the_floor_of_epsilon(sym, scale, gpu_lib):
    """Differences whose 1e-6 v^2 lies on either side of 2^55 times the floor
    of epsilon (where its addition is left out), and below the floor."""
    vals = H.dense_case(sym, seed=5)
    rng = np.random.default_rng(23)
    phi = H.rough_field(rng, H.GB)
    vals["phi"] = np.asfortranarray(phi * scale * 10.0 ** rng.uniform(-1, 1, size=phi.shape))
    want, _ = H.run(H.oracle(), sym, vals)
    got, _ = H.run(gpu_lib, sym, vals)
    L.check()
    for name in H.written_names(sym):
        if name in got and not name.startswith("d"):
            assert H.same(want[name], got[name]), name


def operands(rng, n):
    """Significands as random, with few bits, nearly full and next to powers of
    two; exponents over 2^-40 .. 2^40."""
    m = rng.integers(0, 1 << 52, size=n, dtype=np.uint64)
    kind = rng.integers(0, 6, size=n)
    m = np.where(kind == 1, m & np.uint64(0xfffff80000000), m)
    m = np.where(kind == 2, m | np.uint64(0xfffffff000000), m)
    m = np.where(kind == 3, m % np.uint64(5), m)
    m = np.where(kind == 4, np.uint64((1 << 52) - 1) - m % np.uint64(5), m)
    e = rng.integers(1023 - 40, 1023 + 41, size=n).astype(np.uint64)
    return np.asfortranarray(((e << np.uint64(52)) | m).view(np.float64))


@pytest.mark.gpu
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_device_square_roots(seed, gpu_lib):
    """The root's device form starts from the approximate instruction: a million
    roots per seed, through |grad phi|, against numpy's."""
    import torch
    n = (128, 96, 90)
    rng = np.random.default_rng(seed)
    g = [operands(rng, n) * 2.0 ** 30 for _ in range(3)]  # their squares are above the routine's zero tolerance
    want = np.sqrt((g[0] * g[0] + g[1] * g[1]) + g[2] * g[2])
    if seed == 2:  # roots of squares
        g[1][...] = g[2][...] = 0.0
        want = np.sqrt(g[0] * g[0])
    box = (0, n[0] - 1, 0, n[1] - 1, 0, n[2] - 1)
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
    out = torch.zeros(n[::-1], dtype=torch.float64, device="cuda")
    vals, _ = H.make_call("lsm3dgradientmagnitude_", box, box,
                          arrays=dict(zip(("phi_x", "phi_y", "phi_z"), g), grad_phi_mag=np.zeros(n, order="F")))
    vals.update(phi_x=to(g[0]), phi_y=to(g[1]), phi_z=to(g[2]), grad_phi_mag=out)
    L.invoke(gpu_lib, "lsm3dgradientmagnitude_", vals)
    L.check()
    assert np.array_equal(out.cpu().numpy().T, want)


@pytest.mark.gpu
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_device_quotients(seed, gpu_lib):
    """The quotient likewise: the mean curvature of phi with grad phi = (1, 0, 0)
    is (phi_yy + phi_zz) / |grad phi|^3, |grad phi| being an argument."""
    import torch
    n = (128, 96, 90)
    rng = np.random.default_rng(seed)
    phi, mag = operands(rng, n), operands(rng, n)
    phi *= rng.choice([1.0, -1.0], size=n)
    one, zero = np.ones(n, order="F"), np.zeros(n, order="F")
    gb = (0, n[0] - 1, 0, n[1] - 1, 0, n[2] - 1)
    fb = (1, n[0] - 2, 1, n[1] - 2, 1, n[2] - 2)
    h = 0.5
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a.T)).cuda()
    vals, _ = H.make_call("lsm3dcomputemeancurvatureorder2_", gb, fb,
                          arrays=dict(phi=phi, phi_x=one, phi_y=zero, phi_z=zero, grad_phi_mag=mag,
                                      kappa=np.zeros(n, order="F")), scalars={"dx": h, "dy": h, "dz": h})
    out = torch.zeros(n[::-1], dtype=torch.float64, device="cuda")
    vals.update(phi=to(phi), phi_x=to(one), phi_y=to(zero), phi_z=to(zero), grad_phi_mag=to(mag), kappa=out)
    L.invoke(gpu_lib, "lsm3dcomputemeancurvatureorder2_", vals)
    L.check()
    c = phi[1:-1, 1:-1, 1:-1]
    f = 1.0 / h / h
    yy = ((phi[1:-1, 2:, 1:-1] - 2.0 * c) + phi[1:-1, :-2, 1:-1]) * f
    zz = ((phi[1:-1, 1:-1, 2:] - 2.0 * c) + phi[1:-1, 1:-1, :-2]) * f
    m = mag[1:-1, 1:-1, 1:-1]
    den = (m * m) * m
    want = np.where(den < 1e-11, 0.0, (yy + zz) / den)
    got = out.cpu().numpy().T[1:-1, 1:-1, 1:-1]
    assert np.count_nonzero(den >= 1e-11) > 500000
    assert np.array_equal(got, want)
