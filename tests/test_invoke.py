"""The ctypes call path (lsmlib_gb300.invoke) on the C oracle: scalars by
reference and back, per-call arrays, errors, threads."""
import threading

import numpy as np
import pytest

import lsmlib_gb300 as L
from tests import harness as H

GB, FB = (-1, 4, -1, 3, -1, 2), (0, 3, 0, 2, 0, 1)


def _axpy_call(seed):
    """lsm3drk1step: u_next = u_cur + dt rhs on the fill box."""
    rng = np.random.default_rng(seed)
    u, rhs = (np.asfortranarray(rng.standard_normal(H.shape_of(GB))) for _ in range(2))
    vals, arrays = H.make_call("lsm3drk1step_", GB, FB, arrays={"u_cur": u, "rhs": rhs}, scalars={"dt": 0.1 * seed})
    return vals, arrays["u_next"], u, rhs


def _check(seed):
    vals, out, u, rhs = _axpy_call(seed)
    back = L.invoke(H.oracle(), "lsm3drk1step_", vals)
    inner = (slice(1, 5), slice(1, 4), slice(1, 3))
    assert np.array_equal(out[inner], (u + 0.1 * seed * rhs)[inner])
    assert back == {k: v for k, v in vals.items() if not isinstance(v, np.ndarray)}


def test_scalars_and_arrays_of_each_call():
    for seed in (1, 2, 3):
        _check(seed)


def test_missing_argument_names_the_argument_and_leaves_the_path_usable():
    vals, _, _, _ = _axpy_call(1)
    for name in ("dt", "rhs", "ihi_fb"):
        with pytest.raises(KeyError, match=name):
            L.invoke(H.oracle(), "lsm3drk1step_", {k: v for k, v in vals.items() if k != name})
    with pytest.raises(TypeError):
        L.invoke(H.oracle(), "lsm3drk1step_", dict(vals, rhs="text"))
    _check(4)


def test_out_of_range_scalar_wraps_as_ctypes_does():
    vals, out, u, _ = _axpy_call(1)
    before = out.copy()
    back = L.invoke(H.oracle(), "lsm3drk1step_", dict(vals, ihi_fb=FB[1] + 2 ** 32 - 10))  # -7: an empty box
    assert back["ihi_fb"] == FB[1] - 10
    assert np.array_equal(before, out, equal_nan=True)


def test_threads_do_not_share_a_call():
    errors = []

    def work(seed):
        try:
            for _ in range(200):
                _check(seed)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(q + 1,)) for q in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_two_libraries_called_in_turn_keep_their_plans(monkeypatch):
    """A program that compares two libraries prepares each entry point once per
    library, not once per call."""
    import ctypes
    libs = [ctypes.CDLL(H.oracle()._name) for _ in range(2)]
    made = []

    class Counted(L._Plan):
        def __init__(self, *args):
            made.append(args)
            super().__init__(*args)

    monkeypatch.setattr(L, "_Plan", Counted)
    for seed in range(1, 7):
        vals, out, u, rhs = _axpy_call(seed)
        L.invoke(libs[seed % 2], "lsm3drk1step_", vals)
        inner = (slice(1, 5), slice(1, 4), slice(1, 3))
        assert np.array_equal(out[inner], (u + 0.1 * seed * rhs)[inner])
    assert len(made) == 2
    for _ in range(6):  # any number of libraries
        vals, out, u, rhs = _axpy_call(3)
        L.invoke(ctypes.CDLL(H.oracle()._name), "lsm3drk1step_", vals)
        assert np.array_equal(out[inner], (u + 0.1 * 3 * rhs)[inner])
