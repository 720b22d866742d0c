"""The optimiser kernel: one Adam step, and none from the sums of a training kernel that
gave up (its CTA's share is then missing: what an earlier step left, or uninitialised)."""
import ctypes

import numpy as np
import pytest

from compchan3dmpi_b200 import _lib
from oracle import closure_oracle as C

pytestmark = pytest.mark.gpu


def _step(w, m, v, g, lr, failed):
    L = _lib.load()
    f = [a.ctypes.data_as(ctypes.POINTER(ctypes.c_float)) for a in (w, m, v, g)]
    assert L.chan_selftest_adam(*f, lr, failed, 0) == 0


def _state():
    rng = np.random.default_rng(9)
    w, m, g = (rng.standard_normal(C.N_PARAM).astype(np.float32) for _ in range(3))
    v = rng.random(C.N_PARAM).astype(np.float32)
    return w, m, v, g


def test_one_step():
    """Ten roundings to float (2^-24 each) of numbers no larger than the sums of their terms'
    magnitudes: 16 * 2^-24."""
    w, m, v, g = _state()
    w1, m1, v1 = w.copy(), m.copy(), v.copy()
    lr = np.float32(1e-3)
    _step(w1, m1, v1, g, lr, 0)
    b1, b2 = np.float32(0.9), np.float32(0.999)
    c1, c2 = np.float64(np.float32(1) - b1), np.float64(np.float32(1) - b2)
    w, m, v, g, b1, b2, lr = (np.float64(x) for x in (w, m, v, g, b1, b2, lr))
    mr, vr = b1 * m + c1 * g, b2 * v + c2 * g * g
    step = lr * (mr / c1) / (np.sqrt(vr / c2) + 1e-8)
    tol = 16 * 2.0 ** -24
    mag = b1 * np.abs(m) + c1 * np.abs(g)
    assert np.all(np.abs(m1 - mr) <= tol * mag)
    assert np.all(np.abs(v1 - vr) <= tol * vr)
    assert np.all(np.abs(w1 - (w - step)) <= tol * (np.abs(w) + np.abs(step) * mag / np.abs(mr)))


def test_no_step_from_incomplete_sums():
    w, m, v, g = _state()
    w1, m1, v1 = w.copy(), m.copy(), v.copy()
    _step(w1, m1, v1, g, 1e-3, 1)
    assert np.array_equal(w1, w) and np.array_equal(m1, m) and np.array_equal(v1, v)
