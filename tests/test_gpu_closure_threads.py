"""Two threads that call one closure at the same time get what one thread gets alone."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from compchan3dmpi_b200.closure import Closure
from oracle import closure_oracle as C

pytestmark = pytest.mark.gpu

REPS = 40


def _closure(capacity=0):
    rng = np.random.default_rng(11)
    cl = Closure(capacity=capacity)
    cl.norm = np.concatenate([np.zeros(13), np.ones(13), np.zeros(9), np.ones(9)]).astype(np.float32)
    cl.params = (rng.standard_normal(C.N_PARAM) * 0.4).astype(np.float32)
    return cl


def _both(f, args):
    """f(a) REPS times for each of the two arguments, at the same time."""
    with ThreadPoolExecutor(2) as ex:
        return list(ex.map(lambda a: [f(a) for _ in range(REPS)], args))


def test_normalization():
    """Double sums whose order differs from call to call, rounded to float: 2^-24 and, next
    to a rounding boundary, one float more."""
    rng = np.random.default_rng(3)
    n = 20000
    with _closure(capacity=n) as cl:
        cl.add_data(rng.standard_normal((n, 13)) + 1.0, rng.standard_normal((n, 9)) * 3.0)
        ref = cl.fit_normalization()
        for outs in _both(lambda _: cl.fit_normalization(), (0, 1)):
            for out in outs:
                np.testing.assert_allclose(out, ref, rtol=2.0 ** -22, atol=2e-7)
