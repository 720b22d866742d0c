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


def test_gradients():
    """The same sums but for the order of the CTA's eight float additions per bias: 8 * 2^-24
    of a group's norm, bounded by 1e-5."""
    rng = np.random.default_rng(4)
    data = [(rng.standard_normal((n, 13)).astype(np.float32), rng.standard_normal((n, 9)).astype(np.float32))
            for n in (700, 5000)]
    with _closure() as cl:
        refs = [cl.grad(*d) for d in data]
        for (lo, g), outs in zip(refs, _both(lambda d: cl.grad(*d), data)):
            for l1, g1 in outs:
                assert abs(l1 - lo) <= 1e-5 * abs(lo)
                assert np.linalg.norm(g1 - g) <= 1e-5 * np.linalg.norm(g)


@pytest.mark.parametrize("n", [700, 322639])     # rows of 52 bytes: 16 MB and more is staged
def test_inference(n):
    rng = np.random.default_rng(n)
    X = [rng.standard_normal((m, 13)).astype(np.float32) for m in (n, n + 129)]
    with _closure() as cl:
        refs = [cl.infer(x) for x in X]
        with ThreadPoolExecutor(2) as ex:
            outs = list(ex.map(lambda x: [cl.infer(x) for _ in range(4)], X))
    for ref, out in zip(refs, outs):
        assert all(np.array_equal(y, ref) for y in out)
