"""Closure kernels at the edges of their tiles and launches (128 rows a tile, one CTA per
SM in training with two tiles in flight, six per SM in inference), and the staged host
copies at the edges of their chunks."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from compchan3dmpi_b200.closure import Closure
from oracle import closure_oracle as C

pytestmark = pytest.mark.gpu

SM, TILE = 148, 128
# one row; a tile's edge; one tile per CTA; a group's second tile, partly empty
ROWS = [1, TILE - 1, TILE, TILE + 1, SM * TILE - 1, SM * TILE + 1, 2 * SM * TILE + TILE + 1]


def _closure(seed=5, scale=0.4, capacity=0):
    rng = np.random.default_rng(seed)
    params = (rng.standard_normal(C.N_PARAM) * scale).astype(np.float32)
    norm = np.concatenate([rng.standard_normal(13) * 0.1, 0.5 + rng.random(13),
                           rng.standard_normal(9) * 0.1, 0.5 + rng.random(9)]).astype(np.float32)
    cl = Closure(capacity=capacity)
    cl.norm = norm
    cl.params = params
    return cl, params, norm


@pytest.mark.parametrize("n", ROWS)
def test_gradients_at_launch_edges(n):
    """Device and oracle round to BF16 at the same places; an F32 sum taken in another order
    moves about 1e-4 of the values across a rounding boundary, by one BF16 ulp (2^-8).  Over
    many rows that is ~1e-4 of a group's L2 norm, and the bound is 2e-3; a single row can
    have one flip in each of its two hidden layers, 2 * 2^-8."""
    cl, params, norm = _closure()
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, 13)).astype(np.float32)
    T = rng.standard_normal((n, 9)).astype(np.float32)
    loss, g = cl.grad(X, T)
    lo, go = C.grad(params, norm, X, T)
    tol = 2.0 ** -7 if n == 1 else 2e-3
    assert abs(loss - lo) <= max(tol, 1e-3) * lo
    for name, a, b in (("W1", C.OFF_W1, C.OFF_B1), ("b1", C.OFF_B1, C.OFF_W2), ("W2", C.OFF_W2, C.OFF_B2),
                       ("b2", C.OFF_B2, C.OFF_W3), ("W3", C.OFF_W3, C.OFF_B3), ("b3", C.OFF_B3, C.N_PARAM)):
        e = np.linalg.norm(g[a:b] - go[a:b]) / np.linalg.norm(go[a:b])
        assert e < tol, (name, e)


@pytest.mark.parametrize("n", [1, TILE - 1, TILE, TILE + 1, 6 * SM * TILE + 1])
def test_inference_at_launch_edges(n):
    cl, params, norm = _closure(seed=6)
    X = np.random.default_rng(n).standard_normal((n, 13)).astype(np.float32)
    Y = cl.infer(X)
    ref, _ = C.forward(params, norm, X)
    # as over 1000 rows: BF16 activations, roundings may differ at a boundary
    assert np.max(np.abs(Y - ref)) < 2e-2 * np.max(np.abs(ref))


@pytest.mark.parametrize("n", [2, 255, 257, 2 * SM * 256 + 1])
def test_column_statistics(n):
    """Double sums: the results differ from numpy's by their rounding to float (2^-24) and,
    in the spread, by the cancellation of double sums (far below it)."""
    rng = np.random.default_rng(n)
    X = (rng.standard_normal((n, 13)) + np.arange(13)).astype(np.float32)
    T = (rng.standard_normal((n, 9)) * 3.0).astype(np.float32)
    cl = Closure(capacity=n)
    cl.add_data(X, T)
    out = cl.fit_normalization().astype(np.float64)
    X, T = X.astype(np.float64), T.astype(np.float64)
    ref = np.concatenate([X.mean(0), X.std(0), T.mean(0), T.std(0)])
    scale = np.concatenate([np.abs(X).max(0)] * 2 + [np.abs(T).max(0)] * 2)
    assert np.all(np.abs(out - ref) <= 2e-7 * scale)


# rows of 52 bytes: below and from 16 MB on the copies are staged in 1 MB chunks; whole
# chunks, and one row more
@pytest.mark.parametrize("n", [1, 322638, 322639, 524288, 524289, 700001])
def test_host_copies_round_trip(n):
    rng = np.random.default_rng(n)

    def one(seed):
        X = rng.random((n, 13), dtype=np.float32) if seed == 0 else np.full((n, 13), np.float32(seed))
        T = np.full((n, 9), np.float32(seed)) + np.arange(n, dtype=np.float32)[:, None]
        with Closure(capacity=n) as cl:
            cl.add_data(X, T)
            a, b = cl.data()
        return np.array_equal(a, X) and np.array_equal(b, T)

    assert one(0)
    with ThreadPoolExecutor(3) as ex:      # handles of several threads share the buffers
        assert all(ex.map(one, [1, 2, 3]))
