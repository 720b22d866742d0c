"""Closure samples (filtered fields formed once, features from their ring) against the
oracle where the strides, the filter width and the periods meet: no filter, unequal
strides, strides that leave a remainder, neighbours that wrap once and several times."""
import numpy as np
import pytest

from chan_cases import make_case
from compchan3dmpi_b200 import Channel, RK2
from compchan3dmpi_b200.closure import Closure
from oracle import closure_oracle as C

pytestmark = pytest.mark.gpu

CASES = [((24, 18, 19), (1, 1, 1), 0), ((24, 18, 19), (1, 2, 3), 4), ((24, 18, 19), (4, 3, 3), 4),
         ((23, 17, 20), (5, 2, 4), 2), ((23, 17, 20), (4, 6, 9), 6), ((8, 9, 12), (7, 4, 2), 4),
         ((6, 6, 6), (5, 13, 2), 8), ((6, 7, 6), (1, 1, 1), 2)]


@pytest.mark.parametrize("nP,strides,width", CASES, ids=str)
def test_samples_match_oracle(nP, strides, width):
    """Float results of double sums: 2^-24 of a column's largest value, and where the sums
    cancel (the fluxes, above all without a filter) the roundings of the double products,
    up to 2 (width + 1)^2 + 16 of them; bounds 1e-5 and 1e-13 of the products."""
    p, x3, jac, inv, var = make_case(nP=nP, mesh="tanh", beta=2.2, rk=RK2, istat=2, quantize=False)
    with Channel(p, x3, jac, inv) as g:
        g.init_sol_v(var)
        g.step(4)
        field, (tau, s1, _, _) = g.download(), g.stats()
        with Closure(capacity=nP[0] * nP[1] * nP[2]) as cl:
            n = cl.sample(g, strides=strides, width=width)
            X, T = cl.data()
    Xo, To = C.sample(field, x3, p.dx, p.dy, p.Re, *strides, width, tau, s1)
    assert X.shape == Xo.shape and T.shape == To.shape and n == len(X) > 0
    u = max(np.max(np.abs(field[m])) for m in (1, 2, 3))
    prod = np.max(field[0]) * u * np.array([u] * 6 + [np.max(field[5])] * 3)
    for c in range(13):
        # a gradient's terms: the field's largest value over the spacing
        mag = (u if c < 9 else np.max(field[5])) / min(2 * strides[0] * p.dx, 2 * strides[1] * p.dy, np.min(np.diff(x3)))
        assert np.max(np.abs(X[:, c] - Xo[:, c])) <= 1e-5 * np.max(np.abs(Xo[:, c])) + (1e-13 * mag if c < 12 else 0), c
    for c in range(9):
        assert np.max(np.abs(T[:, c] - To[:, c])) <= 1e-5 * np.max(np.abs(To[:, c])) + 1e-13 * prod[c], c
