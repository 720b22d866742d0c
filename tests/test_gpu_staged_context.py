"""A context's host copies of 16 MB and more, which several threads stage in chunks of
1 MB: upload, download, checkpoint, fluctuations and Q-criterion, every value told from
the others.  The grids give a whole number of chunks, and a part of one at the end."""
import numpy as np
import pytest

from chan_cases import make_case
from compchan3dmpi_b200 import Channel, periodic_coords
from compchan3dmpi_b200.channel import q_criterion

pytestmark = pytest.mark.gpu

# 7 N doubles: 56 and 57 MB; 5 N: 40 MB (up) ; N: 17.0 MB at the third (the Q-criterion)
GRIDS = [(128, 128, 64), (160, 96, 65), (131, 127, 134)]


@pytest.mark.parametrize("nP", GRIDS, ids=str)
def test_values_arrive_where_they_belong(nP, tmp_path):
    p, x3, jac, inv, var = make_case(nP=nP, mesh="tanh", beta=2.0, quantize=False, istat=0)
    rng = np.random.default_rng(nP[0])
    var = var * (1.0 + 1e-3 * rng.standard_normal(var.shape))
    with Channel(p, x3, jac, inv) as g:
        g.init_sol_v(var)
        a = g.download()
        # rho as given; u, v, w, E through rho*u and back: a product, a reciprocal of 1 ulp
        # and a product, at most 3 ulp
        inner = np.s_[1:-1, 1:-1, 1:-1]
        assert np.array_equal(a[0][inner], var[0][inner])
        for m in (1, 2, 3, 4):
            assert np.all(np.abs(a[m][inner] - var[m][inner]) <= 3 * 2.0 ** -52 * np.abs(var[m][inner])), m
        # the wall planes and the corner columns hold what was given, T and p too
        for k in (0, -1):
            assert np.array_equal(a[:, k], var[:, k])
        for j in (0, -1):
            for i in (0, -1):
                assert np.array_equal(a[:, :, j, i], var[:, :, j, i])
        mean = a.mean(axis=(2, 3))
        x1, x2 = periodic_coords(nP[0], p.Lx), periodic_coords(nP[1], p.Ly)
        fl, q = g.fluctuation_q(mean, x1, x2, x3)
        assert np.array_equal(fl, a - mean[:, :, None, None])
        assert np.array_equal(q, q_criterion(fl[1], fl[2], fl[3], x1, x2, x3))
        path = tmp_path / "state.ckp"
        g.checkpoint_write(path)
        with Channel(p, x3, jac, inv) as h:
            h.checkpoint_read(path)
            assert np.array_equal(h.download(), a)
            g.step(2)
            h.step(2)
            assert np.array_equal(h.download(), g.download())
