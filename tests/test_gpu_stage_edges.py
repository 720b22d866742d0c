"""The stage kernel, its images and its march where tiles, pairs and chunks end.

A thread owns one (FP64) or two (float) x columns, a CTA a tile of 32 x 8, 32 x 4,
16 x 16 or 32 x 16 columns and a chunk of wall-normal planes; a plane is completed
one plane later, the last of a chunk after its loop.  The grids put the last
column of the interior on the first, second and last place of a pair and of a tile,
the last row likewise, and the chunks at one plane, two planes and the whole height.

FP64 tolerance: the parity bound of the plain path, 1e-12 per variable after three
steps.  Mixed tolerance, against the same start on the default tile in one chunk: none,
every shape gives the same bits; and against the oracle 2e-6, thirty times the 6e-8
that a float stage rounds by (three steps of three stages, each rounding once).
"""
import numpy as np
import pytest

from chan_cases import make_case, rel_err
from compchan3dmpi_b200 import Channel, RK2, RK3
from oracle import oracle as O

pytestmark = pytest.mark.gpu

GRIDS = [(6, 6, 6), (7, 9, 7), (33, 10, 8), (34, 11, 9), (35, 6, 12), (36, 18, 7), (66, 19, 6), (67, 7, 10)]


def _run(case, tile, chunks, steps=3):
    p, x3, jac, inv, var = case
    with Channel(p, x3, jac, inv) as g:
        g.set_launch(tile, chunks)
        g.init_sol_v(var)
        g.step(steps)
        assert g.debug_canaries() == 0
        return g.download()


@pytest.mark.parametrize("tile", [0, 1, 2, 3])
@pytest.mark.parametrize("nP", GRIDS, ids=str)
def test_fp64_edges_match_oracle(nP, tile):
    for rk in (RK2, RK3):
        case = make_case(nP=nP, mesh="tanh", beta=2.0, rk=rk, Pr=0.72, istat=2, quantize=False)
        p, x3, jac, inv, var = case
        o = O.Oracle(p, x3, jac, inv)
        o.upload(var)
        o.step(3)
        ref = o.download()
        nz = nP[2] - 2
        outs = [_run(case, tile, c) for c in sorted({1, (nz + 1) // 2, nz})]
        assert rel_err(outs[0], ref).max() <= 1e-12, (rk, rel_err(outs[0], ref))
        for out in outs[1:]:
            assert np.array_equal(out, outs[0])


@pytest.mark.parametrize("tile", [0, 1, 2, 3])
@pytest.mark.parametrize("nP", GRIDS, ids=str)
def test_mixed_edges_same_bits_and_near_oracle(nP, tile):
    case = make_case(nP=nP, mesh="tanh", beta=2.0, rk=RK3, Pr=0.72, istat=2, quantize=False, mixed=True)
    p, x3, jac, inv, var = case
    nz = nP[2] - 2
    base = _run(case, 0, 1)
    for c in sorted({1, (nz + 1) // 2, nz}):
        assert np.array_equal(_run(case, tile, c), base)
    o = O.Oracle(p.with_(mixed=False), x3, jac, inv)
    o.upload(var)
    o.step(3)
    ref = o.download()
    scale = max(np.max(np.abs(ref[m])) for m in (1, 2, 3))
    for m in range(7):
        s = scale if m in (1, 2, 3) else np.max(np.abs(ref[m]))
        assert np.max(np.abs(base[m] - ref[m])) <= 2e-6 * s, m


@pytest.mark.parametrize("nP,mixed,tile", [((24, 14, 19), False, 0), ((101, 75, 33), False, 2), ((101, 75, 33), True, 0)])
def test_default_tile_changes_no_bits(nP, mixed, tile):
    """The shape picked at creation against the 32x8 tile: the same results to the bit."""
    p, x3, jac, inv, var = make_case(nP=nP, mesh="tanh", beta=2.2, rk=RK2, istat=2, quantize=False)
    out = []
    for forced in (False, True):
        g = Channel(p.with_(mixed=mixed), x3, jac, inv)
        if forced:
            g.set_launch(0, 0)
        else:
            assert g.launch()[0] == tile
        g.init_sol_v(var)
        g.step(4)
        out.append(g.download())
        g.close()
    assert np.array_equal(out[0], out[1])
