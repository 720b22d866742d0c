"""The persistent ensemble deals its members' wall and image blocks to units of one to
eight, by their number: the members' bits stay those of stepping each alone."""
import numpy as np
import pytest

from chan_cases import make_case
from compchan3dmpi_b200 import Channel, RK3
from compchan3dmpi_b200.ensemble import Ensemble

pytestmark = pytest.mark.gpu


# 202 blocks a member on 296 CTAs: units of 1, 3, 5 and 8, the last one of a member cut short
@pytest.mark.parametrize("mixed", [False, True], ids=["fp64", "mixed"])
@pytest.mark.parametrize("members", [1, 4, 7, 12])
def test_members_match_alone(members, mixed):
    cases = []
    for seed in (1, 2):
        p, x3, jac, inv, var = make_case(nP=(8, 9, 200), mesh="tanh", beta=2.0, rk=RK3, istat=2, quantize=False,
                                         mixed=mixed)
        cases.append((p, x3, jac, inv, var * (1.0 + 1e-3 * np.random.default_rng(seed).standard_normal(var.shape))))

    def start(i):
        p, x3, jac, inv, var = cases[i % 2]
        c = Channel(p, x3, jac, inv)
        c.init_sol_v(var)
        return c

    alone = []
    for i in (0, 1):
        c = start(i)
        c.step(6)
        alone.append((c.download(), c.stats()))
        c.close()
    ch = [start(i) for i in range(members)]
    with Ensemble(ch) as e:
        e.set_mode("persistent")
        assert e.step(6) == [0] * members
        assert e.mode_in_use()[0] == "persistent"
        for i, c in enumerate(ch):
            assert c.debug_canaries() == 0
            assert np.array_equal(c.download(), alone[i % 2][0])
            assert all(np.array_equal(a, b) for a, b in zip(c.stats(), alone[i % 2][1]))
    for c in ch:
        c.close()
