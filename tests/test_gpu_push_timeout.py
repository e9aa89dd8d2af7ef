"""A wait of the pushed exchange that runs out: the solve ends with the status,
no block leaves while copies to it may be in flight, and the context stays
usable."""
import numpy as np
import pytest

from conftest import gen, pkg


def test_argument_checks():
    eaf = pkg()
    for ms in (0.0, -1.0, 10001.0, float("nan")):
        assert eaf.push_timeout_selftest(0, ms) == eaf._lib.EAF_EINVAL


@pytest.mark.gpu
def test_unfinished_exchange():
    import oracle
    eaf, g = pkg(), gen()
    for _ in range(3):
        assert eaf.push_timeout_selftest(0, 20.0) == eaf._lib.EAF_ETIMEOUT
    s = g.make_system(12, 24, 16, 8, seed=1)
    a, b = g.zeros_phi(12, 24, 16), g.zeros_phi(12, 24, 16)
    with eaf.CGSolver(12, 24, 16) as cg:
        res, nit, st = cg.solve(s.arrays(), a, 40, 0.0)
        plan = cg.last_launch()
    assert st == 0 and (res, nit) == oracle.cg(s, b, 40, 0.0, plan=plan)
    assert np.array_equal(a, b)
