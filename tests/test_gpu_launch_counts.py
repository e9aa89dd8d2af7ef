"""Kernels per call as last_timing reports them: every launch of the call, the ones
that clear counters and slots among them."""
import numpy as np
import pytest

from conftest import gen, pkg

pytestmark = pytest.mark.gpu

DIMS = (20, 31, 17)


# pack, what clears the slots (not where the launcher clears by memsets), solver, unpack
@pytest.mark.parametrize("form,kernels", [("LOADS", 4), ("KEEP", 4), ("SLOTS", 4), ("STREAM", 3),
                                          ("cluster", 4), ("resident", 3), ("one", 3),
                                          ("mixed", 3)])
def test_solves(form, kernels):
    eaf, g = pkg(), gen()
    s = g.make_system(*DIMS, 8, seed=1)
    phi = g.zeros_phi(*DIMS)
    with eaf.CGSolver(*DIMS) as cg:
        if form == "mixed":
            cg.solve_mixed(s.arrays(), phi, tol=1e-8)
        else:
            if form == "one":
                cg.set_form(cg.FORM_ONE_REDUCTION)
            elif form == "resident":
                cg.set_launch(512, 16)
                cg.set_cluster(16)
            elif form == "cluster":
                cg.set_launch(256, 32)
                cg.set_cluster(4)
            else:
                cg.set_launch(256, 30)
                cg.set_kernel(getattr(cg, "KERNEL_" + form))
            cg.solve(s.arrays(), phi, 5, 0.0)
        assert cg.last_timing()["kernels"] == kernels


def test_other_calls():
    eaf, g = pkg(), gen()
    t = g.make_transport_system(*DIMS, seed=2)
    phi = np.random.default_rng(0).normal(size=g.halo_shape(*DIMS))
    with eaf.CGSolver(*DIMS) as cg:
        cg.residual(t.arrays(), phi)
        assert cg.last_timing()["kernels"] == 2
        cg.pressure_step(g.make_pressure_state(*DIMS, seed=3), 0.7, 5, 1e-8)
        cluster = len(cg.last_launch()) > 2
        assert cg.last_timing()["kernels"] == 4 + (3 if cluster else 4) + 3
