"""The prefetching kernel beyond L2, with slices of which only a part of the
residual is kept in shared memory and slices that are kept whole, in the
symmetric form (x updated one iteration late) and the seven-array form (in its
own), after any number of iterations and on clusters: the kernel-order oracle's
bits, whole array."""
import numpy as np
import pytest

from conftest import gen, pkg

pytestmark = pytest.mark.gpu

DIMS = (93, 91, 90)  # 761,670 cells; 40 blocks of 1024 threads keep 16,384 of 19,042 each


@pytest.fixture(scope="module", params=["symmetric", "general"])
def system(request):
    s = gen().make_system(*DIMS, 8, seed=2)
    if request.param == "general":
        s.aE[2:-2, 2:-2, 2:-2] *= 1.0 + 1e-13
    return s, request.param == "symmetric"


@pytest.mark.parametrize("grid,cluster", [(40, 1), (148, 1), (40, 4)])
@pytest.mark.parametrize("iters", [0, 1, 2, 5])
def test_forms(system, grid, cluster, iters):
    import oracle
    eaf, g = pkg(), gen()
    s, symmetric = system
    a = np.random.default_rng(1).normal(size=g.halo_shape(*DIMS))
    b = a.copy()
    with eaf.CGSolver(*DIMS) as cg:
        cg.set_launch(1024, grid)
        cg.set_cluster(cluster)
        res, nit, _ = cg.solve(s.arrays(), a, iters, 0.0)
        plan = cg.last_launch()
        assert cg.last_timing()["symmetric"] == symmetric
    assert plan[:2] == (grid, 1024)
    assert (res, nit) == oracle.cg(s, b, iters, 0.0, plan=plan)
    assert np.array_equal(a, b)
