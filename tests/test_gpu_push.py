"""The cluster-resident solver's pushed form (one or two cells a thread in
registers, z and partials pushed between the blocks): bit for bit the
kernel-order oracle's plan (C, B, C) where slices are odd, thinner than a
plane, empty or beyond the form's reach (then the cluster-barrier form runs),
on degenerate meshes, in the symmetric and the 7-array form, at every way out
of the solve."""
import numpy as np
import pytest

from conftest import gen, pkg

pytestmark = pytest.mark.gpu


def both(s, phi0, block, cluster, iters, tol):
    import oracle
    eaf = pkg()
    a, b = phi0.copy(), phi0.copy()
    with eaf.CGSolver(s.nr, s.nth, s.nz) as cg:
        cg.set_launch(block, cluster)
        cg.set_cluster(cluster)
        res, nit, st = cg.solve(s.arrays(), a, iters, tol)
        plan = cg.last_launch()
        sym = cg.last_timing()["symmetric"]
    assert plan == (cluster, block, cluster)
    with np.errstate(all="ignore"):
        ro, no = oracle.cg(s, b, iters, tol, plan=plan)
    return (res, nit, a, st, sym), (ro, no, b)


CASES = [((12, 24, 16), 288, 16), ((12, 24, 16), 160, 16), ((10, 20, 12), 320, 8),
         ((7, 9, 11), 64, 16), ((9, 11, 13), 96, 7), ((5, 1, 9), 64, 4), ((5, 2, 9), 64, 3),
         ((1, 30, 7), 64, 8), ((6, 10, 1), 64, 2), ((1, 1, 33), 64, 16), ((13, 17, 5), 64, 16),
         ((16, 25, 24), 608, 16), ((18, 36, 24), 512, 16), ((11, 19, 20), 384, 6)]


@pytest.mark.parametrize("dims,block,cluster", CASES)
@pytest.mark.parametrize("form", ["symmetric", "general"])
def test_pushed_form_matches_oracle(dims, block, cluster, form):
    g = gen()
    s = g.make_system(*dims, 8, seed=3)
    if form == "general":
        s.aE[2:-2, 2:-2, 2:-2] *= 1.0 + 1e-13
        s.aW[2:-2, 2:-2, 2] = 0.25  # a wall link: multiplies the zero halo
    phi0 = np.random.default_rng(7).normal(size=g.halo_shape(*dims)) * 1e-3
    for iters in (1, 2, 25):
        (res, nit, a, _, sym), (ro, no, b) = both(s, phi0, block, cluster, iters, 0.0)
        assert (nit, res) == (no, ro)
        assert np.array_equal(a, b)
        if form == "general" and dims[0] > 1:
            assert sym == 0


def test_pushed_form_exits():
    """Convergence, breakdown on a zero right-hand side, non-finite input."""
    g = gen()
    dims = (12, 24, 16)
    s = g.make_system(*dims, 8, seed=1)
    z = g.zeros_phi(*dims)
    for tol in (1e-2, 1e-8):
        (res, nit, a, st, _), (ro, no, b) = both(s, z, 288, 16, 5000, tol)
        assert st == 0 and res < tol and (nit, res) == (no, ro) and np.array_equal(a, b)
    s.Su[...] = 0.0
    (res, nit, a, _, _), (ro, no, b) = both(s, z, 288, 16, 50, 1e-8)
    assert (nit, res) == (no, ro) == (0, 0.0) and np.array_equal(a, b)
    s = g.make_system(*dims, 8, seed=1)
    s.Su[6, 7, 8] = np.inf
    (res, nit, a, _, _), (ro, no, b) = both(s, z, 288, 16, 9, 1e-8)
    assert nit == no and np.isnan(res) == np.isnan(ro) and np.array_equal(a, b, equal_nan=True)
