"""Kept operands with one cell a thread (two blocks of different solves may
share an SM): bit for bit the kernel-order oracle's around the largest slice of
one cell a thread, on odd blocks and meshes, symmetric and not, and by handles
that solve at the same time."""
import threading

import numpy as np
import pytest

from conftest import gen, pkg

pytestmark = pytest.mark.gpu


# slices of 512 cells, of 513 (the next variant), of fewer cells than threads
# with empty last blocks, of one cell
@pytest.mark.parametrize("dims,block,grid", [((32, 64, 37), 512, 148), ((32, 64, 37), 512, 147),
                                             ((9, 11, 13), 512, 148), ((5, 7, 3), 512, 148),
                                             ((30, 44, 24), 288, 111), ((17, 31, 29), 416, 37)])
@pytest.mark.parametrize("form", ["symmetric", "general"])
def test_one_cell_a_thread(dims, block, grid, form):
    import oracle
    eaf, g = pkg(), gen()
    s = g.make_system(*dims, 8, seed=6)
    if form == "general":
        s.aE[2:-2, 2:-2, 2:-2] *= 1.0 + 1e-13
    a = np.random.default_rng(3).normal(size=g.halo_shape(*dims)) * 1e-3
    b = a.copy()
    with eaf.CGSolver(*dims) as cg:
        cg.set_launch(block, grid)
        cg.set_kernel(cg.KERNEL_KEEP)
        res, nit, _ = cg.solve(s.arrays(), a, 21, 0.0)
        plan = cg.last_launch()
        assert plan == (grid, block) and cg.last_kernel() == cg.KERNEL_KEEP
    assert (res, nit) == oracle.cg(s, b, 21, 0.0, plan=plan)
    assert np.array_equal(a, b)


def test_an_sm_holds_one_block_of_a_solve():
    """A larger grid is cut to a block per SM, whatever the kept variant's
    registers leave room for."""
    eaf, g = pkg(), gen()
    s = g.make_system(32, 64, 37, 8, seed=6)
    with eaf.CGSolver(32, 64, 37) as cg:
        cg.set_launch(512, 296)
        cg.set_kernel(cg.KERNEL_KEEP)
        cg.solve(s.arrays(), g.zeros_phi(32, 64, 37), 3, 0.0)
        assert cg.last_launch() == (148, 512) and cg.last_kernel() == cg.KERNEL_KEEP


def test_handles_at_the_same_time():
    import oracle
    eaf, g = pkg(), gen()
    dims = (30, 44, 24)
    got = [None] * 4

    def run(t):
        s = g.make_system(*dims, 8, seed=t)
        out = []
        with eaf.CGSolver(*dims) as cg:
            for _ in range(5):
                phi = g.zeros_phi(*dims)
                out.append((cg.solve(s.arrays(), phi, 60, 0.0)[:2], phi, cg.last_launch()))
        got[t] = (s, out)

    threads = [threading.Thread(target=run, args=(t,)) for t in range(len(got))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s, out in got:
        want = g.zeros_phi(*dims)
        r = oracle.cg(s, want, 60, 0.0, plan=out[0][2])
        for res, phi, _ in out:
            assert res == r and np.array_equal(phi, want)
