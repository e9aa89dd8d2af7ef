"""Launch rule of the plain FP64 solve on meshes outside the tuned table: one
block per SM beyond what a cluster holds, own operands kept in shared memory
while they leave the L1 room; the bits are the kernel-order oracle's, and the
no-allocation entry picks the same launch."""
import ctypes

import numpy as np
import pytest

from conftest import gen, pkg

pytestmark = pytest.mark.gpu


# 1 cell beyond 16 x 1,760 (a cluster's capacity is about 28,000), a prime-ish
# mesh, the last and first meshes around the 200 KB a block, and meshes of the
# prefetching kernel (part of the residual kept; a kept residual longer than
# the last block's slice comes with 1024-thread blocks on a smaller mesh)
@pytest.mark.parametrize("dims,kernel,block", [((30, 44, 24), "KEEP", 512),
                                               ((41, 83, 57), "KEEP", 512),
                                               ((69, 139, 98), "KEEP", 512),
                                               ((70, 140, 98), "LOADS", 512),
                                               ((80, 161, 111), "LOADS", 1024)])
def test_untuned_mesh_launch_matches_oracle(dims, kernel, block):
    import oracle
    eaf, g = pkg(), gen()
    s = g.make_system(*dims, 8, seed=3)
    a, b = g.zeros_phi(*dims), g.zeros_phi(*dims)
    with eaf.CGSolver(*dims) as cg:
        res, nit, st = cg.solve(s.arrays(), a, 12, 0.0)
        plan, ran = cg.last_launch(), cg.last_kernel()
        assert ran == getattr(cg, "KERNEL_" + kernel)
    assert plan == (148, block) and st == 0
    assert (res, nit) == oracle.cg(s, b, 12, 0.0, plan=plan)
    assert np.array_equal(a, b)


@pytest.mark.parametrize("iters", [0, 1, 2, 7])
def test_prefetching_kernel_ends_with_its_last_update(iters):
    """The prefetching kernel applies an iteration's update of x in the next
    one: solves that end after any number of iterations, warm-started."""
    import oracle
    eaf, g = pkg(), gen()
    dims = (93, 91, 90)  # 761,670 cells: 1024-thread blocks prefetch
    s = g.make_system(*dims, 8, seed=2)
    a = np.random.default_rng(1).normal(size=g.halo_shape(*dims))
    b = a.copy()
    with eaf.CGSolver(*dims) as cg:
        cg.set_launch(1024, 148)
        res, nit, _ = cg.solve(s.arrays(), a, iters, 0.0)
        plan = cg.last_launch()
    assert (res, nit) == oracle.cg(s, b, iters, 0.0, plan=plan)
    assert np.array_equal(a, b)


def test_noalloc_takes_the_same_launch_beyond_a_cluster():
    torch = pytest.importorskip("torch")
    eaf, g = pkg(), gen()
    dims = (30, 44, 24)
    s = g.make_system(*dims, 8, seed=5)
    dev = [torch.from_numpy(a).cuda() for a in s.arrays()]
    pa = torch.zeros(g.halo_shape(*dims), dtype=torch.float64, device="cuda")
    pb = torch.zeros_like(pa)
    torch.cuda.synchronize()
    with eaf.CGSolver(*dims) as cg:
        res, nit, _ = cg.solve(dev, pa, 60, 1e-8, device_ptrs=True)
    r, n = ctypes.c_double(), ctypes.c_int()
    p = [ctypes.c_void_p(t.data_ptr()) for t in dev + [pb]]
    st = eaf.load().eaf_cg_solve_f64_noalloc(*dims, 0, None, *p, 60, 1e-8, ctypes.byref(r),
                                             ctypes.byref(n))
    assert st == 0 and (r.value, n.value) == (res, nit)
    assert torch.equal(pa, pb)
