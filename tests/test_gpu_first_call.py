"""What a handle allocates in its first calls, and that the calls which share the
handle's memory leave nothing behind for each other."""
import numpy as np
import pytest

from conftest import gen, pkg

pytestmark = pytest.mark.gpu


def grown(call):
    """Device memory that a call takes, in bytes."""
    import torch
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    call()
    return before - torch.cuda.mem_get_info()[0]


def load_sweep_kernels():
    """Sweeps of a small mesh first: a kernel's first launch may take memory too."""
    g = gen()
    s = g.make_transport_system(12, 24, 16, seed=4)
    with pkg().CGSolver(12, 24, 16) as cg:
        cg.tdma(s.arrays(), g.zeros_phi(12, 24, 16), 2)


def fill_device(leave):
    """Tensors that take the device's free memory but about `leave` bytes."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held, step = [], 1 << 60
    while torch.cuda.mem_get_info()[0] > leave + (16 << 20) and step > (1 << 20):
        step = min(step, torch.cuda.mem_get_info()[0] - leave)
        try:
            held.append(torch.empty(step, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            step //= 2
    return held


def on_device(f):
    import torch
    dev = f.copy()
    for k, v in list(dev.__dict__.items()):
        if isinstance(v, np.ndarray):
            setattr(dev, k, torch.from_numpy(v).cuda())
    return dev


def test_assembly_scratch():
    """The device assembly's first call takes fewer than 15 halo arrays."""
    eaf, g = pkg(), gen()
    f = on_device(g.make_assembly_fields(60, 120, 84, seed=1))
    nh = 64 * 124 * 88
    with eaf.CGSolver(60, 120, 84) as cg:
        first = grown(lambda: cg.pressure_assemble(f, device_ptrs=True))
        assert 12 * 8 * nh < first < 15 * 8 * nh
        assert grown(lambda: cg.pressure_assemble(f, device_ptrs=True)) == 0


def test_transport_scratch():
    """One sweep needs no memory of its own, several at most 21 doubles a cell."""
    import torch
    eaf, g = pkg(), gen()
    dims = (60, 120, 84)
    s = g.make_transport_system(*dims, seed=1)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in s.arrays()]
    phi = torch.zeros(g.halo_shape(*dims), dtype=torch.float64, device="cuda")
    load_sweep_kernels()
    with eaf.CGSolver(*dims) as cg:
        for _ in range(2):
            assert grown(lambda: cg.tdma(dev, phi, 1, device_ptrs=True)) == 0
        assert grown(lambda: cg.tdma(dev, phi, 3, device_ptrs=True)) < 21 * 8 * 604800
        assert grown(lambda: cg.tdma(dev, phi, 2, device_ptrs=True)) == 0


def sweeps(dims, phi0, counts, s):
    """phi after sweeps by `counts` on one handle, its kernels, and the oracle's."""
    import oracle
    import torch
    eaf = pkg()
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in s.arrays()]
    a, b = torch.from_numpy(phi0.copy()).cuda(), phi0.copy()
    kernels = []
    with eaf.CGSolver(*dims) as cg:
        for n in counts:
            cg.tdma(dev, a, n, device_ptrs=True)
            kernels.append(cg.last_timing()["kernels"])
            oracle.tdma_3d(s, b, n)
    return a.cpu().numpy(), kernels, b


# (thin meshes, whose scratch is larger than the solver's arrays, among them)
@pytest.mark.parametrize("dims", [(12, 24, 16), (1, 40, 30), (3, 50, 2), (140, 9, 21)])
def test_sweeps_by_turns(dims):
    g = gen()
    s = g.make_transport_system(*dims, seed=4)
    phi0 = np.random.default_rng(2).normal(size=g.halo_shape(*dims))
    a, kernels, b = sweeps(dims, phi0, (1, 3, 1, 2), s)
    assert kernels == [9, 21, 9, 15]
    assert np.array_equal(a, b)


def test_records_built_again_without_room():
    """Several sweeps where the device has no room for all directions' records."""
    import oracle
    import torch
    eaf, g = pkg(), gen()
    dims = (60, 120, 84)
    s = g.make_transport_system(*dims, seed=4)
    phi0 = np.random.default_rng(2).normal(size=g.halo_shape(*dims))
    load_sweep_kernels()

    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in s.arrays()]
    a, b = torch.from_numpy(phi0.copy()).cuda(), phi0.copy()
    with eaf.CGSolver(*dims) as cg:
        held = fill_device(64 << 20)
        assert torch.cuda.mem_get_info()[0] < 90 << 20  # (the records need 94 MB)
        cg.tdma(dev, a, 3, device_ptrs=True)
        assert cg.last_timing()["kernels"] == 27
        del held
        torch.cuda.empty_cache()
        cg.tdma(dev, a, 2, device_ptrs=True)
        assert cg.last_timing()["kernels"] == 15
    oracle.tdma_3d(s, b, 3)
    oracle.tdma_3d(s, b, 2)
    assert np.array_equal(a.cpu().numpy(), b)


@pytest.mark.parametrize("dims", [(17, 26, 19), (40, 41, 42)])
@pytest.mark.parametrize("form", ["auto", "LOADS", "STREAM", "SLOTS", "KEEP", "one", "mixed",
                                  "resident", "mbarrier", "cluster"])
def test_solves_after_sweeps(dims, form):
    """The sweeps' scratch is the solver's arrays: every solver on a handle that
    has swept gives a new handle's bits."""
    eaf, g = pkg(), gen()
    s = g.make_system(*dims, 8, seed=2)
    t = g.make_transport_system(*dims, seed=3)

    def solve(sweep):
        phi = np.random.default_rng(4).normal(size=g.halo_shape(*dims)) * 1e-3
        with eaf.CGSolver(*dims) as cg:
            if form in ("LOADS", "STREAM", "SLOTS", "KEEP"):
                cg.set_launch(256, 60)
                cg.set_kernel(getattr(cg, "KERNEL_" + form))
            elif form == "one":
                cg.set_form(cg.FORM_ONE_REDUCTION)
            elif form in ("resident", "mbarrier"):
                cg.set_launch(1024, 16)
                cg.set_cluster(16)
                cg.set_resident(2 if form == "mbarrier" else 1)
            elif form == "cluster":
                cg.set_launch(256, 64)
                cg.set_cluster(4)
            if sweep:
                for n in (1, 2):
                    q = np.random.default_rng(n).normal(size=phi.shape)
                    cg.tdma(t.arrays(), q, n)
            if form == "mixed":
                r = cg.solve_mixed(s.arrays(), phi, tol=1e-12, inner_tol=0.1, max_outer=5,
                                   max_inner=40)
            else:
                r = cg.solve(s.arrays(), phi, 30, 0.0)
        return r, phi

    (ra, a), (rb, b) = solve(False), solve(True)
    assert ra == rb and np.array_equal(a, b)


def test_calls_of_one_handle_in_any_order():
    """Host-array solves, sweeps and assemblies by turns on one handle (scratch of
    the one is the other's working area): a new handle's results every time."""
    eaf, g = pkg(), gen()
    dims = (17, 26, 19)
    s = g.make_system(*dims, 8, seed=2)
    t = g.make_transport_system(*dims, seed=5)
    f = g.make_assembly_fields(*dims, seed=3)

    def solve(cg):
        phi = g.zeros_phi(*dims)
        return cg.solve(s.arrays(), phi, 30, 0.0)[:2], {"phi": phi}

    def sweep(cg):
        phi = g.zeros_phi(*dims)
        cg.tdma(t.arrays(), phi, 2)
        return cg.residual(t.arrays(), phi), {"phi": phi}

    def assemble(cg):
        out = f.copy()
        return cg.pressure_assemble(out), out.outputs()

    def assemble_device(cg):
        dev, out = on_device(f), f.copy()
        res = cg.pressure_assemble(dev, device_ptrs=True)
        for k in out.outputs():
            setattr(out, k, getattr(dev, k).cpu().numpy())
        return res, out.outputs()

    def alone(call):
        with eaf.CGSolver(*dims) as cg:
            return call(cg)

    calls = [solve, assemble, assemble_device, sweep]
    want = [alone(c) for c in calls]
    with eaf.CGSolver(*dims) as cg:
        for k in (0, 1, 0, 3, 2, 2, 3, 0, 1, 3, 1, 2, 1, 0):
            got = calls[k](cg)
            assert got[0] == want[k][0]
            assert all(np.array_equal(got[1][n], want[k][1][n]) for n in want[k][1])
