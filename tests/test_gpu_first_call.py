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


def test_calls_of_one_handle_in_any_order():
    """Host-array solves and assemblies by turns on one handle (the assembly's
    scratch is the solves' upload area): a new handle's results every time."""
    eaf, g = pkg(), gen()
    dims = (17, 26, 19)
    s = g.make_system(*dims, 8, seed=2)
    f = g.make_assembly_fields(*dims, seed=3)

    def solve(cg):
        phi = g.zeros_phi(*dims)
        return cg.solve(s.arrays(), phi, 30, 0.0)[:2], {"phi": phi}

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

    calls = [solve, assemble, assemble_device]
    want = [alone(c) for c in calls]
    with eaf.CGSolver(*dims) as cg:
        for k in (0, 1, 0, 2, 2, 0, 1, 2, 1, 0):
            got = calls[k](cg)
            assert got[0] == want[k][0]
            assert all(np.array_equal(got[1][n], want[k][1][n]) for n in want[k][1])
