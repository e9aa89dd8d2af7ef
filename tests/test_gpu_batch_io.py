"""Pack and unpack of all systems of a batch in one launch each: bit for bit
the single-system solver's (whole halo array) for meshes of less than one
block, odd sizes and several blocks, asymmetric beside symmetric ones; systems
that share one phi end with the last one's values."""
import numpy as np
import pytest

from conftest import gen, pkg

pytestmark = pytest.mark.gpu

MESHES = [(1, 1, 1), (3, 2, 5), (8, 4, 8), (7, 11, 5), (12, 24, 16), (16, 16, 1)]


def systems():
    g = gen()
    out = []
    for k, d in enumerate(MESHES):
        s = g.make_system(*d, 4, seed=k)
        if k % 2:
            s.aE[2:-2, 2:-2, 2:-2] *= 1.0 + 1e-12
        phi = np.random.default_rng(k).normal(size=g.halo_shape(*d)) * 1e-3
        out.append((s, phi))
    return out


@pytest.mark.parametrize("order", [1, -1])
def test_batch_matches_oracle(order):
    import oracle
    eaf = pkg()
    sl = systems()[::order]
    with eaf.Batch([(s.nr, s.nth, s.nz) for s, _ in sl]) as b:
        phis = [p.copy() for _, p in sl]
        for k, (s, _) in enumerate(sl):
            b.set_system(k, s.arrays(), phis[k])
        b.solve(False, 12, 0.0)
        for k, (s, p) in enumerate(sl):
            want = p.copy()
            with np.errstate(all="ignore"):
                ro, no = oracle.cg(s, want, 12, 0.0, plan=b.system_plan(k))
            got = b.get_phi(k, np.empty_like(p))
            assert b.result(k)[:2] == (ro, no)
            assert np.array_equal(got, want), MESHES[::order][k]


def test_shared_phi_keeps_the_last_system():
    import torch
    eaf = pkg()
    g = gen()
    d = (9, 10, 7)
    s = [g.make_system(*d, 4, seed=k) for k in (1, 2)]
    dev = [[torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in x.arrays()] for x in s]
    phi0 = np.zeros(g.halo_shape(*d))
    alone = torch.from_numpy(phi0.copy()).cuda()
    with eaf.Batch([d]) as b:
        b.set_system(0, dev[1], alone, device_ptrs=True)
        b.solve(False, 20, 0.0)
    both = torch.from_numpy(phi0.copy()).cuda()
    with eaf.Batch([d, d]) as b:
        for k in range(2):
            b.set_system(k, dev[k], both, device_ptrs=True)
        b.solve(False, 20, 0.0)
    assert torch.equal(alone, both)
