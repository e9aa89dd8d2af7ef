"""The batch's tables travel on the batch's own stream. That stream is
non-blocking, so a copy on the default stream is not ordered before the graph
that reads the table, and it waits for whatever else the program runs there."""
import os
import re

import numpy as np
import pytest

from conftest import ROOT, gen, pkg


# (the server's streams are non-blocking too)
@pytest.mark.parametrize("unit", ["batch.cu", "serve.cu"])
def test_no_copy_on_the_default_stream(unit):
    with open(os.path.join(ROOT, "hornofusion-full3d_b200", "csrc", unit)) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    assert "cudaStreamNonBlocking" in code
    assert re.findall(r"\bcuda(?:Memcpy|Memset)\s*\(", code) == []


@pytest.mark.gpu
def test_new_arrays_beside_a_busy_default_stream():
    """A solve of other device arrays (its tables are uploaded again) neither
    waits for the default stream nor touches the arrays it was given before."""
    import oracle
    import torch
    eaf, g = pkg(), gen()
    dims = [(9, 10, 7), (12, 24, 16), (3, 2, 5)]
    sets = []
    for seed in (1, 2):
        sl = [g.make_system(*d, 4, seed=seed + 10 * k) for k, d in enumerate(dims)]
        dev = [[torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in s.arrays()] for s in sl]
        phi = [torch.zeros(g.halo_shape(*d), dtype=torch.float64, device="cuda") for d in dims]
        sets.append((sl, dev, phi))
    src = torch.empty(1 << 28, dtype=torch.uint8, pin_memory=True)
    dst = torch.empty_like(src, device="cuda")
    done = torch.cuda.Event()
    torch.cuda.synchronize()
    with eaf.Batch(dims) as b:
        for sl, dev, phi in sets:
            for k in range(len(dims)):
                b.set_system(k, dev[k], phi[k], device_ptrs=True)
            if sl is sets[1][0]:
                before = [p.clone() for p in sets[0][2]]
                torch.cuda.synchronize()
                for _ in range(160):  # 43 GB over PCIe, well beyond the solve's time
                    dst.copy_(src, non_blocking=True)
                done.record()
            b.solve(False, 20, 0.0)
        assert not done.query()
        plans = [b.system_plan(k) for k in range(len(dims))]
    torch.cuda.synchronize()
    for (sl, _, phi), got in zip(sets, (before, sets[1][2])):
        for k, s in enumerate(sl):
            want = g.zeros_phi(*dims[k])
            oracle.cg(s, want, 20, 0.0, plan=plans[k])
            assert np.array_equal(phi[k].cpu().numpy(), want)
            assert np.array_equal(got[k].cpu().numpy(), want)
