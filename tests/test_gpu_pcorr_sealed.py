"""The sealed-cell mean by blocks that list their sealed cells first: bit for
bit the oracle's where a block's list is empty, full or in between, and at halo
sizes around whole tiles of 1,024 elements."""
import numpy as np
import pytest

from conftest import gen
from test_gpu_pcorr import assert_same, run_gpu, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(4, 4, 12), (4, 4, 13), (12, 12, 4), (13, 6, 3), (1, 1, 1),
                                  (28, 4, 28), (30, 31, 29)])
@pytest.mark.parametrize("share", [0.0, 0.02, 0.5, 1.0])
def test_sealed_share(dims, share):
    f = gen().make_pcorr_fields(*dims, seed=5, sealed_frac=0.0)
    sealed = np.random.default_rng(9).random(f.cell_type.shape) < share
    f.act_l[sealed] = 0
    f.act_g[sealed] = 0
    a, t = run_gpu(f)
    assert_same(a, run_oracle(f))
    assert t["kernels"] == 3
