"""Which form of the cluster-resident kernel ran, as the handle reports it: the
pushed one where a thread's cells fit its registers, the others where they do not
or where they are asked for."""
import numpy as np
import pytest

from conftest import gen, pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,block,cluster,mode,ran", [
    ((12, 24, 16), None, None, 1, "RAN_PUSHED"),           # the tuned launch
    ((12, 24, 16), 288, 16, 1, "RAN_PUSHED"),              # one cell a thread
    ((12, 24, 16), 160, 16, 1, "RAN_PUSHED"),              # two
    ((12, 24, 16), 64, 16, 1, "RAN_CLUSTER_BARRIER"),      # five
    ((20, 40, 30), 1024, 16, 1, "RAN_CLUSTER_BARRIER"),    # blocks without the registers
    ((12, 24, 16), 288, 16, 2, "RAN_MBARRIER"),
    ((12, 24, 16), 288, 16, 0, "RAN_NOT_RESIDENT"),
    ((30, 44, 24), None, None, 1, "RAN_NOT_RESIDENT")])    # beyond a cluster
def test_form(dims, block, cluster, mode, ran):
    import oracle
    eaf, g = pkg(), gen()
    s = g.make_system(*dims, 8, seed=1)
    a, b = g.zeros_phi(*dims), g.zeros_phi(*dims)
    with eaf.CGSolver(*dims) as cg:
        assert cg.last_resident() == cg.RAN_NOT_RESIDENT
        if block:
            cg.set_launch(block, cluster)
            cg.set_cluster(cluster)
        cg.set_resident(mode)
        res, nit, _ = cg.solve(s.arrays(), a, 9, 0.0)
        assert cg.last_resident() == getattr(cg, ran)
        plan = cg.last_launch()
    assert (res, nit) == oracle.cg(s, b, 9, 0.0, plan=plan)
    assert np.array_equal(a, b)
