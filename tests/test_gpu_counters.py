"""The work counters (ps_set_stats) credit work that was needed and done: no
lanes that repeat a sample, no pairs that repeat a pair."""
import ctypes as C

import numpy as np
import pytest

from prismplan_b200 import _lib, workloads

pytestmark = pytest.mark.gpu

PAIRS, EXACT, SAMPLES, JOINTS, SPHERES, SELF, ESDF, CULL = range(8)


def _counted(run):
    import torch

    st = torch.zeros(8, dtype=torch.int64, device="cuda")
    _lib.load().ps_set_stats(C.c_void_p(st.data_ptr()))
    try:
        out = run()
        torch.cuda.synchronize()
    finally:
        _lib.load().ps_set_stats(None)
    return st.cpu().tolist(), out


@pytest.mark.parametrize("G,nodes", [(256, 64), (264, 66), (384, 96), (400, 100)])   # a node is 4 samples
def test_coarse_pass(G, nodes):
    import torch

    from prismplan_b200 import api
    from prismplan_b200.robot import RobotModelBuilder
    from prismplan_b200.scene import SceneTensors, pack_obbs

    asset = workloads.panda_like()
    b = RobotModelBuilder.from_asset(asset).build()
    scene = SceneTensors(*pack_obbs(np.array([[0.1, 0.1, 0.1]]), np.array([[6.0, 0.0, 0.0]]), np.array([[1.0, 0.0, 0.0, 0.0]])))
    n = 40000                                         # enough for the probe and the one-pass queue
    frm, to, _ = workloads.edge_batch(np.random.default_rng(G), asset, n)
    f, t = torch.from_numpy(frm).cuda(), torch.from_numpy(to).cuda()
    g = torch.full((n,), G, dtype=torch.int32, device="cuda")
    st, out = _counted(lambda: api.check_edges(b, scene, f, t, samples=g))
    assert bool(out[0].all())
    assert st[SAMPLES] == n * (nodes + 1)             # and the end-sample probe
    assert st[JOINTS] == st[SAMPLES] * (asset["n_joints"] - 1)
    assert st[PAIRS] == st[SPHERES] == 0              # nothing in reach


@pytest.mark.parametrize("n", [1, 500])
def test_approximate_self_pairs(n):
    import torch

    from prismplan_b200 import api
    from prismplan_b200.robot import RobotModelBuilder

    asset = workloads.generic_chain(n_links=7, spheres_per_link=1)
    asset["spheres_flat"] = [v if k % 4 < 3 else 1e-4 for k, v in enumerate(asset["spheres_flat"])]
    asset = workloads._finish(asset)                  # its approximate spheres are as small, so none overlap
    b = RobotModelBuilder.from_asset(asset).build()
    q = torch.from_numpy(workloads.uniform_configs(np.random.default_rng(n), asset, n)).cuda()
    st, out = _counted(lambda: api.check_configs(b, None, q, check_self=True))
    r = np.asarray(asset["approx_self_cc_ranges_flat"]).reshape(-1, 3)
    assert not bool(out[0].any())
    assert st[SELF] == n * int((r[:, 2] - r[:, 1] + 1).sum())
