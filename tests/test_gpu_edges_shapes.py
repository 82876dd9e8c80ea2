"""The launch-shape fields of the edge parameters ask for the work queue, also
on batches that run one block per edge without them; against the plain path,
bit for bit. (The workspace begins with the queue's item counter.)"""
import numpy as np
import pytest

from conftest import golden_asset
from prismplan_b200 import workloads

pytestmark = pytest.mark.gpu

COUNTS = np.array([0, 1, 15, 16, 31, 32, 33, 64, 65, 129, 257, 600, 1500])


@pytest.mark.parametrize("n", [3, 64, 129, 1024, 2049])
@pytest.mark.parametrize("robot,esdf,self_check", [("panda", 0, False), ("panda", 0, True), ("baxter", 64, True)])
def test_shape_fields(golden, n, robot, esdf, self_check):
    import torch

    from prismplan_b200 import api
    from prismplan_b200.robot import RobotModelBuilder
    from prismplan_b200.scene import SceneTensors

    asset = golden_asset(golden, robot)[0]
    b = RobotModelBuilder.from_asset(asset).build()
    rng = np.random.default_rng(n)
    d, p, e = workloads.random_obbs(rng, 60, -1.2, 1.2, 0.02, 0.1)
    keep = np.linalg.norm(p[:, :3], axis=1) > 0.8
    scene = SceneTensors(d[keep], p[keep], e[keep], *(workloads.random_esdf(rng, n_vox=esdf) if esdf else ()))
    frm, to, _ = workloads.edge_batch(rng, asset, n)
    f, t = torch.from_numpy(frm).cuda(), torch.from_numpy(to).cuda()
    g = torch.from_numpy(COUNTS[rng.integers(0, len(COUNTS), n)].astype(np.int32)).cuda()
    g[0] = 40
    want = api.check_edges(b, scene, f, t, samples=g, params=api.EdgeEvalParams(check_self=self_check), persistent=False)
    ws = api.edges_workspace(n)
    for shape in ({}, {"probe": 1}, {"probe": 2}, {"queue_blocks_per_sm": 2}, {"grab": 1}, {"grab": 32, "probe": 2}):
        params = api.EdgeEvalParams(check_self=self_check, **shape)
        got = api.check_edges(b, scene, f, t, samples=g, params=params, workspace=ws)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
        if shape or n > 2048:
            assert int(ws[:8].view(torch.int64)) > 0, shape   # the queue ran
        elif n <= 64:
            assert int(ws[:8].view(torch.int64)) == 0


def test_tuned_small_batch(golden):
    import torch

    from prismplan_b200 import api
    from prismplan_b200.robot import RobotModelBuilder
    from prismplan_b200.scene import SceneTensors

    asset = golden_asset(golden, "panda")[0]
    b = RobotModelBuilder.from_asset(asset).build()
    rng = np.random.default_rng(1)
    scene = SceneTensors(*workloads.random_obbs(rng, 16, 0.9, 1.4, 0.02, 0.1))
    frm, to, _ = workloads.edge_batch(rng, asset, 200)
    f, t = torch.from_numpy(frm).cuda(), torch.from_numpy(to).cuda()
    p = api.EdgeEvalParams(max_joint_step=0.02, check_self=True)
    tuned, info = api.tune_edges(b, scene, f, t, params=p)
    assert info["candidates"] >= 10
    assert (info["queue_blocks_per_sm"] == 0) == (info["best_ms"] == info["default_ms"])
    # every candidate is a shape of its own: the queue takes some times as long here (110 us against 35)
    assert info["queue_blocks_per_sm"] == 0
    a, c = (api.check_edges(b, scene, f, t, params=x) for x in (tuned, p))
    assert torch.equal(a[0], c[0]) and torch.equal(a[1], c[1])
