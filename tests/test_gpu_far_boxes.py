"""Boxes whose extents are beyond what FP32 can square (half-spaces): the culls
must not drop them. Against the generic kernels (all-ones allowed-collision
masks select them, and change no pair), bit for bit."""
import numpy as np
import pytest

from conftest import golden_asset
from prismplan_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("extent", [1e14, 1e16, 1e20, 1e25, 1e30])
@pytest.mark.parametrize("n", [9, 4737, 33153])   # 16, 4 and 1 lanes a configuration; edges of both routes
def test_half_space(golden, extent, n):
    import torch

    from prismplan_b200 import api
    from prismplan_b200.robot import RobotModelBuilder
    from prismplan_b200.scene import SceneTensors, pack_obbs

    asset, _ = golden_asset(golden, "panda")
    b = RobotModelBuilder.from_asset(asset).build()
    rng = np.random.default_rng(n)
    small = workloads.random_obbs(rng, 5, -1.5, 1.5, 0.02, 0.05)
    turn = rng.normal(size=4)
    large = pack_obbs(np.full((2, 3), 2 * extent), np.array([[0.0, 0.0, -extent], [-extent, extent, 0.0]]),
                      np.array([[1.0, 0.0, 0.0, 0.0], turn / np.linalg.norm(turn)]))
    boxes = [np.concatenate(x) for x in zip(small, large)]
    fast = SceneTensors(*boxes)
    generic = SceneTensors(*boxes, sphere_obb_acm_mask=np.ones((len(b.sphere_to_joint), 7), np.uint8))
    q = torch.from_numpy(workloads.uniform_configs(rng, asset, n)).cuda()
    for clearance in (None, "obb"):
        a, g = (api.check_configs(b, s, q, 0.0, clearance) for s in (fast, generic))
        assert torch.equal(a[0], g[0])
        if clearance:
            assert torch.equal(a[1].view(torch.int32), g[1].view(torch.int32))
    m = min(n, 3000)
    f, t = (torch.from_numpy(x).cuda() for x in workloads.edge_batch(rng, asset, m)[:2])
    params = api.EdgeEvalParams(granularity=40)
    assert torch.equal(*(api.check_edges(b, s, f, t, params=params)[0] for s in (fast, generic)))
    assert torch.equal(*(api.check_edges(b, s, f, t, params=params, persistent=False)[0] for s in (fast, generic)))
