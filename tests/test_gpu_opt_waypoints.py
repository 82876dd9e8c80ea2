"""A waypoint is checked whatever its neighbours hold: seeds whose second or
last but one waypoint is not finite, against the separate waypoint and segment checks
(all-ones allowed-collision masks select those)."""
import numpy as np
import pytest

from conftest import golden_asset
from prismplan_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("T", [3, 40])
@pytest.mark.parametrize("at", [0, -1])
def test_end_beside_a_bad_waypoint(golden, value, T, at):
    import torch

    from prismplan_b200 import api
    from prismplan_b200.robot import RobotModelBuilder
    from prismplan_b200.scene import SceneTensors

    asset, _ = golden_asset(golden, "panda")
    b = RobotModelBuilder.from_asset(asset).build()
    rng = np.random.default_rng(T)
    boxes = workloads.random_obbs(rng, 24, -1.0, 1.0, 0.02, 0.1)
    plain = SceneTensors(*boxes)
    masked = SceneTensors(*boxes, sphere_obb_acm_mask=np.ones((len(b.sphere_to_joint), 24), np.uint8))
    q = workloads.uniform_configs(rng, asset, 4000)
    hit = api.check_configs(b, plain, torch.from_numpy(q).cuda())[0].cpu().numpy() == 1
    theta = np.repeat(q[~hit][:4, None], T, 1)
    theta[:2, at] = q[hit][:2]                            # two requests start (or end) in collision
    theta[[0, 2], 1 if at == 0 else T - 2, 0] = value     # of each kind one with a bad waypoint beside it
    s = api.ChompSettings(num_timesteps=T, num_iterations=1, check_self=False, time_limit_ms=0.0)
    r, m = (api.chomp_optimize(b, scene, torch.from_numpy(theta).cuda(), s) for scene in (plain, masked))
    assert torch.equal(r.solved, m.solved)
    assert not bool(r.solved[:2].any())
    assert torch.equal(r.iterations, m.iterations)
