"""CHOMP's update with several DoFs of a request in a block (large batches)
against a block per DoF (the same requests a few at a time): the same bits."""
import numpy as np
import pytest

from conftest import golden_asset
from prismplan_b200 import workloads

pytestmark = pytest.mark.gpu


# 7 DoFs in blocks of 4 + 3, 7, 3 + 3 + 1, and as many as fit beside long columns; 15 and 8 DoFs
@pytest.mark.parametrize("robot,B,T", [("panda", 150, 33), ("panda", 300, 64), ("panda", 100, 17), ("panda", 300, 700),
                                       ("baxter", 150, 40), ("fetch", 290, 2)])
def test_update_groups_same_bits(golden, robot, B, T):
    import torch

    from prismplan_b200 import api
    from prismplan_b200.robot import RobotModelBuilder
    from prismplan_b200.scene import SceneTensors

    asset, _ = golden_asset(golden, robot)
    b = RobotModelBuilder.from_asset(asset).build()
    rng = np.random.default_rng(B + T)
    sc = SceneTensors(*workloads.random_obbs(rng, 6))
    th = torch.from_numpy(workloads.straight_trajectories(rng, asset, B, T).astype(np.float32)).cuda()
    s = api.ChompSettings(num_iterations=4, num_iterations_after_valid=10 ** 6, convergence_eps=0.0, time_limit_ms=0.0)
    whole = api.chomp_optimize(b, sc, th.clone(), s).theta
    moved = float((whole - th).abs().max())
    assert T == 2 or moved > 0.0
    for part in (slice(0, 5), slice(B // 2, B // 2 + 3), slice(B - 4, B)):
        alone = api.chomp_optimize(b, sc, th[part].clone(), s).theta
        assert torch.equal(whole[part].view(torch.int32), alone.view(torch.int32)), part
