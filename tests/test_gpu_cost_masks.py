"""Costs under allowed-collision masks on models whose joints' sphere counts
leave lanes of a waypoint's group without a sphere (the last joint above all:
there is no mask row past it): all-ones masks change nothing."""
import numpy as np
import pytest

from conftest import golden_asset
from prismplan_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("robot", ["panda", "fetch", "baxter"])
def test_all_ones_masks_change_no_cost(golden, robot):
    import torch

    from prismplan_b200 import api
    from prismplan_b200.robot import RobotModelBuilder
    from prismplan_b200.scene import SceneTensors

    asset, _ = golden_asset(golden, robot)
    b = RobotModelBuilder.from_asset(asset).build()
    rng = np.random.default_rng(5)
    boxes = workloads.random_obbs(rng, 21)
    ones = np.ones((len(b.sphere_to_joint), 21), np.uint8)
    q = torch.from_numpy(workloads.straight_trajectories(rng, asset, 7, 13)).cuda()
    a = api.traj_cost(b, SceneTensors(*boxes), q)
    m = api.traj_cost(b, SceneTensors(*boxes, sphere_obb_acm_mask=ones), q)
    for x, y in zip(a, m):
        assert torch.equal(x, y)
