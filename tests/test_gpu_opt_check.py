"""The optimisers' one-block-per-slice validity check against the waypoint and
segment checks that it replaces (all-ones allowed-collision masks select those,
and change no pair): every field of the result bit for bit."""
import numpy as np
import pytest

from conftest import golden_asset
from prismplan_b200 import workloads

pytestmark = pytest.mark.gpu


# waypoints: one short segment slice, slices of exactly 32 segments, one over, several
@pytest.mark.parametrize("T", [2, 3, 33, 34, 65, 100])
@pytest.mark.parametrize("kind,robot,boxes,esdf,self_check", [("chomp", "panda", 12, 0, True), ("chomp", "panda", 10, 0, False),
                                                              ("chomp", "baxter", 10, 64, True),
                                                              ("chomp", "fetch", 14, 0, True), ("stomp", "panda", 12, 0, True)])
def test_solve_equals_separate_checks(golden, T, kind, robot, boxes, esdf, self_check):
    import torch

    from prismplan_b200 import api
    from prismplan_b200.robot import RobotModelBuilder
    from prismplan_b200.scene import SceneTensors

    asset, _ = golden_asset(golden, robot)
    b = RobotModelBuilder.from_asset(asset).build()
    rng = np.random.default_rng(T + boxes)
    d, p, e = workloads.random_obbs(rng, 20 * boxes, -1.3, 1.3, 0.02, 0.15)
    keep = np.linalg.norm(p[:, :3], axis=1) > 1.2   # |t| = distance of the centre from the base: leave it free
    d, p, e = d[keep][:boxes], p[keep][:boxes], e[keep][:boxes]
    ns = len(b.sphere_to_joint)
    ones = {"sphere_obb_acm_mask": np.ones((ns, len(d)), np.uint8)}
    layers = ()
    if esdf:
        layers = workloads.random_esdf(rng, n_vox=esdf, centre=(0.9, 0.0, 0.5))
        ones["sphere_acm_mask"] = np.ones((ns, 1), np.uint8)
    plain, masked = SceneTensors(d, p, e, *layers), SceneTensors(d, p, e, *layers, **ones)

    def is_free(q):
        return api.check_configs(b, plain, torch.from_numpy(q).cuda(), check_self=True)[0].cpu().numpy() == 0

    starts, goals = workloads.free_pairs(rng, asset, 6, is_free, 64)
    goals[0] = starts[0] + 0.01                      # a request that is valid at once
    if kind == "chomp":
        s = api.ChompSettings(num_timesteps=T, num_iterations=12, check_self=self_check, time_limit_ms=0.0)
        solve = api.chomp_solve
    else:
        s = api.StompSettings(num_timesteps=T, num_iterations=5, check_self=self_check, time_limit_ms=0.0)
        solve = api.stomp_solve
    r, m = (solve(b, sc, starts, goals, s) for sc in (plain, masked))
    for name in ("solved", "iterations", "cost", "path", "theta"):
        x, y = getattr(r, name), getattr(m, name)
        assert torch.equal(x, y), name
