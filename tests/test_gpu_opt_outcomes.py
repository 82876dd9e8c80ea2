"""The optimisers' validity check where it decides something: requests that are
free at once, that become free after some iterates, and that never do, against
the separate waypoint and segment checks (all-ones allowed-collision masks
select those): every field bit for bit."""
import numpy as np
import pytest

from conftest import golden_asset
from prismplan_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,iterations", [("chomp", 40), ("stomp", 8)])
@pytest.mark.parametrize("esdf", [0, 64])
def test_outcomes(golden, kind, iterations, esdf):
    import torch

    from prismplan_b200 import api
    from prismplan_b200.robot import RobotModelBuilder
    from prismplan_b200.scene import SceneTensors

    asset = golden_asset(golden, "panda")[0]
    b = RobotModelBuilder.from_asset(asset).build()
    rng = np.random.default_rng(11)
    d, p, e = workloads.random_obbs(rng, 200, -1.0, 1.0, 0.02, 0.12)
    keep = np.linalg.norm(p[:, :3], axis=1) > 0.6    # |t| = distance of the centre from the base: leave it free
    d, p, e = d[keep][:14], p[keep][:14], e[keep][:14]
    ones = {"sphere_obb_acm_mask": np.ones((len(b.sphere_to_joint), 14), np.uint8)}
    layers = ()
    if esdf:
        layers = workloads.random_esdf(rng, n_vox=esdf, centre=(0.5, 0.3, 0.5))
        ones["sphere_acm_mask"] = np.ones((len(b.sphere_to_joint), 1), np.uint8)
    plain, masked = SceneTensors(d, p, e, *layers), SceneTensors(d, p, e, *layers, **ones)
    starts, goals = workloads.free_pairs(
        rng, asset, 64, lambda q: api.check_configs(b, plain, torch.from_numpy(q).cuda(), check_self=True)[0].cpu().numpy() == 0, 32)
    goals[:4] = starts[:4] + 0.01
    after = 3
    s = {"chomp": api.ChompSettings, "stomp": api.StompSettings}[kind](
        num_timesteps=45, num_iterations=iterations, num_iterations_after_valid=after, time_limit_ms=0.0)
    r, m = ({"chomp": api.chomp_solve, "stomp": api.stomp_solve}[kind](b, sc, starts, goals, s) for sc in (plain, masked))
    for name in ("solved", "iterations", "cost", "path", "theta"):
        assert torch.equal(getattr(r, name), getattr(m, name)), name
    late = r.solved & (r.iterations > after)
    print(kind, esdf, int(r.solved.sum()), int(late.sum()))
    assert 0 < int(r.solved.sum()) < 64 and int(late.sum()) > 0
