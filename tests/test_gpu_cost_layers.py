"""Cost kernels without ESDF lookups (scenes without layers) and with them: a
layer out of every sphere's reach changes no bit, in trajectory costs and
gradients, rollouts and batches of both layouts and all widths, with edges and
without; and with a layer in reach a batch without edges still sees it."""
import numpy as np
import pytest

from conftest import golden_asset
from prismplan_b200 import _lib, workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [_lib.PS_ESDF_NEAREST, _lib.PS_ESDF_TRILINEAR])
@pytest.mark.parametrize("robot,B,T", [("panda", 1, 51), ("panda", 37, 33), ("baxter", 5, 64)])
def test_layer_out_of_reach(golden, mode, robot, B, T):
    import torch

    from prismplan_b200 import api
    from prismplan_b200.robot import RobotModelBuilder
    from prismplan_b200.scene import SceneTensors

    asset = golden_asset(golden, robot)[0]
    b = RobotModelBuilder.from_asset(asset).build()
    rng = np.random.default_rng(T)
    boxes = workloads.random_obbs(rng, 33, -1.0, 1.0, 0.02, 0.2)
    far = workloads.random_esdf(np.random.default_rng(1), n_vox=32, centre=(9.0, 0.0, 0.0))
    near = workloads.random_esdf(np.random.default_rng(1), n_vox=64, centre=(0.3, 0.0, 0.5))
    none, out, seen = SceneTensors(*boxes), SceneTensors(*boxes, *far, esdf_mode=mode), SceneTensors(*boxes, *near, esdf_mode=mode)
    q = torch.from_numpy(workloads.straight_trajectories(rng, asset, B, T)).cuda()
    r = q.transpose(1, 2).contiguous()
    p = api.CostParams(collision_cost_weight=20.0, world_collision_margin=0.05, self_collision_margin=0.01,
                       smoothness_weight=1.0, delta_t=0.1)
    bits = lambda x: x.view(torch.int32)  # noqa: E731
    want = api.traj_cost(b, none, q, p)
    for a, c in zip(want, api.traj_cost(b, out, q, p)):
        assert torch.equal(bits(a), bits(c))
    rolls = api.rollout_costs(b, none, r, p)
    assert torch.equal(bits(rolls), bits(api.rollout_costs(b, out, r, p)))
    lit = api.traj_cost(b, seen, q, p)
    if B > 1:
        assert not torch.equal(want[0], lit[0])
    frm, to, _ = workloads.edge_batch(rng, asset, 20)
    f, t = torch.from_numpy(frm).cuda(), torch.from_numpy(to).cuda()
    for layout, threads in ((0, 128), (0, 256), (1, 128), (1, 256)):
        for edges in (False, True):
            batch = api.MixedBatch(b, 1 if edges else 0, 20 if edges else 0, 2, 2 * B * T + T, T)
            batch.set_shape(layout=layout, work_threads=threads, traj_threads=threads)
            for scene, full in ((none, want), (out, want), (seen, lit)):
                batch.clear()
                if edges:
                    batch.add_edges(f, t)
                wp, tc, g = batch.add_trajectory(q[0].contiguous())
                ro = batch.add_rollouts(r)
                batch.launch(scene, api.EdgeEvalParams(), p)
                assert batch.status() == _lib.PS_OK
                assert torch.equal(bits(wp), bits(full[0][0])) and torch.equal(bits(g), bits(full[2][0]))
                if scene is not seen:
                    assert torch.equal(bits(ro), bits(rolls))
            batch.close()
