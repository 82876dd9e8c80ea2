"""The STOMP update's split kernels where they can go wrong: rollout counts
around a shared-memory batch of 64, waypoint counts around a batch of 64 rows of
the band factor and past the columns that the setup keeps in shared memory, and
totals at or above the selection's mask. Against the dense FP64 restatement of
the update (stomp.cu:257-413) and the literal selection scan (stomp.cu:133-152)."""
import numpy as np
import pytest

from conftest import golden_asset
from prismplan_b200 import workloads

pytestmark = pytest.mark.gpu


def _scan(totals, n):
    cc, out = totals.copy(), []
    for _ in range(n):
        best, value = 0, cc[0]
        for i in range(1, len(cc)):
            if cc[i] < value:
                best, value = i, cc[i]
        out.append(best)
        cc[best] = np.float32(3.0e38)
    return out


@pytest.mark.parametrize("Rn,Ro,T", [(1, 1, 5), (40, 23, 63), (40, 24, 64), (70, 57, 65), (30, 20, 142), (30, 20, 143),
                                     (100, 100, 160)])
def test_update_and_selection(golden, Rn, Ro, T):
    import torch

    from prismplan_b200 import api
    from prismplan_b200.robot import RobotModelBuilder
    from prismplan_b200.scene import SceneTensors
    from stomp_host import stomp_matrices
    from test_gpu_stomp import _free_run, _run, _ws_view

    asset, _ = golden_asset(golden, "panda")
    b = RobotModelBuilder.from_asset(asset).build()
    rng = np.random.default_rng(Rn + Ro + T)
    sc = SceneTensors(*workloads.random_obbs(rng, 16))
    B, D, R = 3, b.n_dof, Rn + Ro + 1
    th0 = workloads.straight_trajectories(rng, asset, B, T).astype(np.float32)
    kw = dict(num_rollouts_new=Rn, num_rollouts_old=Ro, num_timesteps=T)
    s = _free_run(num_iterations=1, **kw)
    res, ws = _run(b, sc, th0, s)
    lay = api.stomp_layout(b, B, T, s)
    roll = _ws_view(ws, lay["rollouts"][1], (R, B, T, D)).astype(np.float64)
    noise = _ws_view(ws, lay["noise"], (R, B, T, D)).astype(np.float64)
    scost = _ws_view(ws, lay["state_cost"][1], (R, B, T)).astype(np.float64)
    Rm, _, M = stomp_matrices(T, s.delta_t, s.noise_scale)
    ctrl = s.control_cost_weight * roll * np.einsum("ts,rbsd->rbtd", Rm, roll)
    c = scost[..., None] + ctrl
    mn, mx = c.min(0), c.max(0)
    u = np.exp(-s.exponentiated_cost_sensitivity * (c - mn) / np.maximum(mx - mn, 1e-8))
    delta = (u / np.maximum(u.sum(0), 1e-12) * noise).sum(0)
    delta[:, [0, -1]] = 0.0
    step = np.einsum("ts,bsd->btd", M, delta)
    step[:, [0, -1]] = 0.0
    # weights: h (c - min) / range <= 10, so some 1e-6 of the noise in FP32, and 200 terms' rounding 1.2e-5
    np.testing.assert_allclose(res.theta.cpu().numpy(), th0 + step, rtol=0, atol=5e-5)
    for weight in (s.collision_cost_weight, 5.0e37):   # the second: most totals at or above the mask, costs finite
        s2 = _free_run(num_iterations=2, collision_cost_weight=weight, world_collision_margin=0.3, **kw)
        _, ws = _run(b, sc, th0, s2)
        tot = _ws_view(ws, lay["row_total"][1], (R, B))
        idx = _ws_view(ws, lay["reuse_index"], (B, Ro), np.int32)
        for i in range(B):
            assert idx[i].tolist() == _scan(tot[:, i], Ro), (weight, i)
