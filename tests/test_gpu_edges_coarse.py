"""The coarse pass over long edges (persistent path with the end-sample probe)
against the plain path, which checks every sample: validity and cost bit for
bit."""
import numpy as np
import pytest

from conftest import golden_asset
from prismplan_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("robot,half_hi,boxes,margin", [("panda", 0.1, 40, 0.0), ("fetch", 0.06, 65, 0.01),
                                                        ("generic_chain", 0.1, 16, -0.005), ("panda_like", 0.3, 33, 0.0)])
def test_coarse_equals_plain(golden, robot, half_hi, boxes, margin):
    import torch

    from prismplan_b200 import api
    from prismplan_b200.robot import RobotModelBuilder
    from prismplan_b200.scene import SceneTensors

    asset = golden_asset(golden, robot)[0] if robot in ("panda", "fetch") else getattr(workloads, robot)()
    b = RobotModelBuilder.from_asset(asset).build()
    rng = np.random.default_rng(boxes)
    d, p, e = workloads.random_obbs(rng, 4 * boxes, -1.0, 1.0, 0.02, half_hi)
    keep = np.linalg.norm(p[:, :3], axis=1) > 0.75   # |t| = distance of the centre from the base: leave it free
    d, p, e = d[keep][:boxes], p[keep][:boxes], e[keep][:boxes]
    p[0, 3:7] *= np.float32(1.001)                    # a stored quaternion off unit norm
    n = 40000                                         # enough for the probe and the one-pass queue
    frm, to, G = workloads.edge_batch(rng, asset, n)
    # sample counts on both sides of the units (128 samples from 256 on), of the chunks and of the padding rule
    edges = np.array([1, 31, 32, 33, 255, 256, 257, 260, 272, 288, 289, 383, 384, 385, 388, 389, 512, 513, 640, 1500])
    G[::2] = np.where(rng.random(n // 2) < 0.5, edges[rng.integers(0, len(edges), n // 2)], G[::2])
    frm[2], to[4] = 20.0, -30.0                       # beyond the angles that the coarse pass judges
    frm[6, 0], to[8, 1] = np.nan, np.inf
    to[10] = frm[10]                                  # no motion at all
    f, t, g = torch.from_numpy(frm).cuda(), torch.from_numpy(to).cuda(), torch.from_numpy(G.astype(np.int32)).cuda()
    sc = SceneTensors(d, p, e)
    params = api.EdgeEvalParams(collision_margin=margin)
    a = api.check_edges(b, sc, f, t, samples=g, params=params)
    q = api.check_edges(b, sc, f, t, samples=g, params=params, persistent=False)
    free = q[0].float()[g >= 256].mean().item()
    assert 0.0 < free < 1.0, free                   # long edges of both kinds
    assert torch.equal(a[0], q[0]) and torch.equal(a[1].view(torch.int32), q[1].view(torch.int32))   # NaN lengths too
