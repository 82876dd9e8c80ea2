"""Small edge batches run one block per edge, with intervals shown clear by a
swept check; against the plain path, which checks every sample: validity and
cost bit for bit."""
import numpy as np
import pytest

from conftest import golden_asset
from prismplan_b200 import workloads

pytestmark = pytest.mark.gpu

# sample counts around the 32 groups (with and without the start sample), the
# interval lengths they set, the quarters, and one far beyond
COUNTS = np.array([0, 1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 96, 97, 128, 129, 130, 255, 600, 5000])


@pytest.mark.parametrize("n", [1, 5, 64, 500, 2048])
@pytest.mark.parametrize("robot,boxes,esdf,self_check", [("panda", 24, 0, True), ("panda", 40, 0, False),
                                                         ("fetch", 33, 0, True), ("baxter", 40, 64, True),
                                                         ("generic_chain", 9, 0, False), ("panda", 0, 0, True)])
def test_path_equals_plain(golden, n, robot, boxes, esdf, self_check):
    import torch

    from prismplan_b200 import api
    from prismplan_b200.robot import RobotModelBuilder
    from prismplan_b200.scene import SceneTensors

    asset = golden_asset(golden, robot)[0] if robot != "generic_chain" else workloads.generic_chain()
    b = RobotModelBuilder.from_asset(asset).build()
    rng = np.random.default_rng(n + boxes)
    d, p, e = workloads.random_obbs(rng, 4 * boxes + 1, -1.2, 1.2, 0.02, 0.1)
    keep = np.linalg.norm(p[:, :3], axis=1) > 0.8   # |t| = distance of the centre from the base: leave it free
    d, p, e = d[keep][:boxes], p[keep][:boxes], e[keep][:boxes]
    if boxes > 2:
        p[0, 3:7] *= np.float32(1.001)               # a stored quaternion off unit norm
        e[1] = 0
    sc = SceneTensors(d, p, e, *(workloads.random_esdf(rng, n_vox=esdf) if esdf else ()))
    frm, to, _ = workloads.edge_batch(rng, asset, n)
    G = COUNTS[rng.integers(0, len(COUNTS), n)].astype(np.int32)
    if n > 20:
        frm[2], to[4] = 20.0, -30.0                  # beyond the angles that the swept check judges
        frm[6, 0], to[8, 1] = np.nan, np.inf
        to[10] = frm[10]
    f, t, g = torch.from_numpy(frm).cuda(), torch.from_numpy(to).cuda(), torch.from_numpy(G).cuda()
    for margin in (0.0, 0.01):
        for samples, granularity in ((g, 16), (None, 16), (None, 40)):
            params = api.EdgeEvalParams(collision_margin=margin, check_self=self_check, granularity=granularity)
            a = api.check_edges(b, sc, f, t, samples=samples, params=params)
            q = api.check_edges(b, sc, f, t, samples=samples, params=params, persistent=False)
            assert torch.equal(a[0], q[0])
            assert torch.equal(a[1].view(torch.int32), q[1].view(torch.int32))   # NaN lengths too
    assert api.edges_status(None) == 0
