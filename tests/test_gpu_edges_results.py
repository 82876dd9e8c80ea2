"""Large batches whose results the queue's launches write themselves (boxes
only, long edges, no self check), with the coarse pass chosen (few end samples
collide) and not, beside the finalize kernel's (with self check): validity, cost
and the clearance output against the plain path, bit for bit, on outputs that
held something else; and closed when the staging gives up."""
import ctypes as C

import numpy as np
import pytest

from conftest import golden_asset
from prismplan_b200 import _lib, workloads

pytestmark = pytest.mark.gpu

FLT_MAX = np.finfo(np.float32).max


@pytest.mark.parametrize("n", [37888, 40001])       # the probe from 37,888 edges on 148 SMs
@pytest.mark.parametrize("boxes,half", [(12, 0.05), (60, 0.3)])   # free at most ends; in collision at most
@pytest.mark.parametrize("self_check", [False, True])
def test_results(golden, n, boxes, half, self_check):
    import torch

    from prismplan_b200 import api
    from prismplan_b200.robot import RobotModelBuilder
    from prismplan_b200.scene import SceneTensors

    asset = golden_asset(golden, "panda")[0]
    b = RobotModelBuilder.from_asset(asset).build()
    rng = np.random.default_rng(boxes)
    d, p, e = workloads.random_obbs(rng, 6 * boxes, -1.0, 1.0, 0.02, half)
    keep = np.linalg.norm(p[:, :3], axis=1) > 0.75  # |t| = distance of the centre from the base: leave it free
    scene = SceneTensors(d[keep][:boxes], p[keep][:boxes], e[keep][:boxes])
    frm, to, _ = workloads.edge_batch(rng, asset, n)
    f, t = torch.from_numpy(frm).cuda(), torch.from_numpy(to).cuda()
    params, view, lib = api.EdgeEvalParams(max_joint_step=0.01, max_samples=600, check_self=self_check), scene.view(), _lib.load()
    ws = api.edges_workspace(n)
    out = []

    def run(persistent, fill):
        valid = torch.full((n,), fill, dtype=torch.uint8, device="cuda")
        cost, clr = torch.full((n,), float(fill), device="cuda"), torch.full((n,), float(fill), device="cuda")
        args = [b.handle, C.byref(view), f.data_ptr(), t.data_ptr(), None, n, C.byref(params.to_c()), valid.data_ptr(),
                cost.data_ptr(), clr.data_ptr()]
        _lib.check(lib.ps_check_edges(*args, ws.data_ptr(), ws.numel(), None) if persistent
                   else lib.ps_check_edges_plain(*args, None))
        torch.cuda.synchronize()
        return valid, cost, clr

    out = [run(False, 1), run(True, 1), run(True, 0), run(True, 7)]
    for got in out[1:]:
        assert all(torch.equal(x, y) for x, y in zip(got, out[0]))
    share = float(out[0][0].float().mean())
    assert share > 0.5 if half < 0.1 else 0.0 < share < 0.5, share
    _lib.check(lib.ps_model_set_wait_limit(b.handle, 0))
    try:
        v, c, _ = run(True, 1)
        assert not bool(v.any()) and bool((c == FLT_MAX).all()) and api.edges_status(ws) == _lib.PS_ETIMEOUT
    finally:
        _lib.check(lib.ps_model_set_wait_limit(b.handle, -1))
    assert all(torch.equal(x, y) for x, y in zip(run(True, 1), out[0]))
