"""Configuration checks with several lanes per configuration and culled boxes,
against the generic kernel (all-ones allowed-collision masks select it, and
change no pair): verdicts and clearances bit for bit."""
import copy

import numpy as np
import pytest

from conftest import golden_asset
from prismplan_b200 import workloads

pytestmark = pytest.mark.gpu


def _robot(name, golden):
    from prismplan_b200.robot import RobotModelBuilder

    if name in ("panda", "baxter"):
        asset, _ = golden_asset(golden, name)
    elif name == "stretched":   # a transform that stretches and a negative radius: the reach must still hold
        asset = copy.deepcopy(workloads.panda_like())
        for k in (0, 1, 2, 4, 5, 6, 8, 9, 10):
            asset["fixed_transforms"][16 * 3 + k] *= 1.25
        asset["spheres_flat"][4 * 7 + 3] = -0.04
    else:
        asset = getattr(workloads, name)()
    return RobotModelBuilder.from_asset(asset).build(), asset


# configuration counts: tile edges of 16, 4 and 1 lanes per configuration and
# both sides of the counts where the lanes change (4736 and 33,152 on 148 SMs)
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 33, 1000, 4736, 4737, 33153])
@pytest.mark.parametrize("robot,boxes,esdf", [("panda", 16, 0), ("panda", 33, 0), ("baxter", 65, 64), ("panda", 0, 64),
                                              ("stretched", 32, 0), ("generic_chain", 1, 0)])
def test_group_equals_generic(golden, n, robot, boxes, esdf):
    import torch

    from prismplan_b200 import api
    from prismplan_b200.scene import SceneTensors

    b, asset = _robot(robot, golden)
    rng = np.random.default_rng(n + boxes)
    d, p, e = workloads.random_obbs(rng, boxes) if boxes else (np.zeros((0, 4)), np.zeros((0, 8)), np.zeros(0))
    if boxes > 3:
        e[2] = 0
        p[1, 3:7] *= np.float32(1.001)   # a stored quaternion off unit norm
    layers = workloads.random_esdf(rng, n_vox=esdf) if esdf else ()
    ns = len(b.sphere_to_joint)
    ones = {}
    if boxes:
        ones["sphere_obb_acm_mask"] = np.ones((ns, boxes), np.uint8)
    if esdf:
        ones["sphere_acm_mask"] = np.ones((ns, 1), np.uint8)
    fast, generic = SceneTensors(d, p, e, *layers), SceneTensors(d, p, e, *layers, **ones)
    q = workloads.uniform_configs(rng, asset, n)
    if n > 30:
        q[3, 0], q[5, 1], q[6] = np.nan, np.inf, 100.0 * q[6]
    q = torch.from_numpy(q).cuda()
    for margin in (0.0, 0.02, -0.005):
        for clearance in (None, "obb") if not esdf else (None,):
            a = api.check_configs(b, fast, q, margin, clearance)
            g = api.check_configs(b, generic, q, margin, clearance)
            assert torch.equal(a[0], g[0])
            if clearance:
                assert torch.equal(a[1].view(torch.int32), g[1].view(torch.int32))


@pytest.mark.parametrize("n", [9, 1000, 4737])
def test_clearances_on_both_sides_of_the_first_bound(golden, n):
    """One box some 2 m from the arm: a warp's configurations disagree on
    whether their clearance is known to be below the level at which the first
    joints stop bounding it by the box centres (2 m)."""
    import torch

    from prismplan_b200 import api
    from prismplan_b200.scene import SceneTensors, pack_obbs

    b, asset = _robot("panda", golden)
    d, p, e = pack_obbs(np.array([[0.2, 0.2, 0.2]]), np.array([[2.4, 0.0, 0.4]]), np.array([[1.0, 0.0, 0.0, 0.0]]))
    ones = np.ones((len(b.sphere_to_joint), 1), np.uint8)
    q = torch.from_numpy(workloads.uniform_configs(np.random.default_rng(n), asset, n)).cuda()
    a = api.check_configs(b, SceneTensors(d, p, e), q, 0.0, "obb")
    g = api.check_configs(b, SceneTensors(d, p, e, sphere_obb_acm_mask=ones), q, 0.0, "obb")
    assert n < 100 or (float(g[1].min()) < 2.0 < float(g[1].max()))
    assert torch.equal(a[0], g[0]) and torch.equal(a[1].view(torch.int32), g[1].view(torch.int32))
