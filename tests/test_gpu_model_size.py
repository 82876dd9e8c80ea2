"""The self check takes every model whose block fits in shared memory with
112 bytes per joint record: models within the last bytes of that limit, against
the FP64 oracle (flips only at contact)."""
import numpy as np
import pytest

from prismplan_b200 import _lib, workloads

pytestmark = pytest.mark.gpu


def _chain(n_joints, n_spheres):
    """Serial chain, one DoF a joint, its spheres spread over the moving joints."""
    n = n_joints - 1
    counts = [n_spheres // n + (k < n_spheres % n) for k in range(n)]
    fts, sph, s2j = workloads._arm(np.random.default_rng(n_spheres), n, counts, 1, (0.0, 0.0, 0.0), 1.0, None)
    parents = [0] + list(range(n))
    asset = {
        "name": "chain", "n_dof": n, "n_joints": n_joints, "joint_types": [workloads.X_ROT] + [workloads.Z_ROT] * n,
        "fixed_transforms": workloads._ft(np.eye(3), (0, 0, 0)) + [v for f in fts for v in f],
        "spheres_flat": [v if k % 4 < 3 else 0.04 * v for k, v in enumerate(sph)], "sphere_to_joint": s2j,
        "joint_lower": [-2.9] * n, "joint_upper": [2.9] * n, "joint_parents": parents,
        "joint_id_to_dof": [-1] + list(range(n)), "t_memory_idx": [0] + [1] * n, "dfs_order": list(range(n_joints)),
    }
    asset["self_cc_ranges_flat"] = workloads._self_ranges(s2j, parents)
    return workloads._finish(asset)


@pytest.mark.parametrize("n_joints,n_spheres", [(9, 283), (11, 280), (13, 277), (15, 274)])
def test_largest_self_checks(n_joints, n_spheres):
    import torch

    import oracle
    from prismplan_b200 import api
    from prismplan_b200.robot import RobotModelBuilder

    asset = _chain(n_joints, n_spheres)
    na = len(asset["approx_sphere_to_joint"])
    up = lambda x: (x + 15) // 16 * 16  # noqa: E731
    core = 64 + 112 * n_joints + up(16 * n_spheres) + up(4 * n_spheres) + up(16 * na) + up(4 * na)
    need = core + 64 * 12 * (n_spheres + na) + 64 * 4 * asset["n_dof"]   # model, positions, configurations of a block
    have = torch.cuda.get_device_properties(0).shared_memory_per_block_optin
    assert 0 <= have - need < 16 * n_joints
    b = RobotModelBuilder.from_asset(asset).build()
    q = workloads.uniform_configs(np.random.default_rng(1), asset, 500)
    h, _ = api.check_configs(b, None, torch.from_numpy(q).cuda(), check_self=True)
    om = oracle.OracleModel(b, np.zeros((0, 4)), np.zeros((0, 8)))
    h64, _, gap = om.check_configs(q, flags=_lib.PS_CHECK_SELF, want_gap=True)
    flips = np.nonzero(h.cpu().numpy() != h64)[0]
    assert np.all(gap[flips] < 1e-5)
    assert 0.0 < h64.mean() < 1.0
