"""The one-block-per-path kernels fail closed when the bounded wait for the
model gives up (limit 0 polls: every launch gives up at once, no fault and no
hang): small edge batches of each route, and both optimisers. Beside it what
else those kernels take: bound centres staged on their own, trilinear ESDF
layers, the clearance output."""
import numpy as np
import pytest

from conftest import golden_asset
from prismplan_b200 import _lib, workloads
from test_gpu_edges_self import _without_last_approx_sphere

pytestmark = pytest.mark.gpu

FLT_MAX = np.finfo(np.float32).max


def _scene(rng, esdf=0, mode=_lib.PS_ESDF_NEAREST, **masks):
    from prismplan_b200.scene import SceneTensors

    d, p, e = workloads.random_obbs(rng, 60, -1.3, 1.3, 0.02, 0.1)
    keep = np.linalg.norm(p[:, :3], axis=1) > 0.9   # |t| = distance of the centre from the base: leave it free
    layers = workloads.random_esdf(rng, n_vox=esdf) if esdf else ()
    return SceneTensors(d[keep], p[keep], e[keep], *layers, esdf_mode=mode, **masks), int(keep.sum())


def _poll(b):
    import ctypes as C

    code = C.c_int(-1)
    _lib.check(_lib.load().ps_model_poll_status(b.handle, C.byref(code)))
    return code.value


@pytest.fixture()
def panda(golden):
    from prismplan_b200.robot import RobotModelBuilder

    asset = golden_asset(golden, "panda")[0]
    b = RobotModelBuilder.from_asset(asset).build()
    yield asset, b
    _lib.check(_lib.load().ps_model_set_wait_limit(b.handle, -1))


# the list at once; a block per edge, then the list; few samples, no list
@pytest.mark.parametrize("n,self_check,granularity", [(5, False, 40), (5, True, 40), (27, False, 0), (200, False, 0),
                                                      (500, True, 0), (1024, True, 0), (500, False, 16)])
@pytest.mark.parametrize("esdf", [0, 64])
def test_edges(panda, n, self_check, granularity, esdf):
    import torch

    from prismplan_b200 import api

    asset, b = panda
    rng = np.random.default_rng(n)
    scene, _ = _scene(rng, esdf)
    n = min(n, 64) if esdf else n
    frm, to, _ = workloads.edge_batch(rng, asset, n)
    f, t = torch.from_numpy(frm).cuda(), torch.from_numpy(to).cuda()
    p = api.EdgeEvalParams(check_self=self_check, **({"granularity": granularity} if granularity else {"max_joint_step": 0.01}))
    ws = api.edges_workspace(n)

    def run():
        v, c, _ = api.check_edges(b, scene, f, t, params=p, workspace=ws)
        torch.cuda.synchronize()
        return v.cpu().numpy(), c.cpu().numpy()

    ok = run()
    assert n < 20 or 0.0 < ok[0].mean() < 1.0
    assert int(ws[:8].view(torch.int64)) == 0        # not the queue
    assert api.edges_status(ws) == _lib.PS_OK and _poll(b) == _lib.PS_OK
    _lib.check(_lib.load().ps_model_set_wait_limit(b.handle, 0))
    v, c = run()
    assert not v.any() and np.all(c == FLT_MAX)
    assert api.edges_status(ws) == _lib.PS_ETIMEOUT and _poll(b) == _lib.PS_ETIMEOUT
    _lib.check(_lib.load().ps_model_set_wait_limit(b.handle, -1))
    again = run()
    assert all(np.array_equal(x, y) for x, y in zip(ok, again)) and api.edges_status(ws) == _lib.PS_OK


@pytest.mark.parametrize("kind", ["chomp", "stomp"])
@pytest.mark.parametrize("step", [0.05, 0.002])   # few samples, and enough for the list
def test_solves(panda, kind, step):
    import torch

    from prismplan_b200 import api

    asset, b = panda
    rng = np.random.default_rng(3)
    scene, _ = _scene(rng)
    q = workloads.free_pairs(rng, asset, 4, lambda q: api.check_configs(b, scene, torch.from_numpy(q).cuda(), check_self=True)[0].cpu().numpy() == 0, 32)[0]
    settings = {"chomp": api.ChompSettings, "stomp": api.StompSettings}[kind](num_timesteps=40, num_iterations=4, time_limit_ms=0.0,
                                                                              collision_check_step=step)
    solve = {"chomp": api.chomp_solve, "stomp": api.stomp_solve}[kind]
    ok = solve(b, scene, q, q + 0.01, settings)      # next to each other: free as they are
    assert bool(ok.solved.all())
    _lib.check(_lib.load().ps_model_set_wait_limit(b.handle, 0))
    r = solve(b, scene, q, q + 0.01, settings)
    torch.cuda.synchronize()
    assert not bool(r.solved.any())
    assert _poll(b) == _lib.PS_ETIMEOUT
    _lib.check(_lib.load().ps_model_set_wait_limit(b.handle, -1))
    again = solve(b, scene, q, q + 0.01, settings)
    assert torch.equal(again.solved, ok.solved) and torch.equal(again.path, ok.path)


@pytest.mark.parametrize("n", [10, 300, 1000])
def test_staged_bound_centres(golden, n):
    """A joint with exact spheres and no approximate one: the self check's second layout."""
    import torch

    from prismplan_b200 import api
    from prismplan_b200.robot import RobotModelBuilder

    asset = _without_last_approx_sphere(golden_asset(golden, "panda")[0])
    b = RobotModelBuilder.from_asset(asset).build()
    rng = np.random.default_rng(n)
    scene, _ = _scene(rng)
    frm, to, _ = workloads.edge_batch(rng, asset, n)
    f, t = torch.from_numpy(frm).cuda(), torch.from_numpy(to).cuda()
    p = api.EdgeEvalParams(check_self=True, max_joint_step=0.005)
    a, c = (api.check_edges(b, scene, f, t, params=p, persistent=x) for x in (True, False))
    assert torch.equal(a[0], c[0]) and torch.equal(a[1], c[1])
    assert n < 100 or 0.0 < float(a[0].float().mean()) < 1.0
    plain, nb = _scene(np.random.default_rng(7))
    masked, _ = _scene(np.random.default_rng(7), sphere_obb_acm_mask=np.ones((len(b.sphere_to_joint), nb), np.uint8))
    starts, goals = workloads.free_pairs(
        rng, asset, 6, lambda q: api.check_configs(b, plain, torch.from_numpy(q).cuda(), check_self=True)[0].cpu().numpy() == 0, 64)
    s = api.ChompSettings(num_timesteps=35, num_iterations=10, time_limit_ms=0.0, collision_check_step=0.004)
    r, m = (api.chomp_solve(b, x, starts, goals, s) for x in (plain, masked))
    for name in ("solved", "iterations", "cost", "path", "theta"):
        assert torch.equal(getattr(r, name), getattr(m, name)), name


@pytest.mark.parametrize("n", [10, 64])
@pytest.mark.parametrize("self_check", [False, True])
@pytest.mark.parametrize("mode", [_lib.PS_ESDF_NEAREST, _lib.PS_ESDF_TRILINEAR])
def test_esdf_modes_and_clearance_output(golden, n, self_check, mode):
    import ctypes as C

    import torch

    from prismplan_b200 import api
    from prismplan_b200.robot import RobotModelBuilder

    asset = golden_asset(golden, "baxter")[0]
    b = RobotModelBuilder.from_asset(asset).build()
    rng = np.random.default_rng(n)
    scene, _ = _scene(rng, 96, mode)
    frm, to, _ = workloads.edge_batch(rng, asset, n)
    f, t = torch.from_numpy(frm).cuda(), torch.from_numpy(to).cuda()
    p, v = api.EdgeEvalParams(check_self=self_check, max_joint_step=0.01), scene.view()
    out = []
    for persistent in (True, False):
        valid = torch.zeros(n, dtype=torch.uint8, device="cuda")
        cost, clr, ws = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda"), api.edges_workspace(n)
        args = [b.handle, C.byref(v), f.data_ptr(), t.data_ptr(), None, n, C.byref(p.to_c()), valid.data_ptr(),
                cost.data_ptr(), clr.data_ptr()]
        lib = _lib.load()
        _lib.check(lib.ps_check_edges(*args, ws.data_ptr(), ws.numel(), None) if persistent
                   else lib.ps_check_edges_plain(*args, None))
        torch.cuda.synchronize()
        out.append((valid, cost, clr))
    assert all(torch.equal(x, y) for x, y in zip(*out))
    assert bool((out[0][2] == FLT_MAX).all())        # not asked for
