"""Samples that the one-block-per-path kernels leave to the whole device: edges
that no swept check can clear (they slide along a box, or by an ESDF layer),
colliding at a few samples or at none. Against the plain path, which checks
every sample: validity and cost bit for bit. And fine steps in the optimisers
against the separate waypoint and segment checks."""
import numpy as np
import pytest

from conftest import golden_asset
from prismplan_b200 import workloads

pytestmark = pytest.mark.gpu


def _robot(golden, name):
    from prismplan_b200.robot import RobotModelBuilder

    asset = golden_asset(golden, name)[0]
    return asset, RobotModelBuilder.from_asset(asset).build()


def _ceiling(b, asset, gap=1e-3, needle=None):
    """A slab `gap` above the robot at mid range, and a 2 mm cube that its outermost sphere touches at `needle` rad of
    the first joint; the configuration."""
    import torch

    from prismplan_b200 import api
    from prismplan_b200.scene import SceneTensors, pack_obbs

    q = ((np.array(asset["joint_lower"]) + np.array(asset["joint_upper"])) / 2).astype(np.float32)
    x = api.fk_spheres(b, torch.from_numpy(q[None]).cuda())[0].cpu().numpy()[:, :3]
    r = np.array(asset["spheres_flat"]).reshape(-1, 4)[:, 3]
    dims, pos = [[4.0, 4.0, 0.2]], [[0.0, 0.0, (x[:, 2] + r).max() + gap + 0.1]]
    if needle is not None:
        out = np.argmax(np.hypot(x[:, 0], x[:, 1]))
        rho, at = np.hypot(*x[out, :2]) + 0.98 * r[out], np.arctan2(x[out, 1], x[out, 0]) + needle - q[0]
        dims.append([0.002] * 3)
        pos.append([rho * np.cos(at), rho * np.sin(at), x[out, 2]])
    return SceneTensors(*pack_obbs(np.array(dims), np.array(pos), np.array([[1.0, 0.0, 0.0, 0.0]] * len(dims)))), q


# edge counts: one, on either side of the tiny batches (14 on 148 SMs), and
# some; samples around the 32 groups, few ones, the units of 32 and longer ones
@pytest.mark.parametrize("n", [1, 14, 15, 40])
@pytest.mark.parametrize("G", [1, 8, 33, 64, 65, 66, 100, 513, 1024, 1025, 1040, 2049, 5000])
@pytest.mark.parametrize("self_check", [False, True])
def test_sliding_edges(golden, n, G, self_check):
    import torch

    from prismplan_b200 import api

    asset, b = _robot(golden, "panda")
    scene, q = _ceiling(b, asset, needle=0.3)
    f = np.repeat(q[None], n, 0)
    t = f.copy()
    f[:, 0], t[:, 0] = -1.5 - 0.013 * np.arange(n), 1.5
    t[1::7, 0] = 0.1                                   # does not reach the cube
    f, t = torch.from_numpy(f).cuda(), torch.from_numpy(t).cuda()
    g = torch.full((n,), G, dtype=torch.int32, device="cuda")
    p = api.EdgeEvalParams(check_self=self_check)
    a = api.check_edges(b, scene, f, t, samples=g, params=p)
    c = api.check_edges(b, scene, f, t, samples=g, params=p, persistent=False)
    assert torch.equal(a[0], c[0]) and torch.equal(a[1], c[1])
    if n == 40 and G >= 513:
        assert 0 < int(a[0].sum()) < n


@pytest.mark.parametrize("n", [14, 15, 64])
@pytest.mark.parametrize("robot,esdf,self_check", [("baxter", 64, False), ("baxter", 64, True), ("panda", 0, True)])
def test_long_edges(golden, n, robot, esdf, self_check):
    import torch

    from prismplan_b200 import api
    from prismplan_b200.scene import SceneTensors

    asset, b = _robot(golden, robot)
    rng = np.random.default_rng(n)
    d, p, e = workloads.random_obbs(rng, 60, -1.2, 1.2, 0.02, 0.08)
    keep = np.linalg.norm(p[:, :3], axis=1) > 0.8
    scene = SceneTensors(d[keep], p[keep], e[keep], *(workloads.random_esdf(rng, n_vox=esdf) if esdf else ()))
    frm, _, _ = workloads.edge_batch(rng, asset, 4000)
    free = api.check_configs(b, scene, torch.from_numpy(frm).cuda(), check_self=self_check)[0].cpu().numpy() == 0
    f = frm[free][:n]
    t = np.clip(f + rng.uniform(-0.4, 0.4, f.shape), asset["joint_lower"], asset["joint_upper"]).astype(np.float32)
    g = torch.from_numpy(rng.choice([0, 16, 40, 200, 777, 1500, 4000], len(f)).astype(np.int32)).cuda()
    f, t = torch.from_numpy(f).cuda(), torch.from_numpy(t).cuda()
    params = api.EdgeEvalParams(check_self=self_check)
    a = api.check_edges(b, scene, f, t, samples=g, params=params)
    c = api.check_edges(b, scene, f, t, samples=g, params=params, persistent=False)
    assert torch.equal(a[0], c[0]) and torch.equal(a[1], c[1])
    if n == 64:
        long = g > 100
        assert 0 < int(a[0][long].sum()) < int(long.sum())


def test_a_long_edge_is_spread_over_the_device(golden):
    """One edge of 20,000 samples along a box, beside the queue path (which a time budget selects): one block alone
    took some 80 times as long."""
    import torch

    from prismplan_b200 import api

    asset, b = _robot(golden, "panda")
    scene, q = _ceiling(b, asset)
    f, t = np.repeat(q[None], 1, 0), np.repeat(q[None], 1, 0)
    f[:, 0], t[:, 0] = -1.5, 1.5
    f, t = torch.from_numpy(f).cuda(), torch.from_numpy(t).cuda()
    for G in (2000, 20000):
        g = torch.full((1,), G, dtype=torch.int32, device="cuda")
        ms = []
        for budget in (0.0, 1000.0):
            p = api.EdgeEvalParams(time_budget_ms=budget)
            ws = api.edges_workspace(1)
            run = lambda: api.check_edges(b, scene, f, t, samples=g, params=p, workspace=ws)  # noqa: E731
            assert int(run()[0]) == 1
            a, z = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(20):
                run()
            z.record()
            z.synchronize()
            ms.append(a.elapsed_time(z))
        assert ms[0] < 4.0 * ms[1], (G, ms)


@pytest.mark.parametrize("robot,boxes,esdf", [("panda", 12, 0), ("baxter", 10, 64)])
@pytest.mark.parametrize("self_check", [False, True])
@pytest.mark.parametrize("T,step", [(6, 0.002), (40, 0.01), (70, 0.002)])
def test_fine_steps_in_a_solve(golden, robot, boxes, esdf, self_check, T, step):
    import torch

    from prismplan_b200 import api
    from prismplan_b200.scene import SceneTensors

    asset, b = _robot(golden, robot)
    rng = np.random.default_rng(T + boxes)
    d, p, e = workloads.random_obbs(rng, 20 * boxes, -1.3, 1.3, 0.02, 0.15)
    keep = np.linalg.norm(p[:, :3], axis=1) > 1.2
    d, p, e = d[keep][:boxes], p[keep][:boxes], e[keep][:boxes]
    ones = {"sphere_obb_acm_mask": np.ones((len(b.sphere_to_joint), len(d)), np.uint8)}
    layers = ()
    if esdf:
        layers = workloads.random_esdf(rng, n_vox=esdf, centre=(0.9, 0.0, 0.5))
        ones["sphere_acm_mask"] = np.ones((len(b.sphere_to_joint), 1), np.uint8)
    plain, masked = SceneTensors(d, p, e, *layers), SceneTensors(d, p, e, *layers, **ones)
    starts, goals = workloads.free_pairs(
        rng, asset, 6, lambda q: api.check_configs(b, plain, torch.from_numpy(q).cuda(), check_self=True)[0].cpu().numpy() == 0, 64)
    goals[0] = starts[0] + 0.01
    s = api.ChompSettings(num_timesteps=T, num_iterations=10, check_self=self_check, time_limit_ms=0.0,
                          collision_check_step=step)
    r, m = (api.chomp_solve(b, sc, starts, goals, s) for sc in (plain, masked))
    for name in ("solved", "iterations", "cost", "path", "theta"):
        assert torch.equal(getattr(r, name), getattr(m, name)), name


@pytest.mark.parametrize("n,self_check", [(10, True), (100, False), (300, True)])
def test_captured_calls(golden, n, self_check):
    """A captured call replayed on other edges, and two streams with a workspace each."""
    import torch

    from prismplan_b200 import api

    asset, b = _robot(golden, "panda")
    scene, _ = _ceiling(b, asset, gap=0.02, needle=0.3)
    params = api.EdgeEvalParams(max_joint_step=0.01, check_self=self_check)
    batches = []
    for seed in range(3):
        frm, to, _ = workloads.edge_batch(np.random.default_rng(seed), asset, n)
        batches.append((torch.from_numpy(frm).cuda(), torch.from_numpy(to).cuda()))
    want = [api.check_edges(b, scene, f, t, params=params, persistent=False)[:2] for f, t in batches]
    f, t = (x.clone() for x in batches[0])
    ws = api.edges_workspace(n)
    api.check_edges(b, scene, f, t, params=params, workspace=ws)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = api.check_edges(b, scene, f, t, params=params, workspace=ws)
    for (a, c), w in zip(batches, want):
        f.copy_(a)
        t.copy_(c)
        g.replay()
        assert torch.equal(got[0], w[0]) and torch.equal(got[1], w[1])
    streams, out = [torch.cuda.Stream() for _ in batches], []
    spaces = [api.edges_workspace(n) for _ in batches]
    torch.cuda.synchronize()
    for _ in range(5):
        for s, (a, c), w in zip(streams, batches, spaces):
            with torch.cuda.stream(s):
                out.append(api.check_edges(b, scene, a, c, params=params, workspace=w))
    torch.cuda.synchronize()
    for k, o in enumerate(out):
        assert torch.equal(o[0], want[k % 3][0]) and torch.equal(o[1], want[k % 3][1])
