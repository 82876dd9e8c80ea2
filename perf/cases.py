"""The work that callers have this library do, as cases that can be timed and compared.

A case is a dict of plain values. ``kind`` names the entry point, ``robot`` and ``field`` the model and the boxes
around it:

  configs      api.check_configs       a batch of configurations (sampling planners, pre-flight checks)
  edges        api.check_edges         a batch of edges on the device, workspace kept by the caller
  bridge       api.EdgeEvalGpu         the same on host arrays, synchronous (the search planners' call)
  cost         api.traj_cost           CHOMP cost and exact gradient of a batch of trajectories
  autograd     api.hinge_cost          the same through torch.autograd, forward and backward
  rollouts     api.rollout_costs       STOMP state costs of noisy rollouts
  chomp_solve, stomp_solve             whole optimiser calls on (start, goal) pairs
  mixed        api.MixedBatch          edge, trajectory and rollout requests queued and launched together

``field``: "dense" boxes (half extents 0.02 to 0.3 m within 1 m of the base: few free edges), "sparse" ones (0.02 to
0.1 m, most edges free) or "wide" ones (as small, within 1.5 m, what the two-arm robot plans among), none of them
touching the robot at mid range. ``esdf``: edge length in voxels of an ESDF layer (5 mm voxels) beside the boxes, 0 for none.
"""
import math
import os

import numpy as np
import torch

from prismplan_b200 import _lib, api, workloads
from prismplan_b200.robot import RobotModelBuilder
from prismplan_b200.scene import SceneTensors

# reach of the centres, smallest and largest half extent (m)
FIELDS = {"dense": (1.0, 0.02, 0.3), "sparse": (1.0, 0.02, 0.1), "wide": (1.5, 0.02, 0.1)}
ASSETS = {}


def listed():
    return [
        # a sampling planner's batch: verdict and clearance of 4096 configurations
        {"name": "configs_4096", "kind": "configs", "robot": "panda_like", "obbs": 16, "field": "dense", "esdf": 0,
         "n": 4096, "clearance": "obb", "self": False, "margin": 0.0},
        # the same for a roadmap's worth of samples: the largest batch
        {"name": "configs_1m", "kind": "configs", "robot": "panda_like", "obbs": 16, "field": "dense", "esdf": 0,
         "n": 1048576, "clearance": "obb", "self": False, "margin": 0.0},
        # verdicts with self collision of a two-arm robot among boxes and a depth camera's ESDF, ragged count
        {"name": "configs_self_esdf", "kind": "configs", "robot": "baxter", "obbs": 128, "field": "wide",
         "esdf": 128, "n": 20011, "clearance": "none", "self": True, "margin": 0.01},
        # one expansion of a search planner: a few edges on host arrays, the smallest call
        {"name": "bridge_27", "kind": "bridge", "robot": "panda", "obbs": 16, "field": "sparse", "esdf": 0, "n": 27,
         "step": 0.0, "self": True, "clearance": False, "margin": 0.0},
        # a planner iteration's candidate edges with self collision, an odd count among small boxes
        {"name": "edges_self_1009", "kind": "edges", "robot": "panda", "obbs": 64, "field": "sparse", "esdf": 0,
         "n": 1009, "step": 0.02, "self": True, "clearance": False, "margin": 0.0},
        # the headline batch: 65,536 uneven edges of 1 to 600 samples
        {"name": "edges_65536", "kind": "edges", "robot": "panda_like", "obbs": 64, "field": "dense", "esdf": 0,
         "n": 65536, "step": 0.01, "self": False, "clearance": False, "margin": 0.0},
        # one trajectory's cost and gradient through autograd: launches and latency
        {"name": "autograd_1x51", "kind": "autograd", "robot": "panda", "obbs": 16, "field": "dense", "esdf": 0,
         "b": 1, "t": 51},
        # CHOMP cost and gradient of many trajectories
        {"name": "cost_256x64", "kind": "cost", "robot": "panda_like", "obbs": 64, "field": "dense", "esdf": 0,
         "b": 256, "t": 64},
        # STOMP: 32 trajectories x 128 rollouts x 100 waypoints of a mobile manipulator
        {"name": "rollouts_4096x100", "kind": "rollouts", "robot": "fetch_like", "obbs": 96, "field": "dense",
         "esdf": 0, "b": 4096, "t": 100},
        # uneven requests of several callers in one launch: edges, trajectories, rollouts, boxes and an ESDF
        {"name": "mixed_24", "kind": "mixed", "robot": "baxter_like", "obbs": 128, "field": "wide", "esdf": 128,
         "edge_requests": 12, "trajectories": 8, "rollout_requests": 4, "step": 0.01},
        # whole optimiser calls: a batch of planning requests, and a few with the default settings
        {"name": "chomp_solve_256", "kind": "chomp_solve", "robot": "panda", "obbs": 16, "field": "dense", "esdf": 0,
         "b": 256, "t": 64},
        {"name": "stomp_solve_16", "kind": "stomp_solve", "robot": "panda", "obbs": 16, "field": "dense", "esdf": 0,
         "b": 16, "t": 51},
    ]


def draw(rng):
    def log(lo, hi):
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(["configs", "configs", "edges", "edges", "bridge", "cost", "autograd", "rollouts", "mixed",
                       "chomp_solve", "stomp_solve"])
    check_self = rng.random() < 0.4   # links of the generated chains overlap: self checks are for the described robots
    c = {"kind": kind, "robot": rng.choice(["panda", "fetch"] if check_self else ["panda_like", "panda", "fetch_like"]), "obbs": log(8, 128), "field": rng.choice(["dense", "sparse"]), "esdf": 0}
    if kind in ("configs", "edges", "bridge") and rng.random() < 0.3:
        c.update(robot="baxter", field="wide", esdf=rng.choice([0, 64, 128]))
    if kind == "configs":
        c.update(n=log(64, 1048576 if c["robot"] != "baxter" and c["obbs"] <= 16 else 100000),
                 clearance=rng.choice(["none", "obb"]), self=check_self, margin=rng.choice([0.0, 0.01]))
    elif kind == "edges":
        c.update(n=log(16, 65536 if c["robot"] != "baxter" else 8192), step=rng.choice([0.01, 0.02, 0.05]),
                 self=check_self, clearance=c["esdf"] > 0 and rng.random() < 0.3, margin=rng.choice([0.0, 0.01]))
        if c["self"] or c["field"] != "dense":
            c["n"] = max(16, c["n"] // 8)   # free edges and self checks cost more: the batch is smaller
    elif kind == "bridge":
        c.update(n=log(1, 2048), step=rng.choice([0.0, 0.02]), self=check_self, clearance=False,
                 margin=rng.choice([0.0, 0.01]))
    elif kind in ("cost", "autograd"):
        c.update(b=log(1, 256), t=rng.randint(16, 64))
    elif kind == "rollouts":
        c.update(b=log(8, 4096), t=rng.randint(16, 100))
    elif kind == "mixed":
        c.update(robot="baxter_like", field="wide", esdf=rng.choice([64, 128]), edge_requests=rng.randint(1, 12),
                 trajectories=rng.randint(1, 8), rollout_requests=rng.randint(1, 4), step=rng.choice([0.01, 0.02]))
    else:
        c.update(robot="panda", field="dense", obbs=log(8, 16), t=rng.randint(32, 64),
                 b=log(1, 256 if kind == "chomp_solve" else 16))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def asset_of(name):
    """The repository's robots: its generators' chains, and the three descriptions that its tests hold."""
    if name not in ASSETS:
        if name in ("panda", "fetch", "baxter"):
            z = np.load(os.path.join("tests", "golden", "reference_golden.npz"))
            a = {k.split("/", 1)[1]: z[k] for k in z.files if k.startswith(name + "/")}
            fields = ("fixed_transforms", "joint_types", "spheres_flat", "sphere_to_joint", "self_cc_ranges_flat",
                      "joint_lower", "joint_upper", "joint_parents", "joint_id_to_dof", "t_memory_idx", "dfs_order",
                      "approx_spheres_flat", "approx_sphere_to_joint", "approx_self_cc_ranges_flat")
            ASSETS[name] = {"name": name, "n_dof": int(a["n_dof"]), "n_joints": int(a["n_joints"]),
                            **{k: a[k].tolist() for k in fields}}
        else:
            ASSETS[name] = getattr(workloads, name)()
    return ASSETS[name]


def link_spheres(asset, q):
    """[N, S, 3] world centres of the collision spheres, in the precision of q [N, D]."""
    n, to = len(q), dict(device=q.device, dtype=q.dtype)
    fixed = torch.tensor(asset["fixed_transforms"], **to).reshape(-1, 4, 4)
    frames = [None] * asset["n_joints"]
    for k, j in enumerate(asset["dfs_order"]):
        if k == 0:   # the root's frame is the base
            frames[j] = torch.eye(4, **to).expand(n, 4, 4)
            continue
        dof, typ = asset["joint_id_to_dof"][j], asset["joint_types"][j]
        v = q[:, dof] if dof >= 0 else torch.zeros_like(q[:, 0])
        one, nil = torch.ones_like(v), torch.zeros_like(v)
        if typ < 3:   # prismatic along x, y, z
            t = [nil, nil, nil]
            t[typ] = v
            rows = [one, nil, nil, t[0], nil, one, nil, t[1], nil, nil, one, t[2]]
        else:
            c, s = torch.cos(v), torch.sin(v)
            rows = [[one, nil, nil, nil, nil, c, -s, nil, nil, s, c, nil],
                    [c, nil, s, nil, nil, one, nil, nil, -s, nil, c, nil],
                    [c, -s, nil, nil, s, c, nil, nil, nil, nil, one, nil]][typ - 3]
        m = torch.stack(rows + [nil, nil, nil, one], -1).reshape(n, 4, 4)
        frames[j] = frames[asset["joint_parents"][j]] @ fixed[j] @ m
    f = torch.stack([frames[j] for j in asset["sphere_to_joint"]], 1)
    centre = torch.tensor(asset["spheres_flat"], **to).reshape(-1, 4)[:, :3]
    return (f[..., :3, :3] @ centre[..., None])[..., 0] + f[..., :3, 3]


def make_esdf(rng, n):
    """workloads.random_esdf's distance field (16 boxes, 5 mm voxels, 2 unobserved outer layers), made on the GPU."""
    voxel, ext = 0.005, (n - 1) * 0.005
    g = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) * voxel - ext * 0.5
    p = torch.stack(torch.meshgrid(g, g, g, indexing="ij"), -1)
    best = torch.full(p.shape[:3], -1e9, device="cuda", dtype=torch.float64)
    for _ in range(16):
        c = torch.from_numpy(rng.uniform(-ext * 0.35, ext * 0.35, 3)).cuda()
        h = torch.from_numpy(rng.uniform(0.02, 0.08, 3)).cuda()
        q = (p - c).abs() - h
        best = torch.maximum(best, -(q.clamp(min=0).norm(dim=-1) + q.amax(-1).clamp(max=0)))
    f = torch.full((n, n, n), -1000.0, device="cuda", dtype=torch.float32)
    f[2:-2, 2:-2, 2:-2] = best.float()[2:-2, 2:-2, 2:-2]
    pose = np.zeros((1, 8), np.float32)
    pose[0, :4] = (-0.45, 0.0, -0.45, 1.0)
    return np.array([[ext, ext, ext, voxel]], np.float32), pose, np.ones(1, np.uint8), f.reshape(1, -1).cpu().numpy()


def rotation(q):
    """Matrix of the quaternion (w, u): v + 2w(u x v) + 2u x (u x v)."""
    K = np.array([[0, -q[3], q[2]], [q[3], 0, -q[1]], [-q[2], q[1], 0]])
    return np.eye(3) + 2 * q[0] * K + 2 * K @ K


def scene_of(case, rng):
    reach, lo, hi = FIELDS[case["field"]]
    asset = asset_of(case["robot"])
    home = (np.array(asset["joint_lower"]) + np.array(asset["joint_upper"])) / 2
    centre = link_spheres(asset, torch.from_numpy(home)[None])[0].numpy()
    radius = np.array(asset["spheres_flat"]).reshape(-1, 4)[:, 3]
    kept = []
    while len(kept) < case["obbs"]:   # boxes clear of the robot with its joints at mid range, its base above all
        for d, p, en in zip(*workloads.random_obbs(rng, case["obbs"], -reach, reach, lo, hi)):
            local = rotation(p[3:7].astype(np.float64)) @ centre.T + p[:3, None]
            gap = np.linalg.norm(np.maximum(np.abs(local) - d[:3, None] / 2, 0), axis=0) - radius
            if gap.min() > 0.05 and len(kept) < case["obbs"]:
                kept.append((d, p, en))
    boxes = [np.stack(x) for x in zip(*kept)]
    layers = make_esdf(rng, case["esdf"]) if case["esdf"] else ()
    # the mixed batch's costs want a gradient of the distance field, so it samples trilinearly
    mode = _lib.PS_ESDF_TRILINEAR if case["kind"] == "mixed" else _lib.PS_ESDF_NEAREST
    return SceneTensors(*boxes, *layers, esdf_mode=mode)


def noisy_rollouts(rng, asset, n_base, n_noisy, T):
    """[n_base * n_noisy, D, T]: noise L z around straight lines, L from the inverse of the smoothness metric."""
    base = torch.from_numpy(workloads.straight_trajectories(rng, asset, n_base, T, 0.0)).cuda().double()
    g = torch.Generator("cuda").manual_seed(int(rng.integers(1 << 31)))
    z = torch.randn((n_base, n_noisy, asset["n_dof"], T), device="cuda", dtype=torch.float64, generator=g)
    q = base.transpose(1, 2)[:, None] + z @ torch.from_numpy(workloads.stomp_noise_L(T, 0.1)).cuda().T
    lo = torch.tensor(asset["joint_lower"], device="cuda", dtype=torch.float64)[:, None]
    hi = torch.tensor(asset["joint_upper"], device="cuda", dtype=torch.float64)[:, None]
    return torch.minimum(hi, torch.maximum(lo, q)).float().reshape(-1, asset["n_dof"], T).contiguous()


def cost_params(case):
    return api.CostParams(collision_cost_weight=20.0, world_collision_margin=0.05, self_collision_margin=0.01,
                          smoothness_weight=0.0 if case["kind"] == "rollouts" else 1.0, delta_t=0.1)


def edge_params(case):
    if case["step"] == 0.0:   # the reference's default: 16 samples an edge
        return api.EdgeEvalParams(check_self=case["self"], collision_margin=case["margin"])
    return api.EdgeEvalParams(max_joint_step=case["step"], max_samples=600, check_self=case.get("self", False),
                              compute_clearance=case.get("clearance", False), collision_margin=case.get("margin", 0.0))


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind, asset = case["kind"], asset_of(case["robot"])
    s = {"case": case, "asset": asset, "robot": RobotModelBuilder.from_asset(asset).build(),
         "scene": scene_of(case, rng)}
    if kind == "configs":
        s["q"] = torch.from_numpy(workloads.uniform_configs(rng, asset, case["n"])).cuda()
    elif kind in ("edges", "bridge"):
        frm, to, _ = workloads.edge_batch(rng, asset, case["n"], case["step"] or 0.01)
        s["params"] = edge_params(case)
        if kind == "bridge":
            s["from"], s["to"] = frm, to
            s["bridge"] = api.EdgeEvalGpu(asset["n_dof"], max(case["n"], 256), s["scene"], s["robot"])
        else:
            s["from"], s["to"] = torch.from_numpy(frm).cuda(), torch.from_numpy(to).cuda()
            s["workspace"] = api.edges_workspace(case["n"])
    elif kind in ("cost", "autograd"):
        s["q"] = torch.from_numpy(workloads.straight_trajectories(rng, asset, case["b"], case["t"])).cuda()
        s["q"].requires_grad_(kind == "autograd")
        s["params"] = cost_params(case)
    elif kind == "rollouts":
        n_noisy = min(case["b"], 128)
        s["q"] = noisy_rollouts(rng, asset, -(-case["b"] // n_noisy), n_noisy, case["t"])[:case["b"]].contiguous()
        s["params"] = cost_params(case)
    elif kind == "mixed":
        sizes = np.random.default_rng(17)   # 16 to 256 edges a request, 32 to 128 waypoints, the same for every seed
        s["edges"] = []
        for n in sizes.integers(16, 257, case["edge_requests"]):
            frm, to, _ = workloads.edge_batch(rng, asset, int(n))
            s["edges"].append((torch.from_numpy(frm).cuda(), torch.from_numpy(to).cuda()))
        s["trajectories"] = [torch.from_numpy(workloads.straight_trajectories(rng, asset, 1, int(t))[0]).cuda()
                             for t in sizes.integers(32, 129, case["trajectories"])]
        s["rollouts"] = [noisy_rollouts(rng, asset, 1, 8, int(t))
                         for t in sizes.integers(32, 129, case["rollout_requests"])]
        s["params"], s["edge_params"] = cost_params(case), edge_params(case)
        s["batch"] = api.MixedBatch(s["robot"], 12, 12 * 256, 12, 8 * 128 + 4 * 8 * 128, 128)
    else:
        def free(q):
            hit, _ = api.check_configs(s["robot"], s["scene"], torch.from_numpy(q).cuda(), check_self=True)
            return hit.cpu().numpy() == 0

        starts, goals = workloads.free_pairs(rng, asset, case["b"], free, 8 + 512 // case["b"])
        s["starts"], s["goals"] = torch.from_numpy(starts).cuda(), torch.from_numpy(goals).cuda()
        settings = api.ChompSettings if kind == "chomp_solve" else api.StompSettings
        s["settings"] = settings(num_timesteps=case["t"])
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "configs":
        hit, clr = api.check_configs(s["robot"], s["scene"], s["q"], case["margin"],
                                     None if case["clearance"] == "none" else case["clearance"], case["self"])
        return {"hit": hit, "clearance": clr}
    if kind == "edges":
        valid, cost, clr = api.check_edges(s["robot"], s["scene"], s["from"], s["to"], params=s["params"],
                                           workspace=s["workspace"])
        return {"valid": valid, "cost": cost, "clearance": clr if case["clearance"] else None}
    if kind == "bridge":
        valid, cost, _ = s["bridge"].evaluate(s["from"], s["to"], case["n"], s["params"])
        return {"valid": valid, "cost": cost}
    if kind == "cost":
        wp, cost, grad = api.traj_cost(s["robot"], s["scene"], s["q"], s["params"])
        return {"waypoint": wp, "cost": cost, "grad": grad}
    if kind == "autograd":
        cost = api.hinge_cost(s["q"], s["robot"], s["scene"], s["params"])
        return {"cost": cost, "grad": torch.autograd.grad(cost.sum(), s["q"])[0]}
    if kind == "rollouts":
        return {"cost": api.rollout_costs(s["robot"], s["scene"], s["q"], s["params"])}
    if kind == "mixed":
        batch = s["batch"]
        batch.clear()
        edges = [batch.add_edges(f, t) for f, t in s["edges"]]
        trajs = [batch.add_trajectory(q) for q in s["trajectories"]]
        rolls = [batch.add_rollouts(r) for r in s["rollouts"]]
        batch.launch(s["scene"], s["edge_params"], s["params"])
        return {"edges": edges, "trajectories": trajs, "rollouts": rolls}
    solve = api.chomp_solve if kind == "chomp_solve" else api.stomp_solve
    r = solve(s["robot"], s["scene"], s["starts"], s["goals"], s["settings"])
    return {"path": r.path, "solved": r.solved, "iterations": r.iterations, "cost": r.cost, "theta": r.theta}


def work(case):
    """Queries read and results written once. Operations: every configuration that the answer rests on has its chain
    walked (90 a joint), its spheres placed (18) and each of them met with its nearest box (30). A free edge rests on
    all its samples, one in collision on one; uniform edges average 200 steps of 0.01 rad, local ones 25, and about
    half of the edges are free. Solves: the usual number of iterations."""
    a, kind = asset_of(case["robot"]), case["kind"]
    D, S = a["n_dof"], len(a["sphere_to_joint"])
    per = 90.0 * (a["n_joints"] - 1) + 48.0 * S
    if kind == "configs":
        return {"bytes": case["n"] * (4.0 * D + 1 + (4 if case["clearance"] != "none" else 0)), "flops": case["n"] * per}
    if kind in ("edges", "bridge"):
        samples = 16 if case["step"] == 0.0 else 112 * 0.01 / case["step"]
        return {"bytes": case["n"] * (8.0 * D + 5), "flops": case["n"] * (1 + 0.5 * samples) * per}
    if kind in ("cost", "autograd", "rollouts"):
        n = case["b"] * case["t"]
        return {"bytes": n * (4.0 * D * (1 if kind == "rollouts" else 2) + 4),
                "flops": n * per * (1 if kind == "rollouts" else 2)}
    if kind == "mixed":
        n_e = case["edge_requests"] * 136
        n_t, n_r = case["trajectories"] * 80, case["rollout_requests"] * 8 * 80
        return {"bytes": n_e * (8.0 * D + 5) + n_t * (8.0 * D + 4) + n_r * (4.0 * D + 4),
                "flops": (n_e * (1 + 0.5 * 1.12 / case["step"]) + 2 * n_t + n_r) * per}
    n = case["b"] * case["t"]
    passes = 60 * 2 if kind == "chomp_solve" else 12 * 30
    return {"bytes": n * 8.0 * D, "flops": n * per * passes}


# ---------------------------------------------------------------------------
# what run() returns, in 64 bits
# ---------------------------------------------------------------------------
class Exact:
    """Spheres, distances and costs of one model and scene in plain 64-bit torch."""

    def __init__(self, s):
        a, f64 = s["asset"], dict(device="cuda", dtype=torch.float64)
        self.a, self.D = a, a["n_dof"]
        self.radius = torch.tensor(a["spheres_flat"], **f64).reshape(-1, 4)[:, 3]
        host = s["scene"].host
        dims = torch.from_numpy(host["obb_dims"]).to(**f64)
        pose = torch.from_numpy(host["obb_pose"]).to(**f64)
        self.half, self.t = dims[:, :3] / 2, pose[:, :3]
        self.R = torch.tensor(np.stack([rotation(q) for q in host["obb_pose"][:, 3:7].astype(np.float64)]), **f64)
        self.layer = None
        if "voxel_params" in host:
            p = host["voxel_params"][0].astype(np.float64)
            n = int(round(p[0] / p[3])) + 1
            self.layer = (p[0], p[3], n, torch.from_numpy(host["voxel_features"][0]).cuda().reshape(n, n, n),
                          torch.from_numpy(host["voxel_pose"][0, :3]).to(**f64))
        r = np.asarray(a["self_cc_ranges_flat"], np.int64).reshape(-1, 3)
        i = np.concatenate([np.full(e - b + 1, k) for k, b, e in r])
        j = np.concatenate([np.arange(b, e + 1) for _, b, e in r])
        self.pairs = torch.from_numpy(i).cuda(), torch.from_numpy(j).cuda()

    def boxes(self, p):
        """[N, S] signed distance of every sphere centre to the nearest box."""
        loc = torch.einsum("bij,nsj->nsbi", self.R, p) + self.t
        q = loc.abs() - self.half
        out = q.clamp(min=0)
        sq = (out * out).sum(-1)
        d = torch.where(sq > 0, torch.where(sq > 0, sq, 1.0).sqrt(), q.amax(-1).clamp(max=0))
        return d.amin(-1).clamp(max=1000.0 + self.radius)

    def self_gap(self, p):
        """[N] smallest distance between the surfaces of two spheres of a pair."""
        i, j = self.pairs
        return ((p[:, i] - p[:, j]).norm(dim=-1) - (self.radius[i] + self.radius[j])).amin(-1)

    def field(self, p):
        """[N, S] trilinear distance of the layer, -1000 where it says nothing ("positive = inside")."""
        ext, voxel, n, f, t = self.layer
        g = (p + t + ext * 0.5) / voxel
        lo = g.detach().floor()
        seen = ((lo > 2) & (lo + 1 < n - 2)).all(-1)
        i = lo.clamp(0, n - 2).long()
        x = g - lo
        d = 0.0
        for cx in (0, 1):
            for cy in (0, 1):
                for cz in (0, 1):
                    v = f[i[..., 0] + cx, i[..., 1] + cy, i[..., 2] + cz].double()
                    seen = seen & (v > -999.0)
                    wx, wy, wz = (x[..., k] if c else 1 - x[..., k] for k, c in enumerate((cx, cy, cz)))
                    d = d + wx * wy * wz * v
        return torch.where(seen, d, -1000.0)

    def cost(self, q, p):
        """[N] weight * (sum of the spheres' hinges + self hinge) of q [N, D]."""
        x = link_spheres(self.a, q)
        m, hinge = p.world_collision_margin, 0.0
        if self.layer is not None:
            hinge = (m + self.field(x) + self.radius).clamp(min=0).sum(-1)
        hinge = hinge + (m - (self.boxes(x) - self.radius)).clamp(min=0).sum(-1)
        return p.collision_cost_weight * (hinge + (p.self_collision_margin - self.self_gap(x)).clamp(min=0))

    def costs(self, q, p, grad):
        """Waypoint costs [N] and, if asked for, their gradients [N, D]."""
        step = max(1, 20_000_000 // (len(self.radius) * len(self.half)))
        cs, gs = [], []
        for k in range(0, len(q), step):
            x = q[k:k + step].detach().double().requires_grad_(grad)
            with torch.set_grad_enabled(grad):
                c = self.cost(x, p)
            cs.append(c.detach())
            if grad:
                gs.append(torch.autograd.grad(c.sum(), x)[0])
        return torch.cat(cs), torch.cat(gs) if grad else None

    def trajectories(self, q, p):
        """Waypoint costs, totals with smoothness_weight * q'Rq, and gradients of q [B, T, D]."""
        B, T, D = q.shape
        c, g = self.costs(q.reshape(-1, D), p, True)
        R = torch.from_numpy(smoothness(T, p.delta_t)).cuda() * p.smoothness_weight
        Rq = torch.einsum("ts,bsd->btd", R, q.detach().double())
        total = c.reshape(B, T).sum(1) + (q.detach().double() * Rq).sum((1, 2))
        return c.reshape(B, T), total, g.reshape(B, T, D) + 2 * Rq

    def hits(self, q, margin, check_self):
        out = [torch.zeros(0, dtype=torch.bool, device="cuda")]
        step = max(1, 20_000_000 // (len(self.radius) * len(self.half)))
        for k in range(0, len(q), step):
            x = link_spheres(self.a, q[k:k + step].double())
            h = (self.boxes(x) < self.radius + margin).any(-1)
            out.append(h | (self.self_gap(x) < 0) if check_self else h)
        return torch.cat(out)


def smoothness(T, dt):
    """dt A'A, A the 5-point second difference on the trajectory padded by 6 on both sides, its T x T centre."""
    A = sum(np.diag(np.full(T + 12 - abs(k), v), k) for k, v in
            {-2: -1 / 12, -1: 16 / 12, 0: -30 / 12, 1: 16 / 12, 2: -1 / 12}.items()) / (dt * dt)
    return (dt * A.T @ A)[6:6 + T, 6:6 + T]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("chomp_solve", "stomp_solve"):
        return None   # iterates of a loop that stops on verdicts
    if case["esdf"] and kind != "mixed":
        return None   # nearest-voxel lookups: a value's voxel is decided by rounding
    s = prepare(case, seed)
    e = Exact(s)
    if kind == "configs":
        if case["clearance"] == "none":
            return None
        clr = [(e.boxes(x) - (e.radius + case["margin"])).amin(-1)
               for x in (link_spheres(e.a, q.double()) for q in s["q"].split(max(1, 20_000_000 // (59 * case["obbs"]))))]
        return {"hit": None, "clearance": torch.cat(clr)}
    if kind in ("edges", "bridge"):
        return {"valid": None, "cost": edge_costs(e, case, torch.as_tensor(s["from"]).cuda(),
                                                  torch.as_tensor(s["to"]).cuda()), "clearance": None}
    if kind in ("cost", "autograd"):
        wp, total, grad = e.trajectories(s["q"], s["params"])
        return {"waypoint": wp, "cost": total, "grad": grad} if kind == "cost" else {"cost": total, "grad": grad}
    if kind == "rollouts":
        B, D, T = s["q"].shape
        c, _ = e.costs(s["q"].transpose(1, 2).reshape(-1, D), s["params"], False)
        return {"cost": c.reshape(B, T)}
    trajs = [e.trajectories(q[None], s["params"]) for q in s["trajectories"]]
    rolls = [e.costs(r.transpose(1, 2).reshape(-1, e.D), s["params"], False)[0].reshape(r.shape[0], -1)
             for r in s["rollouts"]]
    return {"edges": [(None, None) for _ in s["edges"]], "rollouts": rolls,
            "trajectories": [(w[0], c, g[0]) for w, c, g in trajs]}


def edge_costs(e, case, frm, to):
    """Lengths of the free edges, the largest float for the others: samples j/G for j = 1..G, and the start where G
    is no multiple of 16. Few samples of each edge first, so that most in collision are known early."""
    n = len(frm)
    diff = (to - frm).abs().amax(1)
    G = (torch.full((n,), 16, device="cuda") if case["step"] == 0.0
         else (diff / torch.tensor(case["step"], device="cuda")).ceil().long().clamp(1, 600))
    a, d = frm.double(), (to - frm).double()
    live = torch.arange(n, device="cuda")

    def drop(live, edge, t):
        hit = e.hits(a[edge] + t[:, None] * d[edge], case["margin"], case["self"])
        bad = torch.zeros(n, dtype=torch.bool, device="cuda")
        bad[edge[hit]] = True
        return live[~bad[live]]

    for t in (1.0, 0.5, 0.25, 0.75):
        j = (G[live] * t).ceil()
        live = drop(live, live, j / G[live])
    live = drop(live, live[G[live] % 16 != 0], torch.zeros(int((G[live] % 16 != 0).sum()), device="cuda").double())
    edge = torch.repeat_interleave(live, G[live])
    first = torch.repeat_interleave(torch.cumsum(G[live], 0) - G[live], G[live])
    j = torch.arange(len(edge), device="cuda") - first + 1
    live = drop(live, edge, j.double() / G[edge])
    cost = torch.full((n,), float(np.finfo(np.float32).max), device="cuda", dtype=torch.float64)
    cost[live] = d[live].norm(dim=1)
    return cost
