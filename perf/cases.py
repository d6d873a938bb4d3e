"""The work that a program has this library do, case by case, through its Python entry points.

listed() gives named cases, draw() more of the same ranges.  prepare() builds
a case's inputs on the GPU from a seed (uploaded scenes, configurations,
paths, a prepared query array), run() is one call as a program makes it,
work() the bytes and operations the call cannot do without, and exact() the
same results in float64, from the robot model tables and plain torch.

Scenes, planner settings and sizes are those of prrtc_gb300.workloads, the
benchmark and the tests: tabletop and shelf scenes, mixed clutter of 5 to 60
obstacles, 2^20 configurations, 2^14 edges, paths of 64 waypoints, batches of
256 to some thousand queries.
"""
import json
import math
from pathlib import Path

import numpy as np
import torch

from prrtc_gb300 import BatchSettings, Context, Settings, SmoothSettings, autotune, scenes
from prrtc_gb300.workloads import SETTINGS

ROBOT_DIR = Path(scenes.__file__).resolve().parent / "robots"
DOF = {"panda": 7, "fetch": 8, "baxter": 14}
SPHERES = {"panda": 69, "fetch": 125, "baxter": 100}


def listed():
    return [
        # a control loop asks whether a hundred candidate configurations are free
        {"name": "check_panda_100", "op": "check", "robot": "panda", "scene": "tabletop", "n": 100},
        # sampling-based work on one scene: a million random configurations
        {"name": "check_panda_1m", "op": "check", "robot": "panda", "scene": "shelf", "n": 1 << 20},
        # two arms in clutter with every obstacle type, an odd count
        {"name": "check_baxter_200k", "op": "check", "robot": "baxter", "scene": "mixed", "obstacles": 60, "z": 12,
         "n": 200_003},
        # roadmap and path checking: edges at the planner's shelf resolution
        {"name": "edges_panda_16k", "op": "edges", "robot": "panda", "scene": "shelf", "n": 1 << 14, "granularity": 128},
        # a few hundred edges in clutter at a resolution that is no multiple of the block
        {"name": "edges_fetch_1k", "op": "edges", "robot": "fetch", "scene": "mixed", "obstacles": 30, "z": 0, "n": 1001,
         "granularity": 50},
        # kinematics for display, distance queries and learning: every model sphere
        {"name": "fk_panda_100k", "op": "fk", "robot": "panda", "n": 100_000},
        # a trajectory optimiser's gradient: thousands of paths of 64 waypoints
        {"name": "clearance_panda_4k", "op": "clearance", "robot": "panda", "scene": "shelf", "scenes": 32, "paths": 4096,
         "waypoints": 64},
        # the planner's paths repaired, shortened and judged, two robots
        {"name": "smooth_panda_1k", "op": "smooth", "robot": "panda", "scene": "shelf", "scenes": 32, "paths": 1024,
         "waypoints": 64, "steps": 50},
        {"name": "smooth_baxter_32", "op": "smooth", "robot": "baxter", "scene": "tabletop", "scenes": 8, "paths": 32,
         "waypoints": 64, "steps": 50},
        # one query at a time, the reference planner's own call
        {"name": "solve_panda", "op": "solve", "robot": "panda", "scene": "tabletop"},
        # a batch of easy queries, answered as fast as the GPU can
        {"name": "batch_tabletop_1k", "op": "batch", "robot": "panda", "scene": "tabletop", "scenes": 64, "n": 1024,
         "workers": 0, "samples": 1 << 22},
        # a reproducible batch in narrow passages: one worker per query and a bounded number of samples each
        {"name": "batch_shelf_4k", "op": "batch", "robot": "panda", "scene": "shelf", "scenes": 64, "n": 4096,
         "workers": 1, "samples": 6_000},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["check", "check", "edges", "edges", "fk", "clearance", "smooth", "solve", "batch", "batch"])
    robot = rng.choice(["panda", "panda", "fetch", "baxter"])
    scene = "mixed" if robot == "fetch" else rng.choice(["tabletop", "shelf", "mixed"])
    c = {"op": op, "robot": robot, "scene": scene}
    if scene == "mixed":
        c |= {"obstacles": rng.randint(5, 60), "z": rng.choice([0, 0, 6, 12])}
    if op == "check":
        c["n"] = size(16, 1 << 20 if robot == "panda" else 300_000)
    elif op == "edges":
        c["granularity"] = rng.choice([1, 32, 50, 64, 128, 200])
        c["n"] = size(16, (1 << 21 if robot == "panda" else 1 << 19) // max(32, c["granularity"]))
    elif op == "fk":
        c = {"op": op, "robot": robot, "n": size(1, 100_000)}
    elif op == "clearance":
        c["waypoints"] = rng.choice([1, 17, 64, 100])
        c["paths"] = size(1, 262_144 // (64 if robot == "panda" else 400))
        c["scenes"] = min(c["paths"], rng.randint(1, 32))
    elif op == "smooth":
        c["waypoints"], c["steps"] = rng.choice([20, 64, 64, 100]), rng.choice([10, 50])
        c["paths"] = size(1, 1024 if robot == "panda" else 128)
        c["scenes"] = min(c["paths"], rng.randint(1, 16))
    elif op == "solve":
        c = {"op": op, "robot": "panda", "scene": rng.choice(["tabletop", "mixed"]), "obstacles": rng.randint(5, 30), "z": 0}
    else:
        # racing workers only where every query is easy: a query at its sample limit is answered by chance
        racing = robot == "panda" and rng.random() < 0.5
        c = {"op": op, "robot": robot, "scene": "tabletop" if racing else scene, "workers": 0 if racing else 1,
             "samples": 1 << 22 if racing else size(600, 6000 if robot == "panda" else 1500), "n": size(2, 2048 if robot == "panda" else 256)} | {
                 k: v for k, v in c.items() if k in ("obstacles", "z") and not racing}
        c["scenes"] = min(c["n"], rng.randint(1, 64))
    return c


# ---- inputs ----------------------------------------------------------------

_context = None


def context():
    """The process's library context, kept as a program keeps it."""
    global _context
    if _context is None:
        _context = Context(0)
    return _context


def environment(case, seed, k=0):
    s = (seed % (1 << 30)) * 4096 + k
    z = 0.3 if case["robot"] == "baxter" else 0.0
    if case["scene"] == "mixed":
        return scenes.mixed_scene(s, case["obstacles"], n_zaligned=case["z"])
    return scenes.tabletop_scene(s, z) if case["scene"] == "tabletop" else scenes.shelf_scene(s, z)


def ready():
    """The library runs on its own stream: what torch has queued is finished before a call reads it."""
    torch.cuda.current_stream().synchronize()


def generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def random_configs(robot, n, g):
    scale, offset = (torch.tensor(v, dtype=torch.float32, device="cuda") for v in scenes.LIMITS[robot])
    return (torch.rand((n, DOF[robot]), generator=g, device="cuda") * scale + offset).contiguous()


def free_configs(robot, env, n, g, clear=0.0):
    """[n, dof] random collision-free configurations (with `clear`: no leaf test nearer than that)."""
    ctx, got, left = context(), [], n
    while left > 0:
        q = random_configs(robot, 4 * left + 64, g)
        ready()
        q = q[ctx.validate_configs(robot, env, q).bool()]
        if clear and len(q):
            ready()
            q = q[ctx.path_cost_grad(robot, env, q[None], clear)[0][0] == 0]
        got.append(q[:left])
        left -= len(got[-1])
    return torch.cat(got)


def shelf_goals(robot, env, n, seed):
    """[n, dof] free configurations with the hand inside shelf cells."""
    hand, cells = scenes.hand_sphere(robot), scenes.shelf_cells(0.3 if robot == "baxter" else 0.0)
    found, order = [], np.random.default_rng(seed).permutation(len(cells))
    for k, cell in enumerate(order):
        lo, hi = cells[cell]
        found += list(context().sample_goals(robot, env, hand, lo, hi, max_goals=max(1, n // 4), tries=1 << 17, seed=seed + k))
        if len(found) >= n:
            break
    if not found:
        return free_configs(robot, env, n, generator(seed)).cpu().numpy()
    return np.stack([found[i % len(found)] for i in range(n)])


def polylines(robot, env, n, waypoints, g, seed):
    """[n, waypoints, dof] collision-free paths of one to three straight segments, as a planner returns them."""
    rng = np.random.default_rng(seed)
    nodes = free_configs(robot, env, 192, g)
    i, j = (torch.from_numpy(rng.integers(0, 192, 8192)).cuda() for _ in range(2))
    a, b = nodes[i], nodes[j]
    ready()
    ok = context().validate_edges(robot, env, a, b, 64).bool() & (i != j)
    to = [[] for _ in range(192)]
    for a, b in zip(i[ok].tolist(), j[ok].tolist()):
        to[a].append(b)
    starts = [k for k in range(192) if to[k]] or [0]
    walks = np.zeros((n, waypoints, 2), np.int64)   # the segment's ends at every row
    share = np.zeros((n, waypoints), np.float64)
    for p in range(n):
        walk = [starts[int(rng.integers(len(starts)))]]
        for _ in range(int(rng.integers(1, 4))):
            nxt = to[walk[-1]]
            walk.append(nxt[int(rng.integers(len(nxt)))] if nxt else walk[-1])
        at = np.linspace(0.0, len(walk) - 1, waypoints)
        k = np.minimum(at.astype(np.int64), len(walk) - 2)
        w = np.asarray(walk)
        walks[p, :, 0], walks[p, :, 1], share[p] = w[k], w[k + 1], at - k
    a, b = (nodes[torch.from_numpy(walks[:, :, e]).cuda()].double() for e in (0, 1))
    return (a + (b - a) * torch.from_numpy(share).cuda()[..., None]).float().contiguous()


def many_scenes(case, seed):
    return [context().upload_env(environment(case, seed, k)) for k in range(case["scenes"])]


def paths_input(case, seed):
    """Environments (one per path) and paths, interleaved over the scenes."""
    envs, g = many_scenes(case, seed), generator(seed)
    P, S = case["paths"], case["scenes"]
    q = torch.empty((P, case["waypoints"], DOF[case["robot"]]), device="cuda")
    for k, e in enumerate(envs):
        mine = len(range(k, P, S))
        q[k::S] = polylines(case["robot"], e, mine, case["waypoints"], g, seed + k)
    return [envs[i % S] for i in range(P)], q


def plan_settings(case):
    name = {"panda": "panda_shelf" if case["scene"] == "shelf" else "panda_tabletop", "fetch": "fetch_mixed",
            "baxter": "baxter_mixed"}[case["robot"]]
    return name, dict(SETTINGS[name])


def prepare(case, seed):
    op, robot, ctx = case["op"], case["robot"], context()
    s = dict(case)
    if op in ("check", "edges"):
        s["env"], g = ctx.upload_env(environment(case, seed)), generator(seed)
        s["a"] = random_configs(robot, case["n"], g)
        if op == "edges":   # steps of a planner: from free configurations, up to the length of its range
            s["a"] = free_configs(robot, s["env"], case["n"], g)
            way = random_configs(robot, case["n"], g) - s["a"]
            reach = torch.rand((case["n"], 1), generator=g, device="cuda") * 1.5
            s["b"] = (s["a"] + way * (reach / way.norm(dim=1, keepdim=True))).contiguous()
    elif op == "fk":
        s["a"] = random_configs(robot, case["n"], generator(seed))
    elif op == "clearance":
        s["envs"], s["q"] = paths_input(case, seed)
    elif op == "smooth":
        s["envs"], s["q"] = paths_input(case, seed)
        s["settings"] = SmoothSettings(steps=case["steps"])
    elif op == "solve":
        s["env"] = ctx.upload_env(environment(case, seed))
        s["start"], s["goal"] = free_configs(robot, s["env"], 2, generator(seed), 0.002).cpu().numpy()
        s["settings"] = Settings(**plan_settings(case)[1])
    else:
        name, plan = plan_settings(case)
        queries, g, S = [None] * case["n"], generator(seed), case["scenes"]
        for k in range(S):
            env = environment(case, seed, k)
            h, mine = ctx.upload_env(env), len(range(k, case["n"], S))
            q = free_configs(robot, h, 2 * mine, g, 0.002).cpu().numpy()
            ends = shelf_goals(robot, h, mine, seed * 7 + k) if case["scene"] == "shelf" else q[mine:]
            queries[k::S] = [(env, q[i], ends[i]) for i in range(mine)]
        plan["num_new_configs"] = plan.get("num_new_configs", 600)
        plan["max_iters"] = max(1, case["samples"] // plan["num_new_configs"])
        knobs = autotune.load(robot, name)
        if case["workers"] == 1:
            knobs |= {"max_workers_per_attempt": 1, "max_attempts": 1}
        s["settings"] = BatchSettings(Settings(**plan), margin=1e-5, max_nodes_per_tree=16384, **knobs)
        s["prepared"] = ctx.prepare_batch(robot, queries, path_capacity=256)
        s["prepared"].paths.fill(0.0)
    return s


def run(s):
    op, robot, ctx = s["op"], s["robot"], context()
    if op == "check":
        return ctx.validate_configs(robot, s["env"], s["a"])
    if op == "edges":
        return ctx.validate_edges(robot, s["env"], s["a"], s["b"], s["granularity"])
    if op == "fk":
        return ctx.fk_spheres(robot, s["a"])
    if op == "clearance":
        return ctx.path_cost_grad(robot, s["envs"], s["q"])
    if op == "smooth":   # smooths in place: the program keeps its own paths
        q = s["q"].clone()
        ready()
        return ctx.smooth_paths(robot, s["envs"], q, s["settings"])
    if op == "solve":
        # lanes race for the connection: which of the valid paths comes back is a matter of timing, its ends are not
        r = ctx.solve(robot, s["start"], s["goal"], s["env"], s["settings"])
        return {"solved": int(r.solved), "status": r.status, "goal": r.path[:1], "start": r.path[-1:]}
    ctx.solve_prepared(s["prepared"], s["settings"])
    res = s["prepared"].res
    if s["workers"] != 1:   # as above
        each = np.arange(len(res))
        return {"solved": res["solved"], "status": res["status"], "goal": s["prepared"].paths[:, 0],
                "start": s["prepared"].paths[each, np.maximum(res["path_rows"], 1) - 1]}
    return {k: res[k] for k in ("solved", "status", "start_tree_size", "goal_tree_size", "path_length", "iters", "cost",
                                "path_rows", "samples")} | {"paths": s["prepared"].paths}


# ---- what a call cannot do without -----------------------------------------

def env_records(case):
    if case["scene"] == "mixed":
        return 8 * (case["obstacles"] + case["z"]) // 3 + 1
    return 8 + 4 * 5 if case["scene"] == "tabletop" else 20 + 2 * 12 + 4 * 9


def work(case):
    op, robot = case["op"], case["robot"]
    D = DOF[robot]
    kinematics = 2 * (12 * D + 9 * SPHERES[robot])   # one configuration's spheres
    if op == "fk":
        return {"bytes": case["n"] * 4 * (D + 4 * SPHERES[robot]), "flops": case["n"] * kinematics}
    env = 16 * env_records(case)
    if op == "check":
        return {"bytes": env + case["n"] * (4 * D + 1), "flops": case["n"] * kinematics}
    if op == "edges":
        return {"bytes": env + case["n"] * (8 * D + 1), "flops": case["n"] * case["granularity"] * kinematics}
    if op == "clearance":
        rows = case["paths"] * case["waypoints"]
        return {"bytes": case["scenes"] * env + rows * 4 * (2 * D + 1), "flops": 2 * rows * kinematics}
    if op == "smooth":
        rows = case["paths"] * case["waypoints"]
        return {"bytes": case["scenes"] * env + case["paths"] * 9 + rows * 8 * D,
                "flops": rows * kinematics * (2 * (case["steps"] + 2) + 128)}
    if op == "solve":   # a path of some ten nodes, its edges checked once
        return {"bytes": env + 4 * D * 12, "flops": 10 * 32 * kinematics}
    return {"bytes": case["n"] * (env + 4 * D * 12), "flops": case["n"] * 10 * 64 * kinematics}


# ---- the same results in float64 --------------------------------------------

def model(robot):
    """The robot's tables, rounded to float32 as the library compiles them."""
    m = json.loads((ROBOT_DIR / f"{robot}.json").read_text())
    r = lambda v: torch.tensor(np.asarray(v, np.float32).astype(np.float64), device="cuda")  # noqa: E731
    return m, r


def sphere_centres(robot, q):
    """[n, spheres, 3] world centres of float64 configurations q, [spheres] radii."""
    m, r = model(robot)
    n = len(q)
    eye = torch.eye(4, dtype=torch.float64, device="cuda").expand(n, 4, 4)
    T = {-1: eye}
    for jt in m["joints"]:
        F = torch.eye(4, dtype=torch.float64, device="cuda")
        F[:3] = r(jt["F"])
        th = q[:, jt["q"]]
        J = eye.clone()
        if jt["type"] == "revolute":
            J[:, 0, 0], J[:, 0, 1], J[:, 1, 0], J[:, 1, 1] = th.cos(), -th.sin(), th.sin(), th.cos()
        else:
            J[:, 2, 3] = th
        T[jt["q"]] = T[jt["parent"]] @ F @ J
    c = torch.empty((n, len(m["spheres"]), 3), dtype=torch.float64, device="cuda")
    for f in T:
        ids = [i for i, s in enumerate(m["spheres"]) if s["frame"] == f]
        if ids:
            local = r([m["spheres"][i]["c"] for i in ids])
            c[:, ids] = local @ T[f][:, :3, :3].transpose(1, 2) + T[f][:, None, :3, 3]
    return c, r([s["r"] for s in m["spheres"]]), m


def distances(env, c, rad):
    """[n, spheres, obstacles] signed distances of spheres at c to every obstacle."""
    t = lambda a: torch.from_numpy(a.astype(np.float64)).cuda()  # noqa: E731
    length = lambda d: torch.where((d * d).sum(-1) > 0, (d * d).sum(-1), torch.ones_like(d[..., 0])).sqrt() * (  # noqa: E731
        (d * d).sum(-1) > 0)
    x, out = c[:, :, None, :], []
    if len(env.spheres):
        s = t(env.spheres)
        out.append(length(x - s[:, :3]) - (rad[:, None] + s[:, 3]))
    for caps, upright in ((env.capsules, False), (env.z_aligned_capsules, True)):
        if len(caps):
            k = t(caps)
            v = k[:, 3:6] * (torch.tensor([0.0, 0.0, 1.0], device="cuda") if upright else 1.0)
            u = (((x - k[:, :3]) * v).sum(-1) * k[:, 7]).clamp(0.0, 1.0)
            out.append(length(x - k[:, :3] - u[..., None] * v) - (rad[:, None] + k[:, 6]))
    for boxes, upright in ((env.cuboids, False), (env.z_aligned_cuboids, True)):
        if len(boxes):
            k = t(boxes)
            a = k[:, 3:12].reshape(-1, 3, 3).clone()
            if upright:
                a[:, :2, 2] = 0.0
                a[:, 2] = torch.tensor([0.0, 0.0, 1.0], device="cuda", dtype=torch.float64)
            qd = ((x - k[:, :3])[..., None, :] * a).sum(-1).abs() - k[:, 12:15]
            out.append(torch.where((qd > 0).any(-1), length(qd.clamp(min=0.0)), qd.amax(-1)) - rad[:, None])
    return torch.cat(out, -1) if out else None


def clearance_cost(robot, env, q, margin):
    c, rad, m = sphere_centres(robot, q)
    leaves = [i for g in m["env_groups"] for i in g["leaves"]]
    sd = distances(env, c[:, leaves], rad[leaves])
    cost = 0.0 if sd is None else 0.5 * (margin - sd).clamp(min=0.0).square().sum((1, 2))
    pairs = torch.tensor([p for g in m["self_groups"] for p in g["pairs"]], device="cuda")
    d = (c[:, pairs[:, 0]] - c[:, pairs[:, 1]]).square().sum(-1).sqrt() - (rad[pairs[:, 0]] + rad[pairs[:, 1]])
    return cost + 0.5 * (margin - d).clamp(min=0.0).square().sum(1)


def exact(case, seed):
    op, robot = case["op"], case["robot"]
    if op == "fk":
        q = random_configs(robot, case["n"], generator(seed)).double()
        out = []
        for part in q.split(20_000):
            c, rad, _ = sphere_centres(robot, part)
            out.append(torch.cat([c, rad[None, :, None].expand(len(c), -1, 1)], -1).cpu())
        return torch.cat(out)
    if op not in ("clearance", "smooth"):
        return None
    margin = float(np.float32(0.02))
    _, q = paths_input(case, seed)
    P, W, D = q.shape
    cost = torch.empty((P, W), dtype=torch.float64, device="cuda")
    grad = torch.empty((P, W, D), dtype=torch.float64, device="cuda")
    for k in range(case["scenes"]):
        env = environment(case, seed, k)
        mine = q[k::case["scenes"]].reshape(-1, D).double()
        cs, gs = [], []
        for part in mine.split(1024):
            part = part.clone().requires_grad_(op == "clearance")
            v = clearance_cost(robot, env, part, margin)
            cs.append(v.detach())
            if op == "clearance":
                gs.append(torch.autograd.grad(v.sum(), part)[0])
        cost[k::case["scenes"]] = torch.cat(cs).reshape(-1, W)
        if op == "clearance":
            grad[k::case["scenes"]] = torch.cat(gs).reshape(-1, W, D)
    # smoothing's own result depends on which shortcuts the checker allows
    return (cost.cpu(), grad.cpu()) if op == "clearance" else (None, None, cost.sum(1).cpu(), None)
