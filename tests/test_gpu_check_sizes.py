"""The checkers at the sizes where their launches change: edges by warps of 32
points (granularities around 32 and to the largest), small configuration counts
spread over more warps (around every doubling of 8 warps' lanes per SM).
Against the plain checker (prrtc_validate_configs_noalloc, every obstacle, one
configuration per lane); verdicts are equal."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def plain():
    import torch
    from prrtc_gb300 import api
    f = api.lib().prrtc_validate_configs_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_int, C.POINTER(api.EnvDesc), C.c_void_p, C.c_int64, C.c_void_p, C.c_void_p]

    def check(robot, env, q):
        desc, keep = api._env_desc(env)
        qd = torch.from_numpy(q).cuda()
        out = torch.full((len(q),), 7, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        assert f(api.robot_id(robot), C.byref(desc), qd.data_ptr(), len(q), out.data_ptr(), None) == 0
        torch.cuda.synchronize()
        return out.cpu().numpy()
    return check


def _configs(robot, n, seed):
    from prrtc_gb300 import scenes
    sc, off = (np.array(v) for v in scenes.LIMITS[robot])
    return (np.random.default_rng(seed).random((n, len(sc))) * sc + off).astype(np.float32)


@pytest.mark.parametrize("robot", ["panda", "fetch", "baxter"])
@pytest.mark.parametrize("n,g", [(1, 1), (1, 32), (5, 31), (5, 33), (333, 64), (7, 127), (3, 1000), (2, 1024)])
def test_edges_equal_their_points(robot, n, g, ctx, plain):
    from prrtc_gb300 import scenes
    env = scenes.shelf_scene(2, n_zaligned=6)
    a = _configs(robot, n, g)
    b = (a + np.random.default_rng(n).uniform(-0.3, 0.3, a.shape)).astype(np.float32)
    step = (b - a) / np.float32(g)
    k = np.arange(1, g + 1, dtype=np.float32)[None, :, None]
    points = (a[:, None] + k * step[:, None]).astype(np.float32)
    want = plain(robot, env, points.reshape(-1, a.shape[1])).reshape(n, g).all(1)
    assert (ctx.validate_edges(robot, env, a, b, g) == want).all()


@pytest.mark.parametrize("robot", ["panda", "fetch", "baxter"])
def test_counts_around_each_spread(robot, ctx, plain):
    import torch
    from prrtc_gb300 import scenes
    env = scenes.tabletop_scene(1, n_zaligned=8)
    lanes = torch.cuda.get_device_properties(0).multi_processor_count * 8 * 32
    q = _configs(robot, lanes + 1, 5)
    want = plain(robot, env, q)
    for n in sorted({1, 31, 33} | {(lanes >> s) + d for s in range(6) for d in (-1, 0, 1)}):
        assert (ctx.validate_configs(robot, env, q[:n]) == want[:n]).all(), n


@pytest.mark.parametrize("robot,waypoints,paths", [("panda", 32, 3), ("panda", 33, 3), ("panda", 65, 400), ("fetch", 129, 2),
                                                   ("baxter", 256, 1)])
def test_smoothing_at_its_block_sizes(robot, waypoints, paths, ctx, plain):
    """128 and 256 threads, waypoints beyond one pass, the largest environment
    beside the longest path: a path is returned as it came or free edge by edge,
    and its cost before is path_cost_grad's (both sums of the same FP64 terms,
    rounded to float32 at the end, there per waypoint)."""
    from prrtc_gb300 import SmoothSettings
    from prrtc_gb300.env import Environment
    rng = np.random.default_rng(waypoints)
    far = np.column_stack([rng.uniform(1.5, 2.5, (2815, 3)), rng.uniform(0.005, 0.02, 2815)]).astype(np.float32)
    env = ctx.upload_env(Environment(spheres=[[0.6, 0.0, 0.9, 0.1], *far]))
    ends = _configs(robot, 2 * paths, 3).reshape(paths, 2, 1, -1)
    t = np.linspace(0.0, 1.0, waypoints, dtype=np.float32)[None, :, None]
    q = (ends[:, 0] + t * (0.1 * (ends[:, 1] - ends[:, 0]))).astype(np.float32)
    cost, _ = ctx.path_cost_grad(robot, env, q)
    out, acc, before, after = ctx.smooth_paths(robot, env, q, SmoothSettings(steps=2, granularity=5))
    total = cost.astype(np.float64).sum(1)
    assert (np.abs(before - total) <= 2.0 ** -22 * total + 1e-12).all()
    assert (out[acc == 0] == q[acc == 0]).all() and np.isfinite(after).all()
    for p in np.flatnonzero(acc):
        assert ctx.validate_edges(robot, env, out[p, :-1], out[p, 1:], 5).all()
