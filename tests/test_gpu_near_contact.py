"""Verdicts on configurations bisected onto contact: between a free and a
colliding configuration, halved until the two are neighbours in float32, so
that most of them lie within rounding of contact, where the fast form of the
checkers leaves the answer to the exact form.  One configuration has one
verdict, whichever kernel asks: many configurations a call and few, one edge's
points, environments with a clearance grid and without one (the same
obstacles and a crowd out of reach, more than a grid numbers), and the call
that allocates nothing.  (Edges have a form of their own for some robots;
edges are compared with edges.)"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N = 1 << 15     # pairs of neighbours
FEW = 256       # configurations in a small call: spread over warps
KINDS = ("spheres", "capsules", "z_aligned_capsules", "cuboids", "z_aligned_cuboids")


def _crowd(env, n=256):
    """env and n spheres out of every robot's reach: no grid."""
    from prrtc_gb300.env import Environment
    far = np.tile(np.float32([[6.0, 6.0, 6.0, 0.1]]), (n, 1))
    return Environment(**({k: getattr(env, k) for k in KINDS} |
                          {"spheres": np.concatenate([np.asarray(env.spheres, np.float32).reshape(-1, 4), far])}))


def _scene(kind, robot):
    from prrtc_gb300 import scenes
    from prrtc_gb300.env import Environment
    if kind == "empty":
        return Environment()
    return scenes.mixed_scene(7, 60, n_zaligned=12) if kind == "mixed" else \
        scenes.shelf_scene(6, 0.3 if robot == "baxter" else 0.0, n_zaligned=6)


@pytest.fixture(scope="module", params=[(r, k) for r in ("panda", "fetch", "baxter") for k in ("shelf", "mixed", "empty")],
                ids=lambda p: "-".join(p))
def case(request, ctx):
    """(robot, environment, its handle, the handle without a grid, [2 N, dof] configurations, their verdicts)"""
    import torch
    from prrtc_gb300 import scenes
    robot, kind = request.param
    env = _scene(kind, robot)
    h, plain = ctx.upload_env(env), ctx.upload_env(_crowd(env))
    g = torch.Generator(device="cuda").manual_seed(5)
    sc, off = (torch.tensor(v, device="cuda", dtype=torch.float32) for v in scenes.LIMITS[robot])

    def check(q):
        torch.cuda.synchronize()
        return ctx.validate_configs(robot, h, q.contiguous()).bool()
    q = torch.rand((1 << 18, len(sc)), generator=g, device="cuda") * sc + off
    free = check(q)
    a, b = (q[m][torch.arange(N, device="cuda") % int(m.sum())] for m in (free, ~free))
    for _ in range(40):
        m = (a + b) * 0.5
        f = check(m)[:, None]
        a, b = torch.where(f, m, a), torch.where(f, b, m)
    q = torch.cat([a, b]).contiguous()
    torch.cuda.synchronize()
    return robot, env, h, plain, q, ctx.validate_configs(robot, h, q).cpu().numpy()


def test_one_verdict_for_a_configuration(case, ctx):
    import torch
    from prrtc_gb300 import api
    robot, env, h, plain, q, want = case
    assert want[:N].all() and not want[N:].any()     # neighbours on either side of contact
    assert int((q[:N] - q[N:]).abs().amax(1).le(1e-5).sum()) == N
    assert (ctx.validate_configs(robot, plain, q).cpu().numpy() == want).all()
    few = np.concatenate([ctx.validate_configs(robot, e, q[i:i + FEW]).cpu().numpy()
                          for e in (h, plain) for i in range(0, 2 * N, 16 * FEW)])
    assert (few == np.tile(np.concatenate([want[i:i + FEW] for i in range(0, 2 * N, 16 * FEW)]), 2)).all()
    f = api.lib().prrtc_validate_configs_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_int, C.POINTER(api.EnvDesc), C.c_void_p, C.c_int64, C.c_void_p, C.c_void_p]
    desc, keep = api._env_desc(env)
    out = torch.full((len(q),), 7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert f(api.robot_id(robot), C.byref(desc), q.data_ptr(), len(q), out.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert (out.cpu().numpy() == want).all()


@pytest.mark.parametrize("granularity", [1, 33, 96, 97, 128, 200])
def test_one_verdict_for_an_edge(case, granularity, ctx):
    """Edges that stay at one point."""
    robot, _, h, plain, q, want = case
    got = ctx.validate_edges(robot, h, q, q, granularity).cpu().numpy()
    assert (got == ctx.validate_edges(robot, plain, q, q, granularity).cpu().numpy()).all()
    assert (got == want).mean() > 0.9                # the forms differ within rounding at most
    few = ctx.validate_edges(robot, h, q[:5], q[:5], granularity).cpu().numpy()
    assert (few == got[:5]).all()


def test_environments_without_a_grid_hold_no_memory_for_one(ctx):
    """64 environments of more obstacles than a grid numbers take their records (5 KB each) alone."""
    import torch
    from prrtc_gb300.env import Environment
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    held = [ctx.upload_env(_crowd(Environment(), 300)) for _ in range(64)]
    assert before - torch.cuda.mem_get_info()[0] <= 8 << 20
    for h in held:
        h.free()
