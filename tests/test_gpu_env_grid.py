"""The checker with an environment's clearance grid against the checker
without one: prrtc_validate_configs uses the grid that the upload builds,
prrtc_validate_configs_noalloc has none and tests every obstacle.  Verdicts
are equal, configuration by configuration, over obstacles the grid takes
(few, many, more near one cell than it lists, partly or wholly out of its
reach) and obstacles it has to leave to the full test (not boxes, not finite,
too many), with ordinary, extreme and non-finite configurations."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _env(kind):
    from prrtc_gb300 import scenes
    from prrtc_gb300.env import Environment, capsule_row, cuboid_row
    rng = np.random.default_rng(3)
    base = scenes.mixed_scene(11, 24, n_zaligned=8)

    def spheres(n, lo=(0.2, -0.6, 0.0), hi=(0.9, 0.6, 1.2), r=(0.005, 0.05)):
        return np.column_stack([rng.uniform(lo, hi, (n, 3)), rng.uniform(*r, n)]).astype(np.float32)

    def but(**kw):
        return Environment(**({k: getattr(base, k) for k in ("spheres", "capsules", "z_aligned_capsules", "cuboids",
                                                             "z_aligned_cuboids")} | kw))
    bad_box, bad_cap = base.cuboids.copy(), base.capsules.copy()
    if kind == "tabletop":
        return scenes.tabletop_scene(1, n_zaligned=8)
    if kind == "shelf":
        return scenes.shelf_scene(2, n_zaligned=6)
    if kind == "mixed":
        return scenes.mixed_scene(4, 60, n_zaligned=12)
    if kind == "one sphere":
        return Environment(spheres=[[0.5, 0.1, 0.6, 0.2]])
    if kind == "one thin plate":
        return Environment(cuboids=[cuboid_row((0.5, 0.0, 0.5), (0.4, 0.4, 1e-4), (0.3, 0.2, 0.1))])
    if kind == "255 spheres":
        return Environment(spheres=spheres(255))
    if kind == "256 spheres":
        return Environment(spheres=spheres(256))
    if kind == "a crowd in one spot":
        return Environment(spheres=spheres(40, (0.45, -0.05, 0.5), (0.55, 0.05, 0.6)),
                           capsules=[capsule_row((0.4, y, 0.3), (0.4, y, 0.7), 0.01) for y in np.linspace(-0.1, 0.1, 20)])
    if kind == "wide floor and walls":
        return Environment(cuboids=[cuboid_row((0, 0, -0.1), (7, 7, 0.05)), cuboid_row((0.8, 0, 1), (0.02, 7, 2))],
                           spheres=spheres(5))
    if kind == "out of reach":
        return Environment(spheres=[[5.0, 5.0, 5.0, 0.3]], cuboids=[cuboid_row((-8.0, 0.0, 0.0), (0.5, 0.5, 0.5))])
    if kind == "far away":
        return but(spheres=[*base.spheres, [500.0, 0.0, 0.0, 499.7]])
    if kind == "negative sizes":
        bad_box[0, 12:] *= -1
        bad_cap[0, 6] *= -1
        return but(cuboids=bad_box, capsules=bad_cap, spheres=[[0.5, 0.2, 0.6, -0.3]])
    if kind == "skewed axes":
        bad_box[0, 3:6] *= 1.5
        return but(cuboids=bad_box)
    if kind == "wrong rdv":
        bad_cap[0, 7] *= 3.0
        return but(capsules=bad_cap)
    if kind == "zero-length capsules":
        z = [0.5, 0.0, 0.6, 0.0, 0.0, 0.0, 0.1, np.inf]
        return but(capsules=[z], z_aligned_capsules=[z])
    if kind == "tilted z-aligned":
        return but(z_aligned_cuboids=base.cuboids[:3], z_aligned_capsules=base.capsules[:3])
    assert kind == "not finite"
    bad_box[0, 0], bad_cap[0, 2] = np.nan, np.inf
    return but(cuboids=bad_box, capsules=bad_cap, spheres=[[0.5, 0.0, 0.6, np.inf], [np.nan, 0.0, 0.6, 0.1]])


KINDS = ["tabletop", "shelf", "mixed", "one sphere", "one thin plate", "255 spheres", "256 spheres", "a crowd in one spot",
         "wide floor and walls", "out of reach", "far away", "negative sizes", "skewed axes", "wrong rdv",
         "zero-length capsules", "tilted z-aligned", "not finite"]


@pytest.mark.parametrize("kind", KINDS)
def test_grid_verdicts_equal_the_full_test(kind, ctx):
    import torch
    from prrtc_gb300 import api, scenes
    env = _env(kind)
    f = api.lib().prrtc_validate_configs_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_int, C.POINTER(api.EnvDesc), C.c_void_p, C.c_int64, C.c_void_p, C.c_void_p]
    desc, keep = api._env_desc(env)
    for robot in ("sphere", "panda", "fetch", "baxter"):
        sc, off = (np.array(v) for v in scenes.LIMITS[robot])
        rng = np.random.default_rng(len(kind))
        q = (rng.random((60_001, len(sc))) * sc + off).astype(np.float32)
        if robot == "sphere":
            q[::2] = rng.normal(0.5, 0.7, q[::2].shape)   # around the obstacles: its radius is 1 m
        q[-64:] *= 10.0 ** rng.integers(1, 12, (64, 1))
        q[-96:-64, 0] = np.nan
        q[-128:-96] = np.inf
        qd = torch.from_numpy(q).cuda()
        want = torch.full((len(q),), 7, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        assert f(api.robot_id(robot), C.byref(desc), qd.data_ptr(), len(q), want.data_ptr(), None) == 0
        torch.cuda.synchronize()
        got = ctx.validate_configs(robot, env, qd)
        assert int((got != want).sum()) == 0, (kind, robot)
