"""The four-lane evaluation of the clearance cost (clearance_eval.cuh) against
the oracle's float64 cost and adjoint, where it can go wrong: counts of paths
and waypoints that leave lanes of a warp without a configuration, scenes
without obstacles, with more obstacles near one cell than the grid lists and
with too many for a grid, margins beyond the grid's bounds, and
configurations outside the range of its kinematics beside ordinary ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
# relative error of a waypoint's gradient and cost, as for the one-thread form:
# results are float32 of a float64 sum; the 1e-6 floor is for gradients that vanish
TOL = 1e-4


def _env(kind, robot):
    from prrtc_gb300 import scenes
    from prrtc_gb300.env import Environment
    rng = np.random.default_rng(2)
    z = 0.3 if robot == "baxter" else 0.0
    if kind == "empty":
        return Environment()
    if kind == "crowd":
        return Environment(spheres=np.column_stack([rng.normal([0.5, 0.1, 0.6], 0.08, (60, 3)), rng.uniform(0.01, 0.03, 60)]))
    if kind == "many":   # more than a grid numbers
        return Environment(spheres=np.column_stack([rng.uniform(-1, 1.5, (300, 3)), rng.uniform(0.01, 0.05, 300)]))
    if kind == "mixed":
        return scenes.mixed_scene(3, 40, n_zaligned=10)
    return scenes.shelf_scene(1, z, n_zaligned=4)


def _close(cost, grad, c64, g64):
    assert np.all(np.abs(cost - c64) <= TOL * (c64 + 1e-8)), np.abs(cost - c64).max()
    err = np.linalg.norm(grad - g64, axis=-1) / (np.linalg.norm(g64, axis=-1) + 1e-6)
    assert err.max() <= TOL, err.max()


CASES = [("panda", "shelf", 1, 1, 0.02), ("panda", "shelf", 3, 17, 0.02), ("panda", "crowd", 5, 33, 0.02),
         ("panda", "many", 2, 64, 0.02), ("panda", "empty", 2, 7, 0.02), ("panda", "shelf", 2, 9, 0.6),
         ("fetch", "mixed", 3, 21, 0.02), ("fetch", "mixed", 65, 2, 0.0), ("baxter", "shelf", 3, 19, 0.02),
         ("baxter", "many", 1, 65, 0.05), ("sphere", "mixed", 2, 5, 0.02)]


@pytest.mark.parametrize("robot,kind,paths,waypoints,margin", CASES)
def test_cost_and_gradient_match_float64(robot, kind, paths, waypoints, margin, ctx, oracle):
    from prrtc_gb300 import scenes
    env = _env(kind, robot)
    q = scenes._uniform_configs(robot, scenes.Rng(paths * 100 + waypoints), paths * waypoints).astype(np.float32)
    cost, grad = ctx.path_cost_grad(robot, env, q.reshape(paths, waypoints, -1), margin)
    c64, g64 = oracle.cost_grad(robot, env, q.astype(np.float64), float(np.float32(margin)))
    _close(cost.reshape(-1), grad.reshape(q.shape), c64, g64)


def test_configurations_out_of_range_beside_ordinary_ones(ctx, oracle):
    from prrtc_gb300 import scenes
    env = _env("shelf", "panda")
    q = scenes._uniform_configs("panda", scenes.Rng(5), 40).astype(np.float32)
    q[3] *= 1e3          # beyond the range of the fast kinematics
    q[17, 2] = np.nan
    cost, grad = ctx.path_cost_grad("panda", env, q[None], 0.02)
    ok = np.isfinite(q).all(1)
    c64, g64 = oracle.cost_grad("panda", env, q[ok].astype(np.float64), float(np.float32(0.02)))
    _close(cost[0][ok], grad[0][ok], c64, g64)
    assert np.isnan(grad[0, 17]).any()
