"""Cost and gradient of configurations out of the range of the four-lane
kinematics (beyond 100 rad in sum), which a thread each evaluates: any number
of them in a block of 16, among ordinary ones and alone, and the sphere robot,
which has a thread per waypoint throughout.  Against the oracle's float64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-4   # as for the one-thread form: float32 results of float64 sums


@pytest.mark.parametrize("robot", ["sphere", "panda", "fetch", "baxter"])
@pytest.mark.parametrize("rows,far", [(1, "all"), (15, "all"), (17, "all"), (33, "some"), (64, "last"), (100, "none")])
def test_configurations_out_of_range(robot, rows, far, ctx, oracle):
    from prrtc_gb300 import scenes
    env = scenes.mixed_scene(3, 40, n_zaligned=10)
    q = scenes._uniform_configs(robot, scenes.Rng(rows), rows).astype(np.float32)
    pick = {"all": np.ones(rows, bool), "some": np.arange(rows) % 5 < 2, "last": np.arange(rows) == rows - 1,
            "none": np.zeros(rows, bool)}[far]
    for j in scenes.load_model(robot)["joints"]:
        if j["type"] == "revolute":                      # whole turns: the same places, out of range
            q[pick, j["q"]] += np.float32(40 * np.pi)
    cost, grad = ctx.path_cost_grad(robot, env, q[None], 0.03)
    c64, g64 = oracle.cost_grad(robot, env, q.astype(np.float64), float(np.float32(0.03)))
    assert np.all(np.abs(cost[0] - c64) <= TOL * (c64 + 1e-8))
    err = np.linalg.norm(grad[0] - g64, axis=-1) / (np.linalg.norm(g64, axis=-1) + 1e-6)
    assert err.max() <= TOL
