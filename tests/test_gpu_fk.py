"""Sphere centres at the counts where a warp's tile of 32 configurations is
partly filled, against the oracle's float64 kinematics."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 1000])
@pytest.mark.parametrize("robot", ["sphere", "panda", "fetch", "baxter"])
def test_fk_spheres_tile_edges(robot, n, ctx, oracle):
    from prrtc_gb300 import scenes
    q = scenes._uniform_configs(robot, scenes.Rng(n), n).astype(np.float32)
    got = ctx.fk_spheres(robot, q)
    ref = oracle.fk_spheres(robot, q.astype(np.float64))
    assert np.abs(got[..., :3] - ref[..., :3]).max() < 1e-5
    np.testing.assert_array_equal(got[..., 3], ref[..., 3].astype(np.float32))
