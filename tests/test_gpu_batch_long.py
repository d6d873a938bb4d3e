"""A run of many seconds: one query that cannot be solved, one worker, every
other warp of the GPU without work.  They wait until the time budget ends the
run: the query comes back timed out, and the run without an error."""
import pytest

pytestmark = pytest.mark.gpu


def test_idle_warps_wait_for_a_long_query(ctx):
    from prrtc_gb300 import BatchSettings, Settings, scenes
    q = scenes.make_query("panda", "shelf", 3)
    plan = Settings(max_samples=100000, max_iters=4000000, num_new_configs=256, granularity=32, range=1.0, balance=0,
                    dynamic_domain=True, dd_radius=0.001, dd_min_radius=0.0005)
    # (a margin of 0.3 m: no configuration of this scene is free)
    b = ctx.batch("panda", [(q.env, q.start, q.goal)], BatchSettings(plan, margin=0.3, max_workers_per_attempt=1, max_attempts=1,
                                                                     time_budget_ns=int(9e9)))
    b.run()
    r = b.results()[0]
    assert not r.solved and r.status == 3 and b.stats()["error"] == 0
    assert b.stats()["kernel_ns"] > 8.5e9
    b.free()
