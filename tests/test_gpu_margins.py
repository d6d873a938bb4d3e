"""Planning margins around and far above the one that the fast form's leaf
marks allow for (1e-4 m): a batch in scenes with clearance grids explores and
answers as in the same scenes without grids, where every test is made, and the
plain planner's paths clear contact by the margin."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MARGINS = [0.0, 1e-4, 1.1e-4, 5e-3]
CASES = [("panda", "tabletop", None), ("fetch", "mixed", 20), ("baxter", "tabletop", None)]


def _query(robot, kind, seed, nobs):
    from prrtc_gb300 import scenes
    return scenes.make_query(robot, kind, seed, nobs, **({"z_offset": 0.3} if robot == "baxter" else {}))


@pytest.mark.parametrize("margin", MARGINS)
@pytest.mark.parametrize("robot,kind,nobs", CASES)
def test_batches_with_and_without_grids(robot, kind, nobs, margin, ctx):
    from prrtc_gb300 import BatchSettings, Settings
    from test_gpu_near_contact import _crowd
    plan = Settings(max_samples=100000, max_iters=20, num_new_configs=256, granularity=48, range=1.0, balance=0,
                    dynamic_domain=False)
    qs = [_query(robot, kind, 300 + i, nobs) for i in range(24)]
    answers = []
    for shared in (0, 1):
        for env_of in (lambda e: e, _crowd):
            prep = ctx.prepare_batch(robot, [(env_of(q.env), q.start, q.goal) for q in qs], path_capacity=256)
            prep.paths.fill(0.0)
            ctx.solve_prepared(prep, BatchSettings(plan, margin=margin, max_workers_per_attempt=1, max_attempts=1,
                                                   shared_frames=shared))
            answers.append({k: prep.res[k].copy() for k in ("solved", "status", "start_tree_size", "goal_tree_size",
                                                            "path_rows", "iters", "cost", "samples")} | {"paths": prep.paths})
    assert answers[0]["start_tree_size"].max() > 1
    for other in answers[1:]:
        for k, v in answers[0].items():
            np.testing.assert_array_equal(other[k], v, err_msg=k)


@pytest.mark.parametrize("margin", MARGINS[1:])
@pytest.mark.parametrize("robot,kind,nobs", CASES)
def test_plain_paths_clear_contact_by_the_margin(robot, kind, nobs, margin, ctx):
    from prrtc_gb300 import Settings, scenes
    plan = Settings(max_samples=100000, max_iters=100000, num_new_configs=256, granularity=48, range=1.0, balance=0,
                    dynamic_domain=False)
    solved = 0
    ctx.set_planning_margin(margin)
    ctx.set_time_budget(int(1e9))
    try:
        for i in range(6):
            q = _query(robot, kind, 300 + i, nobs)
            r = ctx.solve(robot, q.start, q.goal, q.env, plan)
            if not r.solved:
                continue
            solved += 1
            k = (np.arange(1, 49, dtype=np.float32) / 48)[None, :, None]
            p = r.path.astype(np.float32)
            # the planner's own ends are not inflated: every point between them
            pts = (p[:-1, None] + k * (p[1:] - p[:-1])[:, None]).reshape(-1, p.shape[1])
            pts = pts[(np.abs(pts - q.start).max(1) > 1e-6) & (np.abs(pts - q.goal).max(1) > 1e-6)]
            assert scenes.clearance(robot, q.env, pts.astype(np.float64)).min() > 0.5 * margin, (robot, i)
    finally:
        ctx.set_planning_margin(0.0)
        ctx.set_time_budget(0)
    assert solved >= 2
