"""Batches whose queries share host obstacles: the library packs a scene once
and builds one clearance grid for it, and the answers do not depend on whether
a scene is shared."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KINDS = ("spheres", "capsules", "z_aligned_capsules", "cuboids", "z_aligned_cuboids")


def _copy(env, **kw):
    from prrtc_gb300.env import Environment
    return Environment(**({k: getattr(env, k).copy() for k in KINDS} | kw))


def _settings(**kw):
    """One worker and one attempt per query: results do not depend on timing."""
    from prrtc_gb300 import BatchSettings, Settings
    plan = Settings(max_samples=100000, max_iters=40, num_new_configs=256, granularity=32, range=1.0, balance=0,
                    dynamic_domain=False)
    return BatchSettings(plan, margin=1e-5, max_workers_per_attempt=1, max_attempts=1, **kw)


def _answers(ctx, queries, **kw):
    prep = ctx.prepare_batch("panda", queries, path_capacity=256)
    prep.paths.fill(0.0)
    ctx.solve_prepared(prep, _settings(**kw))
    cols = ("solved", "status", "start_tree_size", "goal_tree_size", "path_length", "iters", "cost", "path_rows", "samples")
    return {k: prep.res[k].copy() for k in cols} | {"paths": prep.paths.copy()}


def test_shared_scenes_give_the_answers_of_separate_ones(ctx):
    from prrtc_gb300 import scenes
    from prrtc_gb300.env import Environment
    base = [scenes.make_query("panda", "tabletop", 40 + i) for i in range(4)]
    base += [scenes.make_query("panda", "mixed", 60 + i, 20) for i in range(2)]
    few = Environment(spheres=base[0].env.spheres[:3])          # the same array, fewer of it
    assert few.spheres.ctypes.data == base[0].env.spheres.ctypes.data
    many = _copy(base[1].env, spheres=np.concatenate([base[1].env.spheres, np.tile(np.float32([[6, 6, 6, 0.1]]), (256, 1))]))
    envs = [q.env for q in base] + [few, Environment(), many]   # (without obstacles; more than a grid numbers)
    queries = [(envs[i % len(envs)], base[i % 6].start, base[i % 6].goal) for i in range(90)]
    apart = [(_copy(e), s, g) for e, s, g in queries]
    handles = {id(e): ctx.upload_env(e) for e in envs}
    uploaded = [(handles[id(e)], s, g) for e, s, g in queries]
    shared = _answers(ctx, queries)
    assert shared["solved"].sum() > 45
    for other in (apart, uploaded, [uploaded[i] if i % 3 else apart[i] for i in range(90)]):
        got = _answers(ctx, other)
        for k in shared:
            np.testing.assert_array_equal(got[k], shared[k], err_msg=k)


@pytest.mark.parametrize("form", ["batch", "solve_batch"])
def test_shared_scenes_hold_one_grid_each(form):
    """2048 queries of two scenes: the path pool is 29 MB and the arena 12 MB;
    a grid of 135 KB per query would be another 277 MB."""
    import torch
    from prrtc_gb300 import BatchSettings, Context, Settings, scenes
    own = Context(0)   # a context that holds nothing yet
    base = [scenes.make_query("panda", "tabletop", 40 + i) for i in range(2)]
    queries = [(base[i % 2].env, base[i % 2].start, base[i % 2].goal) for i in range(2048)]
    s = BatchSettings(Settings(max_samples=100000, max_iters=1, num_new_configs=32, granularity=32, range=1.0, balance=0,
                               dynamic_domain=False), max_nodes_per_tree=64, max_attempts=1)
    own.solve_batch("panda", queries[:2], s)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    if form == "batch":
        b = own.batch("panda", queries, s)
        held = before - torch.cuda.mem_get_info()[0]
        b.free()
    else:
        own.solve_batch("panda", queries, s, path_capacity=16)
        held = before - torch.cuda.mem_get_info()[0]   # what the context keeps
    own.close()
    assert held < 128 << 20, held


def test_a_scene_after_an_empty_one_is_staged(ctx, oracle):
    """One slot, queries in the order given: the warp that answered a query in
    an environment without obstacles takes the next scene's, whose records
    follow at the same place in the batch's memory."""
    from prrtc_gb300 import scenes
    from prrtc_gb300.env import Environment
    first, last = scenes.make_query("panda", "shelf", 80), scenes.make_query("panda", "tabletop", 81)
    empty, rng = Environment(), np.random.default_rng(4)
    sc, off = (np.array(v) for v in scenes.LIMITS["panda"])
    q = (rng.random((400, 7)) * sc + off).astype(np.float32)
    free = q[oracle.check("panda", last.env, q) == 1]
    queries = [(first.env, first.start, first.goal)]
    for i in range(20):
        queries += [(empty, first.start, first.goal), (last.env, free[2 * i], free[2 * i + 1])]
    got = _answers(ctx, queries, max_active=1, admission=1, warps_per_block=1, blocks_per_sm=1)
    mine = np.flatnonzero(got["solved"])[1:]
    assert sum(queries[i][0] is last.env for i in mine) >= 10
    for i in mine:
        p = got["paths"][i][:got["path_rows"][i]]
        assert oracle.check_edges("panda", queries[i][0], p[:-1], p[1:], 32).all(), i
