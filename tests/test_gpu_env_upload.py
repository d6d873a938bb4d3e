"""Uploaded environments and their memory: many at once, freed in any order, by
another context than the one that uploaded them and after that one is gone;
what a context keeps for later uploads is bounded."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _configs(n):
    from prrtc_gb300 import scenes
    sc, off = (np.array(v) for v in scenes.LIMITS["panda"])
    return (np.random.default_rng(1).random((n, 7)) * sc + off).astype(np.float32)


def test_environments_freed_in_any_order_and_used_by_other_contexts(ctx):
    from prrtc_gb300 import Context, api, scenes
    q = _configs(300)
    envs = [scenes.tabletop_scene(i, n_zaligned=i % 5) for i in range(24)]
    want = [ctx.validate_configs("panda", e, q) for e in envs]
    other = Context(0)
    held = [other.upload_env(e) for e in envs]
    for k in np.random.default_rng(2).permutation(24)[:12]:
        held[k].free()
        held[k] = None
    again = {k: other.upload_env(envs[k]) for k in range(24) if held[k] is None}
    for k in range(24):
        h = held[k] or again[k]
        assert (other.validate_configs("panda", h, q) == want[k]).all(), k
        assert (ctx.validate_configs("panda", h, q) == want[k]).all(), k
    handles = [h.handle for h in [*filter(None, held), *again.values()]]
    for h in [*filter(None, held), *again.values()]:
        h.handle = None                       # freed below, through the other context
    for h in handles[:8]:
        assert api.lib().prrtc_env_free(ctx.handle, h) == 0
    other.close()                             # the rest outlives its context
    for h in handles[8:]:
        assert api.lib().prrtc_env_free(ctx.handle, h) == 0
    assert (ctx.validate_configs("panda", envs[3], q) == want[3]).all()


def test_memory_kept_for_environments_is_bounded():
    """400 environments of 0.5 MB, all held, then freed: at most 32 of them stay, and nothing after the context."""
    import torch
    from prrtc_gb300 import Context, scenes
    torch.cuda.synchronize()
    own = Context(0)
    own.validate_configs("panda", scenes.tabletop_scene(0), _configs(10))
    free = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731
    before = free()
    held = [own.upload_env(scenes.tabletop_scene(1)) for _ in range(400)]
    assert before - free() > 100 << 20
    for h in held:
        h.free()
    own.validate_configs("panda", scenes.tabletop_scene(0), _configs(10))
    kept = before - free()
    assert kept <= 40 << 20, kept
    own.close()
    assert free() >= before - (8 << 20)
