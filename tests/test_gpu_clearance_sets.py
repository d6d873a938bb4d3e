"""The four-lane clearance evaluation with more leaf sets than a 32-bit word
has bits: Panda's leaves cut into sets of one to five, against the library's
own call (sets of at most 8).

Both sum the same FP64 terms, in another order, and round once to float32:
a cost (all terms of one sign) differs by at most one float32 step, a gradient
component by one step plus its terms' rounding, at most 1e-15 of their sum,
which a margin of 0.05 m and lever arms of about a metre keep below 1e3."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def sets_call(tmp_path_factory):
    import prrtc_gb300.build as b
    so = tmp_path_factory.mktemp("clearance_sets") / "libclearance_sets.so"
    subprocess.run([b.NVCC, *b.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-cudart", "shared",
                    f"-I{b.CSRC}", f"-I{ROOT / 'include'}", str(ROOT / "tests" / "cuda" / "clearance_sets.cu"), "-o", str(so)],
                   check=True)
    f = C.CDLL(str(so)).clearance_with_sets
    f.restype = C.c_int
    f.argtypes = [C.c_void_p] + [C.c_int] * 5 + [C.c_void_p, C.c_int, C.c_float, C.c_int, C.c_void_p, C.c_void_p]
    return f


@pytest.mark.parametrize("most", [1, 2, 3, 5])
def test_leaf_sets_beyond_a_word(most, ctx, sets_call):
    from prrtc_gb300 import scenes
    from test_gpu_urdf import pack_records
    env = scenes.mixed_scene(3, 40, lo=(-0.6, -0.6, 0.0), hi=(0.8, 0.6, 1.2), n_zaligned=10)
    q = scenes._uniform_configs("panda", scenes.Rng(most), 301).astype(np.float32)
    rec = np.ascontiguousarray(pack_records(env))
    cost, grad = np.zeros(len(q), np.float32), np.zeros_like(q)
    n = sets_call(rec.ctypes.data, len(env.spheres), len(env.capsules), len(env.z_aligned_capsules), len(env.cuboids),
                  len(env.z_aligned_cuboids), q.ctypes.data, len(q), 0.05, most, cost.ctypes.data, grad.ctypes.data)
    assert n > (32 if most == 1 else 0)
    want_c, want_g = ctx.path_cost_grad("panda", env, q[None], 0.05)
    step = 2.0 ** -23
    assert (want_c[0] > 0).mean() > 0.5
    assert (np.abs(cost - want_c[0]) <= step * want_c[0]).all()
    assert (np.abs(grad - want_g[0]) <= step * np.abs(want_g[0]) + 1e-12).all()
