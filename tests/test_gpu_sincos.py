"""Sine and cosine of the checkers' fast form and of the clearance kinematics
against float64, up to the |x| <= 100 they are stated for, with the multiples
of pi / 4 and pi / 2 where their reduction switches.

Fast form: x - k pi / 2 takes two roundings of a value below 1 (2^-25 each),
the series adds at most 2^-25 in its last step and an eighth of that before
it; the cosine's terms are no larger.  In all below 1.75 x 2^-24.
Clearance: the reduction leaves 2^-50, the coefficients below 1 / 9! are
single floats (2^-24 of r^9 / 9!, 2^-45.6), and the steps in pairs round at
2^-47 of terms that shrink: below 2^-44."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]


def test_sines_and_cosines(tmp_path, ctx):
    import torch
    import prrtc_gb300.build as b
    so = tmp_path / "libsincos_units.so"
    subprocess.run([b.NVCC, *b.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-cudart", "shared",
                    f"-I{b.CSRC}", f"-I{ROOT / 'include'}", str(ROOT / "tests" / "cuda" / "sincos_units.cu"), "-o", str(so)],
                   check=True)
    f = C.CDLL(str(so)).units_sincos
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_int, C.c_void_p, C.c_void_p]
    rng = np.random.default_rng(0)
    quarter = (np.arange(-127, 128) * (np.pi / 4)).astype(np.float32)
    near = np.concatenate([quarter] + [np.nextafter(quarter, s, dtype=np.float32) for s in (np.float32(200), np.float32(-200))])
    x = np.concatenate([rng.uniform(-np.pi, np.pi, 1 << 18), rng.uniform(-100, 100, 1 << 18),
                        rng.normal(0, 1, 1000) * 10.0 ** rng.integers(-30, 0, 1000), [0.0, -0.0, 100.0, -100.0],
                        *(near + d for d in (0.0, 1e-6, -1e-6, 1e-3))]).astype(np.float32)
    x = x[np.abs(x) <= 100]
    xd = torch.from_numpy(x).cuda()
    single = torch.zeros((len(x), 2), dtype=torch.float32, device="cuda")
    pair = torch.zeros((len(x), 2), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert f(xd.data_ptr(), len(x), single.data_ptr(), pair.data_ptr()) == 0
    want = np.stack([np.sin(x.astype(np.float64)), np.cos(x.astype(np.float64))], 1)
    assert np.abs(single.cpu().numpy() - want).max() <= 1.75 * 2.0 ** -24
    assert np.abs(pair.cpu().numpy() - want).max() <= 2.0 ** -44
