"""The packed df64 operations on the GPU, where a lane is part of a packed FP32 instruction.

The compiler fuses a packed product that is used once into a following packed sum
(df64.cuh), so the lanes are compared with the scalar operations on the device too,
alone and composed, and the df64 and f32c pairs with the same source compiled on scalar
instructions.  Everything is equal bit for bit."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

OPS = ["add", "sub", "mul", "div", "recip", "sqrt", "log", "atan", "addf", "subf", "mulf", "ab+g", "g-ab", "abg",
       "ab-ag", "(a+b)(a-g)", "2ab+ab", "hypot", "a log a - b/a"]
K4 = np.array([1.0, 1 / (4 * np.pi), 1 / (8 * np.pi), 1 / (4 * np.pi) / (1 - 0.28)])


@pytest.fixture(scope="module")
def libs(pkg, tmp_path_factory):
    """(packed, scalar), compiled with the library's flags of its df64 units."""
    import sys
    sys.path.insert(0, pkg.HERE)
    try:
        import build
    finally:
        sys.path.remove(pkg.HERE)
    out = []
    for name, extra in (("packed", []), ("scalar", ["-DDDD_F2_PLAIN"])):
        so = str(tmp_path_factory.mktemp(name) / "libdf2.so")
        cmd = [build.NVCC] + build.ARCH + build.FLAGS + ["--fmad=false", "-shared", "-I", build.CSRC] + extra + [
            os.path.join(ROOT, "tests", "df_host", "df2_device.cu"), "-o", so]
        out.append(subprocess.Popen(cmd, stderr=subprocess.PIPE, text=True))
        out[-1].so = so
    for p in out:
        err = p.communicate()[1]
        assert p.returncode == 0, err
    return [ctypes.CDLL(p.so) for p in out]


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def test_lanes_equal_scalar_on_device(libs):
    rng = np.random.default_rng(5)
    v = np.exp(rng.uniform(-12, 12, (200000, 6))) * rng.choice([-1.0, 1.0], (200000, 6))
    v[:5000, 1], v[:5000, 3] = v[:5000, 0] * (1 + 1e-9), -v[:5000, 4]  # cancellation
    v[5000:9000, 2] = v[5000:9000, 0] * v[5000:9000, 1]  # of a product and its value
    v[9000:9100, 0] = 1.0
    for lib in libs:
        assert lib.df2_ops() == len(OPS)
        bad = np.zeros(len(OPS), np.int64)
        assert lib.df2_compare(_ptr(v), ctypes.c_int64(len(v)), _ptr(bad)) == 0
        assert dict(zip(OPS, bad)) == dict.fromkeys(OPS, 0)


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("R", [50.0, 1000.0, 20000.0])
def test_pairs_equal_scalar_build(libs, form, R):
    rng = np.random.default_rng(int(R) + form)
    m = 50000
    d = rng.normal(size=(2 * m, 3))
    t = d / np.linalg.norm(d, axis=1)[:, None]
    l = rng.uniform(20.0, 200.0, 2 * m)
    u = rng.normal(size=(m, 3))
    u *= R / np.linalg.norm(u, axis=1)[:, None]
    mid = np.repeat(rng.uniform(0.0, 20000.0, (m, 3)), 2, axis=0)
    mid[1::2] += u
    n1, n2 = mid - 0.5 * l[:, None] * t, mid + 0.5 * l[:, None] * t
    b = rng.normal(size=(2 * m, 3))
    segs = np.ascontiguousarray(np.c_[n1, n2, b / np.linalg.norm(b, axis=1)[:, None], t, 1.0 / l])
    res = []
    for lib in libs:
        F = np.zeros((m, 24), np.float32)
        assert lib.df2_pairs(form, _ptr(K4), _ptr(segs), ctypes.c_int64(m), _ptr(F)) == 0
        res.append(F)
    assert np.isfinite(res[0]).all()
    assert np.array_equal(res[0].view(np.int32), res[1].view(np.int32))
