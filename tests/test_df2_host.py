"""The packed df64 operations on a CPU: both lanes equal the scalar operations bit for bit."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

OPS = ["add", "sub", "mul", "div", "recip", "sqrt", "log", "atan", "addf", "subf", "mulf"]


@pytest.fixture(scope="module")
def bad(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("df2") / "libdf2.so")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-I",
                           os.path.join(ROOT, "ddd.jl_gb300", "csrc"), "-o", out,
                           os.path.join(ROOT, "tests", "df_host", "df2_host.cpp")])
    rng = np.random.default_rng(5)
    v = np.exp(rng.uniform(-12, 12, (50000, 4))) * rng.choice([-1.0, 1.0], (50000, 4))
    v[:2000, 1], v[:2000, 2] = v[:2000, 0] * (1 + 1e-9), -v[:2000, 3]  # cancellation
    v[2000:2100, 0] = 1.0
    counts = np.zeros(len(OPS), np.int64)
    ctypes.CDLL(out).df2_compare(v.ctypes.data_as(ctypes.c_void_p), ctypes.c_int64(len(v)),
                                 counts.ctypes.data_as(ctypes.c_void_p))
    return dict(zip(OPS, counts))


@pytest.mark.parametrize("op", OPS)
def test_lanes_equal_scalar(bad, op):
    assert bad[op] == 0
