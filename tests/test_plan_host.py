"""The launch plans' arithmetic on a CPU (ddd_internal.h): what a kernel gets to index stays inside
a grid, a buffer and a limit, also at sizes that no test can run."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    out = str(tmp_path_factory.mktemp("plan") / "libplan.so")
    # -Bsymbolic: the counting cudaMalloc stays its own beside a loaded CUDA runtime.
    cmd = [cxx, "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", os.path.join(CUDA, "include"),
           "-I", os.path.join(ROOT, "ddd.jl_gb300", "csrc"),
           os.path.join(ROOT, "tests", "plan_host", "plan_host.cpp"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(out)

    def call(name, n, *args):
        o = np.zeros(n, np.int64)
        getattr(lib, name)(*[ctypes.c_int64(int(a)) for a in args], o.ctypes.data_as(ctypes.c_void_p))
        return [int(v) for v in o]

    return call


@pytest.mark.parametrize("n,rows,limit", [(1, 1, 0), (6001, 37, 0), (6001, 6001, 16 << 30),
                                          (2_000_000, 2_000_000, 200 << 30), (16_000_000, 16_000_000, 1 << 40), (100_000, 3_000_000_000, 1 << 42)])
@pytest.mark.parametrize("df64", [0, 1])
def test_row_chunks(plan, df64, n, rows, limit):
    """A chunk's CTAs fit a grid, its partial sums the limit (or 128 rows), and every column has a block."""
    npad = -(-n // 128) * 128
    blocks, m, chunk, threads = plan("plan_rows", 4, npad, rows, limit, df64)
    assert threads == (256 if df64 and m >= 4 else 128)
    assert 1 <= m <= 8 and blocks * m * threads >= npad > (blocks - 1) * m * threads
    assert 1 <= chunk <= rows and chunk * blocks < 2 ** 31
    assert chunk * blocks * 48 <= max(limit, 128 * blocks * 48)
    assert chunk == rows or chunk >= 128 or (chunk + 1) * blocks >= 2 ** 31


@pytest.mark.parametrize("nseg,points", [(1, 1), (4096, 613), (16384, 24575), (65536, 24575), (1_000_000, 1000),
                                         (174_000, 24575), (1_000_000, 24575), (100_000_000, 1), (10 ** 10, 1)])
def test_sigma_chunks(plan, nseg, points):
    """At most 512 launches, each of at least one segment and indexed in 32 bits; 2^19 evaluations
    where that many launches do, none (the point kernel) where 2^23 would not."""
    chunk, scratch, most = plan("plan_sigma", 3, nseg, points)
    assert points < most
    if chunk:
        step = chunk // points
        assert step >= 1 and -(-nseg // step) + 1 <= 512 and 6 * chunk < 2 ** 31
        assert chunk == 2 ** 19 or -(-nseg // (chunk // 2 // points)) + 1 > 512
        assert scratch == 96 * chunk + 24 * (-(-nseg // 128) * 128)
    else:
        assert -(-nseg // (2 ** 23 // points)) + 1 > 512
    assert plan("plan_sigma", 3, nseg, most)[0] == 0


@pytest.mark.parametrize("nb", [1, 10, 153, 253])
def test_store_and_limit(plan, nb):
    """The pair store is taken only when all that the call allocates for it and for the partial sums
    is within the limit; the largest is 285 MB."""
    held = plan("plan_store", 2, nb, nb, 0)[0]
    assert plan("plan_store", 2, nb, nb, held)[1] == 1
    assert plan("plan_store", 2, nb, nb, held - 1)[1] == 0
    assert plan("plan_store", 2, nb, 0, 2 ** 40)[0] <= 285_000_000
