"""Every arithmetic form of the kernels that split small calls: index rows, few-point stress and the
all-pairs force, against the oracle or the form's own kernel for large calls."""
import os

import numpy as np
import pytest

from conftest import k5_of
from test_segseg_gpu import _params, _synthetic, check_forces

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp64_fma", "fp64_fast", "df64", "f32c"])
@pytest.mark.parametrize("n,rows", [(2, 1), (33, 40), (129, 3), (2017, 600)])
def test_index_rows_forms(pkg, synth, oracle, mode, n, rows):
    """One step and seven steps per CTA (600 rows of 2,017 segments; there 256 threads in df64),
    columns that end inside a block, repeated and external rows, under each form's bounds of
    test_segseg_gpu.py."""
    net = _synthetic(pkg, synth, (n + 7) // 8, 7 + n, parallel_fraction=0.2, cube=3000.0)
    net.numSeg = n
    if n > 2:
        net.extSeg[[4, 30]] = 1
    dln, mat = _params(pkg)
    k5 = k5_of(dln, mat)
    idx = np.random.default_rng(n + rows).integers(1, n + 1, rows)
    if n > 2 and rows > 2:
        idx[:3] = [5, n, n]
    ctx = pkg.get_context()
    pkg.calcSegSegForce(dln, mat, net, idx)
    rep_s = dict(ctx.last_report)
    ctx.mode = mode
    try:
        Fi = pkg.calcSegSegForce(dln, mat, net, idx)
        rep = dict(ctx.last_report)
    finally:
        ctx.mode = "fp64"
    for key in ("pairs_general", "pairs_parallel"):
        assert rep[key] == rep_s[key]
    if mode == "f32c":
        nrm = lambda a: np.linalg.norm(a, axis=0)
        ext = oracle.segseg_ser_ld(k5, net, nthreads=os.cpu_count() or 1)
        exti = ext[:, :, idx - 1]
        assert np.linalg.norm(Fi - exti) <= 2e-7 * np.linalg.norm(ext)
        assert np.all(nrm(Fi - exti) <= 1e-4 * nrm(exti) + 1e-6 * nrm(ext).max())
    else:
        factor, normwise = {"fp64_fma": ((8, 6), 1e-10), "fp64_fast": ((4, 3), 1e-10),
                            "df64": ((1000, 1000), 1e-8)}[mode]
        check_forces(Fi, oracle, k5, net, rows=idx - 1, ref=oracle.segseg_idx(k5, net, idx), factor=factor,
                     normwise=normwise)
