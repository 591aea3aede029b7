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


@pytest.mark.parametrize("num_loops,cube,npts", [(1, 2000.0, 1), (64, 2000.0, 613), (300, 20000.0, 333)])
def test_fma_stress_few_points(pkg, synth, oracle, num_loops, cube, npts):
    """σ̃ in DDD_MODE_FP64_FMA at few points (a thread per segment and point): the strict form's
    per-point bound against the oracle, and within 10x the reference arithmetic's own distance from
    the long-double evaluation, as test_sigma_gpu.py asks of the fast form; with a limit that leaves
    no room for its scratch, the point kernel under the same bounds."""
    from test_sigma_gpu import assert_sigma_close
    p, b = synth.square_loops(num_loops, 3, 20.0, 200.0, cube, 0.5, 0.1)
    net = pkg.DislocationNetwork(*synth.network_arrays(p, b))
    pts = np.asfortranarray(np.random.default_rng(npts).uniform(0, cube, (3, npts)))
    dln, mat = _params(pkg)
    k5 = k5_of(dln, mat)
    nt = os.cpu_count() or 1
    ref, ld = oracle.sigma_tilde(k5, pts, net, nthreads=nt), oracle.sigma_tilde_ld(k5, pts, net, nthreads=nt)
    ctx = pkg.get_context()
    ctx.mode = "fp64_fma"
    try:
        for limit in (0, 1):
            ctx.partial_limit = limit
            S = ctx.sigma_tilde(pkg.consts_of(dln, mat), pts, net)
            assert_sigma_close(S, ref)
            assert np.linalg.norm(S - ld) <= 10 * np.linalg.norm(ref - ld) + 1e-15 * np.linalg.norm(ld)
    finally:
        ctx.mode, ctx.partial_limit = "fp64", 0


@pytest.mark.parametrize("mode,rel", [("fp64", 0.0), ("fp64_fast", 1e-12), ("f32c", 1e-11)])
@pytest.mark.parametrize("nseg,npts", [(31, 1), (1000, 1), (1000, 77), (8000, 3000)])
def test_stress_slices_against_list_order(pkg, synth, mode, rel, nseg, npts):
    """σ̃ at few points against the kernels that add the segments in list order (a limit without room
    for scratch): the bits in strict FP64; in the fast and mixed forms a sum regrouped into slices
    (8,000 x 2^-53 and 8,000 x 2^-47 of sums that cancel by less than a factor of ten)."""
    net = _synthetic(pkg, synth, (nseg + 7) // 8, 3, cube=2000.0)
    net.numSeg = nseg
    dln, mat = _params(pkg)
    k = pkg.consts_of(dln, mat)
    x0 = np.asfortranarray(np.random.default_rng(nseg).uniform(0.0, 2000.0, (3, npts)))
    rel = rel * max(1, nseg // 1000)
    ctx = pkg.get_context()
    ctx.mode = mode
    try:
        S = ctx.sigma_tilde(k, x0, net)
        assert np.array_equal(ctx.sigma_tilde(k, x0, net), S)
        ctx.partial_limit = 1
        T = ctx.sigma_tilde(k, x0, net)
    finally:
        ctx.mode, ctx.partial_limit = "fp64", 0
    assert np.all(np.abs(S - T) <= rel * np.abs(T).max())


@pytest.mark.parametrize("n", [24, 1001, 2176, 3298])
def test_fma_form_keeps_the_tile_kernel(pkg, synth, n):
    """The FMA form's all-pairs force never takes the expanded kernels, which would move it: the bits
    do not depend on the room for their store."""
    net = _synthetic(pkg, synth, (n + 7) // 8, 90 + n, parallel_fraction=0.2, cube=3000.0)
    net.numSeg = n
    net.extSeg[5::17] = 1
    dln, mat = _params(pkg)
    ctx = pkg.get_context()
    nt = -(-n // 128)
    ctx.mode = "fp64_fma"
    try:
        F = pkg.calcSegSegForce(dln, mat, net)
        ctx.partial_limit = nt * (nt + 1) // 2 * 12288
        T = pkg.calcSegSegForce(dln, mat, net)
    finally:
        ctx.mode, ctx.partial_limit = "fp64", 0
    assert np.array_equal(F, T)
