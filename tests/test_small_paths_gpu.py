"""The kernels whose unit of work is a step of pairs: small all-pairs networks (every pair's forces
stored, then folded) and the index list.

The fold adds in the tile kernel's order, so with a partial-sum limit that
leaves room for the tile kernel's slots but not for the pair store (the tile
kernel then runs) the forces are equal bit for bit, in every arithmetic."""
import numpy as np
import pytest

from conftest import k5_of
from test_segseg_gpu import _params, _synthetic, check_forces

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp64", "fp64_fma", "fp64_fast", "df64", "f32c"])
@pytest.mark.parametrize("n", [1, 2, 24, 33, 128, 129, 1001, 2176])
def test_expanded_equals_tile_kernel(pkg, synth, mode, n):
    net = _synthetic(pkg, synth, (n + 7) // 8, 90 + n, parallel_fraction=0.2, cube=3000.0)
    net.numSeg = n
    net.extSeg[5::17] = 1
    dln, mat = _params(pkg)
    ctx = pkg.get_context()
    nt = -(-n // 128)
    ctx.mode = mode
    try:
        F = pkg.calcSegSegForce(dln, mat, net)
        rep = dict(ctx.last_report)
        ctx.partial_limit = nt * (nt + 1) // 2 * 12288
        T = pkg.calcSegSegForce(dln, mat, net)
        rep_t = dict(ctx.last_report)
    finally:
        ctx.mode, ctx.partial_limit = "fp64", 0
    if mode == "fp64_fma":  # the compiler contracts each kernel on its own
        assert np.linalg.norm(F - T) <= 1e-10 * np.linalg.norm(T)
    else:
        assert np.array_equal(F, T)
    for key in ("pairs_general", "pairs_parallel", "core_sides"):
        assert rep[key] == rep_t[key]


@pytest.mark.parametrize("mode", ["fp64", "fp64_fma", "fp64_fast", "df64", "f32c"])
@pytest.mark.parametrize("nt", [18, 24, 25, 28, 40])
def test_expanded_rest_equals_tile_kernel(pkg, synth, mode, nt):
    """171 tile pairs (two chunks of the pair store), 300 (strict only), one wave of
    304 and 21 or 102, two and 212; the tile kernel alone under a
    limit that the store does not fit."""
    n = 128 * nt - 37
    net = _synthetic(pkg, synth, (n + 7) // 8, nt, parallel_fraction=0.1, cube=12000.0)
    net.numSeg = n
    net.extSeg[5::17] = 1
    dln, mat = _params(pkg)
    ctx = pkg.get_context()
    ctx.mode = mode
    try:
        F = pkg.calcSegSegForce(dln, mat, net)
        rep = dict(ctx.last_report)
        ctx.partial_limit = nt * (nt + 1) // 2 * 12288
        T = pkg.calcSegSegForce(dln, mat, net)
        rep_t = dict(ctx.last_report)
    finally:
        ctx.mode, ctx.partial_limit = "fp64", 0
    if mode == "fp64_fma":
        assert np.linalg.norm(F - T) <= 1e-10 * np.linalg.norm(T)
    else:
        assert np.array_equal(F, T)
    for key in ("pairs_general", "pairs_parallel", "core_sides"):
        assert rep[key] == rep_t[key]


@pytest.mark.parametrize("n,rows", [(2, 1), (33, 40), (2017, 1), (2017, 600)])
def test_index_rows(pkg, synth, oracle, n, rows):
    """One step and seven steps per CTA (600 rows of 2,017 segments), columns
    that end inside a block, repeated and external rows."""
    net = _synthetic(pkg, synth, (n + 7) // 8, 7 + n, parallel_fraction=0.2, cube=3000.0)
    net.numSeg = n
    if n > 2:
        net.extSeg[[4, 30]] = 1
    dln, mat = _params(pkg)
    k5 = k5_of(dln, mat)
    idx = np.random.default_rng(n + rows).integers(1, n + 1, rows)
    if n > 2 and rows > 2:
        idx[:3] = [5, n, n]
    Fi = pkg.calcSegSegForce(dln, mat, net, idx)
    check_forces(Fi, oracle, k5, net, rows=idx - 1, ref=oracle.segseg_idx(k5, net, idx))


@pytest.mark.parametrize("mode,rel", [("fp64", 0.0), ("fp64_fast", 1e-12), ("f32c", 1e-11)])
@pytest.mark.parametrize("nseg", [1, 31, 1000])
def test_sigma_few_points(pkg, synth, mode, rel, nseg):
    """σ̃ with too few points for a thread each (1 point shared by a whole warp or
    CTA, 33, 100, and 24,575, the most that the FP64 store takes) against the same
    points inside a call that has enough.  FP64 keeps the segment order, so the
    bits; the other forms regroup a sum of 1,000 terms (1,000 x 2^-53 and
    1,000 x 2^-47, of sums that cancel by less than a factor of ten)."""
    net = _synthetic(pkg, synth, 125, 3, cube=2000.0)
    net.numSeg = nseg
    dln, mat = _params(pkg)
    k = pkg.consts_of(dln, mat)
    M = 122880 if mode != "fp64" else 24576
    x0 = np.asfortranarray(np.random.default_rng(nseg).uniform(0.0, 2000.0, (3, M)))
    ctx = pkg.get_context()
    ctx.mode = mode
    try:
        whole = ctx.sigma_tilde(k, x0, net)
        for m in (1, 33, 100, 24575):
            part = ctx.sigma_tilde(k, np.asfortranarray(x0[:, :m]), net)
            assert np.all(np.abs(part - whole[:, :m]) <= rel * np.abs(whole).max())
    finally:
        ctx.mode = "fp64"


@pytest.mark.parametrize("mode,rel", [("fp64", 1e-12), ("fp64_fast", 1e-12)])
@pytest.mark.parametrize("nseg", [1, 8, 9, 2000])
def test_u_tilde_few_points(pkg, synth, mode, rel, nseg):
    """calc_uTilde at 1, 33 and 1,023 points (one-warp CTAs, chunks from 8
    triangles) against the same points inside a call of 1,024 (128-point CTAs,
    other chunks): the same triangles in another grouping of at most 2,000 terms."""
    from ddd_gb300 import fem
    net = _synthetic(pkg, synth, 250, 11, cube=2000.0)
    net.numSeg = nseg
    mat = pkg.MaterialParameters(mu=1.0, nu=0.28)
    mesh = fem.RegularCuboidMesh(2000.0, 2000.0, 2000.0, 4, 4, 4)
    pts = np.asfortranarray(np.random.default_rng(nseg).uniform(-500.0, 2500.0, (3, 1024)))
    ctx = pkg.get_context()
    ctx.mode = mode
    try:
        whole = ctx.u_tilde(mat.omνInv8π, mat.om2νomνInv8π, mesh, pts, net)
        for m in (1, 33, 1023):
            part = ctx.u_tilde(mat.omνInv8π, mat.om2νomνInv8π, mesh, np.asfortranarray(pts[:, :m]), net)
            assert np.all(np.abs(part - whole[:3 * m]) <= rel * np.abs(whole).max())
    finally:
        ctx.mode = "fp64"
