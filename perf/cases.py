"""The workloads this library is timed on, each through its public entry points.

listed() names them, draw() gives more of the same ranges, prepare() makes what
a program has in hand before the call, run() makes one pass, work() counts what
a pass cannot do without and exact() evaluates the same quantity in 64 bits with
plain torch and none of the library's arithmetic.

Networks come from the library's seeded generator (closed 8-segment square
loops on the BCC slip systems, 5 % near-parallel neighbours), cut to the stated
segment count; `ext` marks every `ext`-th segment external.
"""
import math
import os

import numpy as np
import torch

from __graft_entry__ import load_package

pkg = load_package()
import ddd_gb300.synth as synth  # noqa: E402
from ddd_gb300 import fem  # noqa: E402

MODES = ("fp64", "fp64_fast", "fp64_fma", "df64", "f32c")
CHECKPOINT = os.path.join(pkg.HERE, "data", "surrogate_gpu65k_nu028.bin")

# Floating-point operations per unit of work: one general pair with the forces
# on both segments or on one, one field point of one segment, one triangle at
# one point, one far pair by quadrature (6 field points) or by the network.
FLOP_PAIR, FLOP_ROW, FLOP_SIGMA, FLOP_TRIANGLE, FLOP_QUAD, FLOP_NETWORK = 1511, 1000, 289, 350, 700, 98304


def listed():
    return [
        # A Frank-Read study: a few loops, thousands of calls, nothing but latency.
        {"name": "force_24_strict", "kind": "force", "segments": 24, "mode": "fp64", "ext": 0},
        # One time step of the 512-segment workload: calcSegForce!, dlnMobility!, detectCollision.
        {"name": "step_512", "kind": "step", "segments": 512},
        # calcSegSegForce of a grown network between remeshing steps: ragged, some segments outside the volume.
        {"name": "force_5k_strict", "kind": "force", "segments": 5003, "mode": "fp64", "ext": 13},
        # The 32,768-segment workload kept on the device, in the fast FP64 form.
        {"name": "force_32k_fast", "kind": "force_device", "segments": 32768, "mode": "fp64_fast", "ext": 0},
        # The same in the FP32 form with compensated terms.
        {"name": "force_32k_f32c", "kind": "force_device", "segments": 32768, "mode": "f32c", "ext": 0},
        # calcSegSegForce(idx): the segments that a topology operation touched.
        {"name": "rows_37_of_6k", "kind": "rows", "segments": 6001, "rows": 37, "mode": "fp64", "ext": 13},
        # calc_sigmaTilde at the FE nodes that carry the traction.
        {"name": "sigma_nodes_strict", "kind": "sigma", "segments": 4096, "points": 613, "mode": "fp64"},
        # A stress map for plotting: a 32^3 grid in the mixed form.
        {"name": "sigma_grid_mixed", "kind": "sigma", "segments": 16384, "points": 32768, "mode": "f32c"},
        # The 65,536-segment workload, far field by quadrature, f32c near pairs, 1 % audit.
        {"name": "far_quad_65k", "kind": "far", "segments": 65536, "far": "quad3", "mode": "f32c"},
        # The learned far field (the committed checkpoint).
        {"name": "far_network_32k", "kind": "far", "segments": 32768, "far": "network", "mode": "f32c"},
        # An ensemble of independent networks of uneven sizes in one call.
        {"name": "batch_48_f32c", "kind": "batch", "networks": 48, "smallest": 64, "largest": 4096, "mode": "f32c"},
        # calc_uTilde at the displacement nodes of a cantilever.
        {"name": "u_tilde_8k", "kind": "u_tilde", "segments": 8192, "cells": 24, "mode": "fp64"},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("force", "force", "step", "force_device", "force_device", "rows", "sigma", "sigma", "far",
                       "batch", "u_tilde"))
    if kind == "force":
        return {"kind": kind, "segments": _log_int(rng, 8, 8192), "mode": rng.choice(MODES),
                "ext": rng.choice((0, 0, 7, 13))}
    if kind == "step":
        return {"kind": kind, "segments": 8 * _log_int(rng, 2, 500)}
    if kind == "force_device":
        mode = rng.choice(MODES)
        return {"kind": kind, "segments": _log_int(rng, 64, 16384 if mode == "fp64" else 32768), "mode": mode,
                "ext": rng.choice((0, 11))}
    if kind == "rows":
        return {"kind": kind, "segments": _log_int(rng, 64, 16384), "rows": _log_int(rng, 1, 64),
                "mode": rng.choice(MODES), "ext": rng.choice((0, 13))}
    if kind == "sigma":
        return {"kind": kind, "segments": _log_int(rng, 24, 16384), "points": _log_int(rng, 1, 32768),
                "mode": rng.choice(("fp64", "fp64_fast", "f32c"))}
    if kind == "far":
        far = rng.choice(("quad3", "quad3", "quad2", "network"))
        return {"kind": kind, "segments": _log_int(rng, 4096, 32768 if far == "network" else 65536), "far": far,
                "mode": rng.choice(("f32c", "fp64_fast"))}
    if kind == "batch":
        return {"kind": kind, "networks": _log_int(rng, 4, 64), "smallest": _log_int(rng, 16, 128),
                "largest": _log_int(rng, 256, 4096), "mode": rng.choice(("fp64", "fp64_fast", "df64", "f32c"))}
    return {"kind": kind, "segments": _log_int(rng, 64, 16384), "cells": rng.randint(4, 32),
            "mode": rng.choice(("fp64", "fp64_fast"))}


# ---------------------------------------------------------------------------
# Inputs.

def _params():
    dln = pkg.DislocationParameters(coreRad=synth.CORE_RAD, minSegLen=20.0, maxSegLen=400.0,
                                    dragCoeffs={"line": 1e-4})
    return dln, pkg.MaterialParameters(mu=synth.MU, nu=synth.NU)


def _loops(segments, seed):
    """Loops of the 512-segment workload up to 1,024 segments, of the 20,000^3 one above."""
    name = "cpu512" if segments <= 1024 else "gpu32k"
    p, b, cfg = synth.make(name, seed=seed, num_loops=(segments + 7) // 8)
    return p, b, cfg["cube"]


def _network(segments, seed, ext=0):
    p, b, cube = _loops(segments, seed)
    coord, bvec, seg = synth.network_arrays(p, b)
    flags = np.zeros(seg.shape[0], np.uint8)
    if ext:
        flags[::ext] = 1
    return pkg.DislocationNetwork(coord, bvec, seg, numSeg=segments, extSeg=flags), cube


def _packed(segments, seed):
    p, b, cube = _loops(segments, seed)
    return torch.from_numpy(np.ascontiguousarray(synth.packed_soa(p, b)[:, :segments])).cuda()


def _ext_device(segments, every):
    if not every:
        return None
    e = torch.zeros(segments, dtype=torch.uint8, device="cuda")
    e[::every] = 1
    return e


def _batch_sizes(case):
    """Segment counts log-spaced from smallest to largest, in an order that mixes them."""
    n = case["networks"]
    lo, hi = math.log(case["smallest"]), math.log(case["largest"])
    sizes = [int(round(math.exp(lo + (hi - lo) * ((7 * k) % n) / max(1, n - 1)))) for k in range(n)]
    return sizes


def _sigma_points(case, seed, cube):
    rng = np.random.default_rng(seed + 1000)
    side = round(case["points"] ** (1.0 / 3.0))
    if side > 1 and side ** 3 == case["points"]:  # a grid, shifted by the seed
        return np.asfortranarray(synth.grid_points(side, cube) + rng.uniform(-20.0, 20.0, (3, 1)))
    return np.asfortranarray(rng.uniform(0.0, cube, (3, case["points"])))


_stream = []


def _user_stream():
    if not _stream:
        _stream.append(torch.cuda.Stream())
    return _stream[0]


def prepare(case, seed):
    dln, mat = _params()
    kind = case["kind"]
    s = {"case": case, "dln": dln, "mat": mat, "k": pkg.consts_of(dln, mat)}
    if kind in ("force", "rows", "sigma"):
        s["net"], cube = _network(case["segments"], seed, case.get("ext", 0))
        if kind == "rows":
            rng = np.random.default_rng(seed + 2000)
            s["idx"] = rng.integers(1, case["segments"] + 1, case["rows"])
        if kind == "sigma":
            s["x0"] = _sigma_points(case, seed, cube)
        if case["mode"] != "fp64":
            s["ctx"] = pkg.Context()
            s["ctx"].mode = case["mode"]
    elif kind == "step":
        s["net"], _ = _network(case["segments"], seed)
        s["sigma_hat"] = np.asfortranarray(np.random.default_rng(seed + 3000).normal(0, 1e-3, (6, case["segments"])))
    elif kind == "force_device":
        n = case["segments"]
        s["ctx"] = pkg.Context()
        s["ctx"].mode = case["mode"]
        s["segs"], s["ext"] = _packed(n, seed), _ext_device(n, case["ext"])
        s["force"] = torch.empty((n, 6), dtype=torch.float64, device="cuda")
    elif kind == "far":
        s["ctx"] = pkg.Context()
        s["far"] = pkg.Surrogate(s["ctx"])
        if case["far"] == "network":
            s["far"].load(CHECKPOINT)
        s["segs"] = _packed(case["segments"], seed)
        s["force"] = torch.empty((case["segments"], 6), dtype=torch.float64, device="cuda")
    elif kind == "batch":
        sizes = _batch_sizes(case)
        s["ctx"] = pkg.Context()
        s["batch"] = pkg.Batch(s["ctx"], sizes, mode=case["mode"])
        s["segs"] = torch.cat([_packed(n, 1000 * seed + q) for q, n in enumerate(sizes)], dim=1).contiguous()
        s["force"] = torch.empty((sum(sizes), 6), dtype=torch.float64, device="cuda")
    elif kind == "u_tilde":
        s["net"], cube = _network(case["segments"], seed)
        n = case["cells"]
        s["mesh"] = fem.RegularCuboidMesh(cube, cube, cube, n, n, n)
        s["bnd"] = fem.cantilever_boundaries(s["mesh"])
        s["points"] = np.asfortranarray(s["mesh"].coord[:, s["bnd"].uGammaDln - 1])
        if case["mode"] != "fp64":
            s["ctx"] = pkg.Context()
            s["ctx"].mode = case["mode"]
    torch.cuda.synchronize()
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "force":
        if "ctx" in s:
            return s["ctx"].segseg_force(s["k"], s["net"])
        return pkg.calcSegSegForce(s["dln"], s["mat"], s["net"])
    if kind == "rows":
        if "ctx" in s:
            return s["ctx"].segseg_force(s["k"], s["net"], s["idx"])
        return pkg.calcSegSegForce(s["dln"], s["mat"], s["net"], s["idx"])
    if kind == "sigma":
        if "ctx" in s:
            return s["ctx"].sigma_tilde(s["k"], s["x0"], s["net"])
        return pkg.calc_σTilde(s["x0"], s["dln"], s["mat"], s["net"]).reshape(6, -1, order="F")
    if kind == "step":
        net = s["net"]
        pkg.calcSegForce_inplace(s["dln"], s["mat"], s["sigma_hat"], net)
        pkg.dlnMobility_inplace(s["dln"], s["mat"], net)
        hit = pkg.detectCollision(s["dln"], net)
        return {"force": net.segForce, "node_force": net.nodeForce, "node_velocity": net.nodeVel,
                "collision": [int(hit[0]), ("null", "hinge", "twoLine").index(hit[1])] + [int(v) for v in hit[2:8]],
                "places": [float(v) for v in hit[8:10]]}
    if kind == "force_device":
        n = case["segments"]
        s["ctx"].segseg_force_device(s["k"], s["segs"].data_ptr(), n, n, s["force"].data_ptr(),
                                     ext_ptr=None if s["ext"] is None else s["ext"].data_ptr(),
                                     stream=_user_stream().cuda_stream)
        return s["force"]
    if kind == "far":
        return s["far"].force(s["k"], s["segs"], exact_mode=case["mode"], far=case["far"], out=s["force"],
                              stream=_user_stream().cuda_stream)[0]
    if kind == "batch":
        s["batch"].run(s["k"], s["segs"].data_ptr(), s["force"].data_ptr(), stream=_user_stream().cuda_stream)
        return s["force"]
    if "ctx" in s:
        return s["ctx"].u_tilde(s["mat"].omνInv8π, s["mat"].om2νomνInv8π, s["mesh"], s["points"], s["net"])
    return pkg.calc_uTilde(s["mesh"], s["bnd"], s["mat"], s["net"])


def _active(case):
    n, e = case["segments"], case.get("ext", 0)
    return n - (-(-n // e) if e else 0)


def work(case):
    """Each input read once, each output written once; the operations of the formulas."""
    kind = case["kind"]
    if kind == "batch":
        sizes = _batch_sizes(case)
        return {"bytes": 120 * sum(sizes), "flops": FLOP_PAIR * sum(n * (n - 1) // 2 for n in sizes)}
    n = case["segments"]
    pairs = _active(case) * (_active(case) - 1) // 2
    if kind in ("force", "force_device"):
        return {"bytes": 120 * n, "flops": FLOP_PAIR * pairs}
    if kind == "step":
        return {"bytes": 48 * n + 24 * n + 24 * n + 48 * n + 96 * n + 72 * n, "flops": FLOP_PAIR * pairs + 800 * n}
    if kind == "rows":
        return {"bytes": 72 * n + 56 * case["rows"], "flops": FLOP_ROW * case["rows"] * _active(case)}
    if kind == "sigma":
        return {"bytes": 72 * n + 72 * case["points"], "flops": FLOP_SIGMA * n * case["points"]}
    if kind == "far":
        return {"bytes": 120 * n, "flops": (FLOP_NETWORK if case["far"] == "network" else FLOP_QUAD) * pairs}
    points = (case["cells"] + 1) ** 2 + case["cells"] + 1
    return {"bytes": 72 * n + 48 * points, "flops": FLOP_TRIANGLE * n * points}


# ---------------------------------------------------------------------------
# The same quantities in 64 bits with plain torch (vectors are 3 x P tensors).
# Formulas: Arsenlis et al. 2007, App. A.1, in the reference's near-parallel
# form (DislocationForces.jl:879-1561), and DislocationFEM.jl:135-299, :583-660.

SQRT_EPS = 2.0 ** -26
HCOT = math.sqrt((1.0 - SQRT_EPS * 1.01) / (SQRT_EPS * 1.01)) / 2.0


def _dot(a, b):
    return (a * b).sum(0)


def _cross(a, b):
    return torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])


def _norm(a):
    return torch.sqrt(_dot(a, a))


def _corner(aa, den, c, q, x, y):
    """The 19 integrals of a general pair at one corner; aa = a^2 + d^2 (1 - c^2), q = 1 / (1 - c^2)."""
    R = torch.sqrt(aa + x * x + y * y + 2.0 * x * y * c)
    RI = 1.0 / R
    u, v = R + y + x * c, R + x + y * c
    lu, lv = torch.log(u), torch.log(v)
    p, r = RI / u, RI / v
    xp, yr = x * p, y * r
    xxp, yyr = x * xp, y * yr
    i1 = -2.0 * den * torch.atan((1.0 + c) * (R + x + y) * den)
    c1 = aa * i1
    c56 = (c * R - c1) * q
    i2, i3, i4 = (c * lv - lu) * q, (c * lu - lv) * q, (c * c1 - R) * q
    i5, i6 = y * lv + c56, x * lu + c56
    c11 = i1 - c * RI
    c15 = c * xp - RI
    x13 = x * c15
    c19 = c * yr - RI
    y13 = y * c19
    cc = c * c
    c16 = lv - (x - c * y) * RI - cc * yyr
    z15 = y * c16
    c17 = lu - (y - c * x) * RI - cc * xxp
    d = 2.0 * i4
    return [i1, i2, i3, i4, i5, i6, (i1 - xp - yr) / aa, (p - c * r) * q, (r - c * p) * q,
            (RI - c * (xp + yr + i1)) * q, (xp + cc * yr + c11) * q, (yr + cc * xp + c11) * q,
            (i3 - x13 + c * (y13 - i2)) * q, (i2 - y13 + c * (x13 - i3)) * q,
            (i5 - z15 + c * (x * x * c15 - d)) * q, (xxp + c * c16 + 2.0 * i2) * q, (yyr + c * c17 + 2.0 * i3) * q,
            (d - x * x * c15 + c * (z15 - i5)) * q, (d - y * y * c19 + c * (x * c17 - i6)) * q]


def _weighted(V, F):
    s = V[0] * F[0]
    for k in range(1, len(V)):
        s = s + V[k] * F[k]
    return s


def _general(K, b1, n11, n12, t1, s1, b2, n21, n22, t2, s2, c, need12=True, need34=True):
    """Forces on the nodes of segment 1 and of segment 2 (None where not needed); s = 1 / length."""
    a2, m4, m8, m4n = K["a2"], K["m4"], K["m8"], K["m4n"]
    m8a, m4na = a2 * m8, a2 * m4n
    omc = 1.0 - c * c
    q = 1.0 / omc
    t21 = _cross(t2, t1)
    t12 = -t21
    b22, b11 = _cross(b2, t2), _cross(b1, t1)
    t2b2, t2b1, t1b2, t1b1 = _dot(t2, b2), _dot(t2, b1), _dot(t1, b2), _dot(t1, b1)
    t21b2, t12b1, b11b2, b22b1 = _dot(t21, b2), _dot(t12, b1), _dot(b11, b2), _dot(b22, b1)
    t212, t121 = t1 - c * t2, t2 - c * t1
    t2b1t2, t1b2t1 = b1 - t2b1 * t2, b2 - t1b2 * t1
    b1t1t2, b2t2t1 = t2b1 * t1 - c * b1, t1b2 * t2 - c * b2
    e1, e2 = t2b1 - t1b1 * c, t1b2 - t2b2 * c
    e12 = t2b1 * t1b2 - t1b1 * t2b2
    R1, R2 = n21 - n11, n22 - n12
    d = _dot(R2, t21) * q
    m4d, m4nd = m4 * d, m4n * d
    m4ndd = m4nd * d
    m4nddd = m4ndd * d
    m4nad, m8ad = m4na * d, m8a * d
    l11, l12, l21, l22 = _dot(R1, t1), _dot(R1, t2), _dot(R2, t1), _dot(R2, t2)
    x1, x2, y1, y2 = (l12 - c * l11) * q, (l22 - c * l21) * q, (l11 - c * l12) * q, (l21 - c * l22) * q
    aa = a2 + d * d * omc
    den = 1.0 / torch.sqrt(omc * aa)
    I = _corner(aa, den, c, q, x1, y1)
    for x, y, add in ((x1, y2, False), (x2, y1, False), (x2, y2, True)):
        for k, v in enumerate(_corner(aa, den, c, q, x, y)):
            I[k] = I[k] + v if add else I[k] - v
    F1 = F2 = F3 = F4 = None
    if need12:
        V1 = (t1b2 * t2b1 + e12) * t21
        V2 = b11 * e2
        V3 = t12 * b11b2 - t1b2t1 * t2b1
        V4 = -b11 * t21b2
        V5 = b2t2t1 * t2b1 - t12 * b22b1
        V = [m4d * V1 - m4nd * V2 + (m4nd * t12b1) * b2t2t1 + (m4nd * b22b1) * t121,
             m4 * V5 - (m4n * t2b1) * b2t2t1 + (m4n * b22b1) * t12,
             -(m4n * t1b1) * b2t2t1 + m4 * V3 - m4n * V4,
             m8ad * V1 - m4nad * V2 - (m4nddd * e2 * t12b1) * t121,
             m8a * V5 + (m4ndd * e2 * t2b1) * t121 - (m4ndd * e2 * t12b1) * t12,
             m8a * V3 - m4na * V4 + (m4ndd * (t21b2 * t12b1 + e2 * t1b1)) * t121,
             (m4nd * (e2 * t1b1 + t21b2 * t12b1)) * t12 - (m4nd * t21b2 * t2b1) * t121,
             (m4nd * e2 * t2b1) * t12,
             -(m4nd * t21b2 * t1b1) * t121]
        tv = m4n * t21b2 * t12
        V += [-tv * t2b1, -tv * t1b1]
        up, lo = (2, 3, 5, 8, 9, 11, 13, 12, 16, 14, 18), (0, 1, 2, 6, 7, 8, 9, 10, 11, 12, 13)
        F1 = _weighted(V, [I[u] - y2 * I[w] for u, w in zip(up, lo)]) * s1
        F2 = _weighted(V, [y1 * I[w] - I[u] for u, w in zip(up, lo)]) * s1
    if need34:
        V1 = (t2b1 * t1b2 + e12) * t12
        V2 = b22 * e1
        V3 = t21 * b11b2 - b1t1t2 * t1b2
        V5 = t2b1t2 * t1b2 - t21 * b22b1
        V6 = b22 * t12b1
        V = [m4d * V1 - m4nd * V2 + (m4nd * t21b2) * b1t1t2 + (m4nd * b11b2) * t212,
             (m4n * t2b2) * b1t1t2 + m4 * V5 - m4n * V6,
             m4 * V3 + (m4n * t1b2) * b1t1t2 - (m4n * b11b2) * t21,
             m8ad * V1 - m4nad * V2 - (m4nddd * e1 * t21b2) * t212,
             m8a * V5 - m4na * V6 - (m4ndd * (t12b1 * t21b2 + e1 * t2b2)) * t212,
             m8a * V3 - (m4ndd * e1 * t1b2) * t212 + (m4ndd * e1 * t21b2) * t21,
             (m4nd * (e1 * t2b2 + t12b1 * t21b2)) * t21 - (m4nd * t12b1 * t1b2) * t212,
             -(m4nd * t12b1 * t2b2) * t212,
             (m4nd * e1 * t1b2) * t21]
        tv = m4n * t12b1 * t21
        V += [tv * t2b2, tv * t1b2]
        up, lo = (1, 4, 3, 7, 10, 9, 12, 15, 13, 17, 14), (0, 1, 2, 6, 7, 8, 9, 10, 11, 12, 13)
        F3 = _weighted(V, [x2 * I[w] - I[u] for u, w in zip(up, lo)]) * s2
        F4 = _weighted(V, [I[u] - x1 * I[w] for u, w in zip(up, lo)]) * s2
    return F1, F2, F3, F4


def _direction(n1, n2):
    v = n2 - n1
    s = 1.0 / _norm(v)
    return v * s, s


def _par_corner(aa, aai, x, y):
    w, z = x + y, x - y
    R = torch.sqrt(aa + w * w)
    RI = 1.0 / R
    g = torch.log(R + w)
    h = z * R * aai
    i9 = -aai * w * RI
    return [R * aai, -0.5 * (g - h), -0.5 * (g + h), -g, y * g - R, x * g - R, aai * (2.0 * aai * R - RI),
            aai * (h - x * RI), -aai * (h + y * RI), i9, RI - y * i9, RI - x * i9]


def _par_side(K, first, na1, na2, ta, sa, ba, nb1, nb2, bb):
    """Forces on the nodes of segment a by the near-parallel segment b, b projected onto a's line."""
    a2, m4, m8, m4n = K["a2"], K["m4"], K["m8"], K["m4n"]
    nm2 = nb1 + _dot(nb2 - nb1, ta) * ta
    diff = nb2 - nm2
    mag = _norm(diff)
    h, pull = 0.5 * diff, HCOT * mag * ta
    nm1 = nb1 + h + pull
    nm2 = nm2 + h - pull
    if first:
        R = nm1 - na1
        x1, x2, y1, y2 = _dot(nm1, ta), _dot(nm2, ta), -_dot(na1, ta), -_dot(na2, ta)
    else:
        R = na1 - nm1
        x1, x2, y1, y2 = _dot(na1, ta), _dot(na2, ta), -_dot(nm1, ta), -_dot(nm2, ta)
    nd = R - _dot(R, ta) * ta
    aa = a2 + _dot(nd, nd)
    aai = 1.0 / aa
    tabb, taba, ndba = _dot(ta, bb), _dot(ta, ba), _dot(nd, ba)
    bbta, bata, ndta = _cross(bb, ta), _cross(ba, ta), _cross(nd, ta)
    bbtaba, bbtand = _dot(bbta, ba), _dot(bbta, nd)
    bbtata = tabb * ta - bb
    I = _par_corner(aa, aai, x1, y1)
    for x, y, add in ((x1, y2, False), (x2, y1, False), (x2, y2, True)):
        for k, v in enumerate(_par_corner(aa, aai, x, y)):
            I[k] = I[k] + v if add else I[k] - v
    w1, w2 = (taba * tabb) * nd, bbtand * bata
    V = [m4n * (ndba * bbtata + bbtaba * ndta - w2) - m4 * w1, ((m4n - m4) * taba) * bbtata,
         -(a2 * m8) * w1 - (a2 * m4n) * w2 - (m4n * bbtand * ndba) * ndta,
         -((a2 * m8) * taba) * bbtata - (m4n * bbtand * taba) * ndta]
    if first:
        F2 = _weighted(V, [I[k + 2] - y1 * I[k] for k in (0, 3, 6, 9)]) * sa
        F1 = _weighted(V, [y2 * I[k] - I[k + 2] for k in (0, 3, 6, 9)]) * sa
    else:
        F2 = _weighted(V, [I[k + 1] - x1 * I[k] for k in (0, 3, 6, 9)]) * sa
        F1 = _weighted(V, [x2 * I[k] - I[k + 1] for k in (0, 3, 6, 9)]) * sa
    core = torch.nonzero(mag * mag > SQRT_EPS * (_dot(nm1, nm1) + _dot(nm2, nm2)))[:, 0]
    if core.numel():
        na1, na2, ta, sa, ba = na1[:, core], na2[:, core], ta[:, core], sa[core], ba[:, core]
        for p, r in ((nb1, nm1), (nm2, nb2)):
            p, r = p[:, core], r[:, core]
            tc, sc = _direction(p, r)
            _, _, G3, G4 = _general(K, bb[:, core], p, r, tc, sc, ba, na1, na2, ta, sa, _dot(tc, ta), need12=False)
            F1[:, core] += G3
            F2[:, core] += G4
    return F1, F2


def _near_parallel(K, b1, n11, n12, t1, s1, b2, n21, n22, t2, s2, c, need34):
    flip = c < 0.0
    m11, m12 = torch.where(flip, n12, n11), torch.where(flip, n11, n12)
    sg = torch.where(flip, -1.0, 1.0)
    u1, g1 = t1 * sg, b1 * sg
    F1, F2 = _par_side(K, True, m11, m12, u1, s1, g1, n21, n22, b2)
    F3, F4 = _par_side(K, False, n21, n22, t2, s2, b2, m11, m12, g1) if need34 else (None, None)
    return torch.where(flip, F2, F1), torch.where(flip, F1, F2), F3, F4


def _pair_forces(K, segs, i, j, need34):
    n1, n2, b, t, s = segs
    c = _dot(t[:, i], t[:, j])
    out = None
    for near, sel in ((False, torch.nonzero(1.0 - c * c > SQRT_EPS)[:, 0]),
                      (True, torch.nonzero(~(1.0 - c * c > SQRT_EPS))[:, 0])):
        if not sel.numel():
            continue
        p, r = i[sel], j[sel]
        a = (K, b[:, p], n1[:, p], n2[:, p], t[:, p], s[p], b[:, r], n1[:, r], n2[:, r], t[:, r], s[r], c[sel])
        F = _near_parallel(*a, need34) if near else _general(*a, need34=need34)
        out = (out or []) + [(p, r, F)]
    return out or []


def _consts(case_nu=synth.NU):
    m4 = synth.MU / (4.0 * math.pi)
    return {"a2": synth.CORE_RAD ** 2, "m4": m4, "m8": m4 / 2.0, "m4n": m4 / (1.0 - case_nu),
            "nm4n": case_nu * (m4 / (1.0 - case_nu)), "nu": case_nu}


def _segments(n1, n2, b):
    t, s = _direction(n1, n2)
    return n1, n2, b, t, s


def _of_network(net):
    n = net.numSeg
    si = net.segIdx[:n]
    f = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    return _segments(f(net.coord[:, si[:, 1] - 1]), f(net.coord[:, si[:, 2] - 1]), f(net.bVec[:, si[:, 0] - 1]))


CHUNK = 1 << 22


def _all_forces(segs, ext=None):
    """n x 6 node forces of all pairs i < j; ext: n flags of the segments left out."""
    K, n = _consts(), segs[0].shape[1]
    out = torch.zeros((n, 6), dtype=torch.float64, device="cuda")
    act = torch.arange(n, device="cuda") if ext is None else torch.nonzero(ext == 0)[:, 0]
    m, a0 = act.numel(), 0
    while a0 < m:
        rows = max(1, min(m - a0, CHUNK // max(1, m - a0)))
        i = torch.arange(a0, a0 + rows, device="cuda")[:, None].expand(rows, m - a0)
        j = torch.arange(a0, m, device="cuda")[None, :].expand(rows, m - a0)
        keep = j > i
        i, j = act[i[keep]], act[j[keep]]
        for p, r, (F1, F2, F3, F4) in _pair_forces(K, segs, i, j, True):
            out.index_add_(0, p, torch.cat([F1, F2]).T)
            out.index_add_(0, r, torch.cat([F3, F4]).T)
        a0 += rows
    return out


def _row_forces(segs, idx, ext):
    K, n = _consts(), segs[0].shape[1]
    out = torch.zeros((len(idx), 6), dtype=torch.float64, device="cuda")
    act = torch.nonzero(ext == 0)[:, 0]
    for q, r in enumerate(idx):
        if ext[r - 1]:
            continue
        j = act[act != r - 1]
        i = torch.full_like(j, r - 1)
        for _, _, (F1, F2, _, _) in _pair_forces(K, segs, i, j, False):
            out[q] += torch.cat([F1, F2]).sum(1)
    return out


def _host(F):
    """n x 6 -> the 3 x 2 x n array of the host calls."""
    return np.asfortranarray(F.cpu().numpy().reshape(-1, 2, 3).transpose(2, 1, 0))


def _stress(segs, x0):
    K = _consts()
    n1, n2, b, t, _ = segs
    N, M = n1.shape[1], x0.shape[1]
    a2, a2m8, m4, m4n = K["a2"], K["a2"] * K["m8"], K["m4"], K["m4n"]
    out = torch.zeros((6, M), dtype=torch.float64, device="cuda")
    step = max(1, CHUNK // M)
    for s0 in range(0, N, step):
        e = lambda v: v[:, s0:s0 + step, None]  # noqa: E731
        p, r, bb, tt, x = e(n1), e(n2), e(b), e(t), x0[:, None, :]
        R = x - p
        Rt = _dot(R, tt)
        nd = R - Rt * tt
        aa = a2 + _dot(nd, nd)
        ai = 1.0 / aa

        def ends(s):
            RI = 1.0 / torch.sqrt(aa + s * s)
            R3 = RI * RI * RI
            s03 = s * RI * ai
            return s03, -RI, (2.0 * s03 + s * R3) * ai, -R3, s03 - s * R3
        S03, S13, S05, S15, S25 = [v - u for u, v in zip(ends(-Rt), ends(-_dot(x - r, tt)))]
        tb, db = _cross(tt, bb), _cross(nd, bb)
        com = m4n * _dot(db, tt)
        for c, (u, v) in enumerate(((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))):
            sym = lambda f, g: f[u] * g[v] + f[v] * g[u]  # noqa: E731
            dd, ttp, td = nd[u] * nd[v], tt[u] * tt[v], sym(tt, nd)
            ttb, dtb, tdb = sym(tt, tb), sym(nd, tb), sym(tt, db)
            one = com if u == v else 0.0
            I = ((one + m4n * dtb - m4 * tdb) * S03 - K["nm4n"] * ttb * S13
                 + (com * ((a2 if u == v else 0.0) + dd) - a2m8 * tdb) * S05
                 + (a2m8 * ttb - com * td) * S15 + com * ttp * S25)
            out[c] += I.sum(0)
    return out


def _unit(v):
    n = _norm(v)
    ok = n > 2.0 ** -52
    return torch.where(ok, v / torch.where(ok, n, 1.0), 0.0), torch.where(ok, n, 2.0 ** -52)


def _displacements(segs, closure, points):
    """Barnett triangles (segment, closure) of segments inside the volume."""
    K = _consts()
    om = 1.0 / (1.0 - K["nu"])
    k1, k2 = om / (8.0 * math.pi), (1.0 - 2.0 * K["nu"]) * (om / (8.0 * math.pi))
    A, B, b = segs[:3]
    C = closure[:, None].expand_as(A)
    P = points[:, None, :]
    out = torch.zeros_like(points)
    step = max(1, CHUNK // points.shape[1])
    for s0 in range(0, A.shape[1], step):
        e = lambda v: v[:, s0:s0 + step, None]  # noqa: E731
        a, q, r, bb = e(A), e(B), e(C), e(b)
        AB, BC, CA = _unit(q - a)[0], _unit(r - q)[0], _unit(a - r)[0]
        (RA, la), (RB, lb), (RC, lc) = _unit(a - P), _unit(q - P), _unit(r - P)
        ab, bc, ca = [torch.clamp(_dot(u, v), -1.0, 1.0) for u, v in ((RA, RB), (RB, RC), (RC, RA))]
        x, y, z = torch.acos(ab), torch.acos(bc), torch.acos(ca)
        h = (x + y + z) / 2.0
        f = torch.clamp(torch.tan(h / 2) * torch.tan((h - x) / 2) * torch.tan((h - y) / 2) * torch.tan((h - z) / 2),
                        min=0.0)
        omega = -torch.sign(_dot(RA, _cross(CA, AB).expand_as(RA))) * 4.0 * torch.atan(torch.sqrt(f))
        u = -bb * omega / (4.0 * math.pi)

        def line(E, R0, l0, R1, l1):
            return _cross(bb, E) * torch.log((l1 / l0) * (1.0 + _dot(R1, E)) / (1.0 + _dot(R0, E)))

        def turn(R0, R1, d01):
            return _dot(bb, _cross(R0, R1)) * (R0 + R1) / (1.0 + d01)
        u = u - k2 * (line(AB, RA, la, RB, lb) + line(BC, RB, lb, RC, lc) + line(CA, RC, lc, RA, la)) \
            + k1 * (turn(RA, RB, ab) + turn(RB, RC, bc) + turn(RC, RA, ca))
        out += u.sum(1)
    return out


def _step(net, sigma_hat):
    """segForce and nodeForce of a step: seg-seg, self and Peach-Koehler forces, then their sums at the nodes."""
    K = _consts()
    segs = _of_network(net)
    n1, n2, b, t, _ = segs
    L = _norm(n2 - n1)
    a = math.sqrt(K["a2"])
    La = torch.sqrt(L * L + K["a2"])
    core = 1.0 / (4.0 * math.pi) * math.log(a / 0.1)
    om = 1.0 / (1.0 - K["nu"])
    sc = _dot(t, b)
    be = b - sc * t
    tor = K["m4"] * sc * (K["nu"] * om * (torch.log((La + L) / a) - 2.0 * (La - a) / L) - (La - a) ** 2 / (2.0 * La * L))
    own = (tor + 2.0 * core * K["nu"] * om * sc) * be - (sc * sc + _dot(be, be) * om) * core * t
    g = torch.from_numpy(np.ascontiguousarray(sigma_hat)).cuda()
    sb = torch.stack([g[0] * b[0] + g[3] * b[1] + g[4] * b[2], g[3] * b[0] + g[1] * b[1] + g[5] * b[2],
                      g[4] * b[0] + g[5] * b[1] + g[2] * b[2]])
    pk = _cross(sb, n2 - n1)
    F = _all_forces(segs)
    F[:, :3] += (0.5 * pk - own).T
    F[:, 3:] += (0.5 * pk + own).T
    nodes = torch.zeros((net.coord.shape[1], 3), dtype=torch.float64, device="cuda")
    si = torch.from_numpy(np.ascontiguousarray(net.segIdx)).cuda()
    nodes.index_add_(0, si[:, 1] - 1, F[:, :3])
    nodes.index_add_(0, si[:, 2] - 1, F[:, 3:])
    return _host(F), np.asfortranarray(nodes.T.cpu().numpy())


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind in ("force", "rows"):
        ext = torch.from_numpy(s["net"].extSeg[:case["segments"]].copy()).cuda()
        segs = _of_network(s["net"])
        return _host(_all_forces(segs, ext) if kind == "force" else _row_forces(segs, s["idx"].tolist(), ext))
    if kind == "sigma":
        return np.asfortranarray(_stress(_of_network(s["net"]), torch.from_numpy(s["x0"]).cuda()).cpu().numpy())
    if kind == "step":
        F, N = _step(s["net"], s["sigma_hat"])
        # The velocity solve has a condition number of 1e9 and more (climb
        # drag against glide and line drag): 64 bits give no exact value of it.
        # The collision's places are those of whichever pair came last.
        return {"force": F, "node_force": N, "node_velocity": None, "collision": None, "places": None}
    if kind in ("force_device", "far"):
        v = s["segs"]
        return _all_forces(_segments(v[0:3], v[3:6], v[6:9]), s.get("ext"))
    if kind == "batch":
        out, at = [], 0
        for n in _batch_sizes(case):
            v = s["segs"][:, at:at + n]
            out.append(_all_forces(_segments(v[0:3], v[3:6], v[6:9])))
            at += n
        return torch.cat(out)
    u = _displacements(_of_network(s["net"]), torch.from_numpy(s["mesh"].closure).cuda(),
                       torch.from_numpy(s["points"]).cuda())
    return u.T.contiguous().cpu().numpy().ravel()
