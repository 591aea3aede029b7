"""The context's shared scratch (pair store of the small all-pairs forces, partial stresses of σ̃ at
few points) under several streams and under stream capture.

Both tests compare with the same call made alone: the order between streams and
the capture change no bit, except that a captured σ̃ of the fast and mixed forms
sums its segments in list order instead of in slices (1,000 terms, of sums that
cancel by less than a factor of ten: 1,000 x 2^-53 and 1,000 x 2^-47)."""
import numpy as np
import pytest

from test_segseg_gpu import _params

pytestmark = pytest.mark.gpu

CUBE = 4000.0


@pytest.fixture(scope="module")
def torch_():
    return pytest.importorskip("torch")


def _segs(torch, synth, n, seed):
    p, b = synth.square_loops((n + 7) // 8, seed, 50.0, 200.0, CUBE, 0.5, 0.1)
    return torch.from_numpy(np.ascontiguousarray(synth.packed_soa(p, b)[:, :n])).cuda()


class Calls:
    """Device-form calls on one context, each with its own inputs and outputs."""

    def __init__(self, torch, pkg, synth, mode):
        dln, mat = _params(pkg)
        self.torch, self.synth, self.k, self.ctx = torch, synth, pkg.consts_of(dln, mat), pkg.Context()
        self.ctx.mode = mode

    def force(self, n, seed=1):
        s = _segs(self.torch, self.synth, n, seed)
        F = self.torch.zeros((n, 6), dtype=self.torch.float64, device="cuda")
        return F, lambda st: self.ctx.segseg_force_device(self.k, s.data_ptr(), n, n, F.data_ptr(), stream=st.cuda_stream)

    def sigma(self, n, M, seed=1):
        s = _segs(self.torch, self.synth, n, seed)
        x = self.torch.from_numpy(np.random.default_rng(seed).uniform(0.0, CUBE, (M, 3))).cuda()
        S = self.torch.zeros((M, 6), dtype=self.torch.float64, device="cuda")
        return S, lambda st: self.ctx.sigma_tilde_device(self.k, x.data_ptr(), M, s.data_ptr(), n, n, S.data_ptr(),
                                                         stream=st.cuda_stream)


@pytest.mark.parametrize("mode", ["fp64", "fp64_fast", "f32c"])
def test_streams_share_the_scratch(torch_, pkg, synth, mode):
    """A force and two σ̃ calls of one network, each on a stream of its own and nothing waited for
    in between, then one on the context's stream (NULL) while they run."""
    torch = torch_
    c = Calls(torch, pkg, synth, mode)
    calls = [c.force(1500), c.sigma(1500, 700), c.sigma(1500, 3000)]
    st = [torch.cuda.Stream() for _ in calls]
    alone = []
    for out, go in calls:
        go(st[0])
        torch.cuda.synchronize()
        alone.append(out.clone())
    own = type("Own", (), {"cuda_stream": None})
    for rep in range(3):
        for out, _ in calls:
            out.zero_()
        torch.cuda.synchronize()
        for _ in range(2):
            for (out, go), s in zip(calls, st):
                go(s)
        calls[rep][1](own)
        torch.cuda.synchronize()
        for (out, _), a in zip(calls, alone):
            assert torch.equal(out, a)


@pytest.mark.parametrize("mode,rel", [("fp64", 0.0), ("fp64_fast", 1e-12), ("f32c", 1e-11)])
def test_capture_after_a_larger_call(torch_, pkg, synth, mode, rel):
    """After one eager call with more segments, smaller calls can be captured; the graph's results
    stay right after later calls that need more scratch."""
    torch = torch_
    c = Calls(torch, pkg, synth, mode)
    st = torch.cuda.Stream()
    c.force(9400)[1](st)  # past the sizes that store pairs
    c.sigma(9400, 130000)[1](st)  # past the points that take scratch
    torch.cuda.synchronize()
    calls = [c.force(24), c.force(2000), c.force(3298), c.sigma(1000, 1), c.sigma(1000, 700)]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        for out, go in calls:
            go(st)
    g.replay()
    torch.cuda.synchronize()
    captured = [out.clone() for out, _ in calls]
    for out, go in calls:
        out.zero_()
        go(st)
    torch.cuda.synchronize()
    for k, ((out, _), cap) in enumerate(zip(calls, captured)):
        if k < 3:
            assert torch.equal(out, cap)
        else:
            assert (out - cap).abs().max() <= rel * out.abs().max()
    c.force(2176)[1](st)
    c.sigma(1000, 20000)[1](st)
    torch.cuda.synchronize()
    for out, _ in calls:
        out.zero_()
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    for (out, _), cap in zip(calls, captured):
        assert torch.equal(out, cap)


@pytest.mark.parametrize("nseg", [16384, 65536])
def test_many_segments_few_points(torch_, pkg, synth, nseg):
    """σ̃ just below the points that a thread each takes (24,575; chunks of 2^20 and 2^22 evaluations):
    the bits of the kernel above that line, and the call returns while most of it is still to run."""
    import time
    torch = torch_
    c = Calls(torch, pkg, synth, "fp64")
    st = torch.cuda.Stream()
    S, go = c.sigma(nseg, 24576)
    x = torch.from_numpy(np.random.default_rng(1).uniform(0.0, CUBE, (24576, 3))).cuda()
    segs = _segs(torch, synth, nseg, 1)
    T = torch.zeros((24575, 6), dtype=torch.float64, device="cuda")
    few = lambda: c.ctx.sigma_tilde_device(c.k, x.data_ptr(), 24575, segs.data_ptr(), nseg, nseg, T.data_ptr(),
                                           stream=st.cuda_stream)
    go(st)
    few()
    torch.cuda.synchronize()
    assert torch.equal(S[:24575], T)
    t0 = time.perf_counter()
    few()
    t1 = time.perf_counter()
    torch.cuda.synchronize()
    t2 = time.perf_counter()
    assert t1 - t0 < 0.25 * (t2 - t0)


@pytest.mark.parametrize("mode", ["fp64", "fp64_fast", "f32c"])
def test_stress_without_scratch(torch_, pkg, synth, mode):
    """Under a limit that no scratch fits, σ̃ of few points is what the same points give in a call
    with a thread each: the bits of the kernel without slices."""
    torch = torch_
    c = Calls(torch, pkg, synth, mode)
    c.ctx.partial_limit = 1
    st = torch.cuda.Stream()
    S, go = c.sigma(1000, 700000)
    T, few = c.sigma(1000, 700)
    go(st)
    few(st)
    torch.cuda.synchronize()
    assert torch.equal(S[:700], T)
