"""Standalone primitives of one problem queued on several streams without waiting: those of
instances beyond one SM share the problem's scratch."""
import numpy as np
import pytest

import analogsat_b200 as A
from analogsat_b200.instances import make_instance

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def problem(kind):
    # rows and masks; the one-CTA-per-state form of the tanh variant and the bias term
    n, m, k = (40000, 170000, 3) if kind == "wide" else (4000, 17000, 3)
    lits, lens, _ = make_instance("fast", n, m, k, seed=3)
    p = A.SatProblem.from_arrays(lits, lens)
    return p.set_model(tanh=True).set_bias(0.1) if kind == "tanh" else p


def states(p, batch, seed, dtype):
    g = torch.Generator(device="cuda").manual_seed(seed)
    s = torch.rand(batch, p.n, generator=g, device="cuda", dtype=dtype) * 2 - 1
    return torch.cat([s, torch.rand(batch, p.m, generator=g, device="cuda", dtype=dtype) + 0.5], dim=1).contiguous()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("kind", ["wide", "compact", "tanh"])
def test_calls_on_two_streams(kind, dtype):
    p = problem(kind)
    batches = [3, 200, 17, 90, 1, 60]  # the scratch grows on the way
    xs = [states(p, b, i, dtype) for i, b in enumerate(batches)]
    fresh = problem(kind)
    want = []
    for x in xs:
        want.append((A.get_derivatives(fresh, x), A.clause_violation_counts(fresh, x)))
        torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.default_stream()]
    for rnd in range(3):
        got = []
        for i, x in enumerate(xs):
            a, b = streams[(i + rnd) % 3], streams[(i + rnd + 1) % 3]
            out = torch.full_like(x, 7.0)
            a.wait_stream(torch.cuda.default_stream())  # out is filled there
            with torch.cuda.stream(a):
                A.get_derivatives(p, x, out=out)
            with torch.cuda.stream(b):
                cnt = A.clause_violation_counts(p, x)
            got.append((out, cnt))
        torch.cuda.synchronize()
        for (d, c), (wd, wc) in zip(got, want):
            assert torch.equal(d, wd) and torch.equal(c, wc)


@pytest.mark.parametrize("kind", ["wide", "compact", "tanh"])
def test_captured_call_outlives_larger_ones(kind):
    """The graph of a captured call keeps its scratch when a later call needs more."""
    p = problem(kind)
    x, big = states(p, 4, 1, torch.float32), states(p, 300, 2, torch.float32)
    want = A.get_derivatives(p, x)
    counts = A.clause_violation_counts(p, x)
    out = torch.empty_like(x)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        A.get_derivatives(p, x, out=out)
        cnt = A.clause_violation_counts(p, x)
    wbig = A.get_derivatives(problem(kind), big)
    assert torch.equal(A.get_derivatives(p, big), wbig)  # a larger scratch
    for _ in range(2):
        out.zero_()
        cnt.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want) and torch.equal(cnt, counts)
        assert torch.equal(A.get_derivatives(p, big), wbig)
        torch.cuda.synchronize()
