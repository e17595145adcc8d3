"""Standalone primitives in a captured graph: once one of them has laid out a problem's
tables, the others need no more allocations on instances that fit one SM."""
import numpy as np
import pytest

import analogsat_b200 as A
from analogsat_b200.instances import make_instance

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype,n,m,k", [(torch.float64, 200, 840, 3), (torch.float64, 150, 1200, 4),
                                         (torch.float32, 1500, 6300, 3), (torch.float32, 700, 5300, 4)])
def test_first_derivatives_under_capture(dtype, n, m, k):
    lits, lens, _ = make_instance("fast", n, m, k, seed=n)
    p, q = (A.SatProblem.from_arrays(lits, lens) for _ in range(2))
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(-1, 1, (9, p.n)), rng.uniform(0.5, 3, (9, p.m))], axis=1)
    x = torch.from_numpy(x).to(dtype).cuda()
    want = A.get_derivatives(q, x)
    counts = A.clause_violation_counts(p, x)  # the tables of p
    out = torch.empty_like(x)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        A.get_derivatives(p, x, out=out)
        again = A.clause_violation_counts(p, x)
    for _ in range(2):
        out.zero_()
        again.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want) and torch.equal(again, counts)
    A.rhs_check(p)
