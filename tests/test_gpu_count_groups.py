"""Unsat counts on both sides of every line in the choice of groups: states an SM, one to 32
to a group, small and large instances."""
import numpy as np
import pytest

import analogsat_b200 as A
from test_gpu_primitives import counts, formula

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n,m,lens", [(40, 150, [3]), (1024, 1024, [4]), (1025, 900, [3]), (600, 1025, [2, 5]),
                                      (20000, 700, [3])])
def test_counts_at_the_lines(n, m, lens, dtype):
    lits, length = formula(n, m, lens, seed=n + m)
    p = A.SatProblem.from_arrays(lits, length)
    assert p.layout_stats()["compact"]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    batches = [sms - 1, sms, sms + 1, 4 * sms, 4 * sms + 1, 5 * sms + 3, 29 * sms, 32 * sms, 32 * sms + 1]
    top = max(batches) if n < 10000 else 5 * sms + 3
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.zeros(top, p.n + p.m, device="cuda", dtype=getattr(torch, dtype))
    x[:, :p.n] = torch.rand(top, p.n, generator=g, device="cuda", dtype=x.dtype) * 2 - 1
    x[::7, 3] = float("nan")
    want = np.concatenate([counts(lits, length, c.cpu().numpy()) for c in x[:, :p.n].split(500)])
    for b in batches:
        if b <= top:
            assert np.array_equal(A.clause_violation_counts(p, x[:b]).cpu().numpy(), want[:b]), b
