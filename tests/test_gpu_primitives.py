"""Standalone primitives over many states at the edges of their launch shapes: group
sizes and remainders, instances that fit one SM and instances that do not."""
import numpy as np
import pytest

import analogsat_b200 as A
from analogsat_b200.instances import make_instance

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def formula(n, m, lens, seed):
    """Random clauses with lengths drawn from `lens`."""
    rng = np.random.default_rng(seed)
    length = rng.choice(lens, m)
    length[0] = max(lens)
    lits = [int(v) * (1 if rng.random() < 0.5 else -1) for k in length for v in rng.choice(n, k, replace=False) + 1]
    lits[0] = n  # every variable index up to n is declared
    return np.array(lits, np.int32), length.astype(np.int32)


def counts(lits, lens, spins):
    """Unsat clauses of every state: TRUE is s > 0."""
    truth = spins > 0
    v = np.abs(lits) - 1
    ok = np.where(lits > 0, truth[:, v], ~truth[:, v])
    start = np.concatenate([[0], np.cumsum(lens)[:-1]])
    return (np.add.reduceat(ok.astype(np.int64), start, axis=1) == 0).sum(axis=1)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n,m,lens,batch", [
    (1, 1, [1], 1), (5, 3, [1, 2], 33), (50, 210, [3], 31), (50, 210, [3], 1200), (257, 1025, [4], 601),
    (100, 40000, [1], 3), (300, 1000, [2, 3, 7, 12], 150), (31000, 2000, [3], 700), (3000, 33000, [3], 70),
    (40000, 5000, [3, 5], 64), (33000, 300, [4], 2)])
def test_violation_counts_over_groups(n, m, lens, batch, dtype):
    lits, length = formula(n, m, lens, seed=n + m)
    p = A.SatProblem.from_arrays(lits, length)
    rng = np.random.default_rng(1)
    x = rng.uniform(-1, 1, (batch, p.n + p.m)).astype(dtype)
    special = rng.integers(0, 40, x.shape)
    for code, val in enumerate([0.0, -0.0, np.nan, np.inf, -np.inf, 1.0, -1.0, 1e-45]):
        x[special == code] = val
    got = A.clause_violation_counts(p, torch.from_numpy(x).cuda()).cpu().numpy()
    assert np.array_equal(got, counts(lits, length, x[:, :p.n]))

