"""Second rounds of loops that small inputs leave after one: counter flushes of the unsat
counts, chunks of the row kernels, and uneven solves with stop-on-first that nothing stops."""
import numpy as np
import pytest

import analogsat_b200 as A
from analogsat_b200.instances import initial_states, make_instance
from test_gpu_primitives import formula, rhs

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,m,batch,compact", [
    (100, 40000, 700, True),      # CTAs of 256 threads, 127 clauses a thread between flushes
    (100, 70000, 18960, False)])  # two slices of 35,000 clauses for each of 593 groups
def test_counts_beyond_one_flush(n, m, batch, compact):
    lits, length = formula(n, m, [1], seed=m)
    p = A.SatProblem.from_arrays(lits, length)
    assert p.layout_stats()["compact"] == compact
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.zeros(batch, n + m, device="cuda")
    x[:, :n] = torch.rand(batch, n, generator=g, device="cuda") * 2 - 1
    got = A.clause_violation_counts(p, x).cpu().numpy()
    truth = (x[:, :n] > 0).cpu().numpy()
    pos = np.bincount(lits[lits > 0] - 1, minlength=n)
    neg = np.bincount(-lits[lits < 0] - 1, minlength=n)
    assert np.array_equal(got, np.where(truth, neg, pos).sum(axis=1))


@pytest.mark.parametrize("dtype,logspace", [("float32", True), ("float32", False), ("float64", False)])
@pytest.mark.parametrize("lens", [[3], [1, 5]])
def test_rows_beyond_one_chunk(dtype, logspace, lens):
    """A chunk holds 64 MB of rows, here about 60 groups: 480 FP32 or 240 FP64 states."""
    lits, length = formula(33000, 400, lens, seed=5)
    p = A.SatProblem.from_arrays(lits, length)
    batch = 507
    rng = np.random.default_rng(2)
    x = np.concatenate([rng.uniform(-1, 1, (batch, p.n)), rng.uniform(0.5, 3, (batch, p.m))], axis=1).astype(dtype)
    xs = torch.from_numpy(x).cuda()
    got = A.get_derivatives(p, xs, logspace=logspace)
    parts = torch.cat([A.get_derivatives(p, c.contiguous(), logspace=logspace) for c in xs.split(100)])
    assert torch.equal(got, parts)  # groups cut elsewhere: the same operations
    rows = list(range(222, 246)) + list(range(462, 486)) + [batch - 1]
    want = rhs(lits, length, x[rows], p.n, p.k, logspace)
    deg = np.bincount(np.abs(lits) - 1).max()
    big = np.abs(want).max(axis=1, keepdims=True)
    err = np.abs(got[rows].cpu().numpy() - want)
    assert (err <= (2 * max(lens) + deg + 8) * np.finfo(dtype).eps * big).all()


@pytest.mark.parametrize("precision,sizes", [(A.AS_PREC_F32_LOGA, [40, 1500, 300, 2000, 70]),
                                             (A.AS_PREC_F64, [33, 900, 200, 700])])
def test_stop_on_first_that_nothing_stops(precision, sizes):
    """Far above the threshold no start finds a solution, so stop-on-first, whose queue is dealt
    another way, ends every trajectory as a solve without it does."""
    problems = [A.SatProblem.from_arrays(*make_instance("random", n, int(5.5 * n), 3, seed=n)[:2]) for n in sizes]
    dt = np.float32 if precision == A.AS_PREC_F32_LOGA else np.float64
    index = np.tile(np.arange(len(sizes)), 4).astype(np.int32)
    x = np.concatenate([initial_states(problems[i].n, problems[i].m, 1, seed=t)[0].astype(dt)
                        for t, i in enumerate(index)])
    out = []
    for flag in (False, True, False):
        s = A.SatSolver(problems, precision=precision, device=0)
        s.SetEpsilon(1e-6)
        s.SetMaxTime(1e8)
        s.SetMaxSteps(40)
        s.SetBatchSize(20)
        s.SetStopOnFirst(flag)
        s.SetSatStates(index, x)
        s.Solve()
        out.append((s.results(), s.GetSatStates(dt)))
    for r, z in out:
        assert not (r["status"] == 0).any()
        assert np.array_equal(z, out[0][1])
        assert all(np.array_equal(r[k], out[0][0][k]) for k in r)
