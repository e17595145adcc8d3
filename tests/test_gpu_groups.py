"""One call over instances of several launch shapes: the groups run side by side and the
largest instances first, and every trajectory ends as it does when its instance is solved
alone."""
import numpy as np
import pytest

import analogsat_b200 as A
from analogsat_b200.instances import initial_states, make_instance

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def solver(problems, precision):
    s = A.SatSolver(problems, precision=precision)
    s.SetEpsilon(1e-6)
    s.SetMaxTime(1e8)
    s.SetMaxSteps(40)
    s.SetBatchSize(20)
    return s


@pytest.mark.parametrize("precision,sizes", [(A.AS_PREC_F32_LOGA, [40, 1500, 300, 2000, 70]),
                                             (A.AS_PREC_F64, [33, 900, 200, 700]), (A.AS_PREC_F32_LOGA, [64, 65])])
def test_groups_equal_instances_alone(precision, sizes):
    raw = [make_instance("planted", n, int(4.2 * n), 3, seed=n)[:2] for n in sizes]
    problems = [A.SatProblem.from_arrays(*r) for r in raw]
    dt = np.float32 if precision == A.AS_PREC_F32_LOGA else np.float64
    index, parts = [], []
    for t in range(3):  # starts of an instance spread over the call
        for i, p in enumerate(problems):
            index.append(i)
            parts.append(initial_states(p.n, p.m, 1, seed=10 * i + t)[0].astype(dt))
    s = solver(problems, precision)
    alone = [solver([p], precision) for p in problems]
    want = []
    for i, x in zip(index, parts):
        alone[i].SetSatStates([0], x)
        alone[i].Solve()
        want.append((alone[i].GetSatState(0, dt), {k: v[0] for k, v in alone[i].results().items()}))
    stream = torch.cuda.Stream()
    for how in ("solve", "again", "stream", "stop on first"):
        s.SetStopOnFirst(how == "stop on first")  # rebuilds the queue; nothing is solved in 40 steps
        s.SetSatStates(index, np.concatenate(parts))
        if how == "stream":
            s.SolveAsync(stream)
            s.Sync()
        else:
            s.Solve()
        r = s.results()
        for t, (x, w) in enumerate(want):
            if how == "stop on first" and (r["status"] == 0).any():
                break
            assert np.array_equal(s.GetSatState(t, dt), x), (how, t)
            assert all(r[k][t] == w[k] for k in w), (how, t)


@pytest.mark.parametrize("n", [1400, 2500])
def test_few_starts_of_a_large_instance_match_clusters(n):
    """One CTA per trajectory is taken where a cluster of CTAs was; the results are equal."""
    lits, lens, _ = make_instance("planted", n, int(4.2 * n), 3, seed=n)
    p = A.SatProblem.from_arrays(lits, lens)
    x = initial_states(p.n, p.m, 2, seed=1).astype(np.float32)
    out = []
    for ctas in (0, 4, 8):
        s = solver([p], A.AS_PREC_F32_LOGA)
        s.SetClusterSize(ctas)
        s.SetSatStates([0, 0], x)
        s.Solve()
        out.append((s.GetSatStates(np.float32), s.results(), s.kernel_name()))
    assert out[0][2] == "solve_kernel_fast" and out[1][2] == "solve_kernel"
    for o in out[1:]:
        assert np.array_equal(o[0], out[0][0])
        assert all(np.array_equal(o[1][k], out[0][1][k]) for k in o[1])
