"""Asynchronous solves, settings and state copies take effect in the order of the calls."""
import numpy as np
import pytest

import analogsat_b200 as A
from analogsat_b200.instances import initial_states, make_instance

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SETTINGS = {
    "stop on first": lambda s: s.SetStopOnFirst(True),
    "threads": lambda s: s.ForceThreads(128),
    "kernel": lambda s: s.SetKernel(A._abi.AS_KERNEL_GENERIC),
    "storage": lambda s: s.SetStorageMode(2),
}


def uneven():
    """Two sizes and more trajectories than run at once, none of them solved."""
    raw = [make_instance("random", n, int(4.5 * n), 3, seed=n)[:2] for n in (300, 420)]
    problems = [A.SatProblem.from_arrays(*r) for r in raw]
    index = np.tile([0, 1], 700).astype(np.int32)
    states = [initial_states(p.n, p.m, 700, seed=p.n).astype(np.float32) for p in problems]
    return problems, index, np.concatenate([states[i][t // 2] for t, i in enumerate(index)])


@pytest.mark.parametrize("own_stream", [True, False])
@pytest.mark.parametrize("what", list(SETTINGS))
def test_setting_changed_between_two_queued_solves(what, own_stream):
    """The second solve rebuilds the work queue; the first, still running, keeps its own."""
    problems, index, x = uneven()
    stream = None if own_stream else torch.cuda.Stream()
    out = []
    for wait in (True, False):
        s = A.SatSolver(problems, precision=A.AS_PREC_F32_LOGA, device=0)
        s.SetEpsilon(1e-6)
        s.SetMaxTime(1e8)
        s.SetMaxSteps(30)
        s.SetBatchSize(30)
        s.SetSatStates(index, x)
        s.SolveAsync(stream)
        if wait:
            s.Sync()
        SETTINGS[what](s)
        s.SolveAsync(stream)
        s.Sync()
        out.append((s.results(), s.GetSatStates(np.float32)))
    (r0, x0), (r1, x1) = out
    assert not (r0["status"] == 0).any()
    assert np.array_equal(x0, x1)
    assert all(np.array_equal(r0[k], r1[k]) for k in r0)


def test_trajectories_replaced_behind_a_queued_solve():
    """Fewer and other trajectories set while a solve runs: the buffers are its own until it ends."""
    problems, index, x = uneven()
    s = A.SatSolver(problems, precision=A.AS_PREC_F32_LOGA, device=0)
    s.SetEpsilon(1e-6)
    s.SetMaxTime(1e8)
    s.SetMaxSteps(30)
    s.SetBatchSize(30)
    y = initial_states(problems[1].n, problems[1].m, 50, seed=9).astype(np.float32)
    one = np.ones(50, np.int32)
    s.SetSatStates(one, y)
    s.Solve()
    want = s.results(), s.GetSatStates(np.float32)
    for _ in range(3):
        s.SetSatStates(index, x)
        s.SolveAsync()
        s.SetSatStates(one, y)
        s.SolveAsync()
        s.Sync()
        r, z = s.results(), s.GetSatStates(np.float32)
        assert np.array_equal(z, want[1])
        assert all(np.array_equal(r[k], want[0][k]) for k in r)
