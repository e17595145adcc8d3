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


@pytest.mark.parametrize("own", [False, True])
def test_device_states_follow_their_stream(own):
    """States that work queued on the caller's stream still writes are the ones copied in, and
    the tensor may be overwritten right after the call."""
    lits, lens, _ = make_instance("planted", 200, 840, 3, seed=1)
    p = A.SatProblem.from_arrays(lits, lens)
    x = torch.from_numpy(initial_states(p.n, p.m, 64, seed=2).astype(np.float32)).cuda()
    s = A.SatSolver([p], precision=A.AS_PREC_F32_LOGA, device=0)
    index = np.zeros(64, np.int32)
    s.SetSatStates(index, x)  # the buffers are there before
    big = torch.zeros(1 << 28, device="cuda")
    late = torch.zeros_like(x)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream() if own else torch.cuda.default_stream()):
        for _ in range(8):
            big += 1  # milliseconds of work in front
        late.copy_(x)
        s.SetSatStates(index, late)
        late.zero_()
    assert np.array_equal(s.GetSatStates(np.float32), x.cpu().numpy().reshape(-1))


def test_device_states_set_behind_a_queued_solve():
    """The states of the next solve do not reach the one that is running."""
    problems, index, x = uneven()
    s = A.SatSolver(problems, precision=A.AS_PREC_F32_LOGA, device=0)
    s.SetEpsilon(1e-6)
    s.SetMaxTime(1e8)
    s.SetMaxSteps(30)
    s.SetBatchSize(30)
    a = torch.from_numpy(x).cuda()
    b = a.roll(1).clamp(-0.9, 0.9).abs() + 0.05
    torch.cuda.synchronize()
    want = []
    for y in (a, b):
        s.SetSatStates(index, y)
        s.Solve()
        want.append((s.results(), s.GetSatStates(np.float32)))
    for stream in (None, torch.cuda.Stream()):
        s.SetSatStates(index, a, stream=stream)
        s.SolveAsync()
        s.SetSatStates(index, b, stream=stream)
        s.SolveAsync()
        s.Sync()
        r, z = s.results(), s.GetSatStates(np.float32)
        assert np.array_equal(z, want[1][1])
        assert all(np.array_equal(r[k], want[1][0][k]) for k in r)
