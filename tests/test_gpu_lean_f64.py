"""The lean FP64 solver (rows in shared memory or in a global slab) against the general
kernel: the same operations in the same order, so counters and states are equal."""
import numpy as np
import pytest

import analogsat_b200 as A
from analogsat_b200 import _abi
from analogsat_b200.instances import initial_states, make_instance

pytestmark = pytest.mark.gpu


def run(problems, index, x, kernel, mode, threads=0):
    s = A.SatSolver(problems, precision=A.AS_PREC_F64)
    s.SetEpsilon(1e-6)
    s.SetMaxTime(1e8)
    s.SetMaxSteps(60)
    s.SetBatchSize(20)
    s.SetTrackBest(True)
    s.SetKernel(kernel)
    s.SetStorageMode(mode)
    s.ForceThreads(threads)
    s.SetSatStates(index, x)
    s.Solve()
    return s.results(), s.GetSatStates(), [s.GetBestAssignment(t) for t in range(len(index))], s.kernel_name()


@pytest.mark.parametrize("n,m,k,mode,threads", [
    (3, 5, 3, 0, 0), (31, 130, 3, 0, 0), (32, 134, 3, 2, 0), (33, 140, 3, 0, 32), (64, 600, 4, 0, 0), (65, 601, 4, 2, 0),
    (500, 2100, 3, 0, 0), (620, 2600, 3, 0, 0), (1000, 4250, 3, 0, 0), (1023, 4351, 3, 0, 992), (1700, 7000, 3, 0, 0)])
def test_lean_f64_follows_the_general_kernel(n, m, k, mode, threads):
    lits, lens, _ = make_instance("planted", n, m, k, seed=n)
    p = A.SatProblem.from_arrays(lits, lens)
    x = initial_states(p.n, p.m, 3, seed=7)
    x[1, p.n:] = np.random.default_rng(1).uniform(0.1, 4, p.m)
    a = run([p], [0, 0, 0], x, _abi.AS_KERNEL_AUTO, mode, threads)
    b = run([p], [0, 0, 0], x, _abi.AS_KERNEL_GENERIC, 0)
    assert a[3] == "solve_kernel_fast" and b[3] == "solve_kernel"
    for key in a[0]:
        assert np.array_equal(a[0][key], b[0][key]), key
    assert np.array_equal(a[1], b[1])
    assert all(np.array_equal(u, v) for u, v in zip(a[2], b[2]))
