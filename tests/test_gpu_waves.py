"""FP64 instances of one SM: the kernel of a call follows from its waves of trajectories, the
results do not."""
import numpy as np
import pytest

import analogsat_b200 as A
from analogsat_b200._abi import AS_KERNEL_AUTO, AS_KERNEL_GENERIC
from analogsat_b200.instances import initial_states, make_instance

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def run(problems, index, x, kernel):
    s = A.SatSolver(problems, precision=A.AS_PREC_F64, device=0)
    s.SetEpsilon(1e-6)
    s.SetMaxTime(1e8)
    s.SetMaxSteps(20)
    s.SetBatchSize(20)
    s.SetKernel(kernel)
    s.SetSatStates(index, x)
    s.Solve()
    shape = s.launch_shape()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    waves = -(-len(index) // (sms * shape["ctas_per_sm"]))
    return s.results(), s.GetSatStates(), s.kernel_name(), waves


@pytest.mark.parametrize("n,trajectories", [(200, 3), (200, 700), (200, 1500), (150, 700), (150, 1500), (400, 300)])
def test_no_more_waves_than_the_general_kernel(n, trajectories):
    lits, lens, _ = make_instance("random", n, int(4.2 * n), 3, seed=n)
    p = A.SatProblem.from_arrays(lits, lens)
    x = initial_states(p.n, p.m, trajectories, seed=1)
    index = np.zeros(trajectories, np.int32)
    r, z, name, waves = run([p], index, x, AS_KERNEL_AUTO)
    rg, zg, general, waves_g = run([p], index, x, AS_KERNEL_GENERIC)
    assert general == "solve_kernel" and waves <= waves_g
    assert name == "solve_kernel_fast" or waves == waves_g
    assert np.array_equal(z, zg) and all(np.array_equal(r[k], rg[k]) for k in r)


def test_several_instances_in_one_call():
    raw = [make_instance("random", n, int(4.2 * n), 3, seed=n)[:2] for n in (60, 200, 190)]
    problems = [A.SatProblem.from_arrays(*f) for f in raw]
    index = np.tile([0, 1, 2], 400).astype(np.int32)
    x = np.concatenate([initial_states(problems[i].n, problems[i].m, 1, seed=t)[0] for t, i in enumerate(index)])
    r, z, _, waves = run(problems, index, x, AS_KERNEL_AUTO)
    rg, zg, _, waves_g = run(problems, index, x, AS_KERNEL_GENERIC)
    assert waves <= waves_g
    assert np.array_equal(z, zg) and all(np.array_equal(r[k], rg[k]) for k in r)
