"""A start's trajectory does not depend on how many others are solved in the same call."""
import numpy as np
import pytest

import analogsat_b200 as A
from analogsat_b200.instances import initial_states, make_instance

pytestmark = pytest.mark.gpu

KEYS = ("status", "time", "steps", "rhs", "attempts", "violations", "min_violations", "last_step")


def run(p, precision, states):
    s = A.SatSolver([p], precision=precision, device=0)
    s.SetEpsilon(1e-6)
    s.SetBatchSize(20)
    s.SetMaxSteps(60)
    s.SetMaxTime(1e8)
    s.SetSatStates(np.zeros(len(states), np.int32), states)
    s.Solve()
    dtype = np.float64 if precision == A.AS_PREC_F64 else np.float32
    return s.results(), s.GetSatStates(dtype).reshape(len(states), -1)


@pytest.mark.parametrize("precision", [A.AS_PREC_F64, A.AS_PREC_F32_LOGA])
@pytest.mark.parametrize("tanh", [False, True])
@pytest.mark.parametrize("b", [0.0, 0.05])
@pytest.mark.parametrize("n,m", [(50, 210), (200, 840)])
def test_one_start_alone_and_among_many(precision, tanh, b, n, m):
    """Bit for bit: with the bias term the clause weights are summed over the threads of a CTA,
    so its rounding follows the CTA's size."""
    lits, lens, _ = make_instance("planted", n, m, 3, seed=21)
    p = A.SatProblem.from_arrays(lits, lens)
    p.set_model(tanh=tanh)
    p.set_bias(b)
    x = initial_states(p.n, p.m, 700, seed=5)
    x = x if precision == A.AS_PREC_F64 else x.astype(np.float32)
    many, xm = run(p, precision, x)
    few, xf = run(p, precision, x[:3])
    alone, xa = run(p, precision, x[:1])
    assert np.array_equal(xf, xm[:3]) and np.array_equal(xa, xm[:1])
    for k in KEYS:
        assert np.array_equal(few[k], many[k][:3]) and np.array_equal(alone[k], many[k][:1]), k
