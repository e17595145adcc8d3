"""The allocation-free solve runs in the launch shape that as_solver_solve picks for the same
trajectories, whether they are few or many."""
import ctypes as C

import numpy as np
import pytest

import analogsat_b200 as A
from analogsat_b200.instances import initial_states, make_instance

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("precision", [A.AS_PREC_F32_LOGA, A.AS_PREC_F64])
@pytest.mark.parametrize("n,trajectories", [(50, 1), (50, 16), (50, 300), (50, 2000), (200, 16), (400, 3)])
@pytest.mark.parametrize("b", [0.0, 0.1])
def test_launch_shape_of_the_allocating_solve(n, trajectories, precision, b):
    lits, lens, _ = make_instance("planted", n, int(4.2 * n), 3, seed=n)
    p = A.SatProblem.from_arrays(lits, lens).set_bias(b)
    dt = np.float32 if precision == A.AS_PREC_F32_LOGA else np.float64
    x = initial_states(p.n, p.m, trajectories, seed=1).astype(dt)
    s = A.SatSolver([p], precision=precision, device=0)
    s.SetMaxSteps(3)
    s.SetSatStates(np.zeros(trajectories, np.int32), x)
    s.Solve()
    want = s.launch_shape(), s.kernel_name()
    t = A.SatSolver([p], precision=precision, device=0)
    t.SetMaxSteps(3)
    xd = torch.from_numpy(x).cuda()
    res = torch.zeros(trajectories * 48, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    rc = A.load().as_solver_solve_noalloc(t._h, 0, trajectories, C.c_void_p(xd.data_ptr()),
                                          C.c_void_p(res.data_ptr()), None)
    assert rc == 0
    torch.cuda.synchronize()
    assert (t.launch_shape(), t.kernel_name()) == want
    assert np.array_equal(xd.cpu().numpy().reshape(-1), s.GetSatStates(dt))
