"""Repeated adjoint calls on one solver: what is kept between them and at what sizes they
are taken."""
import numpy as np
import pytest

import analogsat_b200 as A
from analogsat_b200.instances import initial_states, make_instance

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def setup(precision, n=60, m=250, starts=5):
    lits, lens, _ = make_instance("random", n, m, 3, seed=3)
    p = A.SatProblem.from_arrays(lits, lens)
    s = A.SatSolver([p], precision=precision, device=0)
    s.SetEpsilon(1e-6)
    dt = np.float32 if precision == A.AS_PREC_F32_LOGA else np.float64
    return s, initial_states(p.n, p.m, starts, seed=1).astype(dt)


def gradients(s, x, **kw):
    s.SetSatStates(np.zeros(len(x), np.int32), x)
    return s.Adjoint(2.0, **kw)


def same(a, b):
    return (all(np.array_equal(a[k], b[k]) for k in ("loss", "grad_x0", "grad_w", "nsteps"))
            and all(np.array_equal(u, v) for u, v in zip(a["step_sizes"], b["step_sizes"])))


@pytest.mark.parametrize("precision", [A.AS_PREC_F32_LOGA, A.AS_PREC_F64])
def test_first_and_later_calls_agree(precision):
    """The first call of a size, later ones, fewer and more trajectories after that."""
    s, x = setup(precision, starts=40)
    want = {b: gradients(setup(precision)[0], x[:b]) for b in (1, 7, 40)}
    for b in (7, 7, 7, 1, 40, 7, 40, 40, 1):
        assert same(gradients(s, x[:b]), want[b])


@pytest.mark.parametrize("precision", [A.AS_PREC_F32_LOGA, A.AS_PREC_F64])
@pytest.mark.parametrize("max_steps,starts", [(2 ** 28 + 3, 2), (2 ** 31 - 1, 1)])
def test_any_step_limit(precision, max_steps, starts):
    """A limit that stands for "no limit": tables of gigabytes, of which a few rows are used."""
    s, x = setup(precision, starts=starts)
    want = gradients(s, x)
    assert same(gradients(setup(precision)[0], x, max_steps=max_steps), want)
    with pytest.raises(A.AnalogSatError):
        gradients(s, x, max_steps=int(want["nsteps"].max()) - 1)
    assert same(gradients(s, x), want)


def test_little_memory_left():
    """The room for checkpoints that a first call takes on a guess is not needed for its result."""
    s, x = setup(A.AS_PREC_F64, n=200, m=850, starts=2000)
    want = gradients(s, x)
    steps = int(want["nsteps"].max())
    need = 8 * x.size * (steps + 2)
    guess = 8 * x.size * 48
    assert need < guess - (200 << 20)  # the case that matters
    s = setup(A.AS_PREC_F64, n=200, m=850)[0]
    s.SetSatStates(np.zeros(len(x), np.int32), x)
    torch.cuda.synchronize()
    tables = 16 * 2000 * 4097 + 4 * 8 * x.size
    room = need + tables + (64 << 20)
    hold = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
    try:
        got = s.Adjoint(2.0)
    finally:
        del hold
        torch.cuda.empty_cache()
    assert same(got, want)
