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


def rhs(lits, lens, x, n, k, logspace):
    """ds/dt and da/dt (or d log2 a / dt) of every state in 64 bits."""
    x = x.astype(np.float64)
    s, a = x[:, :n], np.exp2(x[:, n:]) if logspace else x[:, n:]
    start = np.concatenate([[0], np.cumsum(lens)[:-1]])
    idx = np.repeat(np.arange(len(lens)), lens)
    v, c = np.abs(lits) - 1, np.sign(lits).astype(np.float64)
    f = 1 - c * s[:, v]
    # the factors of missing literals are 1 - (-1) = 2
    scale = 2.0 ** (k - lens) * 2.0 ** -k
    K = np.multiply.reduceat(f, start, axis=1) * scale
    out = np.zeros_like(x)
    out[:, n:] = K * K / np.log(2) if logspace else a * K * K
    for i in range(len(lits)):  # leave-one-out products
        j = idx[i]
        others = np.prod(np.delete(f[:, start[j]:start[j] + lens[j]], i - start[j], axis=1), axis=1) * scale[j]
        out[:, v[i]] += 2 * a[:, j] * c[i] * others * K[:, j]
    return out


@pytest.mark.parametrize("dtype,logspace", [("float32", True), ("float32", False), ("float64", False)])
@pytest.mark.parametrize("n,m,lens,batch", [
    (33000, 250, [3], 1), (33000, 250, [4], 2), (40001, 333, [2, 3, 5], 3), (33000, 257, [3], 4),
    (35000, 255, [3], 5), (33001, 400, [4], 8), (33000, 129, [1, 12], 9), (34000, 301, [3], 37)])
def test_rhs_of_instances_beyond_one_sm(n, m, lens, batch, dtype, logspace):
    lits, length = formula(n, m, lens, seed=n + m)
    p = A.SatProblem.from_arrays(lits, length)
    assert not p.layout_stats()["compact"]
    rng = np.random.default_rng(2)
    x = np.concatenate([rng.uniform(-1, 1, (batch, p.n)), rng.uniform(0.5, 3, (batch, p.m))], axis=1).astype(dtype)
    got = A.get_derivatives(p, torch.from_numpy(x).cuda(), logspace=logspace).cpu().numpy()
    want = rhs(lits, length, x, p.n, p.k, logspace)
    # each contribution is a product of 2 k + 2 rounded factors (ex2.approx: 2 ulp more);
    # a variable adds up at most its degree of them
    deg = np.bincount(np.abs(lits) - 1).max()
    eps = np.finfo(dtype).eps
    big = np.abs(want).max(axis=1, keepdims=True)
    assert (np.abs(got - want) <= (2 * max(lens) + deg + 8) * eps * big).all()
    if dtype == "float64" and batch > 1:  # a state alone takes rows of one lane, the same operations
        one = A.get_derivatives(p, torch.from_numpy(x[-1:]).cuda()).cpu().numpy()
        assert np.array_equal(one[0], got[-1])


@pytest.mark.parametrize("dtype,logspace", [("float32", True), ("float32", False), ("float64", False)])
@pytest.mark.parametrize("n,m,k,batch,shift", [
    (3, 1, 3, 1, 0), (50, 210, 3, 301, 1), (256, 1280, 3, 7, 0), (257, 1280, 3, 7, 1), (200, 1281, 3, 8, 0),
    (255, 700, 4, 2, 1), (512, 2560, 3, 301, 0), (513, 2160, 3, 5, 1), (400, 2561, 4, 3, 0), (999, 4251, 3, 298, 1),
    (1024, 4100, 3, 4, 0)])
def test_rhs_of_staged_states(n, m, k, batch, shift, dtype, logspace):
    lits, lens, _ = make_instance("fast", n, m, k, seed=n + m)
    p = A.SatProblem.from_arrays(lits, lens)
    rng = np.random.default_rng(3)
    x = np.concatenate([rng.uniform(-1, 1, (batch, p.n)), rng.uniform(0.5, 3, (batch, p.m))], axis=1).astype(dtype)
    # rows off a 16-byte boundary, and an output that shares or does not share its offset
    buf = torch.zeros(2, x.size + 4, dtype=getattr(torch, dtype), device="cuda")
    xs = buf[0, shift:shift + x.size].view(x.shape)
    xs.copy_(torch.from_numpy(x))
    out = buf[1, 1:1 + x.size].view(x.shape)
    A.get_derivatives(p, xs, out=out, logspace=logspace)
    A.rhs_check(p)
    got = out.cpu().numpy()
    rows = [0, batch // 2, batch - 1]
    want = rhs(lits, lens, x[rows], p.n, p.k, logspace)
    deg = np.bincount(np.abs(lits) - 1).max()
    big = np.abs(want).max(axis=1, keepdims=True)
    assert (np.abs(got[rows] - want) <= (2 * k + deg + 8) * np.finfo(dtype).eps * big).all()
    assert float(buf[1, 0]) == 0 and not buf[1, 1 + x.size:].any()  # nothing written around the output
    for r in rows:  # a state alone: the same operations
        one = A.get_derivatives(p, xs[r:r + 1].clone(), logspace=logspace).cpu().numpy()
        assert np.array_equal(one[0], got[r])


@pytest.mark.parametrize("dtype,logspace", [("float32", True), ("float32", False), ("float64", False)])
@pytest.mark.parametrize("n,m,k,batch", [(1025, 4200, 3, 3), (1500, 6300, 3, 150), (600, 5200, 4, 2), (2048, 6145, 3, 5),
                                         (4000, 16500, 3, 11)])
def test_rhs_of_larger_compact_instances(n, m, k, batch, dtype, logspace):
    """One FP32 state per staged pass, the one-state kernel, and rows over the whole GPU with
    clauses out of public order."""
    lits, lens, _ = make_instance("fast", n, m, k, seed=n + m)
    p = A.SatProblem.from_arrays(lits, lens)
    rng = np.random.default_rng(4)
    x = np.concatenate([rng.uniform(-1, 1, (batch, p.n)), rng.uniform(0.5, 3, (batch, p.m))], axis=1).astype(dtype)
    xs = torch.from_numpy(x).cuda()
    got = A.get_derivatives(p, xs, logspace=logspace).cpu().numpy()
    A.rhs_check(p)
    rows = [0, batch - 1]
    want = rhs(lits, lens, x[rows], p.n, p.k, logspace)
    deg = np.bincount(np.abs(lits) - 1).max()
    big = np.abs(want).max(axis=1, keepdims=True)
    assert (np.abs(got[rows] - want) <= (2 * k + deg + 8) * np.finfo(dtype).eps * big).all()
    for r in rows:  # a state alone: the same operations
        one = A.get_derivatives(p, xs[r:r + 1].clone(), logspace=logspace).cpu().numpy()
        assert np.array_equal(one[0], got[r])
