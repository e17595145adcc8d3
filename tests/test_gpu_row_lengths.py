"""Right-hand side beyond one SM at every line of its clause lengths and batch sizes."""
import numpy as np
import pytest

import analogsat_b200 as A

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def formula(n, m, lens, seed):
    """Random clauses (a variable may come twice in one) with lengths drawn from `lens`."""
    rng = np.random.default_rng(seed)
    length = rng.choice(lens, m).astype(np.int32)
    length[0] = max(lens)
    lits = rng.integers(1, n + 1, length.sum()) * rng.choice([-1, 1], length.sum())
    lits[0] = n
    return lits.astype(np.int32), length


def rhs(lits, lens, x, n, k, logspace):
    """ds/dt and da/dt (or d log2 a / dt) of every state in 64 bits; absent literals are factors
    of 1 here and of 2, against 2^-k, in the definition."""
    x = x.astype(np.float64)
    s, a = x[:, :n], np.exp2(x[:, n:]) if logspace else x[:, n:]
    there = np.arange(k) < lens[:, None]
    lit = np.zeros((len(lens), k), np.int64)
    lit[there] = lits
    v, c = np.abs(lit) - there, np.sign(lit)
    f = np.where(there, 1 - c * s[:, v], 1.0)
    scale = 2.0 ** -lens.astype(np.float64)
    K = f.prod(axis=2) * scale
    out = np.zeros_like(x)
    out[:, n:] = K * K / np.log(2) if logspace else a * K * K
    for q in range(k):
        g = f.copy()
        g[:, :, q] = 1.0
        d = np.where(there[:, q], 2 * a * c[:, q] * g.prod(axis=2) * scale * K, 0.0)
        for b in range(len(x)):
            out[b, :n] += np.bincount(v[:, q], d[b], n)
    return out


def check(p, lits, length, x, got, rows, logspace):
    want = rhs(lits, length, x[rows], p.n, p.k, logspace)
    # each contribution is a product of 2 k + 2 rounded factors (ex2.approx: 2 ulp more); a
    # variable adds up at most its degree of them
    deg = np.bincount(np.abs(lits) - 1).max()
    big = np.abs(want).max(axis=1, keepdims=True)
    assert (np.abs(got[rows] - want) <= (2 * p.k + deg + 8) * np.finfo(x.dtype).eps * big).all()


@pytest.mark.parametrize("dtype,logspace", [("float32", True), ("float32", False), ("float64", False)])
@pytest.mark.parametrize("lens", [[1], [2], [1, 2], [4, 5], [5], [8], [2, 8], [9], [3, 16]])
@pytest.mark.parametrize("n", [33000, 5000])
def test_every_compiled_length(n, lens, dtype, logspace):
    m = 300 if n == 33000 else int(60000 / np.mean(lens))  # wide words; compact ones beyond one SM
    lits, length = formula(n, m, lens, seed=n + m)
    p = A.SatProblem.from_arrays(lits, length)
    rng = np.random.default_rng(2)
    x = np.concatenate([rng.uniform(-1, 1, (11, p.n)), rng.uniform(0.5, 3, (11, p.m))], axis=1).astype(dtype)
    xs = torch.from_numpy(x).cuda()
    got = A.get_derivatives(p, xs, logspace=logspace).cpu().numpy()
    check(p, lits, length, x, got, [0, 7, 10], logspace)
    for b in (1, 2, 5):  # rows of other widths: the same operations
        part = A.get_derivatives(p, xs[:b].contiguous(), logspace=logspace).cpu().numpy()
        check(p, lits, length, x, part, [b - 1], logspace)
        if dtype == "float64":
            assert np.array_equal(part, got[:b])


@pytest.mark.parametrize("k", [8, 9, 12])
def test_large_batches_of_long_clauses(k):
    """FP64 clauses of more than eight literals go to one CTA per state from eight states an SM on;
    both sides give the reference's products and sums bit for bit."""
    lits, length = formula(2500, 4000, [3, k], seed=k)
    p = A.SatProblem.from_arrays(lits, length)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(3)
    x = np.concatenate([rng.uniform(-1, 1, (8 * sms, p.n)), rng.uniform(0.5, 3, (8 * sms, p.m))], axis=1)
    xs = torch.from_numpy(x).cuda()
    at = A.get_derivatives(p, xs)
    below = A.get_derivatives(p, xs[:-1].contiguous())
    assert torch.equal(at[:-1], below)
    assert torch.equal(A.get_derivatives(p, xs[-1:].contiguous())[0], at[-1])
    check(p, lits, length, x, at.cpu().numpy(), [0, 8 * sms - 1], False)
