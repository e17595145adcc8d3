"""The work that users of this library have it do, case by case, through its public
Python entry points: sizes, inputs, one pass of each, and the same results in plain
64-bit torch.

Five kinds of pass:

* rhs      get_derivatives on a [batch, N + M] tensor of states
* viol     clause_violation_counts on such a tensor
* solve    SatSolver: set states, Solve, read the results and the final states
* maxsat   the same on one instance far beyond one SM, random starts drawn on the
           device and the best assignment seen kept
* adjoint  gradients of the final potential

Every solve ends by itself or at its step limit (no start stops another), so that a
pass has one outcome.
"""
import math

import numpy as np
import torch

import analogsat_b200 as A
from analogsat_b200.instances import make_instance

PREC = {"f32": A.AS_PREC_F32_LOGA, "f64": A.AS_PREC_F64}
TORCH = {"f32": torch.float32, "f64": torch.float64}
SIZE = {"f32": 4, "f64": 8}


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one right-hand side of a small formula: a caller with its own integrator, where
        # the call's latency is all there is
        dict(name="rhs_one", kind="rhs", dtype="f64", log=False, n=50, m=210, k=3, batch=1),
        # the standalone right-hand side at the benchmark's size: 64 x 256 states in HBM
        dict(name="rhs_f32", kind="rhs", dtype="f32", log=True, n=1000, m=4250, k=3, batch=16384),
        # the same in the reference's precision, at sizes that divide nothing
        dict(name="rhs_f64", kind="rhs", dtype="f64", log=False, n=777, m=3301, k=3, batch=1999),
        # a few states of an instance that no SM holds (the large 4-SAT formula)
        dict(name="rhs_large", kind="rhs", dtype="f32", log=True, n=100000, m=1000000, k=4, batch=4),
        # unsatisfied clauses of many states: the check that any outer search makes
        dict(name="viol_f32", kind="viol", dtype="f32", n=1000, m=4250, k=3, batch=16384),
        # one small formula, 16 starts to their solutions in the reference's precision
        dict(name="solve_small_f64", kind="solve", dtype="f64", n=50, n_max=50, m=210, k=3, instances=1, starts=16,
             steps=2000, check=50),
        # planted 3-SAT at the threshold, N = 1000, FP32 with log-space weights: the
        # benchmark's instances and starts, fewer of each
        dict(name="solve_f32", kind="solve", dtype="f32", n=1000, n_max=1000, m=4250, k=3, instances=32, starts=16,
             steps=300, check=50),
        # instances of uneven size in one call, N from 100 to 5000 (most beyond one SM)
        dict(name="solve_uneven_f32", kind="solve", dtype="f32", n=100, n_max=5000, m=0, k=3, instances=24, starts=11,
             steps=100, check=50),
        # N = 1000 in FP64: bit for bit the reference's integration
        dict(name="solve_f64", kind="solve", dtype="f64", n=1000, n_max=1000, m=4250, k=3, instances=16, starts=16,
             steps=100, check=50),
        # gradients w.r.t. initial state and clause weights, N = 200, T = 5, FP32
        dict(name="adjoint_f32", kind="adjoint", dtype="f32", n=200, m=850, k=3, instances=64, starts=16, t_end=5.0,
             weighted=False),
        # the same in FP64 with clause weights, a smaller and odd batch
        dict(name="adjoint_f64", kind="adjoint", dtype="f64", n=151, m=643, k=3, instances=17, starts=9, t_end=4.0,
             weighted=True),
        # MAXSAT: one 4-SAT instance of a million clauses, 32 random starts
        dict(name="maxsat_f32", kind="maxsat", dtype="f32", n=100000, m=1000000, k=4, starts=32, steps=20, check=10),
    ]


def _spread(rng, lo, hi):
    """A whole number, uniform over its logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5))))))


def draw(rng):
    kind = rng.choice(["rhs", "rhs", "viol", "solve", "solve", "adjoint", "adjoint", "maxsat"])
    k = rng.choice([3, 3, 3, 4])
    alpha = rng.uniform(3.8, 4.26) if k == 3 else rng.uniform(8.0, 10.0)
    dtype = rng.choice(["f32", "f64"])
    if kind in ("rhs", "viol"):
        n = _spread(rng, 30, 100000)
        m = round(alpha * n)
        batch = _spread(rng, 1, max(1, min(16384, 86_000_000 * 4 // SIZE[dtype] // (n + m))))
        case = dict(kind=kind, dtype=dtype, n=n, m=m, k=k, batch=batch)
        return dict(case, log=dtype == "f32" and rng.random() < 0.7) if kind == "rhs" else case
    if kind == "solve":
        n = _spread(rng, 40, 5000 if dtype == "f32" else 1500)
        n_max = n if rng.random() < 0.7 else min(5000, 2 * n)
        steps = _spread(rng, 20, 300)
        units = max(1, int((1.5e8 if dtype == "f32" else 2.5e7) / (steps * n_max * (1 if k == 3 else 3))))
        instances = _spread(rng, 1, min(16, units))
        starts = _spread(rng, 1, max(1, min(64, units // instances)))
        return dict(kind="solve", dtype=dtype, n=n, n_max=n_max, m=0 if n_max > n else round(alpha * n), k=k,
                    instances=instances, starts=starts, steps=steps, check=rng.choice([10, 20, 50]))
    if kind == "adjoint":
        n = _spread(rng, 30, 250 if k == 3 else 110)
        instances = _spread(rng, 1, 48)
        return dict(kind="adjoint", dtype=dtype, n=n, m=round(alpha * n), k=k, instances=instances,
                    starts=_spread(rng, 1, max(1, (1000 if dtype == "f32" else 400) // instances)),
                    t_end=round(rng.uniform(1.0, 5.0), 2), weighted=rng.random() < 0.5)
    n = _spread(rng, 53000, 100000)
    return dict(kind="maxsat", dtype="f32", n=n, m=10 * n, k=4, starts=_spread(rng, 3, 32), steps=rng.choice([10, 20]),
                check=10)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _sizes(case, seed):
    """(N, M) of every instance of a case."""
    if case["kind"] != "solve":
        return [(case["n"], case["m"])] * case.get("instances", 1)
    if case["n_max"] == case["n"]:
        return [(case["n"], case["m"])] * case["instances"]
    # uneven: N ~ U{n..n_max}, drawn evenly over the range so that seeds differ in the
    # instances and not in the amount of work; alpha ~ U(3.8, 4.26)
    rng = np.random.default_rng(1234)
    at = (np.arange(case["instances"]) + rng.random(case["instances"])) / case["instances"]
    ns = case["n"] + (at * (case["n_max"] - case["n"])).astype(int)
    lo, hi = (3.8, 4.26) if case["k"] == 3 else (8.0, 9.5)
    return [(int(n), int(round(n * a))) for n, a in zip(ns, rng.uniform(lo, hi, len(ns)))]


def _formulas(case, seed):
    """[(literals, lengths)] of a case: planted instances for solving, random ones otherwise."""
    out = []
    for i, (n, m) in enumerate(_sizes(case, seed)):
        kind = "planted" if case["kind"] == "solve" and m < 40000 else "random" if m < 40000 else "fast"
        lits, lens, _ = make_instance(kind, n, m, case["k"], seed=1000 * (seed + 1) + i)
        out.append((lits, lens))
    return out


def _nm(formula):
    return int(np.abs(formula[0]).max()), len(formula[1])


def _rhs_states(case, seed, n, m):
    """States as an integration meets them: spins in (-1, 1), some of them close to +-1,
    weights that have grown from 1 (as log2 a in log space)."""
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    dt = TORCH[case["dtype"]]
    s = torch.rand(case["batch"], n, generator=g, device="cuda", dtype=dt) * 2 - 1
    s = torch.sin(s * (math.pi / 2))
    u = torch.rand(case["batch"], m, generator=g, device="cuda", dtype=dt) * 3
    if not case.get("log", False):
        u = torch.exp2(u)
    return torch.cat([s, u], dim=1).contiguous()


def _starts(case, seed, formulas, dtype):
    """Problem index of every trajectory and their initial states, one after another:
    s ~ U(-1, 1), a = 1."""
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    index, parts = [], []
    for i, f in enumerate(formulas):
        n, m = _nm(f)
        x = torch.ones(case["starts"], n + m, device="cuda", dtype=dtype)
        x[:, :n] = torch.rand(case["starts"], n, generator=g, device="cuda", dtype=torch.float64) * 2 - 1
        parts.append(x.reshape(-1))
        index += [i] * case["starts"]
    return np.array(index, np.int32), torch.cat(parts)


def _weights(case, seed, count):
    return 0.5 + np.random.default_rng(seed + 7).random(count) if case["weighted"] else None


def prepare(case, seed):
    formulas = _formulas(case, seed)
    problems = [A.SatProblem.from_arrays(*f) for f in formulas]
    st = {"case": case, "problems": problems}
    kind = case["kind"]
    if kind in ("rhs", "viol"):
        p = problems[0]
        st["x"] = _rhs_states(case, seed, p.n, p.m)
        if kind == "rhs":
            st["out"] = torch.empty_like(st["x"])
        return st
    s = A.SatSolver(problems, precision=PREC[case["dtype"]], device=0)
    s.SetEpsilon(1e-6)
    s.SetMaxTime(1e8)
    st["solver"] = s
    if kind == "adjoint":
        st["index"], x = _starts(case, seed, formulas, TORCH[case["dtype"]])
        s.SetSatStates(st["index"], x)
        st["weights"] = _weights(case, seed, sum(problems[i].m for i in st["index"]))
        return st
    s.SetBatchSize(case["check"])
    s.SetMaxSteps(case["steps"])
    if kind == "maxsat":
        s.SetTrackBest(True)
        st["index"] = np.zeros(case["starts"], np.int32)
        st["seed"] = seed + 1
        total = case["starts"] * (problems[0].n + problems[0].m)
    else:
        st["index"], st["x"] = _starts(case, seed, formulas, TORCH[case["dtype"]])
        total = st["x"].numel()
    st["host"] = torch.empty(total, dtype=TORCH[case["dtype"]], pin_memory=True).numpy()
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "rhs":
        return A.get_derivatives(st["problems"][0], st["x"], out=st["out"], logspace=case["log"])
    if kind == "viol":
        return A.clause_violation_counts(st["problems"][0], st["x"])
    s = st["solver"]
    if kind == "adjoint":
        g = s.Adjoint(case["t_end"], weights=st["weights"], max_steps=512)
        dt = np.float32 if case["dtype"] == "f32" else np.float64
        # in the states' own precision, as a caller's autograd function hands them on
        return {"loss": g["loss"].astype(dt), "grad_x0": g["grad_x0"].astype(dt), "grad_w": g["grad_w"].astype(dt),
                "nsteps": g["nsteps"]}
    if kind == "maxsat":
        s.SetRandomInitialState(st["index"], st["seed"])
        s.Solve()
        best = np.stack([s.GetBestAssignment(t) for t in range(case["starts"])])
        return {"results": s.results(), "best": best, "states": s.GetSatStates(out=st["host"])}
    s.SetSatStates(st["index"], st["x"])
    s.Solve()
    return {"results": s.results(), "states": s.GetSatStates(out=st["host"])}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _rhs_flops(m, k):
    # per clause: k factors, their product, k leave-one-out products and contributions
    # (one multiply and one add each), the weight's derivative
    return m * (2 * k + max(0, k - 2) * k + 2 * k + 4)


def work(case):
    size, kind, k = SIZE[case["dtype"]], case["kind"], case["k"]
    sizes = _sizes(case, 0)
    lits = sum(4 * k * m for _, m in sizes)
    if kind == "rhs":
        n, m = sizes[0]
        return {"bytes": 2 * case["batch"] * (n + m) * size + lits, "flops": case["batch"] * _rhs_flops(m, k)}
    if kind == "viol":
        n, m = sizes[0]
        return {"bytes": case["batch"] * (n * size + 4) + lits, "flops": case["batch"] * m * k}
    starts = case["starts"]
    if kind == "adjoint":
        steps = 6 + 7 * case["t_end"]
        rhs = sum(_rhs_flops(m, k) for _, m in sizes) * starts
        vals = sum(n + 2 * m for n, m in sizes) * starts
        # forward 6 evaluations a step; backward 5 again and 6 vector-Jacobian products
        # of about three times the operations
        return {"bytes": 2 * vals * size + lits, "flops": steps * (11 + 18) * rhs}
    steps = min(case["steps"], 250)  # a small instance is solved after some 250 steps
    per = sum(6 * _rhs_flops(m, k) + 60 * (n + m) for n, m in sizes) * starts
    states = sum(n + m for n, m in sizes) * starts * size
    return {"bytes": (1 if kind == "maxsat" else 2) * states + lits, "flops": steps * per}


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------
class _Formula:
    def __init__(self, formula, k):
        lits = torch.from_numpy(formula[0].reshape(-1, k)).cuda().long()
        self.n, self.m = _nm(formula)
        self.k = k
        self.var, self.sign = lits.abs() - 1, lits.sign().double()

    def factors(self, s):
        return [1 - self.sign[:, q] * s[:, self.var[:, q]] for q in range(self.k)]

    def derivative(self, s, a, w=None):
        """ds/dt and K^2 for a batch of states."""
        f = self.factors(s)
        norm = 2.0 ** -self.k
        K = norm * math.prod(f)
        ds = torch.zeros_like(s)
        r = 2 * a * K if w is None else 2 * w * a * K
        for q in range(self.k):
            others = norm * math.prod([f[l] for l in range(self.k) if l != q])
            ds = ds.index_add(1, self.var[:, q], r * others * self.sign[:, q])
        return ds, K * K


_B = [[], [1 / 5], [3 / 40, 9 / 40], [3 / 10, -9 / 10, 6 / 5], [-11 / 54, 5 / 2, -70 / 27, 35 / 27],
      [1631 / 55296, 175 / 512, 575 / 13824, 44275 / 110592, 253 / 4096]]
_C = [37 / 378, 0, 250 / 621, 125 / 594, 0, 512 / 1771]
_D = [37 / 378 - 2825 / 27648, 0, 250 / 621 - 18575 / 48384, 125 / 594 - 13525 / 55296, -277 / 14336,
      512 / 1771 - 1 / 4]


def _step(f, x, h, w):
    """Cash-Karp stages of one step of every trajectory (linear weights)."""
    ks = []
    for row in _B:
        y = x
        if row:
            y = x + h[:, None] * sum(b * k for b, k in zip(row, ks))
        s, a = y[:, : f.n], y[:, f.n :]
        ds, k2 = f.derivative(s, a, w)
        ks.append(torch.cat([ds, a * k2], dim=1))
    return ks


def _exact_adjoint(f, x0, w, t_end, eps):
    """The adaptive integration to t_end and the gradients of the recorded steps."""
    B = x0.shape[0]
    t = torch.zeros(B, dtype=torch.float64, device="cuda")
    hnext = torch.full_like(t, 1e-9)
    x, hs = x0.clone(), []
    with torch.no_grad():
        while bool((t < t_end).any()):
            live = t < t_end
            hnext = torch.where(t + hnext > t_end, t_end - t, hnext)
            h, h0, todo = torch.where(live, hnext, 0 * t), hnext.clone(), live.clone()
            xn = x
            while bool(todo.any()):
                ks = _step(f, x, h, w)
                err = h[:, None] * sum(d * k for d, k in zip(_D, ks))
                scale = x.abs() + (ks[0] * h0[:, None]).abs() + 1e-20
                e = (err / scale).abs().amax(dim=1) / eps
                ok = todo & (e <= 1)
                new = x + h[:, None] * sum(c * k for c, k in zip(_C, ks))
                xn = torch.where(ok[:, None], new, xn)
                grow = torch.where(e > 1.89e-4, 0.9 * h * e.clamp_min(1e-300) ** -0.2, 5 * h)
                hnext = torch.where(ok, grow, hnext)
                todo = todo & ~ok
                h = torch.where(todo, torch.maximum(0.9 * h * e.clamp_min(1e-300) ** -0.25, 0.1 * h), h)
            hs.append(torch.where(live, h, 0 * h))
            x, t = xn, torch.where(live, t + h, t)
    ck = [x0]
    with torch.no_grad():
        for h in hs:
            ks = _step(f, ck[-1], h, w)
            ck.append(ck[-1] + h[:, None] * sum(c * k for c, k in zip(_C, ks)))
    xT, wT = ck[-1].requires_grad_(), w.clone().requires_grad_()
    loss = (wT * xT[:, f.n :] * (2.0 ** -f.k * math.prod(f.factors(xT[:, : f.n]))) ** 2).sum(dim=1)
    lam, gw = torch.autograd.grad(loss.sum(), [xT, wT])
    for x, h in zip(reversed(ck[:-1]), reversed(hs)):
        x, wi = x.detach().requires_grad_(), w.clone().requires_grad_()
        new = x + h[:, None] * sum(c * k for c, k in zip(_C, _step(f, x, h, wi)))
        lam, g = torch.autograd.grad(new, [x, wi], lam)
        gw = gw + g
    return loss.detach(), lam, gw


def exact(case, seed):
    kind, k = case["kind"], case["k"]
    if kind in ("solve", "maxsat"):
        return None  # adaptive integrations of many steps: a rounding decides the next step size
    formulas = _formulas(case, seed)
    if kind in ("rhs", "viol"):
        f = _Formula(formulas[0], k)
        x = _rhs_states(case, seed, f.n, f.m)
        rows = max(1, 6_000_000 // f.m)
        out = []
        for c in x.split(rows):
            s, a = c[:, : f.n].double(), c[:, f.n :].double()
            if kind == "viol":
                true = (s > 0).double() * 2 - 1
                open_ = math.prod([(true[:, f.var[:, q]] != f.sign[:, q]).int() for q in range(k)])
                out.append(open_.sum(dim=1).int())
            else:
                ds, k2 = f.derivative(s, torch.exp2(a) if case["log"] else a)
                out.append(torch.cat([ds, k2 / math.log(2) if case["log"] else a * k2], dim=1))
        return torch.cat(out)
    index, x = _starts(case, seed, formulas, TORCH[case["dtype"]])
    wts = _weights(case, seed, sum(_nm(formulas[i])[1] for i in index))
    res, ox, ow = [], 0, 0
    for fm in formulas:
        f = _Formula(fm, k)
        B = case["starts"]
        x0 = x[ox : ox + B * (f.n + f.m)].view(B, -1).double()
        w = torch.ones(B, f.m, dtype=torch.float64, device="cuda")
        if wts is not None:
            w = torch.from_numpy(wts[ow : ow + B * f.m]).cuda().view(B, f.m)
        ox, ow = ox + x0.numel(), ow + w.numel()
        res.append(_exact_adjoint(f, x0, w, case["t_end"], 1e-6))
    return {"loss": torch.cat([r[0] for r in res]), "grad_x0": torch.cat([r[1].reshape(-1) for r in res]),
            "grad_w": torch.cat([r[2].reshape(-1) for r in res]), "nsteps": None}
