"""The work that users of this package have it do, as cases that can be timed
and compared: whole solver calls and differentiable losses, through the public
entry points (``regot`` and ``regot.torch``), from the README's example to the
large dense problems, in both storage types.

A case is a dict of plain values. ``kind`` says which entry point it calls:

    call       regot.<solver>(M, a, b, reg, ...) on host arrays, plan returned:
               what the README shows
    resident   Problem.<solver>(reg, ..., plan=False) on a cost matrix that is
               on the GPU already: what a program with a large problem does
    batched    regot.sinkhorn_bcd_batched(..., grad=True): many small problems,
               costs on the fly, forward and backward
    ot_cost    regot.torch.sqeuclid_ot_cost and its backward: a training loss
    ot_plan    regot.torch.ot_plan and its backward: a loss on the plan

``problem`` says what the cost matrix is made of:

    readme     1-D supports on [0, 5], exponential against a mixture of two
               normals (the README's example, on random supports)
    points     squared distances of 3-D Gaussian clouds over their largest,
               marginals uniform in (0.5, 1.5) (the large dense EROT workload)
    square     squared distances of points in the unit square, Dirichlet
               marginals (the large QROT workload)
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "regot-python_gb300"))

import regot  # noqa: E402
import regot.torch as regot_torch  # noqa: E402

BATCH_DIMS = (2, 3, 4, 6, 8, 12, 16)


def listed():
    return [
        # The README's example: a first call, an interactive session, a unit
        # test of a user's program. Launches and latency.
        dict(name="readme-100x80", kind="call", solver="sinkhorn_bcd", problem="readme",
             n=100, m=80, dtype="f64", reg=0.1, tol=1e-6, max_iter=1000),
        # The same at an ordinary size and a tight tolerance: some hundreds of
        # sweeps over a matrix that fits on the chip.
        dict(name="bcd-1000x800-f64", kind="call", solver="sinkhorn_bcd", problem="readme",
             n=1000, m=800, dtype="f64", reg=0.1, tol=1e-8, max_iter=1000),
        # The headline workload: a large dense problem in the default mode of
        # FP32 costs, duals only.
        dict(name="bcd-8192x8192-f32", kind="resident", solver="sinkhorn_bcd", problem="points",
             n=8192, m=8192, dtype="f32", reg=0.01, tol=1e-6, max_iter=1000),
        # A ragged problem in double precision, NumPy's and so most users'
        # default type.
        dict(name="bcd-3001x2503-f64", kind="resident", solver="sinkhorn_bcd", problem="points",
             n=3001, m=2503, dtype="f64", reg=0.01, tol=1e-6, max_iter=1000),
        # Newton's method at a large size: conjugate gradients on the dense
        # Hessian, one product with the plan a step.
        dict(name="newton-4096x4096-f32", kind="resident", solver="sinkhorn_newton",
             problem="points", n=4096, m=4096, dtype="f32", reg=0.01, tol=1e-6, max_iter=100),
        # Newton's method from host arrays in double precision.
        dict(name="newton-1000x800-f64", kind="call", solver="sinkhorn_newton", problem="points",
             n=1000, m=800, dtype="f64", reg=0.02, tol=1e-8, max_iter=100),
        # The sparsified Newton method, the reference's fastest solver.
        dict(name="ssns-1000x800-f64", kind="call", solver="sinkhorn_ssns", problem="points",
             n=1000, m=800, dtype="f64", reg=0.02, tol=1e-8, max_iter=200),
        # Quadratic regularisation at the size it is used at, a part of the
        # solve's iterations.
        dict(name="qrot-lbfgs-4096x4096-f32", kind="resident", solver="qrot_lbfgs_dual",
             problem="square", n=4096, m=4096, dtype="f32", reg=0.1, tol=1e-6, max_iter=100),
        # The semi-smooth Newton method for the same, ragged, in double
        # precision.
        dict(name="qrot-assn-1023x769-f64", kind="call", solver="qrot_assn", problem="square",
             n=1023, m=769, dtype="f64", reg=0.1, tol=1e-6, max_iter=20),
        # A batch of uneven point-cloud problems, forward and backward.
        dict(name="batched-64-grad", kind="batched", count=64, nmin=64, nmax=2048, reg=0.05,
             tol=1e-6, max_iter=20000),
        # A training loss on two clouds of embeddings.
        dict(name="ot-cost-4096x64-f32", kind="ot_cost", n=4096, m=4096, d=64, dtype="f32",
             reg=0.05, tol=1e-6),
        # A loss on the transport plan, differentiated through the solve.
        dict(name="ot-plan-1024x777-f64", kind="ot_plan", problem="points", n=1024, m=777,
             dtype="f64", reg=0.05, tol=1e-10),
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("call", "bcd", "newton", "ssns", "lbfgs", "assn", "batched", "ot_cost",
                       "ot_plan"))
    dtype = rng.choice(("f32", "f64"))
    if kind == "call":  # small problems from host arrays, in double precision
        problem, reg = rng.choice((("readme", 0.1), ("points", 0.05), ("points", 0.01)))
        return dict(kind="call", solver="sinkhorn_bcd", problem=problem,
                    n=_log_size(rng, 40, 1500), m=_log_size(rng, 40, 1500), dtype="f64", reg=reg,
                    tol=rng.choice((1e-6, 1e-8)), max_iter=1000)
    if kind == "bcd":
        return dict(kind="resident", solver="sinkhorn_bcd", problem="points",
                    n=_log_size(rng, 200, 8192), m=_log_size(rng, 200, 8192), dtype=dtype,
                    reg=rng.choice((0.05, 0.02, 0.01)), tol=1e-6, max_iter=1000)
    if kind == "newton":
        return dict(kind="resident", solver="sinkhorn_newton", problem="points",
                    n=_log_size(rng, 200, 4096), m=_log_size(rng, 200, 4096), dtype=dtype,
                    reg=rng.choice((0.05, 0.02, 0.01)), tol=1e-6, max_iter=100)
    if kind == "ssns":
        return dict(kind="call", solver="sinkhorn_ssns", problem="points",
                    n=_log_size(rng, 100, 1500), m=_log_size(rng, 100, 1500), dtype="f64",
                    reg=rng.choice((0.05, 0.02)), tol=1e-8, max_iter=200)
    if kind == "lbfgs":
        return dict(kind="resident", solver="qrot_lbfgs_dual", problem="square",
                    n=_log_size(rng, 200, 4096), m=_log_size(rng, 200, 4096), dtype=dtype,
                    reg=0.1, tol=1e-6, max_iter=rng.randint(30, 100) if dtype == "f32" else 30)
    if kind == "assn":
        return dict(kind="call", solver="qrot_assn", problem="square",
                    n=_log_size(rng, 100, 1200), m=_log_size(rng, 100, 1200), dtype="f64",
                    reg=0.1, tol=1e-6, max_iter=rng.randint(5, 20))
    if kind == "batched":
        return dict(kind="batched", count=rng.randint(4, 64), nmin=64,
                    nmax=rng.choice((500, 1000, 2048)), reg=0.05, tol=1e-6, max_iter=20000)
    if kind == "ot_cost":
        top = 4096 if dtype == "f32" else 1024
        return dict(kind="ot_cost", n=_log_size(rng, 128, top), m=_log_size(rng, 128, top),
                    d=_log_size(rng, 2, 64), dtype=dtype, reg=0.05, tol=1e-6)
    return dict(kind="ot_plan", problem="points", n=_log_size(rng, 100, 1024),
                m=_log_size(rng, 100, 1024), dtype="f64", reg=rng.choice((0.05, 0.02)), tol=1e-10)


# ------------------------------------------------------------------ inputs --

def _normal_pdf(x, loc, scale):
    return torch.exp(-0.5 * ((x - loc) / scale) ** 2) / (scale * math.sqrt(2 * math.pi))


def _distances(x, y):
    M = torch.zeros((x.shape[0], y.shape[0]), dtype=x.dtype, device=x.device)
    for k in range(x.shape[1]):
        M += (x[:, k, None] - y[None, :, k]) ** 2
    return M


def _problem(case, seed):
    """Cost matrix and marginals of a case, on the GPU, the marginals in
    float64 and the costs in the case's type."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    kw = dict(generator=g, device="cuda", dtype=torch.float64)
    n, m = case["n"], case["m"]
    if case["problem"] == "readme":
        x = 5.0 * torch.sort(torch.rand(n, **kw)).values
        y = 5.0 * torch.sort(torch.rand(m, **kw)).values
        a = torch.exp(-x)
        b = 0.2 * _normal_pdf(y, 1.0, 0.2) + 0.8 * _normal_pdf(y, 3.0, 0.5)
        b = torch.clamp(b, min=1e-12)
        M = _distances(x[:, None], y[:, None])
    elif case["problem"] == "points":
        x = torch.randn((n, 3), **kw)
        y = torch.randn((m, 3), **kw) + 0.5
        a = torch.rand(n, **kw) + 0.5
        b = torch.rand(m, **kw) + 0.5
        M = _distances(x, y)
        M /= M.max()
    else:
        x = torch.rand((n, 2), **kw)
        y = torch.rand((m, 2), **kw)
        # Dirichlet(1): normalised exponential variates
        a = torch.clamp(-torch.log1p(-torch.rand(n, **kw)), min=1e-6 * n)
        b = torch.clamp(-torch.log1p(-torch.rand(m, **kw)), min=1e-6 * m)
        M = _distances(x, y)
    if case["dtype"] == "f32":
        M = M.float()
    return M, a / a.sum(), b / b.sum()


def _batch(case, seed):
    """Point clouds of uneven sizes and their marginals, as host arrays; costs
    over the dimension."""
    rng = np.random.default_rng(seed)
    lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
    # sizes and dimensions belong to the case, points and marginals to the seed
    shape = np.random.default_rng(case["count"] * 7919 + case["nmax"])
    xs, ys, as_, bs, scale = [], [], [], [], []
    for _ in range(case["count"]):
        n, m = (int(round(math.exp(shape.uniform(lo, hi)))) for _ in range(2))
        d = int(shape.choice(BATCH_DIMS))
        xs.append(rng.standard_normal((n, d), dtype=np.float32))
        ys.append(rng.standard_normal((m, d), dtype=np.float32) + np.float32(0.3))
        a, b = rng.uniform(0.5, 1.5, n), rng.uniform(0.5, 1.5, m)
        as_.append(a / a.sum())
        bs.append(b / b.sum())
        scale.append(1.0 / d)
    return xs, ys, as_, bs, scale


def _clouds(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = torch.float32 if case["dtype"] == "f32" else torch.float64
    x = torch.randn((case["n"], case["d"]), generator=g, device="cuda", dtype=dt)
    y = torch.randn((case["m"], case["d"]), generator=g, device="cuda", dtype=dt)
    y += 0.2
    a = torch.full((case["n"],), 1.0 / case["n"], dtype=torch.float64, device="cuda")
    b = torch.full((case["m"],), 1.0 / case["m"], dtype=torch.float64, device="cuda")
    return x, y, a, b


def _weights(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed + 77)
    return torch.rand((case["n"], case["m"]), generator=g, device="cuda", dtype=torch.float64)


def prepare(case, seed):
    state = dict(case)
    if case["kind"] == "batched":
        state["inputs"] = _batch(case, seed)
    elif case["kind"] == "ot_cost":
        state["inputs"] = _clouds(case, seed)
    else:
        M, a, b = _problem(case, seed)
        if case["kind"] == "call":
            state["inputs"] = tuple(t.cpu().numpy() for t in (M, a, b))
        elif case["kind"] == "resident":
            torch.cuda.synchronize()  # the package copies M on its own stream
            state["problem"] = regot.Problem(M, a.cpu().numpy(), b.cpu().numpy())
        else:
            state["inputs"] = (M, a, b)
            state["weights"] = _weights(case, seed)
    return state


# ------------------------------------------------------------------- a pass --

def run(state):
    kind = state["kind"]
    if kind == "call":
        M, a, b = state["inputs"]
        r = getattr(regot, state["solver"])(M, a, b, state["reg"], tol=state["tol"],
                                            max_iter=state["max_iter"])
        return {"dual": r.dual, "plan": r.plan, "objective": r.obj_vals[-1]}
    if kind == "resident":
        r = getattr(state["problem"], state["solver"])(state["reg"], tol=state["tol"],
                                                       max_iter=state["max_iter"], plan=False)
        return {"dual": r.dual, "objective": r.obj_vals[-1]}
    if kind == "batched":
        xs, ys, as_, bs, scale = state["inputs"]
        r = regot.sinkhorn_bcd_batched(xs, ys, as_, bs, state["reg"], tol=state["tol"],
                                       max_iter=state["max_iter"], cost_scale=scale, grad=True)
        # one array each for all problems: a list of 64 would be too many outputs
        return {"duals": np.concatenate(r.duals), "costs": r.costs,
                "grad_x": np.concatenate([v.ravel() for v in r.grad_x]),
                "grad_y": np.concatenate([v.ravel() for v in r.grad_y])}
    if kind == "ot_cost":
        x, y, a, b = (t.detach().requires_grad_(True) for t in state["inputs"])
        loss = regot_torch.sqeuclid_ot_cost(x, y, a, b, state["reg"], scale=float(state["d"]),
                                            tol=state["tol"])
        loss.backward()
        return {"loss": loss.detach(), "x": x.grad, "y": y.grad, "a": a.grad, "b": b.grad}
    M, a, b = (t.detach().requires_grad_(True) for t in state["inputs"])
    T = regot_torch.ot_plan(M, a, b, state["reg"], tol=state["tol"])
    (T * state["weights"]).sum().backward()
    return {"plan": T.detach(), "M": M.grad, "a": a.grad, "b": b.grad}


# -------------------------------------------------------------------- work --

# Passes over the n x m entries that the solves of the listed problems take
# (sweeps of two reductions for BCD; conjugate gradient steps, gradients and
# line searches for Newton; trials for L-BFGS). They give the arithmetic, one
# multiplication and one addition an entry and reduction; the bytes are the
# inputs and outputs, once.
_REDUCTIONS = {"sinkhorn_bcd": 40, "sinkhorn_newton": 2 * 300, "sinkhorn_ssns": 60,
               "qrot_lbfgs_dual": 2 * 100, "qrot_assn": 2 * 20}


def work(case):
    kind = case["kind"]
    if kind == "batched":
        xs, ys, as_, bs, _ = _batch(case, 0)
        points = sum(x.size + y.size for x, y in zip(xs, ys))
        duals = sum(a.size + b.size for a, b in zip(as_, bs))
        pairs = sum(a.size * b.size for a, b in zip(as_, bs))
        return {"bytes": 2 * 4 * points + 2 * 8 * duals, "flops": 2.0 * 2 * 100 * pairs}
    n, m = case["n"], case["m"]
    size = 4 if case["dtype"] == "f32" else 8
    if kind == "ot_cost":
        return {"bytes": 2 * size * (n + m) * case["d"] + 2 * 8 * (n + m),
                "flops": 2.0 * n * m * (2 * 100 + 3 * case["d"])}
    if kind == "ot_plan":
        return {"bytes": n * m * (2 * size + 2 * 8) + 2 * 8 * (n + m), "flops": 2.0 * n * m * 400}
    plan = 8 * n * m if kind == "call" else 0
    return {"bytes": size * n * m + plan + 2 * 8 * (n + m),
            "flops": 2.0 * n * m * _REDUCTIONS[case["solver"]]}


# -------------------------------------------------------------- in 64 bits --

def _plan(M, alpha, beta, reg):
    return torch.exp((alpha[:, None] + beta[None, :] - M) / reg)


def _lse_beta(M, alpha, b, reg):
    return reg * (torch.log(b) - torch.logsumexp((alpha[:, None] - M) / reg, 0))


def _objective(M, a, b, alpha, beta, reg, r):
    return float(reg * r.sum() - (a * alpha).sum() - (b * beta).sum())


def _bcd(M, a, b, reg, tol, max_iter):
    """Block coordinate descent in the log domain; stops on the norm of the
    dual gradient at the start of a sweep."""
    alpha = torch.zeros_like(a)
    beta = _lse_beta(M, alpha, b, reg)
    for k in range(max_iter + 1):
        lse = torch.logsumexp((beta[None, :] - M) / reg, 1)
        r = torch.exp(lse + alpha / reg)
        if float(torch.linalg.norm(r - a)) < tol or k == max_iter:
            break
        alpha = reg * (torch.log(a) - lse)
        beta = _lse_beta(M, alpha, b, reg)
    obj = _objective(M, a, b, alpha, beta, reg, r)
    return alpha + beta[-1], beta - beta[-1], obj


def _hessian(T, reg):
    n, m = T.shape
    H = torch.zeros((n + m - 1, n + m - 1), dtype=T.dtype, device=T.device)
    H[:n, n:] = T[:, :-1]
    H[n:, :n] = T[:, :-1].T
    H.diagonal()[:n] = T.sum(1)
    H.diagonal()[n:] = T.sum(0)[:-1]
    return H / reg


def _newton(M, a, b, reg, tol, max_iter):
    """Newton's method with a dense factorisation and the Armijo rule."""
    n, m = M.shape
    beta = _lse_beta(M, torch.zeros_like(a), b, reg)
    alpha, beta = torch.zeros_like(a) + beta[-1], beta - beta[-1]
    for _ in range(max_iter):
        T = _plan(M, alpha, beta, reg)
        r = T.sum(1)
        obj = _objective(M, a, b, alpha, beta, reg, r)
        g = torch.cat([r - a, (T.sum(0) - b)[:-1]])
        if float(torch.linalg.norm(g)) < tol:
            break
        L = torch.linalg.cholesky(_hessian(T, reg))
        d = -torch.cholesky_solve(g[:, None], L)[:, 0]
        da, db = d[:n], torch.cat([d[n:], d.new_zeros(1)])
        slope, step = float(g @ d), 1.0
        for _ in range(20):
            w = step * (da[:, None] + db[None, :]) / reg
            # e^w - 1 - w without cancellation
            phi = torch.where(w.abs() < 1e-3, w * w * (0.5 + w * (1 / 6 + w / 24)),
                              torch.expm1(w) - w)
            if step * slope + reg * float((T * phi).sum()) <= 0.5 * step * slope:
                break
            step *= 0.5
        alpha, beta = alpha + step * da, beta + step * db
    return alpha, beta, obj


def _exact_batched(case, seed):
    xs, ys, as_, bs, scale = _batch(case, seed)
    out = {"duals": [], "costs": [], "grad_x": [], "grad_y": []}
    for x, y, a, b, s in zip(xs, ys, as_, bs, scale):
        x, y, a, b = (torch.from_numpy(v).cuda().double() for v in (x, y, a, b))
        M = s * _distances(x, y)
        alpha, beta, obj = _bcd(M, a, b, case["reg"], case["tol"], case["max_iter"])
        T = _plan(M, alpha, beta, case["reg"])
        out["duals"].append(torch.cat([alpha, beta[:-1]]))
        out["costs"].append(torch.tensor([-obj], dtype=torch.float64, device="cuda"))
        out["grad_x"].append((2 * s * (T.sum(1)[:, None] * x - T @ y)).ravel())
        out["grad_y"].append((2 * s * (T.sum(0)[:, None] * y - T.T @ x)).ravel())
    return {k: torch.cat(v) for k, v in out.items()}


def exact(case, seed):
    kind, reg, tol = case["kind"], case["reg"], case["tol"]
    if kind == "batched":
        # a problem takes up to some hundreds of sweeps of a dozen launches
        return _exact_batched(case, seed) if case["count"] <= 64 else None
    if kind == "ot_cost":
        x, y, a, b = (t.double() for t in _clouds(case, seed))
        M = _distances(x, y) / case["d"]
        alpha, beta, obj = _newton(M, a, b, reg, tol, 100)
        T = _plan(M, alpha, beta, reg)
        return {"loss": torch.tensor(-obj, dtype=torch.float64, device="cuda"),
                "x": 2 * (T.sum(1)[:, None] * x - T @ y) / case["d"],
                "y": 2 * (T.sum(0)[:, None] * y - T.T @ x) / case["d"],
                "a": alpha - alpha.mean(), "b": beta - beta.mean()}
    if kind == "ot_plan":
        M, a, b = _problem(case, seed)
        W = _weights(case, seed)
        n = case["n"]
        alpha, beta, _ = _newton(M, a, b, reg, tol, 100)
        T = _plan(M, alpha, beta, reg)
        WT = W * T / reg
        v = torch.cat([WT.sum(1), WT.sum(0)[:-1]])
        u = torch.linalg.solve(_hessian(T, reg), v)
        ua, ub = u[:n], torch.cat([u[n:], u.new_zeros(1)])
        return {"plan": T, "M": T / reg * (ua[:, None] + ub[None, :] - W), "a": ua, "b": ub}
    if case["solver"] not in ("sinkhorn_bcd", "sinkhorn_newton"):
        return None  # the iterate at which these stop depends on the path taken
    M, a, b = _problem(case, seed)
    solve = _bcd if case["solver"] == "sinkhorn_bcd" else _newton
    alpha, beta, obj = solve(M.double(), a, b, reg, tol, case["max_iter"])
    out = {"dual": torch.cat([alpha, beta[:-1]]), "objective": obj}
    if kind == "call":
        out["plan"] = _plan(M.double(), alpha, beta, reg)
    return out
