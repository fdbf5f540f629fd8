"""The work a user of this framework gives it, as measurable cases.

A case names one public entry point, a problem and its sizes:

  solve       pof.solver.solve of a built-in field (host arrays in, the whole IEKS loop)
  pass        pof.parallel_filtsmooth.linear_filtsmooth: one filter + smoother pass
  nonuniform  linear_noiseless_filtering, then smoothing, with one transition model per step
  sequential  pof.solver.sequential_eks_solve: the sequential extended Kalman smoother
  batch       pof.batch.run_batch of a prepared batch of uneven problems
  dense       linear_filtsmooth at a large state dimension (reaction-diffusion system)

Square-root factors come back as covariances L L^T: a factor's column signs and, where a
noiseless observation makes it rank-deficient, the rotation of its null columns are rounding
noise.  So is sigma^2 for systems of two or more dimensions (it whitens with the observation
factor's transpose, which depends on those signs), so calibrated covariances come back per
unit sigma^2.  The log-likelihood of exact observations sums squared innovations that cancel
to rounding, so those come back rounded to float32, as do covariances of mixed-precision
solves, whose linearization point carries the float32 phase's rounding.  A dense float32 pass
returns its means, the part that the mixed-precision loop takes from it.
"""

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "parallel-in-time-ode-filters_gb300"))

from pof import batch as pbatch  # noqa: E402
from pof import ivp as pivp  # noqa: E402
from pof import parallel_filtsmooth, solver  # noqa: E402
from pof import _lib  # noqa: E402
from pof.observations import AffineModel  # noqa: E402
from pof.transitions import IWP, TransitionModel, discretize_transitions  # noqa: E402
from pof.utils import MVNSqrt  # noqa: E402


def listed():
    return [
        # an interactive solve: a scalar problem on a short grid; launches and host work count
        {"name": "solve_logistic_short", "kind": "solve", "field": "logistic", "q": 2, "n": 100, "precision": "float64"},
        # the everyday solve: a planar oscillator on a grid of about a thousand points
        {"name": "solve_vanderpol", "kind": "solve", "field": "vanderpol", "q": 3, "n": 1000, "precision": "float64"},
        # the same, float32 iterations with float64 polish, on a longer grid
        {"name": "solve_vanderpol_mixed", "kind": "solve", "field": "vanderpol", "q": 4, "n": 8191, "precision": "mixed"},
        # a three-dimensional system on a long, odd grid (D = 12)
        {"name": "solve_rigid_body", "kind": "solve", "field": "rigid_body", "q": 3, "n": 12001, "precision": "float64"},
        # the scan-length sweep's long end: a scalar problem, a quarter of a million points
        {"name": "solve_logistic_long", "kind": "solve", "field": "logistic", "q": 3, "n": 262143, "precision": "float64"},
        # one pass at the headline benchmark's size (FitzHugh-Nagumo, q = 3, N = 2^16)
        {"name": "pass_fhn", "kind": "pass", "field": "fhn_classic", "q": 3, "n": 65535, "dtype": "float64"},
        # one float32 pass, as a caller's own mixed-precision loop runs it
        {"name": "pass_f32", "kind": "pass", "field": "fhn_classic", "q": 2, "n": 2000, "dtype": "float32"},
        # a grid with its own step sizes and observation noise, filter and smoother called one by one
        {"name": "nonuniform_noisy", "kind": "nonuniform", "field": "lotkavolterra", "q": 2, "n": 3001},
        # the sequential baseline (and the coarse initialization) of every parallel solve
        {"name": "sequential_eks", "kind": "sequential", "field": "vanderpol", "q": 2, "n": 400},
        # many uneven problems in one call
        {"name": "batch_vanderpol", "kind": "batch", "field": "vanderpol", "q": 3, "b": 192, "lo": 128, "hi": 4096,
         "precision": "float64"},
        # a dense state dimension in float64
        {"name": "dense_f64", "kind": "dense", "cells": 16, "q": 3, "n": 150, "dtype": "float64"},
        # the reaction-diffusion system of 64 cells in float32 (D = 384, d = 128)
        {"name": "dense_f32", "kind": "dense", "cells": 64, "q": 2, "n": 256, "dtype": "float32"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "pass", "pass", "nonuniform", "sequential", "batch", "dense", "dense"])
    if kind == "solve":
        field = rng.choice(["logistic", "vanderpol", "rigid_body"])
        mixed = rng.random() < 0.3 and field == "vanderpol"
        q = rng.choice([3, 4] if mixed else {"logistic": [1, 2, 3], "vanderpol": [2, 3, 4], "rigid_body": [2, 3]}[field])
        return {"kind": kind, "field": field, "q": q, "precision": "mixed" if mixed else "float64",
                "n": _log_int(rng, 1000 if mixed else 100, {"logistic": 200000, "vanderpol": 16000, "rigid_body": 12000}[field])}
    if kind == "pass":
        f32 = rng.random() < 0.3
        field = "fhn_classic" if f32 else rng.choice(["fhn_classic", "lotkavolterra", "vanderpol"])
        return {"kind": kind, "field": field, "q": rng.choice([1, 2] if f32 else [1, 2, 3]),
                "n": _log_int(rng, 300, 3000) if f32 else _log_int(rng, 4000 if field == "fhn_classic" else 200, 60000),
                "dtype": "float32" if f32 else "float64"}
    if kind == "nonuniform":
        return {"kind": kind, "field": rng.choice(["lotkavolterra", "vanderpol"]), "q": rng.choice([1, 2]),
                "n": _log_int(rng, 100, 5000)}
    if kind == "sequential":
        return {"kind": kind, "field": rng.choice(["logistic", "vanderpol", "rigid_body"]), "q": rng.choice([1, 2]),
                "n": _log_int(rng, 50, 450)}
    if kind == "batch":
        hi = _log_int(rng, 512, 4096)
        mixed = rng.random() < 0.5
        return {"kind": kind, "field": "vanderpol", "q": 3 if mixed else rng.choice([2, 3]), "b": rng.randint(20, 190),
                "lo": rng.randint(64, 256), "hi": hi, "precision": "mixed" if mixed else "float64"}
    f32 = rng.random() < 0.5
    return {"kind": kind, "cells": rng.randint(6, 48 if f32 else 16), "q": 2 if f32 else rng.choice([2, 3]),
            "n": _log_int(rng, 20, 200), "dtype": "float32" if f32 else "float64"}


# ---------------------------------------------------------------------------
# the problems, in numpy (for inputs and for the 64-bit reference)
# ---------------------------------------------------------------------------
_SPAN = {"logistic": 10.0, "vanderpol": 6.3, "rigid_body": 20.0, "lotkavolterra": 7.0, "fhn_classic": 100.0}


def _problem(field, rng):
    """(parameters, y0) near the field's usual ones."""
    j = lambda v, s=0.05: tuple(float(x) * (1.0 + s * rng.uniform(-1, 1)) for x in v)  # noqa: E731
    if field == "logistic":
        return j((1.0,)), j((0.01,))
    if field == "vanderpol":
        return j((1.0,)), (2.0 + 0.05 * rng.uniform(-1, 1), 0.05 * rng.uniform(-1, 1))
    if field == "rigid_body":
        return j((-2.0, 1.25, -0.5), 0.02), j((1.0,)) + (0.0,) + j((0.9,))
    if field == "lotkavolterra":
        return j((1.5, 1.0, 3.0, 1.0)), j((1.0, 1.0))
    return j((0.2, 0.2, 3.0)), j((-1.0, 1.0))


def _rhs(field, p, y, mul, one):
    """f(y) for the components y, with the product `mul` and the constant `one` (numbers, arrays or Taylor series)."""
    if field == "logistic":
        return [p[0] * (y[0] - mul(y[0], y[0]))]
    if field == "vanderpol":
        return [y[1], p[0] * (y[1] - mul(mul(y[0], y[0]), y[1]) - y[0])]
    if field == "rigid_body":
        return [p[0] * mul(y[1], y[2]), p[1] * mul(y[0], y[2]), p[2] * mul(y[0], y[1])]
    if field == "lotkavolterra":
        return [p[0] * y[0] - p[1] * mul(y[0], y[1]), p[3] * mul(y[0], y[1]) - p[2] * y[1]]
    cube = mul(mul(y[0], y[0]), y[0])
    return [p[2] * (y[0] - cube / 3.0 + y[1]), (p[0] * one - y[0] - p[1] * y[1]) / p[2]]


def _jac(field, p, y):
    """Jacobians (n, d, d) at the states y (n, d)."""
    y = np.asarray(y)
    J = np.zeros(y.shape + (y.shape[1],))
    if field == "logistic":
        J[:, 0, 0] = p[0] * (1 - 2 * y[:, 0])
    elif field == "vanderpol":
        J[:, 0, 1] = 1.0
        J[:, 1, 0] = p[0] * (-2 * y[:, 0] * y[:, 1] - 1)
        J[:, 1, 1] = p[0] * (1 - y[:, 0] ** 2)
    elif field == "rigid_body":
        J[:, 0, 1], J[:, 0, 2] = p[0] * y[:, 2], p[0] * y[:, 1]
        J[:, 1, 0], J[:, 1, 2] = p[1] * y[:, 2], p[1] * y[:, 0]
        J[:, 2, 0], J[:, 2, 1] = p[2] * y[:, 1], p[2] * y[:, 0]
    elif field == "lotkavolterra":
        J[:, 0, 0], J[:, 0, 1] = p[0] - p[1] * y[:, 1], -p[1] * y[:, 0]
        J[:, 1, 0], J[:, 1, 1] = p[3] * y[:, 1], p[3] * y[:, 0] - p[2]
    else:
        J[:, 0, 0], J[:, 0, 1] = p[2] * (1 - y[:, 0] ** 2), p[2]
        J[:, 1, 0], J[:, 1, 1] = -1.0 / p[2], -p[1] / p[2]
    return J


def _f(field, p, y):
    return np.stack(_rhs(field, p, [y[:, i] for i in range(y.shape[1])], np.multiply, np.ones(len(y))), 1)


def _taylor(field, p, y0, q):
    """(d, q + 1) derivatives of the solution at the initial time, by its power series."""
    K = q + 1
    d = len(y0)
    c = np.zeros((d, K))
    c[:, 0] = y0
    one = np.zeros(K)
    one[0] = 1.0
    for k in range(q):
        f = _rhs(field, p, list(c), lambda a, b: np.convolve(a, b)[:K], one)
        for i in range(d):
            c[i, k + 1] = f[i][k] / (k + 1)
    return c * np.array([math.factorial(k) for k in range(K)])


def _trajectory(field, p, y0, span, n):
    """(n + 1, d) states on a uniform grid: classical Runge-Kutta on a coarse grid, interpolated."""
    m = 4000
    h = span / m
    f = lambda y: np.array(_rhs(field, p, y, lambda a, b: a * b, 1.0))  # noqa: E731
    ys = [np.array(y0, dtype=float)]
    for _ in range(m):
        y = ys[-1]
        k1 = f(y)
        k2 = f(y + 0.5 * h * k1)
        k3 = f(y + 0.5 * h * k2)
        k4 = f(y + h * k3)
        ys.append(y + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4))
    ys = np.array(ys)
    t, tt = np.linspace(0, span, m + 1), np.linspace(0, span, n + 1)
    return np.stack([np.interp(tt, t, ys[:, i]) for i in range(ys.shape[1])], 1)


def _nordsieck(q, h):
    pw = np.arange(q, -1, -1)
    return abs(h) ** (pw + 0.5) / np.array([math.factorial(k) for k in pw])


def _prior(d, q):
    A = np.array([[math.comb(q - i, q - j) if j >= i else 0 for j in range(q + 1)] for i in range(q + 1)], dtype=float)
    Q = np.array([[1.0 / (2 * q + 1 - i - j) for j in range(q + 1)] for i in range(q + 1)])
    return np.kron(np.eye(d), A), np.kron(np.eye(d), np.linalg.cholesky(Q))


def _linear_model(field, p, y, q, scale):
    """EK1 model (H, c) of y' = f(y) at the states y (n, d): H = E1 - J E0 in coordinates scaled by `scale` (q + 1)."""
    n, d = y.shape
    J = _jac(field, p, y)
    H = np.zeros((n, d, d, q + 1))
    H[:, :, :, 0] = -J * scale[0]
    for i in range(d):
        H[:, i, i, 1] += scale[1]
    c = np.einsum("nij,nj->ni", J, y) - _f(field, p, y)
    return H.reshape(n, d, d * (q + 1)), c


# ---------------------------------------------------------------------------
# preparation
# ---------------------------------------------------------------------------
def _dev(x, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=dtype, device="cuda")


def _pass_inputs(case, seed):
    """(m0, L0, F, QL, H, c) in numpy: a linear model along a solution, noiseless, preconditioned."""
    rng = np.random.default_rng(seed)
    field, q, n = case["field"], case["q"], case["n"]
    p, y0 = _problem(field, rng)
    d = len(y0)
    span = _SPAN[field]
    ps = _nordsieck(q, span / n)
    y = _trajectory(field, p, y0, span, n)
    F, QL = _prior(d, q)
    H, c = _linear_model(field, p, y[1:], q, ps)
    m0 = (_taylor(field, p, y0, q) / ps).reshape(-1)
    L0 = np.zeros((len(m0), len(m0)))
    if case["dtype"] == "float32":  # rows of a noiseless model scale freely: unit norm, as the mixed solver gives them
        s = np.linalg.norm(H, axis=-1)
        H, c = H / s[..., None], c / s
        return [x.astype(np.float32) for x in (m0, L0, F, QL, H, c)]
    return [m0, L0, F, QL, H, c]


def _nonuniform_inputs(case, seed):
    """(m0, L0, steps, H, c, R): plain coordinates, steps of their own size, noisy observations."""
    rng = np.random.default_rng(seed)
    field, q, n = case["field"], case["q"], case["n"]
    p, y0 = _problem(field, rng)
    d = len(y0)
    span = _SPAN[field]
    steps = rng.uniform(0.5, 1.5, n)
    steps *= span / steps.sum()
    fine = _trajectory(field, p, y0, span, 4000)
    t = np.cumsum(steps)
    y = np.stack([np.interp(t, np.linspace(0, span, 4001), fine[:, i]) for i in range(d)], 1)
    H, c = _linear_model(field, p, y, q, np.ones(q + 1))
    R = 1e-3 * np.eye(d) * rng.uniform(0.5, 1.5, (n, 1, 1))
    m0 = _taylor(field, p, y0, q).reshape(-1)
    return m0, 1e-3 * np.eye(len(m0)), steps, H, c, R


def _dense_inputs(case, seed):
    """(m0, L0, F, QL, H, c) of the reaction-diffusion FitzHugh-Nagumo system along a solution."""
    rng = np.random.default_rng(seed)
    m, q, n = case["cells"], case["q"], case["n"]
    d = 2 * m
    a, b, cc, kv, kw = 0.2, 0.2, 3.0, 0.5, 0.05
    h = 0.02  # about the step of the system's usual grids
    ps = _nordsieck(q, h)
    lap = np.roll(np.eye(m), 1, 0) + np.roll(np.eye(m), -1, 0) - 2 * np.eye(m)

    def rhs(y):
        v, w = y[..., :m], y[..., m:]
        return np.concatenate([cc * (v - v**3 / 3 + w) + kv * v @ lap, -(v - a + b * w) / cc + kw * w @ lap], -1)

    x = 2 * np.pi * np.arange(m) / m + rng.uniform(0, 2 * np.pi)
    k, fine = 4, []  # classical Runge-Kutta, four steps per grid step
    y, dt = np.concatenate([-1 + 0.5 * np.sin(x), np.ones(m)]) + 0.02 * rng.standard_normal(d), h / k
    for i in range(n * k + 1):
        if i % k == 0:
            fine.append(y)
        k1 = rhs(y)
        k2 = rhs(y + 0.5 * dt * k1)
        k3 = rhs(y + 0.5 * dt * k2)
        y = y + dt / 6 * (k1 + 2 * k2 + 2 * k3 + rhs(y + dt * k3))
    y = np.array(fine)
    f, v = rhs(y), y[:, :m]
    J = np.zeros((n, d, d))
    J[:, :m, :m] = kv * lap
    J[:, np.arange(m), np.arange(m)] += cc * (1 - v[1:] ** 2)
    J[:, :m, m:] = cc * np.eye(m)
    J[:, m:, :m] = -np.eye(m) / cc
    J[:, m:, m:] = kw * lap - b / cc * np.eye(m)
    H = np.zeros((n, d, d, q + 1))
    H[:, :, :, 0] = -J * ps[0]
    H[:, np.arange(d), np.arange(d), 1] += ps[1]
    H = H.reshape(n, d, d * (q + 1))
    c = np.einsum("nij,nj->ni", J, y[1:]) - f[1:]
    m0 = np.zeros((d, q + 1))
    m0[:, 0], m0[:, 1] = y[0], f[0]
    m0 = (m0 / ps).reshape(-1)
    F, QL = _prior(d, q)
    s = np.linalg.norm(H, axis=-1)
    H, c = H / s[..., None], c / s
    out = [m0, np.zeros((len(m0), len(m0))), F, QL, H, c]
    return [x.astype(np.float32) for x in out] if case["dtype"] == "float32" else out


def _make_ivp(field, p, y0):
    y0 = list(y0)
    if field == "logistic":
        return pivp.logistic(y0=y0, r=p[0])
    if field == "vanderpol":
        return pivp.vanderpol(y0=y0, stiffness_constant=p[0])
    return pivp.rigid_body(y0=y0, p=p)


def _batch_problems(case, seed):
    rng, sizes = np.random.default_rng(seed), np.random.default_rng(case["b"])  # the grid sizes belong to the case
    out = []
    for _ in range(case["b"]):
        p, y0 = _problem(case["field"], rng)
        n = int(round(math.exp(sizes.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        out.append((case["field"], p, list(y0), np.linspace(0.0, _SPAN[case["field"]], n)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("solve", "sequential"):
        p, y0 = _problem(case["field"], np.random.default_rng(seed))
        return {"case": case, "ivp": _make_ivp(case["field"], p, y0),
                "ts": np.linspace(0.0, _SPAN[case["field"]], case["n"] + 1)}
    if kind == "pass":
        dt = getattr(torch, case["dtype"])
        m0, L0, F, QL, H, c = (_dev(x, dt) for x in _pass_inputs(case, seed))
        n, d = c.shape
        R = torch.zeros((n, d, d), dtype=dt, device="cuda")  # as linearize gives it
        return {"case": case, "x0": MVNSqrt(m0, L0), "dtm": TransitionModel(F.expand(n, *F.shape), QL.expand(n, *F.shape)),
                "dom": AffineModel(H, c, R)}
    if kind == "nonuniform":
        m0, L0, steps, H, c, R = _nonuniform_inputs(case, seed)
        iwp = IWP(num_derivatives=case["q"], wiener_process_dimension=c.shape[1])
        return {"case": case, "x0": MVNSqrt(_dev(m0), _dev(L0)), "dtm": discretize_transitions(iwp, steps=steps),
                "dom": AffineModel(_dev(H), _dev(c), _dev(R))}
    if kind == "batch":
        prep = pbatch.prepare_batch(_batch_problems(case, seed), case["q"])
        G, D = prep["means0"].shape
        return {"case": case, "prep": prep, "chols": torch.empty((G, D, D), dtype=torch.float64, device="cuda"),
                "info": torch.zeros((prep["B"], _lib.I_COUNT), dtype=torch.float64, device="cuda"),
                "info32": torch.zeros((prep["B"], 2), dtype=torch.float64, device="cuda"), "ws": None}
    dt = getattr(torch, case["dtype"])
    m0, L0, F, QL, H, c = (_dev(x, dt) for x in _dense_inputs(case, seed))
    return {"case": case, "x0": MVNSqrt(m0, L0), "dtm": TransitionModel(F, QL), "dom": (H, c, None)}


def _cov(L):
    return L @ L.transpose(-1, -2)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve":
        ys, info = solver.solve(f=state["ivp"].f, y0=state["ivp"].y0, ts=state["ts"], order=case["q"], init="constant",
                                maxiters=1000, precision=case["precision"])
        s = info["sigma_squared"]
        if case["precision"] == "mixed":
            return {"mean": ys.mean, "cov": _cov(ys.chol / s).float()}
        return {"mean": ys.mean, "cov": _cov(ys.chol / s), "nll": info["nll"].float(), "iterations": info["iterations"]}
    if kind == "sequential":
        ys, info = solver.sequential_eks_solve(f=state["ivp"].f, y0=state["ivp"].y0, ts=state["ts"], order=case["q"])
        return {"mean": ys.mean, "cov": _cov(ys.chol) / info["sigma_squared"], "nll": info["nll"]}
    if kind == "nonuniform":
        filt, nll, obj, _ = parallel_filtsmooth.linear_noiseless_filtering(state["x0"], state["dtm"], state["dom"])
        smo, sobj = parallel_filtsmooth.smoothing(state["dtm"], filt)
        return {"filt_mean": filt.mean, "filt_cov": _cov(filt.chol), "mean": smo.mean, "cov": _cov(smo.chol), "nll": nll}
    if kind == "batch":
        prep = state["prep"]
        means = prep["means0"].clone()
        state["ws"] = pbatch.run_batch(prep, means, state["chols"], state["info"], maxiters=1000, calibrate=False,
                                       workspace=state["ws"], precision=case["precision"], info_f32=state["info32"])
        ym, yc = pbatch.project(prep, means, state["chols"])
        if case["precision"] == "mixed":
            return {"mean": ym, "cov": _cov(yc).float()}
        return {"mean": ym, "cov": _cov(yc), "nll": state["info"][:, _lib.I_NLL].float(),
                "iterations": state["info"][:, _lib.I_ITERATIONS].to(torch.int64)}
    out, nll, obj, ssq = parallel_filtsmooth.linear_filtsmooth(state["x0"], state["dtm"], state["dom"])
    if case["dtype"] == "float32":
        return {"mean": out.mean} if kind == "dense" else {"mean": out.mean, "cov": _cov(out.chol)}
    return {"mean": out.mean, "cov": _cov(out.chol), "nll": nll.float()}


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------
def _step_flops(D, d):
    """One step of the square-root Kalman filter and Rauch-Tung-Striebel smoother: the predict's factorization with
    the smoother gain's rows below it, the update's, the gain, the smoothed factor, and F L, E L."""
    lq = lambda m, w, below: sum(4 * w * (m - 1 - j + below) + 3 * w for j in range(m))  # noqa: E731
    return lq(D, D + 1, D) + lq(d, D, D) + lq(D, D / 2, 0) + D**3 + lq(D, D + 1, 0) + 2 * D**3 + 2 * d * D * D


def work(case):
    kind, q = case["kind"], case["q"]
    es = 4 if case.get("dtype") == "float32" else 8
    if kind == "dense":
        d = 2 * case["cells"]
    else:
        d = {"logistic": 1, "rigid_body": 3}.get(case["field"], 2)
    D = d * (q + 1)
    if kind == "batch":
        lo, hi = case["lo"], case["hi"]
        n = case["b"] * (hi - lo) / max(math.log(hi / lo), 1e-9)
    else:
        n = case["n"]
    its = {"solve": 10, "batch": 10}.get(kind, 1)
    flops = n * _step_flops(D, d) * its
    out_bytes = n * es * ((d + d * d) if kind in ("solve", "sequential", "batch") else (D + D * D))
    in_bytes = n * 8 if kind in ("solve", "sequential") else n * es * D if kind == "batch" else n * es * (d * D + d)
    if kind == "nonuniform":
        in_bytes += n * es * (2 * D * D + d * d)
        out_bytes *= 2
    return {"bytes": in_bytes + out_bytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same in plain 64-bit numpy, step after step
# ---------------------------------------------------------------------------
def _lower(X):
    return np.linalg.qr(X.T, mode="r").T


def _filter(m, L, model, n):
    """Square-root Kalman filter; model(k, predicted mean) gives (F, QL, H, c, R or None).  (means, factors, nll)."""
    ms, Ls, nll = [m], [L], 0.0
    for k in range(n):
        F, QL, (H, c, R) = model(k, m)
        mp = F @ m
        Lp = _lower(np.concatenate([F @ L, QL], 1))
        d = len(c)
        top = H @ Lp if R is None else np.concatenate([H @ Lp, R], 1)
        low = Lp if R is None else np.concatenate([Lp, np.zeros((len(m), d))], 1)
        X = np.concatenate([top, low])
        if X.shape[0] > X.shape[1]:
            X = np.concatenate([X, np.zeros((X.shape[0], X.shape[0] - X.shape[1]))], 1)
        T = _lower(X)
        S, K, L = T[:d, :d], T[d:, :d], T[d:, d:]
        w = np.linalg.solve(S, H @ mp + c)
        nll += 0.5 * w @ w + np.log(np.abs(np.diag(S))).sum() + 0.5 * d * math.log(2 * math.pi)
        m = mp - K @ w
        ms.append(m)
        Ls.append(L)
    return np.array(ms), np.array(Ls), nll


def _smoother(ms, Ls, trans):
    n = len(ms) - 1
    m, L = ms[n], Ls[n]
    om, oL = [m], [L]
    D = len(m)
    for k in range(n - 1, -1, -1):
        F, QL = trans(k)
        X = np.concatenate([np.concatenate([F @ Ls[k], QL], 1), np.concatenate([Ls[k], np.zeros((D, D))], 1)])
        T = _lower(X)
        E = np.linalg.solve(T[:D, :D].T, T[D:, :D].T).T
        m = ms[k] + E @ (m - F @ ms[k])
        L = _lower(np.concatenate([E @ L, T[D:, D:]], 1))
        om.append(m)
        oL.append(L)
    return np.array(om[::-1]), np.array(oL[::-1])


def _t(x):
    return torch.from_numpy(np.ascontiguousarray(x))


def _covs(L):
    return _t(L @ np.swapaxes(L, -1, -2))


def exact(case, seed):
    kind, q = case["kind"], case["q"]
    n = case.get("n", 0)
    # about 0.2 ms a step, filter and smoother, at small state dimensions
    if kind == "batch" or (kind == "solve" and n > 1500) or n > 45000:
        return None
    if kind == "dense":
        D = 2 * case["cells"] * (q + 1)
        if n * (D / 640.0) ** 3 > 30:
            return None
    if kind in ("pass", "dense"):
        m0, L0, F, QL, H, c = (x.astype(np.float64) for x in (_pass_inputs if kind == "pass" else _dense_inputs)(case, seed))
        ms, Ls, nll = _filter(m0, L0, lambda k, m: (F, QL, (H[k], c[k], None)), n)
        sm, sL = _smoother(ms, Ls, lambda k: (F, QL))
        out = {"mean": _t(sm), "cov": _covs(sL), "nll": _t(np.float64(nll))}
        if case["dtype"] == "float32":
            return {k: out[k] for k in (("mean",) if kind == "dense" else ("mean", "cov"))}
        return out
    if kind == "nonuniform":
        m0, L0, steps, H, c, R = _nonuniform_inputs(case, seed)
        d = c.shape[1]
        A, Q = _prior(d, q)

        def trans(k):
            P = np.tile(_nordsieck(q, steps[k]), d)
            return P[:, None] * A / P, P[:, None] * Q

        ms, Ls, nll = _filter(m0, L0, lambda k, m: trans(k) + ((H[k], c[k], R[k]),), n)
        sm, sL = _smoother(ms, Ls, trans)
        return {"filt_mean": _t(ms), "filt_cov": _covs(Ls), "mean": _t(sm), "cov": _covs(sL),
                "nll": _t(np.float64(nll))}
    field = case["field"]
    p, y0 = _problem(field, np.random.default_rng(seed))
    d = len(y0)
    ts = np.linspace(0.0, _SPAN[field], n + 1)
    ps = _nordsieck(q, ts[1] - ts[0])
    F, QL = _prior(d, q)
    D = d * (q + 1)
    m0 = (_taylor(field, p, y0, q) / ps).reshape(-1)
    if kind == "sequential":
        def model(k, m):
            H, c = _linear_model(field, p, (F @ m).reshape(d, q + 1)[:, 0][None] * ps[0], q, ps)
            return F, QL, (H[0], c[0], None)

        ms, Ls, nll = _filter(m0, np.zeros((D, D)), model, n)
        sm, sL = _smoother(ms, Ls, lambda k: (F, QL))
        nll = -nll
    else:
        row = np.zeros((d, q + 1))
        row[:, 0] = y0
        row[:, 1] = _f(field, p, np.array([y0]))[0]
        sm = np.tile((row / ps).reshape(-1), (n + 1, 1))
        obj_old, its = 0.0, 0
        Qi = np.linalg.inv(QL)
        while True:
            old = sm
            H, c = _linear_model(field, p, sm[1:, :: q + 1] * ps[0], q, ps)
            ms, Ls, nll = _filter(m0, np.zeros((D, D)), lambda k, m: (F, QL, (H[k], c[k], None)), n)
            sm, sL = _smoother(ms, Ls, lambda k: (F, QL))
            its += 1
            r = (sm[:-1] - sm[1:] @ F.T) @ Qi.T
            obj = (r * r).sum()
            close = np.abs(old - sm) <= 1e-8 + 1e-13 * np.abs(sm)
            if abs(obj_old - obj) <= 1e-9 + 1e-6 * abs(obj) or close.all() or its > 100:
                break
            obj_old = obj
    ym, yL = sm[:, :: q + 1] * ps[0], sL[:, :: q + 1, :] * ps[0]
    out = {"mean": _t(ym), "cov": _covs(yL)}
    if kind == "sequential" or case["precision"] == "float64":
        out["nll"] = _t(np.float64(nll))
    if kind == "solve" and case["precision"] == "float64":
        out["iterations"] = None
    return out
