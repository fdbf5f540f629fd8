"""Solver set-up (pof/convenience.py)."""

import numpy as np
import torch

from . import initialization as init
from .observations import NonlinearModel, linearize
from .transitions import (
    IWP,
    TransitionModel,
    _nordsieck_1d_np,
    _preconditioned_1d_np,
    get_transition_model,
    projection_matrix,
)
from .utils import MVNSqrt, default_device, gmul_stack


def linearize_observation_model(observation_model, trajectory):
    """vmap(linearize) over a trajectory (pof/convenience.py:9-10)."""
    return linearize(observation_model, trajectory)


def _ts(ts):
    return torch.as_tensor(ts, dtype=torch.float64).to(default_device())


def _to_device(arrays, dev):
    """Small host matrices on the device with one copy, each 256-byte aligned."""
    sizes = [-(-a.size // 32) * 32 for a in arrays]
    flat = np.zeros(sum(sizes))
    at = np.concatenate([[0], np.cumsum(sizes)])
    for a, o in zip(arrays, at):
        flat[o:o + a.size] = a.reshape(-1)
    buf = torch.from_numpy(flat).to(dev)
    return [buf[o:o + a.size].view(a.shape) for a, o in zip(arrays, at)]


def set_up_solver(*, f, y0, ts, order):
    """pof/convenience.py:13-45: preconditioned IWP prior, Nordsieck P/PI,
    projections E0 P and E1 P, the residual model E1 x - f(E0 x) and the
    Taylor-mode x0 (times PI).  The N-1 identical transition models are
    exposed as a stride-0 expand of one (D, D) pair."""
    ts = torch.as_tensor(ts, dtype=torch.float64)
    dt = float(ts[1] - ts[0])  # uniform grid assumed, as in the reference (its check is commented out)
    dev = default_device()
    ts = ts.to(dev)
    y0 = torch.as_tensor(y0, dtype=torch.float64)
    d = y0.shape[0]
    n = ts.shape[0] - 1
    iwp = IWP(num_derivatives=order, wiener_process_dimension=d)
    x0 = init.taylor_mode_init(f, y0, order, device=torch.device("cpu"))
    # the set-up matrices are small: formed on the host, one copy to the device
    A1, QL1 = _preconditioned_1d_np(order)
    P1, PI1 = _nordsieck_1d_np(order, dt)
    I = np.eye(d)
    A, QL, P, PI = (np.kron(I, x) for x in (A1, QL1, P1, PI1))
    E0, E1 = (np.kron(I, np.eye(1, order + 1, k)) @ P for k in (0, 1))
    A, QL, P, PI, E0, E1, m0, L0 = _to_device([A, QL, P, PI, E0, E1, PI @ x0.mean.numpy(), PI @ x0.chol.numpy()], dev)
    D = A.shape[0]
    dtm = TransitionModel(A.expand(n, D, D), QL.expand(n, D, D))

    def om_fn(x, f=f, E0=E0, E1=E1):
        return E1 @ x - f(None, E0 @ x)

    setup = {
        "f": f,
        "y0": y0,
        "ts": ts,
        "dt": dt,
        "dtm": dtm,
        "E0": E0,
        "E1": E1,
        "P": P,
        "PI": PI,
        "order": order,
        "iwp": iwp,
    }
    om = NonlinearModel(om_fn, field=getattr(f, "pof_field", None), setup=setup)
    setup["om"] = om
    setup["x0"] = MVNSqrt(m0, L0)
    return setup


def set_up_solver_no_precond(*, f, y0, ts, order):
    """pof/convenience.py:48-73: per-step non-preconditioned transitions."""
    ts = _ts(ts)
    y0 = torch.as_tensor(y0, dtype=torch.float64)
    d = y0.shape[0]
    iwp = IWP(num_derivatives=order, wiener_process_dimension=d)
    steps = (ts[1:] - ts[:-1]).cpu()
    Fs, QLs = zip(*[get_transition_model(iwp, float(h)) for h in steps])
    dtm = TransitionModel(torch.stack(Fs), torch.stack(QLs))
    E0, E1 = projection_matrix(iwp, 0), projection_matrix(iwp, 1)

    def om_fn(x):
        return E1 @ x - f(None, E0 @ x)

    x0 = init.taylor_mode_init(f, y0, order)
    D = x0.mean.shape[0]
    I = torch.eye(D, dtype=torch.float64, device=x0.mean.device)
    return {"ts": ts, "dtm": dtm, "om": NonlinearModel(om_fn), "x0": x0, "E0": E0, "P": I, "PI": I,
            "order": order, "iwp": iwp, "f": f, "y0": y0}


def get_initial_trajectory(setup, method="prior"):
    """pof/convenience.py:76-92 ("prior" keeps the reference's behaviour: no PI)."""
    f, y0, order = setup["f"], setup["y0"], setup["order"]
    ts = setup["ts"]
    PI = setup["PI"]
    if method == "coarse":
        states = init.coarse_ekf_init(y0=y0, order=order, ts=ts, f=f, N=100)
        return gmul_stack(PI, states)
    elif method == "constant":
        # one row, repeated (PI times a zero chol is zero)
        row = init.constant_init(y0=y0, order=order, ts=ts[:1], f=f, device=ts.device)
        N, D = ts.shape[0], row.mean.shape[1]
        return MVNSqrt((row.mean @ PI.T).repeat(N, 1), torch.zeros((N, D, D), dtype=torch.float64, device=ts.device))
    elif method == "prior":
        return init.prior_init(f=f, y0=y0, order=order, ts=ts)
    else:
        raise Exception(f"method={method} not found")
