"""Models far from one in size.  With the state's unit taken as 2^k (initial
mean and factor, Q_L, c and the observation noise times 2^k) the smoothed means
and factors are those of the model itself times 2^k, through every kernel: the
thread-per-chunk and team levels, the sequential block, the dense panels.  The
squared row norms then lie around 2^2k, at the ends of the type's range, where
the reflectors must stay as accurate as near one.  Bounds: 1e-9 and, in
float32, 2e-3 of the largest entry, what two orders of the same sums may differ
by after n steps of the random models below."""

import numpy as np
import pytest
import torch

from pof import parallel_filtsmooth as pfs, sequential_filtsmooth as sfs
from pof.observations import AffineModel
from pof.transitions import IWP, TransitionModel, preconditioned_discretize
from pof.utils import MVNSqrt

pytestmark = pytest.mark.gpu


def T(x, dtype):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=dtype, device="cuda")


def _model(D, d, n, dtype, noise, k):
    """k: the exponent of the state's unit."""
    rng = np.random.default_rng(D + n)
    u = 2.0**k
    if D < 32:
        F, QL = preconditioned_discretize(IWP(num_derivatives=D // d - 1, wiener_process_dimension=d), device="cpu")
        F, QL = F.numpy(), QL.numpy()
    else:
        F = np.eye(D) + (0.1 / np.sqrt(D)) * rng.standard_normal((D, D))
        QL = np.tril((0.3 / np.sqrt(D)) * rng.standard_normal((D, D))) + 0.25 * np.eye(D)
    H = rng.standard_normal((n, d, D)) / np.sqrt(D)
    c = rng.standard_normal((n, d)) * u
    R = 0.3 * np.tile(np.eye(d), (n, 1, 1)) * u if noise else None
    x0 = MVNSqrt(T(rng.standard_normal(D) * u, dtype), T(0.5 * np.eye(D) * u, dtype))
    return x0, TransitionModel(T(F, dtype), T(QL * u, dtype)), AffineModel(T(H, dtype), T(c, dtype),
                                                                         None if R is None else T(R, dtype))


def _check(run, args, ks, dtype):
    tol = 1e-9 if dtype == torch.float64 else 2e-3
    cov = lambda L: L @ L.mT  # noqa: E731
    ref = run(*_model(*args, 0))[0]
    for k in ks:
        out = run(*_model(*args, k))[0]
        assert torch.isfinite(out.mean).all() and torch.isfinite(out.chol).all(), k
        m, L = out.mean * 2.0**-k, out.chol * 2.0**-k
        assert float((m - ref.mean).abs().max() / ref.mean.abs().max()) <= tol, k
        assert float((cov(L) - cov(ref.chol)).abs().max() / cov(ref.chol).abs().max()) <= tol, k


KS = {torch.float64: (-300, -490, -505, 470, 500), torch.float32: (-40, -58, 50)}


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("D,d,n,noise", [(2, 1, 40, False), (4, 1, 33, True), (6, 2, 25, False), (8, 2, 21, True),
                                         (12, 3, 9, False)])
def test_passes_far_from_one(D, d, n, noise, dtype):
    """(The parallel pass also carries the information's factor, in units of 2^-k
    and growing along the grid: its squares overflow a little before k = -512,
    where the state's still hold.)"""
    _check(pfs.linear_filtsmooth, (D, d, n, dtype, noise), KS[dtype], dtype)
    ks = KS[dtype] + ((-512, -514, 505) if dtype == torch.float64 else ())
    _check(sfs.linear_filtsmooth, (D, d, n, dtype, noise), ks, dtype)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("D,d,n,noise", [(40, 4, 9, True), (150, 10, 5, False)])
def test_dense_passes_far_from_one(D, d, n, noise, dtype):
    _check(pfs.linear_filtsmooth, (D, d, n, dtype, noise), KS[dtype], dtype)


@pytest.mark.parametrize("D,cluster", [(40, "1"), (1300, "0"), (1300, "1")])
def test_dense_float32_pivots_whose_square_overflows(D, cluster, monkeypatch):
    """The filter from an initial factor of 1e20 I with Q_L of order one: alpha^2 is
    beyond float32, the norm is not.  D = 1300: beyond the register panels (2600
    columns), one CTA or a cluster per matrix.  Bound: the float64 filter to 1e-3
    of each array's largest entry."""
    monkeypatch.setenv("POF_DENSE_CLUSTER", cluster)
    n = 2
    H = np.zeros((n, 1, D))
    H[:, 0, 0] = 1.0
    m0 = np.linspace(-1.0, 1.0, D)

    def run(dtype):
        out = pfs.linear_noiseless_filtering(MVNSqrt(T(m0, dtype), T(1e20 * np.eye(D), dtype)),
                                             TransitionModel(T(np.eye(D), dtype), T(0.25 * np.eye(D), dtype)),
                                             AffineModel(T(H, dtype), T(np.full((n, 1), -2.0), dtype), None))[0]
        return out.mean.double(), out.chol.double() @ out.chol.double().mT

    m, C = run(torch.float32)
    m64, C64 = run(torch.float64)
    assert torch.isfinite(m).all() and torch.isfinite(C).all()
    assert float((m - m64).abs().max()) <= 1e-3 * float(m64.abs().max())
    assert float((C - C64).abs().max()) <= 1e-3 * float(C64.max())
