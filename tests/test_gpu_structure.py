"""The zero structure that the level-0 kernels find in a model -- block-diagonal
F, triangular QL, the last column that H reaches, steps without noise, columns
of the state's factor that are zero -- against the NumPy float64 oracle, with
every combination present and absent, at the smallest step counts, across the
end of a chunk, and with square roots that are not triangular.  Means and
L L^T (normwise relative) within the parity tests' bound: 1e-10, or ten times
the spread between the oracle's own two orders (its associative scan and the
sequential filter and smoother), which is what the model's conditioning makes
of rounding (q = 5); sums over the structure only leave out exact zeros."""

import numpy as np
import pytest
import torch

from oracle import core, filtsmooth as ofs
from pof import parallel_filtsmooth as pfs, sequential_filtsmooth as sfs
from pof.observations import AffineModel
from pof.transitions import TransitionModel
from pof.utils import MVNSqrt

pytestmark = pytest.mark.gpu

TOL = 1e-10
SHAPES = [(2, 1), (4, 1), (4, 2), (5, 1), (6, 1), (6, 2), (6, 3), (8, 2), (8, 4), (9, 3), (10, 2), (12, 2), (12, 3)]


def T(x):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device="cuda")


def N_(x):
    return x.detach().cpu().numpy()


def rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


def cov(L):
    return L @ np.swapaxes(L, -1, -2)


def model(D, d, n, prior, noise, full_h, x0, seed):
    rng = np.random.default_rng(seed)
    q = D // d - 1
    if prior:
        F, QL = core.preconditioned_discretize(d, q)
    else:
        F = np.eye(D) + 0.1 * rng.standard_normal((D, D))
        QL = 0.5 * np.eye(D) + 0.1 * rng.standard_normal((D, D))  # not triangular
    H = rng.standard_normal((n, d, D))
    if not full_h:  # rows reach the first two columns of each block only
        keep = np.zeros(D, bool)
        keep[:: q + 1] = keep[1 :: q + 1] = True
        H[:, :, ~keep] = 0.0
    c = rng.standard_normal((n, d))
    R = {"none": np.zeros((n, d, d)), "zeros": np.zeros((n, d, d)),
         "some": 0.2 * np.tril(rng.standard_normal((n, d, d)) + 2 * np.eye(d)) * (np.arange(n) % 3 == 1)[:, None, None],
         "all": 0.2 * np.tril(rng.standard_normal((n, d, d)) + 2 * np.eye(d))}[noise]
    L0 = np.zeros((D, D)) if x0 == "point" else 0.3 * np.eye(D) + 0.1 * rng.standard_normal((D, D))
    return (rng.standard_normal(D), L0), (F, QL), (H, c, R)


@pytest.mark.parametrize("D,d", SHAPES)
@pytest.mark.parametrize("prior,noise,full_h,x0,n", [
    (True, "none", False, "point", 23), (True, "zeros", False, "full", 9), (True, "some", False, "point", 10),
    (True, "all", False, "full", 7), (True, "zeros", True, "point", 1), (True, "none", False, "full", 2),
    (False, "zeros", True, "full", 11), (False, "some", True, "point", 3), (False, "all", False, "full", 8),
])
def test_level0_structure(D, d, prior, noise, full_h, x0, n):
    st, (F, QL), dom = model(D, d, n, prior, noise, full_h, x0, 100 * D + d + n)
    rep = lambda A: np.broadcast_to(A, (n, D, D)).copy()  # noqa: E731
    dtm = (rep(F), rep(QL))
    (fm, fL), _, _, _ = ofs.linear_noiseless_filtering(st, dtm, dom)
    (om, oL), _, _, _ = ofs.linear_filtsmooth(st, dtm, dom)
    (sm_, sL), _, _, _ = ofs.sequential_linear_filtsmooth(st, dtm, dom)
    tol_m = max(TOL, 10 * rel(sm_, om))
    tol_c = max(TOL, 10 * rel(cov(sL), cov(oL)))
    x0 = MVNSqrt(T(st[0]), T(st[1]))
    gdom = AffineModel(T(dom[0]), T(dom[1]), None if noise == "none" else T(dom[2]))
    for gdtm in (TransitionModel(T(F), T(QL)), TransitionModel(T(dtm[0]), T(dtm[1]))):  # shared and per step
        filt, _, _, _ = pfs.linear_noiseless_filtering(x0, gdtm, gdom)
        assert rel(N_(filt.mean), fm) <= tol_m and rel(cov(N_(filt.chol)), cov(fL)) <= tol_c
        out, _, _, _ = pfs.linear_filtsmooth(x0, gdtm, gdom)
        assert rel(N_(out.mean), om) <= tol_m and rel(cov(N_(out.chol)), cov(oL)) <= tol_c
        # the smoother alone, from filtered factors turned by an orthogonal matrix
        turn = np.linalg.qr(np.random.default_rng(n).standard_normal((D, D)))[0]
        sm, _ = pfs.smoothing(gdtm, MVNSqrt(filt.mean, filt.chol @ T(turn)))
        assert rel(N_(sm.mean), om) <= tol_m and rel(cov(N_(sm.chol)), cov(oL)) <= tol_c


@pytest.mark.parametrize("D,d", SHAPES + [(3, 4)])
@pytest.mark.parametrize("prior,noise,x0,n", [(True, "none", "point", 12), (True, "some", "full", 5),
                                              (False, "all", "full", 1), (True, "all", "point", 2)])
def test_sequential_twin_structure(D, d, prior, noise, x0, n):
    """The sequential twin (one block, the same step operations) on the same
    models, filtered and smoothed, within the bound of the test above."""
    if d > D:  # more rows than states: noise on all of them
        prior, noise = False, "all"
    st, (F, QL), dom = model(D, d, n, prior, noise, d > D, x0, 7 * D + d + n)
    rep = lambda A: np.broadcast_to(A, (n, D, D)).copy()  # noqa: E731
    dtm = (rep(F), rep(QL))
    (om, oL), oell, oobj, _ = ofs.sequential_linear_filtsmooth(st, dtm, dom)
    (pm, pL), pnll, pobj, _ = ofs.linear_filtsmooth(st, dtm, dom)
    tol_m = max(TOL, 10 * rel(pm, om))
    tol_c = max(TOL, 10 * rel(cov(pL), cov(oL)))
    gx0 = MVNSqrt(T(st[0]), T(st[1]))
    gdom = AffineModel(T(dom[0]), T(dom[1]), None if noise == "none" else T(dom[2]))
    shared = TransitionModel(T(F).expand(n, D, D), T(QL).expand(n, D, D))
    for gdtm in (shared, TransitionModel(T(dtm[0]), T(dtm[1]))):
        out, ell, obj, _ = sfs.linear_filtsmooth(gx0, gdtm, gdom)
        assert rel(N_(out.mean), om) <= tol_m and rel(cov(N_(out.chol)), cov(oL)) <= tol_c
        assert abs(float(ell) - oell) <= max(TOL * abs(oell), 10 * abs(oell + pnll))
        assert abs(float(obj) - oobj) <= max(TOL * abs(oobj), 10 * abs(oobj - pobj))
