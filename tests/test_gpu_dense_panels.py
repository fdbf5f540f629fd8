"""The dense panels beyond the register panels' columns (768 in float64, 1280 in
float32), one CTA or a cluster of four per matrix, and a shared Q_L that is not
triangular, against the oracle's segmented schedule."""

import numpy as np
import pytest
import torch

from .test_gpu_dense import _chunk_plan, _expected, _gpu, _random_problem, covrel, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cluster", ["0", "1"])
@pytest.mark.parametrize("dtype,D,tol", [(torch.float64, 400, 1e-10), (torch.float32, 656, 2e-3)])
def test_panels_beyond_the_registers(monkeypatch, dtype, D, tol, cluster):
    """Q_L per step: trias of 2 D columns without known structure.  float32: a
    sum of 2 D products rounds by up to 2 D 6e-8 = 8e-5 of its terms, over the
    few dependent factorizations of a step."""
    monkeypatch.setenv("POF_DENSE_CLUSTER", cluster)
    n, d = 3, 16
    x0, dtm, dom = _random_problem(D, n, D, d, False)
    C0, P = _chunk_plan(n, 2)
    m, L, sc = _gpu("filtsmooth", x0, dtm, dom, 2, dtype=dtype)
    _, (sm, sL), nll, _, _, _ = _expected(x0, dtm, dom, C0, P)
    assert rel(m, sm) <= tol and covrel(L, sL) <= tol
    assert abs(sc[0] - nll) <= tol * abs(nll)


@pytest.mark.parametrize("n,D,d,noise", [(9, 40, 4, False), (7, 70, 6, True), (4, 150, 10, False)])
def test_shared_ql_that_is_not_triangular(n, D, d, noise):
    x0, (F, QL), dom = _random_problem(D + 1, n, D, d, noise)
    rng = np.random.default_rng(D)
    F = np.broadcast_to(F[0], F.shape).copy()
    QL = np.broadcast_to(QL[0] + np.triu((0.3 / np.sqrt(D)) * rng.standard_normal((D, D)), 1), QL.shape).copy()
    C0, P = _chunk_plan(n, 3)
    m, L, sc = _gpu("filtsmooth", x0, (F, QL), dom, 3, per_step=False)
    _, (sm, sL), nll, _, _, _ = _expected(x0, (F, QL), dom, C0, P)
    assert rel(m, sm) <= 1e-10 and covrel(L, sL) <= 1e-10
    assert abs(sc[0] - nll) <= 1e-10 * abs(nll)
