"""The chunk rule of level 0: problems that fitted the allocation-free entry
point's scratch with power-of-two chunks still fit it, and a pass at the edges
where the rule takes one more step per chunk equals the same pass in chunks of
4 (both bracket the same associative scan; 1e-9 relative is the distance that
two orders of it may have in float64 at these lengths)."""

import numpy as np
import pytest
import torch

SCRATCH = 16 * 1024 * 1024


@pytest.mark.parametrize("dtype,n,D,d", [(0, 100000, 2, 1), (0, 136000, 2, 1), (1, 131500, 3, 1), (1, 133500, 3, 4),
                                         (1, 18200, 6, 2), (1, 8700, 9, 3)])
def test_scratch_sized_passes_still_fit(dtype, n, D, d, lib):
    assert 0 < lib.pof_filtsmooth_workspace_bytes(dtype, n, D, d) <= SCRATCH


@pytest.fixture(scope="module")
def lib():
    from pof import _lib
    return _lib.lib()


def _pass(n, q, d):
    from pof import parallel_filtsmooth as pfs
    from pof.observations import AffineModel
    from pof.transitions import IWP, TransitionModel, preconditioned_discretize
    from pof.utils import MVNSqrt
    rng = np.random.default_rng(n)
    D = d * (q + 1)
    F, QL = preconditioned_discretize(IWP(num_derivatives=q, wiener_process_dimension=d), device="cuda")
    t = lambda x: torch.as_tensor(x, dtype=torch.float64, device="cuda")  # noqa: E731
    H = np.zeros((n, d, D))
    for i in range(d):
        H[:, i, i * (q + 1) + 1] = 1.0
        H[:, i, i * (q + 1)] = 0.1 * rng.uniform(0.5, 1.0, size=n)
    x0 = MVNSqrt(t(rng.normal(size=D)), t(0.1 * np.eye(D)))
    dom = AffineModel(t(H), t(0.1 * rng.normal(size=(n, d))), t(np.zeros((n, d, d))))
    (m, L), *_ = pfs.linear_filtsmooth(x0, TransitionModel(F, QL), dom)
    return m, L @ L.mT


@pytest.mark.gpu
@pytest.mark.parametrize("n,q,d", [(12160, 2, 2), (12161, 2, 2), (18241, 2, 2), (6081, 4, 2), (9121, 3, 3),
                                   (77824, 2, 1), (77825, 2, 1)])
def test_edges_of_the_rule(n, q, d, monkeypatch):
    m, C = _pass(n, q, d)
    monkeypatch.setenv("POF_C0", "4")
    m4, C4 = _pass(n, q, d)
    assert float((m - m4).norm() / m4.norm()) <= 1e-9
    assert float((C - C4).norm() / C4.norm()) <= 1e-9
