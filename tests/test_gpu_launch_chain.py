"""The tree levels' overlapped launches against ordinary ones: the profiler
gives every kernel a launch of its own, so a pass with it on must equal one
without it bit for bit, at one step, at one and several levels, and where the
lower levels' launches are ordinary and the upper ones' overlapped.  Each size
runs several times in a row on changing inputs: a kernel that read its inputs
before they were written would show the pass before."""

import numpy as np
import pytest
import torch

from pof import _lib, parallel_filtsmooth as pfs
from pof.observations import AffineModel
from pof.transitions import IWP, TransitionModel, preconditioned_discretize
from pof.utils import MVNSqrt

pytestmark = pytest.mark.gpu


def _inputs(n, q, d, dtype, seed):
    rng = np.random.default_rng(seed)
    D = d * (q + 1)
    F, QL = (x.to(dtype) for x in preconditioned_discretize(IWP(num_derivatives=q, wiener_process_dimension=d),
                                                            device="cuda"))
    t = lambda x: torch.as_tensor(x, dtype=dtype, device="cuda")  # noqa: E731
    x0 = MVNSqrt(t(rng.normal(size=D)), t(0.1 * np.eye(D)))
    H = np.zeros((n, d, D))
    for i in range(d):
        H[:, i, i * (q + 1) + 1] = 1.0
        H[:, i, i * (q + 1)] = 0.1 * rng.normal(size=n)
    dom = AffineModel(t(H), t(0.1 * rng.normal(size=(n, d))), t(np.zeros((n, d, d))))
    return x0, TransitionModel(F, QL), dom


def _pass(args):
    (m, L), nll, obj, ssq = pfs.linear_filtsmooth(*args)
    return [x.detach().clone() for x in (m, L, nll, obj, ssq)]


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("q,d", [(2, 1), (2, 2), (3, 2)])
@pytest.mark.parametrize("n", [1, 2, 9, 700, 20011])
def test_overlapped_launches_equal_ordinary_ones(n, q, d, dtype):
    cases = [_inputs(n, q, d, dtype, seed) for seed in range(3)]
    lib = _lib.lib()
    lib.pof_profile_enable(1)
    try:
        ordinary = [_pass(a) for a in cases]
        torch.cuda.synchronize()
        _lib.profile_read()
    finally:
        lib.pof_profile_enable(0)
    overlapped = [_pass(a) for a in cases * 2]
    for k, got in enumerate(overlapped):
        for x, y in zip(got, ordinary[k % 3]):
            assert torch.isfinite(y).all() and torch.equal(x, y)
