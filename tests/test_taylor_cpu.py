"""libpof's power-series Taylor mode (pof_taylor) of every built-in field
against nested torch.func.jvp of the same field as a plain function, and its
refusals.  Both evaluate the same expressions in float64 with at most ~(q + 1)^2
operations per coefficient: 1e-12 of each derivative's largest entry leaves two
orders for cancellation inside the fields."""

import numpy as np
import pytest
import torch

from pof import _lib, initialization, ivp

CTORS = ["logistic", "lotkavolterra", "vanderpol", "fitzhughnagumo", "fhn_classic", "rober", "rigid_body", "seir",
         "threebody", "henonheiles", "fhn_reaction_diffusion"]


@pytest.mark.parametrize("ctor", CTORS)
@pytest.mark.parametrize("q", [1, 2, 5])
def test_power_series_equals_nested_jvp(ctor, q):
    p = getattr(ivp, ctor)(**({"cells": 5} if ctor == "fhn_reaction_diffusion" else {}))
    a = initialization.taylor_derivatives(p.f, p.y0, q).numpy()
    b = initialization.taylor_derivatives(lambda t, y: p.f(t, y), p.y0, q).numpy()
    assert a.shape == b.shape == (q + 1, len(p.y0))
    assert (np.abs(a - b) <= 1e-12 * np.abs(b).max(axis=1, keepdims=True) + 1e-300).all()


def test_refusals():
    lib = _lib.lib()
    p, y, out = np.ones(5), np.ones(4), np.empty(400)
    call = lambda f, d, q: lib.pof_taylor(f, d, q, p.ctypes.data, y.ctypes.data, out.ctypes.data)  # noqa: E731
    assert call(_lib.FIELDS["logistic"], 2, 3) == -5 and call(_lib.FIELDS["fhn_rd"], 3, 3) == -5
    assert call(0, 1, 3) == -5 and call(99, 1, 3) == -5
    assert call(_lib.FIELDS["logistic"], 1, -1) == -1 and call(_lib.FIELDS["logistic"], 1, 65) == -1
    assert call(_lib.FIELDS["logistic"], 1, 64) == 0
    assert lib.pof_taylor(_lib.FIELDS["logistic"], 1, 2, None, y.ctypes.data, out.ctypes.data) == -1
    assert torch.isfinite(initialization.taylor_derivatives(ivp.logistic().f, [0.01], 0)).all()
