"""The dense schedule with the triangular structure that the GPU's context
exploits (tests/dense_struct_cpu.cpp): the leading rows' factorization of Phi,
Psi and Xi, and reflectors that end with the triangular block, against the
oracle's segmented schedule, bounds-checked, with scratch that starts as NaN.
A shared Q_L that is not triangular takes the general form."""

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from .test_dense_cpu import CSRC, ROOT, _check, _covd, _expected, _p, _random_problem


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    so = str(tmp_path_factory.mktemp("dstruct") / "dense_struct_cpu.so")
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-shared", "-fPIC", "-I", CSRC,
                    os.path.join(ROOT, "tests", "dense_struct_cpu.cpp"), "-o", so],
                   check=True, capture_output=True, text=True)
    return ctypes.CDLL(so)


def _run(lib, which, x0, dtm, fts, dom, chunks, n, D, d):
    H, c, R = dom
    om, oL, osc = np.zeros((n + 1, D)), np.zeros((n + 1, D, D)), np.zeros(8)
    msg = ctypes.create_string_buffer(256)
    i64 = ctypes.c_int64
    a = [None if x is None else np.ascontiguousarray(x) for x in (*x0, *dtm, H, c, R)]
    rc = lib.dense_struct_filtsmooth(which, i64(n), D, d, *[_p(x) for x in a[:4]], i64(fts), *[_p(x) for x in a[4:]],
                                     i64(0 if R is None else d * d), _p(om), _p(oL), _p(osc), chunks, msg, 256)
    assert rc >= 0, msg.value.decode()
    return rc, om, oL, osc


@pytest.mark.parametrize("n,D,d,chunks,noise,ql", [
    (23, 20, 3, 5, True, "shared"), (23, 20, 3, 4, False, "shared"), (16, 33, 4, 4, False, "dense"),
    (9, 24, 24, 3, True, "dense"), (33, 16, 2, 4, True, "shared"), (12, 12, 5, 12, False, "per step"),
    (97, 12, 3, 33, False, "shared"), (1, 18, 2, 0, False, "shared")])
def test_structured_schedule_matches_oracle(lib, n, D, d, chunks, noise, ql):
    rng = np.random.default_rng(n * 1000 + D)
    x0, (F, QL), (H, c, R) = _random_problem(rng, n, D, d, noise)
    if ql != "per step":
        Q1 = QL[0] + (0.05 * np.triu(rng.standard_normal((D, D)), 1) if ql == "dense" else 0.0)
        F, QL = np.broadcast_to(F[0], F.shape).copy(), np.broadcast_to(Q1, QL.shape).copy()
    shared = ql != "per step"
    dtm, fts = ((F[0], QL[0]), 0) if shared else ((F, QL), D * D)
    low, om, oL, osc = _run(lib, 1, x0, dtm, fts, (H, c, R), chunks, n, D, d)
    assert low == (ql == "shared")
    C0 = -(-n // min(n, chunks or 64))
    (fm, fL), (sm, sL), nll, _, _, _ = _expected(x0, (F, QL), (H, c, R), C0, -(-n // C0))
    _check(om, sm, 1e-10, "smoothed means")
    assert _covd(oL, sL) <= 1e-10
    _check(osc[0], nll, 1e-10, "nll")
    _, om0, oL0, _ = _run(lib, 0, x0, dtm, fts, (H, c, R), chunks, n, D, d)
    _check(om0, fm, 1e-10, "filtered means")
    assert _covd(oL0, fL) <= 1e-10
    _, om2, oL2, _ = _run(lib, 2, (om0, oL0), dtm, fts, (None, None, None), chunks, n, D, d)
    _check(om2, sm, 1e-10, "smoother alone")
    assert _covd(oL2, sL) <= 1e-10
