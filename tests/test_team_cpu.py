"""The team kernels (csrc/pof_team*.cuh, pof_seq.cuh) on the host, every thread
of a block a fiber (tests/team_cpu.cpp), no GPU: results must not depend on the
order in which the lanes run between two barriers, nor on what shared memory
and scratch held before, and agree with the oracle."""

import ctypes
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

from oracle import core, filtsmooth as ofs

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "parallel-in-time-ode-filters_gb300", "csrc")
# PTX statements and shared-memory declarations of the headers, and their host forms
SUBST = [
    (r'asm\("rcp\.approx\.ftz\.f32 %0, %1;" : "=f"\(y\) : "f"\(x\)\);', "y = 1.0f / x;"),
    (r'asm\("rsqrt\.approx\.ftz\.f32 %0, %1;" : "=f"\(y\) : "f"\(x\)\);', "y = 1.0f / sqrtf(x);"),
    (r'asm volatile\("[^"]*"(?: : "\+l"\(p\))?\s*::: ?"memory"\);', ""),
    (r'asm volatile\("" : "\+l"\(p\)::"memory"\);', ""),
    (r"extern __shared__ __align__\(16\) unsigned char smem_raw_\[\];", "unsigned char* smem_raw_ = host_smem;"),
    (r"__shared__ ", "static "),
]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("team")
    for name in os.listdir(CSRC):
        if name.endswith((".cuh", ".h")):
            with open(os.path.join(CSRC, name)) as f:
                text = f.read()
            for pat, rep in SUBST:
                text = re.sub(pat, rep, text)
            if name != "pof_dense.cuh":
                assert "asm" not in re.sub(r"//.*", "", text), name
            (d / name).write_text(text)
    (d / "cuda_runtime.h").write_text("")
    dense = (d / "pof_dense.cuh").read_text()
    kern = re.search(r"constexpr int kTrsmBlock = \d+;", dense).group(0) + "\n" + \
        re.search(r"template <typename T>\n__global__ void k_trsm_diag\(.*?\n}\n", dense, re.S).group(0)
    (d / "trsm_diag.h").write_text("namespace pof {\nnamespace dense {\n%s}\n}\n" % kern)
    so = str(d / "team_cpu.so")
    subprocess.run([cxx, "-std=c++17", "-O1", "-ffp-contract=off", "-w", "-shared", "-fPIC", "-I", str(d),
                    os.path.join(ROOT, "tests", "team_cpu.cpp"), "-o", so], check=True, capture_output=True, text=True)
    return ctypes.CDLL(so)


def _p(a):
    return None if a is None else a.ctypes.data_as(ctypes.c_void_p)


def _model(D, d, n, prior, noise, per_step, seed, dtype):
    rng = np.random.default_rng(seed)
    q = D // d - 1
    if prior:
        F, QL = core.preconditioned_discretize(d, q)
    else:
        F = np.eye(D) + 0.1 * rng.standard_normal((D, D))
        QL = 0.5 * np.eye(D) + 0.1 * rng.standard_normal((D, D))
    H = rng.standard_normal((n, d, D))
    if prior:  # observation rows of the solver: the first two columns of each block
        keep = np.zeros(D, bool)
        keep[:: q + 1] = keep[1 :: q + 1] = True
        H[:, :, ~keep] = 0.0
    R = {"none": None, "some": 0.2 * np.tril(rng.standard_normal((n, d, d)) + 2 * np.eye(d))
         * (np.arange(n) % 3 == 1)[:, None, None]}[noise]
    if per_step:
        F, QL = np.tile(F, (n, 1, 1)), np.tile(QL, (n, 1, 1))
    c = rng.standard_normal((n, d))
    m0, L0 = rng.standard_normal(D), 0.3 * np.eye(D) + 0.1 * rng.standard_normal((D, D))
    return [None if x is None else np.ascontiguousarray(x, dtype) for x in (F, QL, H, c, R, m0, L0)]


def _pass(lib, dtype, order, poison, n, C0, D, d, model):
    F, QL, H, c, R, m0, L0 = model
    out = [np.zeros((n + 1, D), dtype), np.zeros((n + 1, D, D), dtype), np.zeros((n + 1, D), dtype),
           np.zeros((n + 1, D, D), dtype), np.zeros(4)]
    rc = lib.team_cpu_pass(int(dtype == np.float32), order, poison, ctypes.c_int64(n), C0, D, d, _p(F), _p(QL),
                           ctypes.c_int64(D * D if F.ndim == 3 else 0), _p(H), _p(c), _p(R), _p(m0), _p(L0),
                           *[_p(x) for x in out])
    assert rc == 0 and not lib.team_cpu_deadlock()
    return out


def _sequential(lib, dtype, order, poison, n, D, d, model, field=0, params=None, p0=0.0, p1=0.0):
    F, QL, H, c, R, m0, L0 = model
    out = [np.zeros((n + 1, D), dtype), np.zeros((n + 1, D, D), dtype), np.zeros(3)]
    rc = lib.team_cpu_sequential(int(dtype == np.float32), order, poison, ctypes.c_int64(n), D, d, _p(F), _p(QL),
                                 ctypes.c_int64(D * D if F.ndim == 3 else 0), _p(H), _p(c), _p(R), field, _p(params),
                                 ctypes.c_double(p0), ctypes.c_double(p1), _p(m0), _p(L0), *[_p(x) for x in out])
    assert rc == 0 and not lib.team_cpu_deadlock()
    return out


ORDERS = [(0, 0xff), (1, 0xff), (2, 0xff), (3, 0x3f), (0, 0)]  # (order of the lanes, what memory held)


def _same(a, b):
    return all(x.tobytes() == y.tobytes() for x, y in zip(a, b))


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("D,d,n,C0,prior,noise,per_step", [
    (6, 2, 19, 2, True, "none", False), (8, 2, 13, 3, True, "none", False), (8, 2, 9, 2, True, "some", True),
    (9, 3, 11, 2, False, "some", False), (12, 3, 7, 1, True, "none", True)])
def test_pass_does_not_depend_on_lane_order(lib, dtype, D, d, n, C0, prior, noise, per_step):
    model = _model(D, d, n, prior, noise, per_step, D + n, dtype)
    ref = _pass(lib, dtype, *ORDERS[0], n, C0, D, d, model)
    for o in ORDERS[1:]:
        assert _same(ref, _pass(lib, dtype, *o, n, C0, D, d, model)), o
    if dtype == np.float64:
        F, QL, H, c, R, m0, L0 = model
        rep = lambda A: np.broadcast_to(A, (n, D, D))  # noqa: E731
        (om, oL), nll, _, _ = ofs.sequential_linear_filtsmooth(
            (m0, L0), (rep(F), rep(QL)), (H, c, np.zeros((n, d, d)) if R is None else R))
        assert np.abs(ref[2] - om).max() <= 1e-8 * np.abs(om).max()
        cov = lambda L: L @ np.swapaxes(L, -1, -2)  # noqa: E731
        assert np.abs(cov(ref[3]) - cov(oL)).max() <= 1e-8 * np.abs(cov(oL)).max()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("D,d,prior,noise,per_step", [
    (2, 1, True, "none", False), (4, 1, True, "some", True), (8, 2, True, "none", False), (9, 3, False, "some", True),
    (12, 3, True, "none", False), (3, 4, False, "some", False), (3, 4, False, "none", False)])
def test_sequential_twin_does_not_depend_on_lane_order(lib, dtype, D, d, prior, noise, per_step):
    """(3, 4) without noise has more exact observations than states: not a
    number, whatever memory held."""
    n = 6
    model = _model(D, d, n, prior, noise, per_step, D + 10 * d, dtype)
    ref = _sequential(lib, dtype, *ORDERS[0], n, D, d, model)
    for o in ORDERS[1:]:
        out = _sequential(lib, dtype, *o, n, D, d, model)
        if d > D:
            ok = [np.isnan(a) == np.isnan(b) for a, b in zip(ref, out)]
            assert all(x.all() for x in ok)
        else:
            assert _same(ref, out), o
    if d > D:
        assert not np.isfinite(ref[2][0])


def test_sequential_ekf_does_not_depend_on_lane_order(lib):
    D, d, n = 8, 2, 6  # Van der Pol, q = 3
    F, QL, _, _, _, m0, L0 = _model(D, d, n, True, "none", False, 3, np.float64)
    params = np.array([1.0])
    args = (n, D, d, (F, QL, None, None, None, m0, L0), 3, params, 0.1, 0.3)
    ref = _sequential(lib, np.float64, *ORDERS[0], *args)
    assert all(np.isfinite(x).all() for x in ref)
    for o in ORDERS[1:]:
        assert _same(ref, _sequential(lib, np.float64, *o, *args)), o


# rows of [P | W; Yp | Yw] scaled by powers of two: the factors scale with them
SCALES = {np.float64: [0, -300, -495, -505, -512, -518, -530, 490, 505, 509], np.float32: [0, -40, -55, 50, 60]}


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("which", [0, 1, 2, 3])
@pytest.mark.parametrize("rows", ["all", "first", "pivot zero"])
def test_factorizations_of_rows_far_from_one(lib, dtype, which, rows):
    """lq_rows, lq_pivot and t_lq (8 and 32 lanes) of a matrix with rows times
    2^k equal the factors of the matrix itself with rows times 2^k.  Bound: 64
    roundings of the entries' sums, and what the squared norm and the dot
    products lose to underflow (units of the smallest number, 16 of them) where
    they are small."""
    M, MB, NW = 4, 3, 4
    rng = np.random.default_rng(5)
    X = rng.standard_normal((M + MB, M + NW))
    X[:, :M] = np.tril(X[:, :M])
    X[M:, :M] = 0.0 if which else X[M:, :M]
    if rows == "pivot zero":  # the factors of an updated state
        X[:M, :M][np.diag_indices(M)] = 0.0
    X = X.astype(dtype)
    tiny = {np.float64: -1074, np.float32: -149}[dtype]
    for k in SCALES[dtype]:
        s = np.ones((M + MB, 1), dtype)
        s[: 1 if rows == "first" else M + MB] = np.ldexp(dtype(1), k)
        out = []
        for A in (X, X * s):
            A = A.copy()
            assert lib.team_cpu_factor(int(dtype == np.float32), which, 0, _p(A)) == 0
            out.append(np.concatenate([np.tril(A[:M, :M]), A[M:, :M]]))  # L and the pivot columns below
            if which:  # the rows below, all columns
                out[-1] = np.concatenate([out[-1], A[M:, M:].reshape(-1, M)])
        ref = out[0].astype(np.longdouble)
        sc = np.concatenate([s, s[M:]]) if which else s
        assert np.isfinite(out[1]).all(), k
        err = np.abs(out[1].astype(np.longdouble) / sc - ref).max() / np.abs(ref).max()
        assert err <= 64 * np.finfo(dtype).eps + 16 * 2.0 ** (tiny - 2 * k), (k, err)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("upper", [0, 1])
def test_dense_diagonal_solves_round_like_divisions(lib, dtype, upper):
    """k_trsm_diag with a diagonal matrix: the quotients, bit for bit, also of
    zeros, infinities and entries at the ends of the range."""
    rng = np.random.default_rng(1)
    n, K = 32, 200
    big = {np.float64: 1000, np.float32: 120}[dtype]
    x = (rng.standard_normal((n, K)) * np.exp2(rng.integers(-5, 5, (n, K)))).astype(dtype)
    diag = (rng.uniform(1, 2, n) * np.exp2(rng.integers(-8, 8, n))).astype(dtype)
    diag[:6] = np.array([0.0, np.inf, -0.0, np.finfo(dtype).tiny / 4, 2.0**big, 2.0**-big], dtype)
    x[6, :5] = [np.inf, -np.inf, 0.0, np.nan, np.finfo(dtype).max]
    with np.errstate(all="ignore"):
        ref = x / diag[:, None]

    def solve(r0, r1):
        b = np.ascontiguousarray(x[r0:r1])
        lib.team_cpu_trsm_diag(int(dtype == np.float32), r1 - r0, upper, K,
                               _p(np.ascontiguousarray(np.diag(diag[r0:r1]))), _p(b))
        return b

    for i in range(7):  # one by one: what is not finite would reach other rows as 0 * inf
        assert np.array_equal(solve(i, i + 1), ref[i : i + 1], equal_nan=True), diag[i]
    assert np.array_equal(solve(7, n), ref[7:])


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("D,d", [(4, 1), (8, 2)])
def test_infinite_observation(lib, dtype, D, d):
    """c infinite in the last step: sigma^2 and -log L are infinite, in float32
    (compensated sums) as in float64, and the filtered mean is not a number only
    where it is in float64."""
    n = 5
    model = _model(D, d, n, True, "some" if d == 1 else "none", False, D, dtype)
    model[3][-1, 0] = np.inf
    m, L, s = _sequential(lib, dtype, 0, 0, n, D, d, model)
    m64 = _sequential(lib, np.float64, 0, 0, n, D, d, [None if x is None else x.astype(np.float64) for x in model])
    if d == 1:
        assert s[0] == -np.inf and s[2] == np.inf
    assert np.array_equal(np.isnan(m), np.isnan(m64[0])) and np.array_equal(np.isnan(s), np.isnan(m64[2]))
