"""The device math of csrc/mpm_math.cuh and csrc/mpm_svd.cuh on the host, against numpy."""
from __future__ import annotations

import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "diffskill_gb300", "csrc")


INCLUDE = ["-I", os.path.join(HERE, "host_math"), "-I", CSRC]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("host_math") / "host_math.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-Wno-unknown-pragmas",
                    *INCLUDE, os.path.join(HERE, "host_math", "host_math.cpp"),
                    "-o", out], check=True)
    return ctypes.CDLL(out)


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _svd(lib, name, A):
    """U, s, V of each matrix of A by the device function ``name``, and who took the plain form."""
    n, T = len(A), A.dtype
    U, s, V, plain = np.zeros((n, 3, 3), T), np.zeros((n, 3), T), np.zeros((n, 3, 3), T), np.zeros(n, np.int32)
    D = np.ascontiguousarray(A - np.eye(3, dtype=T) if name.endswith("32") else A)
    getattr(lib, name)(ctypes.c_long(n), _ptr(D), _ptr(U), _ptr(s), _ptr(V), _ptr(plain))
    return U, s, V, plain


def _rotations(rng, n):
    q = np.linalg.qr(rng.normal(size=(n, 3, 3)))[0]
    q[:, :, 2] *= np.linalg.det(q)[:, None]
    return q


def _matrices(rng, s):
    """Matrices with the singular values s, between random rotations."""
    return (_rotations(rng, len(s)) * s[:, None, :]) @ _rotations(rng, len(s)).transpose(0, 2, 1)


def _errors(A, U, s, V):
    """Per matrix: how far U and V are from orthonormal and U diag(s) V^T from A
    (relative to A), in extended precision."""
    A, U, s, V = (a.astype(np.longdouble) for a in (A, U, s, V))
    eye = np.eye(3, dtype=np.longdouble)

    def mul(a, b):
        return np.einsum("nij,njk->nik", a, b)

    t = (0, 2, 1)
    e = [abs(mul(U.transpose(t), U) - eye), abs(mul(V.transpose(t), V) - eye),
         abs(mul(U * s[:, None, :], V.transpose(t)) - A) / abs(A).max((1, 2), keepdims=True)]
    return np.max([x.max((1, 2)) for x in e], 0).astype(float)


# ranges of the three singular values
SPREADS = {"dough": [(0.97, 1.03)] * 3, "strained": [(0.8, 1.25)] * 3, "short-0.2": [(1.0, 1.6), (0.6, 1.2), (0.2, 0.25)],
           "short-0.35": [(1.0, 1.6), (0.6, 1.2), (0.35, 0.5)], "short-0.5": [(1.0, 1.6), (0.6, 1.2), (0.5, 0.7)],
           "long-3": [(1.5, 3.0), (0.6, 1.4), (0.5, 1.0)], "long-10": [(3.0, 10.0), (0.6, 1.4), (0.5, 1.0)],
           "any": [(0.2, 3.0)] * 3}


@pytest.mark.parametrize("spread", SPREADS)
def test_fp32_left_svd_is_as_exact_as_by_gram_schmidt(lib, spread):
    """No range of deformations loses digits to V = A^T U / s: the errors' median and
    99 % quantile are at most those of an SVD that takes V by Gram-Schmidt (and a tenth,
    for the scatter of quantiles of 20,000 matrices)."""
    rng = np.random.default_rng(3)
    s = np.stack([rng.uniform(lo, hi, 20000) for lo, hi in SPREADS[spread]], 1)
    A = _matrices(rng, s).astype(np.float32)
    left, ref = (_errors(A, *_svd(lib, name, A)[:3]) for name in ("left32", "by_gram_schmidt32"))
    for q in (0.5, 0.99):
        assert np.quantile(left, q) <= 1.1 * np.quantile(ref, q), q


# and two values nearly equal, where the refinement's angle is large
@pytest.mark.parametrize("spread", list(SPREADS) + ["pair-1e-2", "pair-3e-4", "pair-1e-7"])
def test_fp64_left_svd_is_as_exact_as_by_gram_schmidt(lib, spread):
    """The refined FP32 decomposition has no worse matrices than FP64 sweeps: median, 99 %
    quantile and largest error of 20,000 are at most theirs (and a tenth, half for the
    largest)."""
    rng = np.random.default_rng(5)
    s = np.stack([rng.uniform(lo, hi, 20000) for lo, hi in SPREADS.get(spread, [(0.7, 1.3)] * 3)], 1)
    if spread not in SPREADS:
        s[:, 1] = s[:, 0] + float(spread[5:]) * rng.uniform(0.3, 1, 20000)
    A = _matrices(rng, s)
    left, ref = (_errors(A, *_svd(lib, name, A)[:3]) for name in ("left64", "by_gram_schmidt64"))
    for q, more in ((0.5, 1.1), (0.99, 1.1), (1.0, 1.5)):
        assert np.quantile(left, q) <= more * np.quantile(ref, q), q


@pytest.mark.parametrize("name,ulp", [("left32", 2.0 ** -23), ("left64", 2.0 ** -52)])
def test_left_svd_of_inverted_and_singular_matrices(lib, name, ulp):
    """det U = det V = 1 with the sign on the last value, orthonormal vectors and A = U
    diag(s) V^T also where the short vectors have no length of their own; and no NaN for
    matrices of rank 0 and 1.  Products and rotations round at some 30 ulp (of 1), and a
    value near 0 of FP32, the root of a difference, at the root of that."""
    rng = np.random.default_rng(4)
    sing = [(1.2, 1.0, -0.5), (1.3, 1.0, -0.04), (1, 1, -1), (1.1, 0.9, 0.0), (1.1, 0.9, 1e-3), (1, 1, 1), (1, 1, 0.9),
            (1.2, 0.8, 0.8), (2, 0, 0), (0, 0, 0)]
    s = np.array([sing[i % len(sing)] for i in range(2000)], np.float64)
    A = _matrices(rng, s).astype(np.float32 if name == "left32" else np.float64)
    U, got, V, _ = _svd(lib, name, A)
    tol = (30 * ulp) ** (0.5 if name == "left32" else 1)
    some = s.max(1) > 0  # (the zero matrix has no relative error)
    assert _errors(A[some], U[some], got[some], V[some]).max() < tol
    for W in (U, V):
        assert np.abs(np.linalg.det(W.astype(np.float64)) - 1).max() < 30 * ulp
    assert np.abs(np.sort(got, 1) - np.sort(s, 1)).max() < 2 * tol


RCP, RSQRT, SQRT, LOG, EXPM1, CUT, WIDEN, EXACT, ROUND, QUOT, RCP_MID, RSQRT_MID = range(12)
TINY, HUGE = 2.0 ** -1022, 2.0 ** 1023
FTINY = 2.0 ** -126


def _ftz(x):
    """x in FP32 as a conversion under -ftz gives it: rounded to 24 bits, and what is then
    below the normal range a zero of its sign."""
    with np.errstate(over="ignore", invalid="ignore"):
        x = np.asarray(x, np.float64)
        small = (x * 2.0 ** 64).astype(np.float32).astype(np.float64) * 2.0 ** -64
        y = np.where(abs(x) < 2.0 ** -60, small, x.astype(np.float32))
    return np.where(abs(y) < FTINY, np.copysign(0.0, y), y).astype(np.float32)


def _range(rng, lo, hi, n=20000):
    """n values of both signs, their logarithms spread over [lo, hi]; and the two ends."""
    x = np.exp2(rng.uniform(np.log2(lo), np.log2(hi), n)) * rng.choice([-1.0, 1.0], n)
    return np.concatenate([x, [lo, -lo, hi, -hi]])


def check_scalar_helpers(call):
    """``call(which, x)``: the helpers against numpy over the ranges they state."""
    rng = np.random.default_rng(6)
    inf, nan = np.inf, np.nan

    def near(got, want, ulps):
        assert (abs(got - want) <= ulps * 2.0 ** -52 * abs(want)).all()

    def same(got, want):
        assert np.array_equal(np.asarray(got, np.float64).view(np.int64),
                              np.asarray(want, np.float64).view(np.int64))

    # half an ulp of the last rounding, the rounding of e and its cube: below 1.5 ulp
    x = np.concatenate([_range(rng, TINY, 2.0 ** 1021), 2.0 ** np.arange(-40, 40.0), np.linspace(1, 4, 2001)])
    near(call(RCP, x), 1 / x, 1.5)
    near(call(QUOT, x), 3 / x, 2.5)
    near(call(RSQRT, abs(x)), 1 / np.sqrt(abs(x)), 1.5)
    near(call(SQRT, abs(x)), np.sqrt(abs(x)), 2.5)
    x = np.concatenate([_range(rng, FTINY, 2.0 ** 125), np.linspace(1, 4, 2001)])
    near(call(RCP_MID, x), 1 / x, 1.5)
    near(call(RSQRT_MID, abs(x)), 1 / np.sqrt(abs(x)), 1.5)
    same(call(RCP, np.array([0.0, -0.0, inf, -inf])), [inf, -inf, 0.0, -0.0])
    same(call(RCP, np.array([HUGE, -HUGE, 1e-310])), [0.0, -0.0, inf])
    same(call(RSQRT, np.array([0.0, 1e-310, inf])), [inf, inf, 0.0])
    same(call(SQRT, np.array([inf])), [inf])
    for f in (RCP, RSQRT, SQRT):
        assert np.isnan(call(f, np.array([nan, -nan]))).all()
    assert np.isnan(call(RSQRT, np.array([-1.0, -inf]))).all()
    # the series and, from 1/8, the library's functions: some four roundings
    x = np.concatenate([_range(rng, 1e-12, 0.25), [0.125, -0.125, 0.0]])
    s = 1.0 + x
    near(call(LOG, x), np.log1p(s - 1.0), 4)
    near(call(EXPM1, x), np.expm1(x), 4)
    # conversions: exact, or to nearest even
    x = np.concatenate([_range(rng, FTINY, 2.0 ** 127), [0.0, -0.0]])
    same(call(CUT, x), (x.view(np.int64) & ~0x1fffffff).view(np.float64))
    same(call(CUT, np.array([inf, -inf, nan, 2.0 ** 128, FTINY / 2])), [0.0, -0.0, 0.0, 0.0, 0.0])
    f = _ftz(x)
    same(call(WIDEN, f.astype(np.float64)), f)
    f = np.concatenate([f, np.float32([inf, -inf, FTINY / 2, -FTINY / 2])])
    same(call(EXACT, f.astype(np.float64)), _ftz(f))
    assert np.isnan(call(EXACT, np.array([nan]))).all() and np.isnan(call(ROUND, np.array([nan, -nan]))).all()
    one, ulp = np.array([1.0, 1.0 + 2.0 ** -23, 1.5]), 2.0 ** -23
    ties = np.concatenate([one + ulp / 2, one + ulp / 2 + 2.0 ** -52, one + ulp / 2 - 2.0 ** -52, one + ulp / 4])
    edge = np.array([2.0 ** 128, 2.0 ** 128 * (1 - 2.0 ** -25), 2.0 ** 128 * (1 - 2.0 ** -24), 3e38, 1e39, inf,
                     FTINY * (1 - 2.0 ** -30), FTINY * (1 - 2.0 ** -24), FTINY / 2, 1e-60])
    x = np.concatenate([_range(rng, 1e-50, 1e45), ties, -ties, edge, -edge, [0.0, -0.0]])
    same(call(ROUND, x), _ftz(x))


def test_scalar_helpers_on_the_host(lib):
    """Over all of FP64's range, its ends, rounding ties, infinities and NaN."""
    def call(which, x):
        x = np.ascontiguousarray(x, np.float64)
        y = np.zeros_like(x)
        assert lib.scalar(which, len(x), _ptr(x), _ptr(y)) == 0
        return y

    check_scalar_helpers(call)


@pytest.mark.gpu
def test_scalar_helpers_on_the_device(tmp_path):
    """The same with the device's own approximations of 1/x and 1/sqrt(x), compiled with
    the substep's flags."""
    import torch

    from diffskill_gb300 import build

    out = str(tmp_path / "device_math.so")
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", *build._FAST32,
                    "-I", CSRC, "-o", out, os.path.join(HERE, "host_math", "device_math.cu"), "-lcudart"], check=True)
    dev = ctypes.CDLL(out)

    def call(which, x):
        a = torch.as_tensor(np.ascontiguousarray(x, np.float64), device="cuda")
        y = torch.zeros_like(a)
        torch.cuda.synchronize()
        assert dev.scalar(which, a.numel(), ctypes.c_void_p(a.data_ptr()), ctypes.c_void_p(y.data_ptr())) == 0
        return y.cpu().numpy()

    check_scalar_helpers(call)
