"""The device math of csrc/mpm_math.cuh and csrc/mpm_svd.cuh on the host, against numpy."""
from __future__ import annotations

import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "diffskill_gb300", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("host_math") / "host_math.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-Wno-unknown-pragmas",
                    "-I", os.path.join(HERE, "host_math"), "-I", CSRC, os.path.join(HERE, "host_math", "host_math.cpp"),
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
