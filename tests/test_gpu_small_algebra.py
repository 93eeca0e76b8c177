"""The one-CTA L x L routines of the block solvers on matrices of the test's
own: singular ones that complete pivoting has to refuse, and FP64 values whose
reciprocal is beyond its range, for the widths of one warp (up to 8) and of the
whole CTA."""
import ctypes as ct
import os
import subprocess

import numpy as np
import pytest

from bdda.build import nvcc_path
from conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def steps(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("small") / "small_steps.so")
    subprocess.run([nvcc_path(), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
                    "-shared", "-Xcompiler", "-fPIC", "-I", os.path.join(ROOT, "block-dda_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "small_steps.cu"), "-o", so], check=True)
    return ct.CDLL(so)


def _ptr(a):
    return a.ctypes.data_as(ct.POINTER(ct.c_double))


def _lu(steps, A, B, full, df):
    a, x, ok = A.astype(complex, order="F"), B.astype(complex, order="F"), ct.c_int(-1)
    assert steps.lu(_ptr(a), _ptr(x), A.shape[0], int(full), int(df), ct.byref(ok)) == 0
    return x, ok.value


# Powers of two, so that the elimination is exact and the trailing block becomes exactly zero; the largest entry is in
# the last column.
@pytest.mark.parametrize("df", [False, True])
@pytest.mark.parametrize("L", [2, 3, 8, 9, 32])
def test_complete_pivoting_refuses_a_singular_matrix(steps, L, df):
    v = 2.0 ** (np.arange(L) / 4).round()
    A = np.outer(v, v)                                  # rank one
    assert _lu(steps, A, np.eye(L), True, df)[1] == 0
    A = np.zeros((L, L))
    A[:, L - 1] = v                                     # one column
    assert _lu(steps, A, np.eye(L), True, df)[1] == 0
    assert _lu(steps, np.zeros((L, L)), np.eye(L), True, df)[1] == 0
    A = np.diag(v)                                      # rank L - 1
    A[0, 0] = 0
    A[0, L - 1] = v[0]
    assert _lu(steps, A, np.eye(L), True, df)[1] == 0


# Errors: backward stable elimination of a well-conditioned matrix, L eps cond(A), 2^-44 for double-float's eps.
@pytest.mark.parametrize("df", [False, True])
@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("L", [1, 2, 8, 9, 32])
def test_lu_solves(steps, L, full, df):
    rng = np.random.default_rng(L)
    A = rng.standard_normal((L, L)) + 1j * rng.standard_normal((L, L)) + 3 * np.sqrt(L) * np.eye(L)[rng.permutation(L)]
    B = rng.standard_normal((L, L)) + 1j * rng.standard_normal((L, L))
    x, ok = _lu(steps, A, B, full, df)
    assert ok == 1
    want = np.linalg.solve(A, B)
    eps = 2.0 ** -44 if df else 2.0 ** -52
    assert np.linalg.norm(x - want) <= 8 * L * eps * np.linalg.cond(A) * np.linalg.norm(want)


# The Gram sums of a solve whose right-hand sides are about 1e-155 or 1e153: 2^-1034 (40 bits left) and 2^1018.
# Cholesky factor and inverse of s H are those of H times sqrt(s) and its inverse; both are compared with H's.
@pytest.mark.parametrize("L", [1, 2, 8, 9, 32])
@pytest.mark.parametrize("e, eps", [(-1034, 2.0 ** -40), (0, 2.0 ** -52), (1018, 2.0 ** -52)])
def test_cholesky_over_the_range_of_fp64(steps, L, e, eps):
    rng = np.random.default_rng(L)
    W = rng.standard_normal((4 * L, L)) + 1j * rng.standard_normal((4 * L, L))
    H = W.conj().T @ W / L
    h = np.ldexp(H.real, e) + 1j * np.ldexp(H.imag, e)
    H = np.ldexp(h.real, -e) + 1j * np.ldexp(h.imag, -e)            # as rounded
    h, r, ri, ok = np.asfortranarray(h), np.zeros((L, L), complex, "F"), np.zeros((L, L), complex, "F"), ct.c_int(-1)
    assert steps.chol(_ptr(h), _ptr(r), _ptr(ri), L, 0, ct.byref(ok)) == 0
    assert ok.value == 1
    R = np.linalg.cholesky(H).conj().T
    tol = 8 * L * eps * np.linalg.cond(H)
    assert np.linalg.norm(r * 2.0 ** (-e // 2) - R) <= tol * np.linalg.norm(R)
    assert np.linalg.norm(ri * 2.0 ** (e // 2) - np.linalg.inv(R)) <= tol * np.linalg.norm(np.linalg.inv(R))


# A pivot of 2^-520 has a square of 2^-1040, 34 bits; its reciprocal is within FP64.
@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("L", [1, 2, 8, 9, 32])
@pytest.mark.parametrize("e, eps", [(-520, 2.0 ** -32), (-505, 2.0 ** -52), (505, 2.0 ** -52)])
def test_lu_over_the_range_of_fp64(steps, L, full, e, eps):
    rng = np.random.default_rng(L)
    A = rng.standard_normal((L, L)) + 1j * rng.standard_normal((L, L)) + 3 * np.sqrt(L) * np.eye(L)[rng.permutation(L)]
    B = rng.standard_normal((L, L)) + 1j * rng.standard_normal((L, L))
    x, ok = _lu(steps, A * 2.0 ** e, B * 2.0 ** e, full, False)
    assert ok == 1
    want = np.linalg.solve(A, B)
    assert np.linalg.norm(x - want) <= 8 * L * eps * np.linalg.cond(A) * np.linalg.norm(want)
