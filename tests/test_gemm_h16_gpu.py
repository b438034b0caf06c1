"""The mixed form's high-frequency GEMM (two FP16 planes per number under a
power-of-two scale per vector and operator row) on one complex product, against
a long-double product of the same complex64 data, and against the split-TF32
kernel.

Tolerance, per output: hi = FP16(x), lo = FP16(x - hi) leave 2^-22 |x| (unit
roundoff 2^-11 twice) and, where lo is subnormal, 2^-25 on a scale where the
largest component M is at least 2^13, so less than 2^-22 |x| + 2^-38 M.  With
both factors' error and the dropped lo lo <= 2^-22 |a||x| a real product is off
by at most 3.1 2^-22 max|A_row| max|x|; 2k of them make each part, a complex
output sqrt 2 more: 9 k 2^-22 max max.  Sums: 6k products of a part, each
addition off by at most 2^-22 (one FP32 place, truncated) of sum|A||x|, the
output scaling and the final addition 2^-22 |y| more: (6 k + 2) 2^-22 sum|A||x|,
sqrt 2 for the two parts within 9 k + 3."""
import ctypes as C

import numpy as np
import pytest

from ddfmm_b200 import _lib

pytestmark = pytest.mark.gpu
EDGES = [(1, 1, 1), (17, 9, 7), (8, 8, 127), (9, 15, 128), (53, 56, 129), (56, 16, 255), (57, 17, 33), (64, 152, 300), (104, 24, 131),
         (111, 100, 5), (112, 112, 640), (113, 90, 48), (152, 100, 257), (225, 31, 40), (296, 174, 70), (400, 400, 131)]


def product(A, X, path, Y=None):
    m, k = A.shape
    n = X.shape[1]
    A, X = np.asfortranarray(A, dtype=np.complex128), np.asfortranarray(X, dtype=np.complex128)
    Y = np.zeros((m, n), np.complex128, order="F") if Y is None else np.asfortranarray(Y.copy())
    dp = C.POINTER(C.c_double)
    _lib.check(_lib.load().ddfmm_test_gemm(A.ctypes.data_as(dp), m, k, X.ctypes.data_as(dp), n, path,
                                           Y.ctypes.data_as(dp)))
    return Y


def mats(m, k, n, spread=0.0):
    r = np.random.default_rng([m, k, n])
    g = lambda a, b: ((r.standard_normal((a, b)) + 1j * r.standard_normal((a, b)))
                      * 10.0 ** (spread * r.standard_normal((a, b)))).astype(np.complex64).astype(np.complex128)
    return g(m, k), g(k, n)


def part_max(v, axis):
    return np.maximum(np.abs(v.real), np.abs(v.imag)).max(axis=axis, keepdims=True)


def bound(A, X):
    k = A.shape[1]
    return 2.0 ** -22 * (9 * k * part_max(A, 1) * part_max(X, 0) + (9 * k + 3) * (np.abs(A) @ np.abs(X)))


@pytest.mark.parametrize("m,k,n", EDGES)
@pytest.mark.parametrize("spread", [0.0, 1.0])
def test_against_long_double(m, k, n, spread):
    A, X = mats(m, k, n, spread)
    want = A.astype(np.clongdouble) @ X.astype(np.clongdouble)
    err = {p: np.abs((product(A, X, p) - want).astype(np.complex128)) for p in (3, 4)}
    assert np.all(err[3] <= bound(A, X))
    if k >= 16 and spread == 0.0:  # no further off than the split-TF32 kernel
        print("relative 2-norm error", [float(np.linalg.norm(err[p]) / np.linalg.norm(want)) for p in (3, 4)])
        assert np.linalg.norm(err[3]) <= np.linalg.norm(err[4])


def test_adds_into_the_output():
    A, X = mats(57, 33, 130)
    Y = mats(57, 130, 1)[0]
    assert np.all(np.abs(product(A, X, 3, Y) - (Y + A @ X)) <= bound(A, X) + 2.0 ** -22 * np.abs(Y))


@pytest.mark.parametrize("e", [-148, -126, -110, -86, 60, 100, 120])
def test_vector_scales(e):
    """Vectors scaled by a power of two, subnormal ones too (the additions into the
    output flush subnormal terms and sums: 2^-126 each)."""
    A, X = mats(56, 48, 64)
    X /= 8
    Xe = (X * 2.0 ** e).astype(np.complex64).astype(np.complex128)
    A = (A / 64).astype(np.complex64).astype(np.complex128)
    assert np.all(np.abs(product(A, Xe, 3) - A @ Xe) <= bound(A, Xe) + 4 * 2.0 ** -126)


def test_zero_and_nonfinite_columns():
    """A zero vector gives zeros, one with an infinity or a NaN gives no finite
    output, and the others are what they are without it."""
    A, X = mats(60, 40, 140)
    clean = product(A, X, 3)
    X[:, 3] = 0
    X[7, 5] = np.nan
    X[0, 129] = np.inf
    X[39, 130] = complex(0, -np.inf)
    got = product(A, X, 3)
    assert np.all(got[:, 3] == 0)
    for c in (5, 129, 130):
        assert not np.any(np.isfinite(got[:, c]))
    rest = [c for c in range(140) if c not in (3, 5, 129, 130)]
    assert np.array_equal(got[:, rest], clean[:, rest])
