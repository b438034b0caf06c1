"""The plain form's translation kernels on one complex product: the FP64
tensor path (64-column tiles, and the one for few columns) and the int8 tensor path (seven balanced base-256 digits a number,
54 bits below the largest component of a vector or operator row, all sums
exact) against a long-double product.

Tolerance of the int8 path, per output: each factor is rounded to half of
2^(e - 54), 2^e at most twice its vector's (row's) largest component, so to
2^-54 of that component, and the dropped digit products stay below 2^-57 of
the product of both: each of the 2k real products of a part is off by at most
(2 + 1/8) 2^-54 max|A_row| max|x|, a complex output by 2^-51 k max max with
the factor sqrt 2 of its two parts; two FP64 roundings add 2^-51 |y|.  The FP64 path: 2k products and sums at
2^-53 each, three-MMA form with factor-two larger terms; 4 k 2^-52 sum|A||x|."""
import ctypes as C

import numpy as np
import pytest

from ddfmm_b200 import _lib

pytestmark = pytest.mark.gpu
EDGES = [(1, 1, 1), (17, 9, 7), (64, 296, 8), (129, 33, 17), (8, 15, 127), (53, 56, 128), (55, 16, 129), (56, 17, 33), (57, 152, 300), (64, 31, 5),
         (106, 95, 257), (112, 112, 640), (113, 90, 48), (152, 110, 129), (296, 174, 70), (400, 400, 131)]


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
    g = lambda a, b: (r.standard_normal((a, b)) + 1j * r.standard_normal((a, b))) * 10.0 ** (spread * r.standard_normal((a, b)))
    return g(m, k), g(k, n)


def part_max(v, axis):
    return np.maximum(np.abs(v.real), np.abs(v.imag)).max(axis=axis, keepdims=True)


@pytest.mark.parametrize("m,k,n", EDGES)
@pytest.mark.parametrize("spread", [0.0, 1.0])
def test_paths_against_long_double(m, k, n, spread):
    A, X = mats(m, k, n, spread)
    want = A.astype(np.clongdouble) @ X.astype(np.clongdouble)
    err = {p: np.abs((product(A, X, p) - want).astype(np.complex128)) for p in (0, 1, 2)}
    assert np.all(err[1] <= 2.0 ** -51 * (k * part_max(A, 1) * part_max(X, 0) + np.abs(want).astype(float)))
    for p in (0, 2):
        assert np.all(err[p] <= 4 * k * 2.0 ** -52 * (np.abs(A) @ np.abs(X)))
    if k >= 16 and spread == 0.0:  # no further off than the FP64 path, column by column norms apart
        assert np.linalg.norm(err[1]) <= np.linalg.norm(err[0])


def test_adds_into_the_output():
    A, X = mats(57, 33, 130)
    Y = mats(57, 130, 1)[0]
    d = np.abs(product(A, X, 1, Y) - (Y + product(A, X, 1)))
    assert np.all(d <= 2.0 ** -52 * (np.abs(Y) + np.abs(A @ X)))


@pytest.mark.parametrize("scale", [1e-307, 1e-290, 1e-250, 1e250, 1e290])
def test_vector_scales(scale):
    """A power of two on a vector comes out as that power of two."""
    A, X = mats(56, 48, 64)
    s = 2.0 ** np.round(np.log2(scale))
    a, b = product(A, X, 1), product(A, X * s, 1)
    fine = np.abs(a) > 0 if scale > 1e-290 else np.zeros(a.shape, bool)
    assert np.array_equal(b[fine], (a * s)[fine])
    assert np.all(np.abs(b - a * s) <= 2.0 ** -1070 + 1e-13 * np.abs(a * s))


def test_zero_and_nonfinite_columns():
    """A zero vector gives zeros, one with an infinity or a NaN gives no finite
    output, and the others are what they are without it."""
    A, X = mats(60, 40, 140)
    clean = product(A, X, 1)
    X[:, 3] = 0
    X[7, 5] = np.nan
    X[0, 129] = np.inf
    X[39, 130] = complex(0, -np.inf)
    got = product(A, X, 1)
    assert np.all(got[:, 3] == 0)
    for c in (5, 129, 130):
        assert not np.any(np.isfinite(got[:, c]))
    rest = [c for c in range(140) if c not in (3, 5, 129, 130)]
    assert np.array_equal(got[:, rest], clean[:, rest])


def test_largest_digits_do_not_overflow():
    """Every digit at its extreme: the int32 diagonal sums are at their largest."""
    k = 400
    for v in (1.0, -1.0, 1.0 - 2.0 ** -53, 0.50196078431372548, -0.50196078431372548):
        A, X = np.full((56, k), v * (1 + 1j)), np.full((k, 128), v * (1 - 1j))
        want = (A.astype(np.clongdouble) @ X.astype(np.clongdouble)).astype(np.complex128)
        assert np.all(np.abs(product(A, X, 1) - want) <= 2.0 ** -51 * (k + np.abs(want)))
