"""The kernel of two low-frequency products in a row on operators that are not square, as a
truncated rank makes them: Y = A (A^T X), A m x r with r below, above and off multiples of
8 and 16, against a long-double product.  A swap of m and r, of the operators or of
their leading dimensions reads other numbers (tests/test_gemm_pair_gpu.py has m = r only).

Tolerance: the first product's outputs are off by 4 m 2^-52 sum|A^T||x| (three-MMA form, as in the
other FP64 kernels), which the second multiplies by |A|; the second's own is 4 r 2^-52
sum|A||A^T x|, at most as large a sum: 4 (m + r) 2^-52 |A| |A^T| |x|, and once more for the second
order."""
import ctypes as C

import numpy as np
import pytest

from ddfmm_b200 import _lib

pytestmark = pytest.mark.gpu
DP = C.POINTER(C.c_double)


def pair(A, X, Y):
    m, k = A.shape
    A, X = np.asfortranarray(A), np.asfortranarray(X)
    return _lib.load().ddfmm_test_gemm(A.ctypes.data_as(DP), m, k, X.ctypes.data_as(DP), X.shape[1], 8,
                                       Y.ctypes.data_as(DP))


@pytest.mark.parametrize("m,r", [(56, 41), (56, 56), (41, 56), (64, 1), (1, 64), (64, 63), (63, 64), (17, 9), (9, 17), (48, 31),
                                 (31, 48), (7, 3)])
@pytest.mark.parametrize("n", [1, 8, 9, 150])
def test_operators_that_are_not_square(m, r, n):
    rng = np.random.default_rng([m, r, n])
    g = lambda a, b: np.asfortranarray(rng.standard_normal((a, b)) + 1j * rng.standard_normal((a, b)))
    A, X, Y = g(m, r), g(m, n), g(m, n)  # what Y holds is overwritten
    _lib.check(pair(A, X, Y))
    L = A.astype(np.clongdouble)
    want = L @ (L.T @ X.astype(np.clongdouble))
    bound = 5 * (m + r) * 2.0 ** -52 * (np.abs(A) @ (np.abs(A).T @ np.abs(X)))
    assert np.all(np.abs((Y - want).astype(np.complex128)) <= bound)


@pytest.mark.parametrize("m,r", [(65, 8), (8, 65)])
def test_larger_ones_are_refused(m, r):
    A, X = np.zeros((m, r), np.complex128), np.zeros((m, 1), np.complex128)
    assert pair(A, X, X.copy()) != 0
