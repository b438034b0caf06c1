"""The kernel of two low-frequency products in a row (plain form), on the identity
and then a random operator, against a long-double product.  The identity's product
is exact but for the three-MMA form's (xr + xi) - xr - xi, off by at most 2^-52
(|xr| + |xi|) <= 2^-51 |x|; the second product as in the other FP64 kernels,
4 k 2^-52 sum|A||x|: together 2 (2 k + 1) 2^-52 sum|A||x|, doubled for the operator's
own rounding of the perturbed column."""
import ctypes as C

import numpy as np
import pytest

from ddfmm_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 7, 8, 17, 45, 56, 63, 64])
@pytest.mark.parametrize("n", [1, 8, 9, 263])
def test_identity_then_operator(m, n):
    r = np.random.default_rng([m, n])
    g = lambda a, b: np.asfortranarray(r.standard_normal((a, b)) + 1j * r.standard_normal((a, b)))
    A, X, Y = g(m, m), g(m, n), g(m, n)  # what Y holds is overwritten
    want = A.astype(np.clongdouble) @ X.astype(np.clongdouble)
    dp = C.POINTER(C.c_double)
    _lib.check(_lib.load().ddfmm_test_gemm(A.ctypes.data_as(dp), m, m, X.ctypes.data_as(dp), n, 5, Y.ctypes.data_as(dp)))
    assert np.all(np.abs((Y - want).astype(np.complex128)) <= 4 * (2 * m + 1) * 2.0 ** -52 * (np.abs(A) @ np.abs(X)))


def test_larger_operators_are_refused():
    A = np.zeros((65, 65), np.complex128, order="F")
    dp = C.POINTER(C.c_double)
    p = A.ctypes.data_as(dp)
    assert _lib.load().ddfmm_test_gemm(p, 65, 65, p, 65, 5, p) != 0
