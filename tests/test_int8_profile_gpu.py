"""The int8 path on graded vectors: components that differ by many orders of magnitude and
meet operator columns as much smaller, as an outgoing vector and the operators on it do.
With the vectors' profile (powers of two, from the sizes of their components; here the largest
of all vectors) both are flat before they are written as digits.

Tolerance, per output: as in tests/test_gemm_paths_gpu.py for the scaled factors, 2^-51 (k max|A'_row|
max|x'| + |y|).  A' and x' are formed here with the rows' largest components themselves; a power
of two is within a factor of two of its component, so 2^-50.  And no further off than the FP64 kernel, whose error does
not depend on such a scaling, in the 2-norm over all outputs."""
import numpy as np
import pytest

from ddfmm_b200 import _lib
from test_gemm_paths_gpu import mats, part_max, product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n", [(8, 16, 1), (45, 45, 33), (56, 56, 128), (81, 90, 129), (100, 152, 300), (139, 168, 24),
                                   (57, 129, 7), (400, 400, 131)])
@pytest.mark.parametrize("decades", [0.0, 2.0, 4.0])
def test_graded_vectors(m, k, n, decades):
    A, X = mats(m, k, n)
    g = 10.0 ** np.random.default_rng([k, 1]).uniform(-decades, decades, k)
    A, X = A / g, X * g[:, None]
    want = A.astype(np.clongdouble) @ X.astype(np.clongdouble)
    err = {p: np.abs((product(A, X, p) - want).astype(np.complex128)) for p in (0, 6)}
    s = part_max(X, 1)[:, 0]
    bound = 2.0 ** -50 * (k * part_max(A * s, 1) * part_max(X / s[:, None], 0) + np.abs(want).astype(float))
    assert np.all(err[6] <= bound)
    assert np.linalg.norm(err[6]) <= np.linalg.norm(err[0])


def test_rows_of_zeros_and_extremes():
    """A component that is zero in every vector, and vectors near both ends of the range."""
    A, X = mats(60, 40, 33)
    X[7] = 0
    X[:, 5] = 0
    clean = product(A, X, 6)
    want = A.astype(np.clongdouble) @ X.astype(np.clongdouble)
    assert np.all(clean[:, 5] == 0)
    assert np.linalg.norm((clean - want).astype(np.complex128)) <= 1e-15 * np.linalg.norm(want.astype(np.complex128))
    for e in (-1000, -900, 900, 1000):
        got = product(A * 2.0 ** -8, X * 2.0 ** e, 6)
        assert np.all(np.isfinite(got))
        d = np.abs(got - (clean * 2.0 ** -8) * 2.0 ** e)
        assert np.all(d <= 2.0 ** -1070 + 2.0 ** -52 * np.abs(clean * 2.0 ** -8) * 2.0 ** e)
    X[3, 9] = np.nan
    X[0, 20] = np.inf
    got = product(A, X, 6)
    for c in (9, 20):
        assert not np.any(np.isfinite(got[:, c]))
