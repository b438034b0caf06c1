"""The FP16 path on graded vectors (tests/test_int8_profile_gpu.py has the int8 one): with
the vectors' profile, components that differ by many orders of magnitude and meet operator
columns as much smaller keep their bits, as they do in the split-TF32 kernel.

Tolerance, per output: as in tests/test_gemm_h16_gpu.py, for the scaled factors where it has the
largest components of a vector and an operator row; the factors are scaled here by those
components themselves, and a power of two is within a factor of two of them."""
import numpy as np
import pytest

from ddfmm_b200 import _lib
from test_gemm_h16_gpu import mats, part_max, product

pytestmark = pytest.mark.gpu
TF32, PLAIN, PROFILED = 4, 3, 7


def single(v):
    return v.astype(np.complex64).astype(np.complex128)


@pytest.mark.parametrize("m,k,n", [(8, 16, 1), (45, 45, 33), (56, 56, 128), (100, 152, 300), (139, 168, 24), (113, 129, 7),
                                   (400, 400, 131)])
@pytest.mark.parametrize("decades", [0.0, 2.0, 4.0])
def test_graded_vectors(m, k, n, decades):
    A, X = mats(m, k, n)
    g = 10.0 ** np.random.default_rng([k, 1]).uniform(-decades, decades, k)
    A, X = single(A / g), single(X * g[:, None])
    want = A.astype(np.clongdouble) @ X.astype(np.clongdouble)
    err = {p: np.abs((product(A, X, p) - want).astype(np.complex128)) for p in (TF32, PROFILED)}
    s = part_max(X, 1)[:, 0]
    bound = 2.0 ** -22 * (18 * k * part_max(A * s, 1) * part_max(X / s[:, None], 0)
                          + (9 * k + 3) * (np.abs(A) @ np.abs(X)))
    assert np.all(err[PROFILED] <= bound)
    assert np.linalg.norm(err[PROFILED]) <= np.linalg.norm(err[TF32])


def test_rows_of_zeros_and_extremes():
    A, X = mats(60, 40, 33)
    X[7] = 0
    X[:, 5] = 0
    clean = product(A, X, PROFILED)
    assert np.all(clean[:, 5] == 0)
    for e in (-120, -90, 90, 110):
        got = product(single(A / 64), single(X * 2.0 ** e), PROFILED)
        assert np.all(np.isfinite(got))
        assert np.all(np.abs(got - clean / 64 * 2.0 ** e) <= 4 * 2.0 ** -126 + 2.0 ** -22 * np.abs(clean) / 64 * 2.0 ** e)
    X[3, 9] = np.nan
    X[0, 20] = np.inf
    got = product(A, X, PROFILED)
    for c in (9, 20):
        assert not np.any(np.isfinite(got[:, c]))
