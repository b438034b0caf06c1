"""The bounded pipeline waits of the FP16 and int8 GEMM kernels, made to run out on
purpose as in tests/test_failure_gpu.py (which does it to the split-TF32 kernel): block 0
of the next launch withholds the operator copies that its MMA issuer waits on, every
wait being bounded by 2 ms.  The eval fails, within the limit, and the same session, a
fresh one and the batch compute correct matvecs afterwards, so the block gave its
tensor memory back and nothing of it was left in flight."""
import time

import numpy as np
import pytest

import fixtures
from ddfmm_b200 import _lib, geometry, precompute, wave3d
from test_failure_gpu import TOL_MIXED, _rel, _session

pytestmark = pytest.mark.gpu
TF32, FP16, INT8 = 0, 1, 2
TOL_PLAIN = 1e-10


def _plain_int8(tmp_path):
    """A plain session whose evals use the int8 kernel: sphere K = 16, P = 4, with densities."""
    n, K = 20106, 16
    ld, hd = precompute.ensure_operators(str(tmp_path), 0, 1, 2)
    mlib = wave3d.Mlib3d()
    mlib.setup({"-mlib3d_ldname": ld, "-mlib3d_hdname": hd})
    w = wave3d.Wave3d(precision=_lib.PLAIN_FP64)
    w.posptr, w.mlibptr, w.geomprtn = geometry.sphere_points(n, float(K), 2), mlib, geometry.cells_for(K)
    w.setup({"-wave3d_ACCU": "1", "-wave3d_K": repr(float(K)), "-wave3d_maxlevel": str(geometry.maxlevel_for(K))})
    return w, geometry.densities(n, 3)


def _fails_once(w, den, want, tol, kernel):
    lib = _lib.load()
    _lib.check(lib.ddfmm_session_test_gemm_stall_in(w._s, 0.002, kernel))
    t0 = time.perf_counter()
    with pytest.raises(_lib.DDFMMError) as e:
        w.eval(den, np.zeros_like(den))
    assert time.perf_counter() - t0 < 5.0  # the 2 ms limit, not the default 1 s or a hang
    assert e.value.code == 2 and "timed out" in str(e.value)
    v = np.zeros_like(den)
    w.eval(den, v)
    assert _rel(v, want) <= tol


@pytest.mark.parametrize("kernel", [TF32, FP16])
def test_mixed_form(kernel, tmp_path):
    c = fixtures.Case("sphere_k8_n5000_p4_helm")
    w = _session(c, tmp_path, _lib.MIXED)
    for _ in range(2):
        _fails_once(w, c.den, c.val, TOL_MIXED, kernel)
    other = _session(c, tmp_path, _lib.MIXED)
    b = wave3d.Batch([w, other])
    den = [c.den.astype(np.complex64)] * 2
    vals = [np.zeros(len(c.den), np.complex64) for _ in range(2)]
    _lib.check(_lib.load().ddfmm_session_test_gemm_stall_in(w._s, 0.002, kernel))
    with pytest.raises(_lib.DDFMMError) as e:
        b.eval(den, vals)
    assert e.value.code == 2 and "timed out" in str(e.value)
    b.eval(den, vals)
    for v in vals:
        assert _rel(v, c.val) <= TOL_MIXED
    b.close()
    w.close()
    v = np.zeros_like(c.den)
    other.eval(c.den, v)
    assert _rel(v, c.val) <= TOL_MIXED
    other.close()


def test_plain_form(tmp_path):
    w, den = _plain_int8(tmp_path)
    want = np.zeros_like(den)
    w.eval(den, want)
    ids = np.arange(0, len(den), 200, dtype=np.int32)
    assert w.check(den, want, ids) <= 2e-3  # P = 4
    for _ in range(2):
        _fails_once(w, den, want, TOL_PLAIN, INT8)
    w.close()
    w, den = _plain_int8(tmp_path)
    v = np.zeros_like(den)
    w.eval(den, v)
    assert _rel(v, want) <= TOL_PLAIN
    w.close()


def test_refused_where_the_kernel_is_not_launched(tmp_path):
    lib = _lib.load()
    c = fixtures.Case("sphere_k4_n1500_p4_expr")
    w = _session(c, tmp_path, _lib.PLAIN_FP64)  # too small for the int8 kernel
    m = _session(c, tmp_path, _lib.MIXED)
    for s, kernels in ((w, (TF32, FP16, INT8)), (m, (INT8,))):
        for k in kernels:
            assert lib.ddfmm_session_test_gemm_stall_in(s._s, 0.002, k) == 1
    assert lib.ddfmm_session_test_gemm_stall_in(m._s, 0.002, 3) == 1
    assert lib.ddfmm_session_test_gemm_stall_in(m._s, 2.0, FP16) == 1
    w.close()
    m.close()
