"""What an enqueued eval leaves behind when a tensor-core GEMM's bounded wait runs out
(tests/test_failure_gpu.py has the calls that return a status): its values are all NaN,
and the evals after it are none the wiser."""
import ctypes as C

import numpy as np
import pytest

import fixtures
from ddfmm_b200 import _lib, wave3d
from test_failure_gpu import TOL_MIXED, _rel, _session

pytestmark = pytest.mark.gpu
NAME = "sphere_k8_n5000_p4_helm"


def _device(v):
    import torch
    return torch.from_numpy(np.ascontiguousarray(v)).to("cuda")


def _check_failed_then_correct(w, c, stall, call, out):
    """call() fails once after stall(), and not again; the host call in between is correct."""
    import torch
    torch.cuda.synchronize()
    call()
    torch.cuda.synchronize()
    assert _rel(out.cpu().numpy(), c.val) <= TOL_MIXED
    stall()
    call()
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert np.all(np.isnan(got.real)) and np.all(np.isnan(got.imag))
    v = np.zeros_like(c.den)
    w.eval(c.den, v)
    assert _rel(v, c.val) <= TOL_MIXED
    call()
    torch.cuda.synchronize()
    assert _rel(out.cpu().numpy(), c.val) <= TOL_MIXED


@pytest.mark.parametrize("entry", ["eval_device", "eval_device_c64", "noalloc", "batch"])
def test_enqueued_eval_with_a_timed_out_wait_is_nan(entry, tmp_path):
    lib = _lib.load()
    c = fixtures.Case(NAME)
    w = _session(c, tmp_path, _lib.MIXED)
    stall = lambda: _lib.check(lib.ddfmm_session_test_gemm_stall(w._s, 0.002))
    c64 = entry in ("eval_device_c64", "batch")
    den = _device(c.den.astype(np.complex64) if c64 else c.den)
    out = den.clone()
    if entry == "noalloc":
        call = lambda: _lib.check(lib.ddfmm_eval_device_noalloc(w._s, C.c_void_p(den.data_ptr()),
                                                                C.c_void_p(out.data_ptr()), None))
    elif entry == "batch":
        other = _session(c, tmp_path, _lib.MIXED)
        b = wave3d.Batch([other, w])
        out2 = den.clone()  # the hook is for the launch's first block, whose tiles may be either instance's
        call = lambda: b.eval_device([den.data_ptr()] * 2, [out2.data_ptr(), out.data_ptr()])
    else:
        call = lambda: w.eval_device(den.data_ptr(), out.data_ptr(), c64=c64)
    _check_failed_then_correct(w, c, stall, call, out)
    if entry == "batch":
        stall()  # the call with a status
        with pytest.raises(_lib.DDFMMError) as e:
            b.eval([c.den.astype(np.complex64)] * 2, [np.zeros(len(c.den), np.complex64) for _ in range(2)])
        assert e.value.code == 2 and "timed out" in str(e.value)
        b.close()
        other.close()
    w.close()
