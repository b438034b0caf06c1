"""One session's matvec in each way its launches are issued: as the graph built
at setup (a small instance's evals), step by step on one stream (while profiled),
and captured by the caller into a graph of their own and replayed.  All are the
same sums in another order, so each is held to the parity bars of the other GPU
tests: 1e-10 relative l2 for the plain form, 2e-5 for the mixed one."""
import numpy as np
import pytest

import fixtures
from ddfmm_b200 import _lib, wave3d

pytestmark = pytest.mark.gpu
TOL = {_lib.PLAIN_FP64: 1e-10, _lib.MIXED: 2e-5}


def _session(c, tmp_path, precision):
    ldp, hdp = c.write_operators(str(tmp_path))
    p = c.params
    mlib = wave3d.Mlib3d()
    mlib.setup({"-mlib3d_ldname": ldp, "-mlib3d_hdname": hdp})
    w = wave3d.Wave3d(precision=precision)
    w.posptr = c.pos
    w.kernel = p["kernel"]
    w.mlibptr = mlib
    w.geomprtn = p["nc"]
    w.setup({"-wave3d_ACCU": str(p["accu"]), "-wave3d_NPQ": str(p["npq"]), "-wave3d_K": str(p["K"]),
             "-wave3d_ptsmax": str(p["ptsmax"]), "-wave3d_maxlevel": str(p["maxlevel"])})
    return w


@pytest.mark.parametrize("precision", [_lib.PLAIN_FP64, _lib.MIXED])
@pytest.mark.parametrize("name", ["sphere_k8_n5000_p4_helm", "cluster_k4_n1500_p4_helm_m8", "sphere_k4_n1500_p4_expr",
                                  "sphere_k4_n1500_p8_helm"])
def test_every_way_to_issue_an_eval(name, precision, tmp_path):
    import torch
    c = fixtures.Case(name)
    w = _session(c, tmp_path, precision)
    den = torch.from_numpy(np.ascontiguousarray(c.den).view(np.float64)).to("cuda")
    out = torch.empty_like(den)

    def close(scale=1.0):
        torch.cuda.synchronize()
        v = out.cpu().numpy().view(np.complex128)
        rel = np.linalg.norm(v - scale * c.val) / np.linalg.norm(scale * c.val)
        out.fill_(float("nan"))
        return rel <= TOL[precision]

    for _ in range(3):
        w.eval_device(den.data_ptr(), out.data_ptr())
        assert close()
    w.profile(True)
    for _ in range(2):
        w.eval_device(den.data_ptr(), out.data_ptr())
        assert close()
    assert len(w.profile_read()) > 0
    w.profile(False)
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(g, stream=s):
        w.eval_device(den.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    for k in range(3):  # other densities in the same array
        g.replay()
        assert close(2.0 ** k)
        den *= 2
    torch.cuda.synchronize()
    with torch.cuda.stream(s):  # and the session's own graph again, on that stream
        w.eval_device(den.data_ptr(), out.data_ptr(), s.cuda_stream)
    assert close(8.0)
    w.close()
