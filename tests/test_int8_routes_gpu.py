"""The plain form's sessions with products on both GEMM routes.  Which high-frequency
products go to the int8 kernel is a question of their size, and the fixtures' are small;
here every second product of each launch goes there (ddfmm_session_test_create), so
every pass is split between digits and FP64 vectors.  The results are held to the
reference's values at the parity bar of the other GPU tests, 1e-10 in relative l2, in
each way an eval's launches are issued, and the profile has to show both routes."""
import numpy as np
import pytest

import fixtures
from ddfmm_b200 import _lib, geometry, precompute, wave3d
from test_failure_gpu import _session

pytestmark = pytest.mark.gpu
TOL = 1e-10
BY_SIZE, NONE, ALTERNATE = 0, 1, 2


def _force(monkeypatch, rule):
    lib = _lib.load()
    monkeypatch.setattr(lib, "ddfmm_session_create_ex",
                        lambda *a: lib.ddfmm_session_test_create(*a[:-1], rule, a[-1]))


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def _profile(w, den, val):
    w.profile(True)
    w.eval(den, val)
    p = w.profile_read()
    w.profile(False)
    return p


def _routes(p):
    """{(pass, width): kernels} of the high-frequency GEMM passes"""
    out = {}
    for label, e in p.items():
        if label.startswith(("hf_m2m", "hf_m2l", "hf_l2l")):
            out.setdefault(label.replace("_i8", ""), set()).add(e["kernel"])
    return out


@pytest.mark.parametrize("rule", [ALTERNATE, NONE])
@pytest.mark.parametrize("name", ["sphere_k8_n5000_p4_helm", "sphere_k16_n4000_p4_helm", "ellipsoid_k8_n3000_p4_helm",
                                  "sphere_k4_n1500_p4_expr", "sphere_k4_n1500_p6_helm", "sphere_k4_n1500_p8_helm",
                                  "cluster_k4_n1500_p4_helm_m8"])
def test_split_launches_match_the_reference(name, rule, tmp_path, monkeypatch):
    import torch
    _force(monkeypatch, rule)
    c = fixtures.Case(name)
    w = _session(c, tmp_path, _lib.PLAIN_FP64)
    v = np.zeros_like(c.den)
    for _ in range(2):  # the second one on the first one's digits
        w.eval(c.den, v)
        assert _rel(v, c.val) <= TOL
    w.eval(-2.0 * c.den, v)
    assert _rel(v, -2.0 * c.val) <= TOL
    p = _profile(w, c.den, v)
    assert _rel(v, c.val) <= TOL
    routes = _routes(p)
    if w.stats()["hf_up_nodes"]:
        assert {k.split("_w")[0] for k in routes} == {"hf_m2m", "hf_m2l", "hf_l2l"}
    for label, kernels in routes.items():
        fp64 = kernels & {"zgemm_kernel", "zgemm_narrow_kernel"}
        assert fp64 and kernels - fp64 == ({"i8_gemm_kernel"} if rule == ALTERNATE else set()), (label, kernels)
    # captured by the caller
    den = torch.from_numpy(np.ascontiguousarray(c.den)).to("cuda")
    out = torch.zeros_like(den)
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(g, stream=s):
        w.eval_device(den.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        out.fill_(float("nan"))
        g.replay()
        torch.cuda.synchronize()
        assert _rel(out.cpu().numpy(), c.val) <= TOL
    w.close()


@pytest.mark.parametrize("accu", [1, 2])
def test_a_session_that_takes_the_int8_route_by_size(accu, tmp_path, monkeypatch):
    """Sphere K = 16 with 25 points per square wavelength: both routes by the rule itself,
    against the same session without the int8 kernel."""
    n, K = 20106, 16
    ld, hd = precompute.ensure_operators(str(tmp_path), 0, accu, 2)
    pos, den = geometry.sphere_points(n, float(K), 2), geometry.densities(n, 3)
    vals = {}
    for rule in (BY_SIZE, NONE):
        with monkeypatch.context() as m:
            _force(m, rule)
            mlib = wave3d.Mlib3d()
            mlib.setup({"-mlib3d_ldname": ld, "-mlib3d_hdname": hd})
            w = wave3d.Wave3d(precision=_lib.PLAIN_FP64)
            w.posptr, w.mlibptr, w.geomprtn = pos, mlib, geometry.cells_for(K)
            w.setup({"-wave3d_ACCU": str(accu), "-wave3d_K": repr(float(K)),
                     "-wave3d_maxlevel": str(geometry.maxlevel_for(K))})
        v = vals[rule] = np.zeros_like(den)
        w.eval(den, v)
        kernels = {e["kernel"] for e in _profile(w, den, np.zeros_like(den)).values()}
        assert ("i8_gemm_kernel" in kernels) == ("i8_slice_kernel" in kernels) == (rule == BY_SIZE)
        assert kernels & {"zgemm_kernel", "zgemm_narrow_kernel"}
        if rule == NONE:
            assert w.check(den, v, np.arange(0, n, 200, dtype=np.int32)) <= {1: 2e-3, 2: 2e-5}[accu]
        w.close()
    assert _rel(vals[BY_SIZE], vals[NONE]) <= TOL
