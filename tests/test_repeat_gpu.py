"""Root boxes of one and two wavelengths have no high-frequency passes, whose atomic
additions come in no fixed order: their matvecs repeat bit for bit.  (A profiled eval
issues its launches one by one, in an order that adds a box's check values up the
other way round: it repeats itself.)"""
import numpy as np
import pytest

from ddfmm_b200 import _lib, geometry, precompute, wave3d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [_lib.PLAIN_FP64, _lib.MIXED, _lib.MIXED_MMA_SYNC])
@pytest.mark.parametrize("K", [1, 2])
def test_low_frequency_matvec_repeats_bit_for_bit(K, precision, tmp_path):
    import torch
    n = 4000
    pos = geometry.cluster_points(n, float(K), 3)
    ld, hd = precompute.ensure_operators(str(tmp_path), 0, 1, 1)
    mlib = wave3d.Mlib3d()
    mlib.setup({"-mlib3d_ldname": ld, "-mlib3d_hdname": hd})
    w = wave3d.Wave3d(precision=precision)
    w.posptr, w.mlibptr, w.geomprtn = pos, mlib, K
    w.setup({"-wave3d_ACCU": "1", "-wave3d_K": repr(float(K)), "-wave3d_ptsmax": "8", "-wave3d_maxlevel": "8"})
    assert w.stats()["hf_up_nodes"] == 0 and w.stats()["hf_down_nodes"] == 0
    den = geometry.densities(n, 5)
    d, out = torch.from_numpy(den).to("cuda"), torch.zeros(n, dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()

    def values():
        w.eval_device(d.data_ptr(), out.data_ptr())
        torch.cuda.synchronize()
        return out.cpu().numpy()

    def repeats(first, times):
        for _ in range(times):
            assert np.array_equal(values(), first)

    first = values()
    ids = np.arange(0, n, 40, dtype=np.int32)
    assert np.linalg.norm(first[ids] - w.direct(den, ids)) <= 2e-3 * np.linalg.norm(first[ids])  # the method's own error
    repeats(first, 30)
    w.profile(True)
    repeats(values(), 10)
    w.close()
