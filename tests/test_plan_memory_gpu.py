"""Device memory of plain sessions with products on the int8 path.

An operator entry is 16 bytes for the FP64 kernels and 14 x 2 as digits (rows [Ar, -Ai] and
[Ai, Ar]), padded to whole tiles of 8 rows and K blocks of 16, at most 1.4 times as many
entries at the fixtures' ranks (45 and up).  Their sessions are nearly all operators, so with
every second product on the int8 path, and no FP64 copy of those, a session takes at most
(16 + 28 x 1.4) / 32 = 1.725 of what it takes without; vectors' digits (14 bytes beside 2 x 16)
stay below that."""
import numpy as np
import pytest

import fixtures
from ddfmm_b200 import _lib, wave3d, workloads
from test_failure_gpu import _session
from test_int8_routes_gpu import ALTERNATE, BY_SIZE, NONE, TOL, _force, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["sphere_k16_n4000_p4_helm", "sphere_k4_n1500_p8_helm", "sphere_k8_n5000_p4_helm"])
def test_int8_operators_are_not_kept_twice(name, tmp_path, monkeypatch):
    c = fixtures.Case(name)
    size = {}
    for rule in (NONE, ALTERNATE):
        with monkeypatch.context() as m:
            _force(m, rule)
            w = _session(c, tmp_path, _lib.PLAIN_FP64)
        size[rule] = w.stats()["device_bytes"]
        w.close()
    assert size[ALTERNATE] <= 1.725 * size[NONE]


def test_spectra_and_digits_share_memory(monkeypatch):
    """Sphere K = 32, P = 6: the V-list spectra lie in the digits' memory, and the digits of a
    level's outgoing and incoming vectors in one place; without the int8 path nothing is shared."""
    wl = workloads.sphere(32.0, accu=2)
    den = wl.densities()
    vals = {}
    for rule in (NONE, BY_SIZE):
        with monkeypatch.context() as m:
            _force(m, rule)
            w = wave3d.from_workload(wl)
        v = vals[rule] = np.zeros_like(den)
        w.eval(np.conj(den), v)
        w.eval(den, v)  # over the first one's spectra
        assert w.stats()["fft_spectra_bytes"] > 128 << 20
        if rule == NONE:
            assert w.check(den, v, wl.check_ids()) <= 2e-5
        w.close()
    assert _rel(vals[BY_SIZE], vals[NONE]) <= TOL
