"""What a context keeps of a replaced binding: at most 64 MB, nothing that the
bindings since have not used, and nothing once another allocation finds no room."""
import ctypes as C

import numpy as np
import pytest

from effmass_gb300 import system as S

pytestmark = pytest.mark.gpu


def _kept(H):
    from effmass_gb300._lib import load
    out = (C.c_longlong * 5)()
    assert load().hpsi_selftest_memory_state(H.ctx, out) == 0
    return out[4]


def _apply(H, kid, kp, prec):
    psi = S.make_bands(kp, 3)
    out = np.zeros_like(psi)
    H.apply(kid, 3, psi, out, prec)
    return out


def test_spares_are_bounded_and_given_back():
    from effmass_gb300 import build
    from effmass_gb300._lib import load
    from effmass_gb300.hamiltonian import Hamiltonian
    build.build()
    sysm = S.make_system("sc8")
    kp = S.g_sphere(sysm.lattice, (0.1, -0.2, 0.3), sysm.ecut)
    with Hamiltonian(sysm) as H:
        for kid in range(24):
            H.set_kpoint(kid, kp)
            for prec in ("fp64", "fp32", "tc"):
                want = _apply(H, kid, kp, prec)
        assert _kept(H) == 0
        for kid in range(24):
            H.set_kpoint(kid, kp)  # many slots replaced: one binding's buffers stay
            assert 0 < _kept(H) <= 64 << 20
        kept = _kept(H)
        assert np.array_equal(_apply(H, 23, kp, "tc"), want)
        assert 0 < _kept(H) < kept
        H.set_kpoint(23, kp)
        H.set_kpoint(23, kp)  # nothing was built in between
        assert _kept(H) == 0
        _apply(H, 23, kp, "fp64")
        H.set_kpoint(23, kp)
        assert _kept(H) > 0
        assert load().hpsi_selftest_memory(H.ctx, -1, 1) == 0
        H.set_kpoint(99, kp)
        assert _kept(H) == 0
        assert np.array_equal(_apply(H, 99, kp, "tc"), want)
