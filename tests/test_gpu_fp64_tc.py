"""FP64 GEMMs on the tensor cores (csrc/d64_gemm.cu) at the edges of their tiles.

H|psi> in FP64 is compared with hpsi_apply_noalloc, which runs the same local
term and the SIMT projector GEMMs, and the band-pair matrix with numpy's
complex128 product of the gradient.  Tolerance: both sides round sums of
K <= 2 npw or 2 P terms, each relative error at most K 2^-53 of the sums of
absolute products; K <= 10^4 and a cancellation factor of 10 give 1e-11 at
worst and sqrt(K) 2^-53 = 1e-14 typically; 1e-13 is required per band.
"""
import ctypes as C

import numpy as np
import pytest

from effmass_gb300 import abi
from effmass_gb300 import system as S

pytestmark = pytest.mark.gpu
TOL = 1e-13


def _cell(name, k):
    from effmass_gb300 import build
    from effmass_gb300.hamiltonian import Hamiltonian
    build.build()
    sysm = S.make_system(name)
    kp = S.g_sphere(sysm.lattice, k, sysm.ecut)
    H = Hamiltonian(sysm)
    H.set_kpoint(0, kp)
    return H, kp


def _noalloc(H, nb, psi):
    import torch
    from effmass_gb300._lib import load
    out = torch.zeros_like(psi)
    f = abi.HPSI_PREC_FP64 | abi.HPSI_DEVICE_PTRS | abi.HPSI_SYNC
    st = load().hpsi_apply_noalloc(H.ctx, 0, nb, C.c_void_p(psi.data_ptr()), C.c_void_p(out.data_ptr()), f, None)
    assert st == 0, st
    return out


def _per_band(a, b):
    import torch
    return float((torch.linalg.norm(a - b, dim=1) / torch.linalg.norm(b, dim=1)).max())


@pytest.mark.parametrize("name,nb", [("tiny", 1), ("tiny", 9), ("tinyd", 16), ("tinyd", 17), ("fcc2", 1), ("fcc2", 25),
                                     ("fcc2", 33), ("fcc2", 257), ("sc8", 7), ("sc8", 48), ("sc8", 65)])
def test_fp64_apply_matches_simt(name, nb):
    torch = pytest.importorskip("torch")
    H, kp = _cell(name, (0.1, -0.2, 0.3))
    rng = np.random.default_rng(nb)
    psi = rng.standard_normal((nb, kp.npw)) + 1j * rng.standard_normal((nb, kp.npw))
    # bands of very different weight over the sphere, and of very different size
    psi *= (0.1 + kp.kinetic)[None, :] ** rng.uniform(-4.0, 4.0, nb)[:, None]
    psi *= 2.0 ** rng.integers(-300, 300, nb)[:, None]
    psi = torch.from_numpy(psi).cuda()
    out = torch.zeros_like(psi)
    H.apply(0, nb, psi, out, "fp64")
    torch.cuda.synchronize()
    assert _per_band(out, _noalloc(H, nb, psi)) <= TOL
    H.close()


@pytest.mark.parametrize("name,nb", [("tiny", 3), ("tinyd", 33), ("sc8", 129)])
def test_fp64_velocity_matches_numpy(name, nb):
    pytest.importorskip("torch")
    from effmass_gb300.hamiltonian import GradHPsi
    H, kp = _cell(name, (0.1, -0.2, 0.3))
    psi = S.make_bands(kp, nb, seed=nb)
    g = np.zeros((3,) + psi.shape, dtype=np.complex128)
    H.grad_apply(0, nb, psi, GradHPsi(g[0], g[1], g[2]), "fp64")
    m = H.velocity_matrix(0, nb, psi, precision="fp64")
    ref = np.einsum("ig,ajg->aij", psi.conj(), g)
    assert np.linalg.norm(m - ref) <= TOL * np.linalg.norm(ref)
    H.close()


def test_fp64_zero_and_nonfinite_bands():
    """A zero band gives zeros; a band with a NaN or infinity gives NaN in that band alone."""
    torch = pytest.importorskip("torch")
    H, kp = _cell("sc8", (0.1, -0.2, 0.3))
    psi = torch.from_numpy(S.make_bands(kp, 12)).cuda()
    psi[3] = 0
    clean = torch.zeros_like(psi)
    H.apply(0, 12, psi, clean, "fp64")
    psi[5, 17] = complex(float("nan"), 0.0)
    psi[8, 100] = complex(0.0, float("inf"))
    out = torch.zeros_like(psi)
    H.apply(0, 12, psi, out, "fp64")
    torch.cuda.synchronize()
    assert not torch.any(out[3])
    assert torch.isnan(out[5]).all() and not torch.isfinite(out[8]).any()
    keep = [i for i in range(12) if i not in (5, 8)]
    assert torch.equal(out[keep], clean[keep])
    H.close()


def test_fp64_wait_runs_out_then_context_recovers():
    """The MMA issuer's bounded wait gives up (limit 0, nothing faults): the call
    reports HPSI_ERR_TIMEOUT and the next one is correct again."""
    torch = pytest.importorskip("torch")
    from effmass_gb300._lib import HpsiError, load
    H, kp = _cell("sc8", (0.1, -0.2, 0.3))
    psi = S.make_bands(kp, 12)
    good = np.zeros_like(psi)
    H.apply(0, 12, psi, good, "fp64")
    try:
        assert load().hpsi_selftest_wait_limit(0) == abi.HPSI_OK
        with pytest.raises(HpsiError) as ei:
            H.apply(0, 12, psi, np.zeros_like(psi), "fp64")
        assert ei.value.status == abi.HPSI_ERR_TIMEOUT
    finally:
        assert load().hpsi_selftest_wait_limit(-1) == abi.HPSI_OK
    again = np.zeros_like(psi)
    H.apply(0, 12, psi, again, "fp64")
    assert np.array_equal(again, good)
    assert torch.isfinite(torch.from_numpy(again).real).all()
    H.close()
