"""The FP64 velocity matrix of bands of very different norm: an entry depends on its
own two bands alone.

Tolerance, relative to |psi_i| |g_j|: each operand is rounded to 2^-56 of its row's
largest element (which is at most the row's norm), and the sums to 2^-53 per K split
(fewer than 64); 64 x 2^-53 = 7e-15 is required.
"""
import numpy as np
import pytest

from effmass_gb300 import system as S

pytestmark = pytest.mark.gpu
TOL = 7e-15


@pytest.mark.parametrize("big", [1.0, 1e10, 1e120])
def test_entries_depend_on_their_bands_alone(big):
    pytest.importorskip("torch")
    from effmass_gb300 import build
    from effmass_gb300.hamiltonian import GradHPsi, Hamiltonian
    build.build()
    sysm = S.make_system("sc8")
    kp = S.g_sphere(sysm.lattice, (0.1, -0.2, 0.3), sysm.ecut)
    psi = S.make_bands(kp, 6, seed=2)
    psi[0] *= big * (kp.kinetic < 1.0)  # large, and on few G alone
    psi[3] *= 1.0 / big
    g = np.zeros((3,) + psi.shape, dtype=np.complex128)
    with Hamiltonian(sysm) as H:
        H.set_kpoint(0, kp)
        H.grad_apply(0, 6, psi, GradHPsi(g[0], g[1], g[2]), "fp64")
        m = H.velocity_matrix(0, 6, psi, precision="fp64")
    size = np.linalg.norm(psi, axis=1)
    gsize = np.linalg.norm(g, axis=2)
    ref = np.einsum("ig,ajg->aij", psi.conj() / size[:, None], g / gsize[:, :, None])
    assert np.abs(m / size[None, :, None] / gsize[:, None, :] - ref).max() <= TOL
