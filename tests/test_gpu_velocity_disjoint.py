"""FP64 velocity matrix of bands that share little weight: an entry is a sum of small
products, which must not be lost against the bands' largest coefficients.

Tolerance relative to the sum of an entry's absolute products: both operands are held
to 2^-62 of their largest coefficients, an entry that would lose more than 6 bits to
that is summed in FP64, and sums of K <= 6000 terms are rounded to K 2^-53 at worst,
sqrt(K) 2^-53 = 9e-15 typically; 1e-13 is required.
"""
import numpy as np
import pytest

from effmass_gb300 import system as S

pytestmark = pytest.mark.gpu
TOL = 1e-13


@pytest.mark.parametrize("nb", [2, 7, 40])
@pytest.mark.parametrize("tiny", [0.0, 1e-3, 1e-12])
def test_entries_of_nearly_disjoint_bands(nb, tiny):
    from effmass_gb300 import build
    from effmass_gb300.hamiltonian import Hamiltonian
    build.build()
    sysm = S.make_system("sc8")
    sysm = S.System(name="bare", lattice=sysm.lattice, omega=sysm.omega, n1=sysm.n1, n2=sysm.n2, n3=sysm.n3,
                    v_loc=sysm.v_loc, species=[], atom_species=np.zeros(0, np.int32), atom_z=np.zeros(0, np.int32),
                    atom_tau=np.zeros((0, 3)), ecut=sysm.ecut)
    kp = S.g_sphere(sysm.lattice, (0.1, -0.2, 0.3), sysm.ecut)
    rng = np.random.default_rng(nb)
    psi = rng.standard_normal((nb, kp.npw)) + 1j * rng.standard_normal((nb, kp.npw))
    low = kp.kinetic < 0.3 * kp.kinetic.max()
    psi[0::2] *= np.where(low, 1.0, tiny)
    psi[1::2] *= np.where(low, tiny * tiny, 1.0)
    with Hamiltonian(sysm) as H:
        H.set_kpoint(0, kp)
        m = H.velocity_matrix(0, nb, psi, precision="fp64")
    for a in range(3):
        g = kp.kvec[:, a] * psi
        want = (psi.conj().astype(np.clongdouble)[:, None, :] * g[None]).sum(-1)
        size = np.abs(psi) @ np.abs(g).T
        assert (np.abs(m[a] - want) <= TOL * size).all()
