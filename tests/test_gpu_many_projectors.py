"""dH/dk of a cell with 16400 projectors (65600 rows with the derivatives) in FP64.

The projector part is a sum over atoms: the gradient of all atoms is that of
the two halves together, less one kinetic term.  Tolerance: sums of K = 2 P terms
are each off by K 2^-53 = 4e-12 of the sum of absolute products at most.
"""
import numpy as np
import pytest

from effmass_gb300 import system as S

pytestmark = pytest.mark.gpu
TOL = 4e-12


def test_fp64_gradient_of_many_projectors():
    from effmass_gb300 import build
    from effmass_gb300.hamiltonian import GradHPsi, Hamiltonian
    build.build()
    rng = np.random.default_rng(11)
    lat, n, natom = 9.0 * np.eye(3), 12, 4100
    q = 0.01 * np.arange(1200)
    beta = np.stack([np.exp(-q * q / 4), q * np.exp(-q * q / 4)])
    dbeta = np.stack([-0.5 * q * beta[0], (1 - 0.5 * q * q) * np.exp(-q * q / 4)])
    sp = S.Species(z=6, proj_l=np.array([0, 1], np.int32), lam=np.array([0.7, -0.4]), dq=0.01, q_max=11.0, beta_q=beta,
                   dbeta_q=dbeta)
    tau = rng.random((natom, 3))
    kp = S.g_sphere(lat, (0.1, -0.2, 0.3), 3.0)
    psi = S.make_bands(kp, 2)

    def grad(t):
        sysm = S.System(name="many", lattice=lat, omega=729.0, n1=n, n2=n, n3=n, v_loc=np.zeros(n ** 3), species=[sp],
                        atom_species=np.zeros(len(t), np.int32), atom_z=np.full(len(t), 6, np.int32),
                        atom_tau=np.ascontiguousarray(t), ecut=3.0)
        g = np.zeros((3,) + psi.shape, dtype=np.complex128)
        with Hamiltonian(sysm) as H:
            H.set_kpoint(0, kp)
            H.grad_apply(0, 2, psi, GradHPsi(g[0], g[1], g[2]), "fp64")
        return g

    kinetic = kp.kvec.T[:, None, :] * psi[None]
    want = grad(tau[::2]) + grad(tau[1::2]) - kinetic
    got = grad(tau)
    assert np.linalg.norm(got - want) <= TOL * np.linalg.norm(want)
