"""FP64 nonlocal sums of p and d projectors with smooth bands, whose scales are those of
the s projectors at small |k+G| (3 to 5 bits above the sums' own terms, as in
silicon-like cells), against the SIMT FP64 GEMMs, which the context runs when it is
granted no room for digits.

Tolerance: a SIMT sum in chains of at most 192 terms is rounded to sqrt(192) 2^-53 =
1.5e-15 of the 2-norm of its terms, which is about the size of a sum of random terms;
the digit-sliced sums have to be as good: 3e-15 of a band's result.
"""
import numpy as np
import pytest

from effmass_gb300 import system as S

pytestmark = pytest.mark.gpu
TOL = 3e-15
Q = 0.01 * np.arange(1300)


@pytest.mark.parametrize("l", [1, 2])
@pytest.mark.parametrize("steep", [1.0, 2.0, 3.0])
def test_nonlocal_term_as_accurate_as_simt(l, steep):
    from effmass_gb300 import build
    from effmass_gb300._lib import load
    from effmass_gb300.hamiltonian import Hamiltonian
    build.build()
    # the s projector is weak, so that the others' sums are not hidden behind its own
    e = np.exp(-Q * Q / 4)
    beta = np.stack([e, Q ** l * e])
    dbeta = np.stack([-0.5 * Q * e, (l * Q ** (l - 1) - 0.5 * Q ** (l + 1)) * e])
    sp = S.Species(z=14, proj_l=np.array([0, l], np.int32), lam=np.array([1e-12, 1.0]), dq=0.01, q_max=12.0,
                   beta_q=beta, dbeta_q=dbeta)
    sysm = S.System(name="two", lattice=10.26 * np.eye(3), omega=10.26 ** 3, n1=24, n2=24, n3=24,
                    v_loc=np.zeros(24 ** 3), species=[sp], atom_species=np.zeros(1, np.int32),
                    atom_z=np.full(1, 14, np.int32), atom_tau=np.zeros((1, 3)), ecut=18.0)
    kp = S.g_sphere(sysm.lattice, (0.02, 0.01, 0.03), 18.0)
    rng = np.random.default_rng(3)
    psi = rng.standard_normal((64, kp.npw)) + 1j * rng.standard_normal((64, kp.npw))
    psi /= (1.0 + 2.0 * kp.kinetic) ** steep
    kp.kinetic[:] = 0.0
    out = []
    with Hamiltonian(sysm) as H:
        H.set_kpoint(0, kp)
        for room in (-1, 0):
            assert load().hpsi_selftest_memory(H.ctx, room, 0) == 0
            h = np.zeros_like(psi)
            H.apply(0, len(psi), psi, h, "fp64")
            out.append(h)
    err = np.linalg.norm(out[0] - out[1], axis=1) / np.linalg.norm(out[1], axis=1)
    assert err.max() <= TOL, (err.max(), np.sqrt((err ** 2).mean()))
