"""FP64 nonlocal sums whose two operands are large at different places: projectors of
two radii with bands at high |G| (the wide one has decayed there, the narrow one has
not), strengths that differ by many orders, and bands whose coefficients do.  The
digit split (csrc/d64_gemm.cu) would lose the small terms; it forms such sums in FP64.

The reference is the same call on the SIMT FP64 GEMMs, which the context runs when it
is granted no room for digits.  V_loc and the kinetic energies are zero, so that the
nonlocal term stands alone, and results are compared shell by shell in |k+G|, so that
no component hides behind a larger one.  Tolerance: 1e-13 per sum (test_gpu_fp64_tc.py)
and what the digits may lose, 4 bits of that: 16e-13.
"""
import numpy as np
import pytest

from effmass_gb300 import system as S

pytestmark = pytest.mark.gpu
TOL = 16e-13
Q = 0.01 * np.arange(1300)


def _system(radii, lam, natom):
    beta, dbeta, ls = [], [], []
    for l in (0, 1):
        for r in radii:
            e = np.exp(-Q * Q * r * r / 4)
            beta.append(Q ** l * e)
            dbeta.append((l - 0.5 * r * r * Q ** (l + 1)) * e if l == 0 else (1 - 0.5 * r * r * Q * Q) * e)
            ls.append(l)
    sp = S.Species(z=14, proj_l=np.array(ls, np.int32), lam=np.array(lam * 2, float), dq=0.01, q_max=12.0,
                   beta_q=np.stack(beta), dbeta_q=np.stack(dbeta))
    lat = 10.26 * np.eye(3)
    tau = np.random.default_rng(1).random((natom, 3))
    sysm = S.System(name="two", lattice=lat, omega=10.26 ** 3, n1=24, n2=24, n3=24, v_loc=np.zeros(24 ** 3),
                    species=[sp], atom_species=np.zeros(natom, np.int32), atom_z=np.full(natom, 14, np.int32),
                    atom_tau=tau, ecut=18.0)
    kp = S.g_sphere(lat, (0.1, 0.2, 0.05), 18.0)
    kp.kinetic[:] = 0.0
    return sysm, kp


def _bands(kp, nb, kind):
    rng = np.random.default_rng(nb)
    q = np.linalg.norm(kp.kvec, axis=1)
    psi = rng.standard_normal((nb, kp.npw)) + 1j * rng.standard_normal((nb, kp.npw))
    if kind == "high":
        return psi * (q > 5.0)
    if kind == "low":
        return psi * np.exp(-q * q)
    return psi * 10.0 ** (-10.0 * rng.random(nb)[:, None] * q[None, :] / q.max())


def _near(a, b, q):
    """every shell of every band"""
    for lo in np.arange(0.0, q.max(), 0.5):
        s = (q >= lo) & (q < lo + 0.5)
        err, size = np.linalg.norm((a - b)[..., s], axis=-1), np.linalg.norm(b[..., s], axis=-1)
        assert (err <= TOL * size).all(), (lo, (err / np.maximum(size, 1e-300)).max())


@pytest.mark.parametrize("kind", ["high", "low", "mixed"])
@pytest.mark.parametrize("radii,lam,natom,nb", [((0.8, 1.8), [1e-6, 1.0], 2, 4), ((0.8, 1.8), [1e-13, 1.0], 17, 17),
                                                ((1.0, 1.5), [1.0, 1e-9], 9, 33), ((0.7, 2.5), [1.0, 1.0], 5, 1),
                                                ((0.8, 1.8), [1e-6, 1.0], 3, 300)])
def test_sums_of_mismatched_scales(radii, lam, natom, nb, kind):
    pytest.importorskip("torch")
    from effmass_gb300 import build
    from effmass_gb300._lib import load
    from effmass_gb300.hamiltonian import GradHPsi, Hamiltonian
    build.build()
    sysm, kp = _system(radii, lam, natom)
    psi = _bands(kp, nb, kind)
    q = np.linalg.norm(kp.kvec, axis=1)
    got = []
    with Hamiltonian(sysm) as H:
        H.set_kpoint(0, kp)
        for room in (-1, 0):
            assert load().hpsi_selftest_memory(H.ctx, room, 0) == 0
            h, g = np.zeros_like(psi), np.zeros((3,) + psi.shape, dtype=np.complex128)
            e = H.apply_energies(0, nb, psi, h, "fp64")
            H.grad_apply(0, nb, psi, GradHPsi(g[0], None, g[2]), "fp64")
            got.append((h, g - kp.kvec.T[:, None, :] * psi * np.array([1, 0, 1])[:, None, None], e))
    (h, g, e), (hr, gr, er) = got
    _near(h, hr, q)
    assert (np.abs(e - er) <= TOL * np.abs(er)).all()
    # what the kinetic part leaves: it is rounded to 2^-53 of itself
    full = np.abs(kp.kvec.T[:, None, :] * psi)
    s = np.linalg.norm(g - gr, axis=-1)
    assert (s <= TOL * np.linalg.norm(gr, axis=-1) + 2.0 ** -51 * np.linalg.norm(full, axis=-1)).all()
    quiet = (np.abs(psi) == 0).all(axis=0)  # G without kinetic part
    if quiet.any():
        _near(g[..., quiet][[0, 2]], gr[..., quiet][[0, 2]], q[quiet])
