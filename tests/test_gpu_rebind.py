"""Rebinding a k-point slot: its tables and projector buffers are kept for the
next binding, which must give what a fresh context gives, bit for bit.  And the
plane lists of a sphere with several G on one grid point (the last is
scattered, all gather), against numpy.
"""
import numpy as np
import pytest

from effmass_gb300 import system as S

pytestmark = pytest.mark.gpu


def _results(H, kid, kp, prec, grad_first):
    from effmass_gb300.hamiltonian import GradHPsi
    psi = S.make_bands(kp, 5, seed=kp.npw)
    h = np.zeros_like(psi)
    g = np.zeros((3,) + psi.shape, dtype=np.complex128)

    def grad():
        H.gradient().at_k(kid, precision=prec)(psi, GradHPsi(g[0], g[1], g[2]), n_bands=5)

    if grad_first:
        grad()
    H.at_k(kid, precision=prec)(5, psi, h)
    if not grad_first:
        grad()
    return h, g


@pytest.mark.parametrize("prec", ["fp64", "fp32", "tc"])
def test_rebound_slot_equals_fresh_context(prec):
    from effmass_gb300 import build
    from effmass_gb300.hamiltonian import Hamiltonian
    build.build()
    sysm = S.make_system("tinyd")
    # larger, smaller, much smaller (below half), larger again
    kps = [S.g_sphere(sysm.lattice, k, e) for k, e in (((0.1, -0.2, 0.3), 4.0), ((0.0, 0.0, 0.0), 5.0),
                                                       ((0.4, 0.1, 0.2), 4.9), ((0.2, 0.2, 0.0), 1.5),
                                                       ((0.1, 0.0, 0.3), 5.0))]
    with Hamiltonian(sysm) as H:
        for i, kp in enumerate(kps):
            H.set_kpoint(0, kp)
            got = _results(H, 0, kp, prec, i % 2 == 0)
            with Hamiltonian(sysm) as F:
                F.set_kpoint(0, kp)
                want = _results(F, 0, kp, prec, i % 2 == 1)
            for x, y in zip(got, want):
                assert np.array_equal(x, y), i


@pytest.mark.parametrize("n", [(4, 5, 6), (3, 4, 9), (8, 8, 2)])
def test_aliased_sphere(n):
    from effmass_gb300 import build
    from effmass_gb300.hamiltonian import Hamiltonian
    build.build()
    rng = np.random.default_rng(5)
    ax = [np.arange(-(m // 2) - 4, m + 8 - m // 2 - 4) for m in n]  # every index the range check admits
    g = np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    g = g[rng.permutation(len(g))[: 3 * int(np.prod(n))]]
    v = rng.standard_normal(n)
    sysm = S.System(name="box", lattice=np.diag([5.0, 6.0, 7.0]), omega=210.0, n1=n[0], n2=n[1], n3=n[2],
                    v_loc=v.reshape(-1), species=[], atom_species=np.zeros(0, np.int32), atom_z=np.zeros(0, np.int32),
                    atom_tau=np.zeros((0, 3)), ecut=1.0)
    kin = rng.uniform(0.0, 2.0, len(g))
    kp = S.KPoint(npw=len(g), k_frac=np.zeros(3), g_idx=np.ascontiguousarray(g, dtype=np.int32),
                  kvec=np.ascontiguousarray(g, dtype=np.float64), kinetic=kin)
    psi = rng.standard_normal((3, len(g))) + 1j * rng.standard_normal((3, len(g)))
    at = tuple(g[:, d] % n[d] for d in range(3))
    want = np.empty_like(psi)
    for b in range(3):
        grid = np.zeros(n, complex)
        for i, c in enumerate(psi[b]):  # the last write wins
            grid[at[0][i], at[1][i], at[2][i]] = c
        want[b] = kin * psi[b] + np.fft.fftn(v * np.fft.ifftn(grid))[at]
    with Hamiltonian(sysm) as H:
        H.set_kpoint(0, kp)
        for prec, tol in (("fp64", 1e-14), ("fp32", 1e-6)):
            out = np.zeros_like(psi)
            H.at_k(0, precision=prec)(3, psi, out)
            assert np.linalg.norm(out - want) <= tol * np.linalg.norm(want)
