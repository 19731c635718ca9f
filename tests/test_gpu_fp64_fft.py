"""FP64 local term (csrc/local64.cu, 64-bit fixed-point transforms) against numpy's
complex128 transforms, on grids of every radix, unequal axes, one-point axes and
the largest planes, for H|psi>, band energies and the density.

Tolerance: complex128 transforms of N points carry about eps log2(N) with eps =
2^-53, the 3-D round trip of V psi three times that: 19 x 3 x 1.1e-16 = 6e-15
for the largest grid here, and the fixed-point form is below it; 1e-14 of the
band's norm.
"""
import numpy as np
import pytest

from effmass_gb300 import system as S

pytestmark = pytest.mark.gpu
TOL = 1e-14
GRIDS = [(1, 1, 1), (2, 3, 4), (1, 8, 1), (5, 7, 9), (11, 13, 8), (26, 21, 22), (25, 27, 16), (512, 2, 3), (3, 500, 10),
         (10, 48, 50), (72, 36, 24), (9, 60, 64), (4, 84, 84), (6, 90, 78)]


def _case(n, seed=3, nb=5):
    rng = np.random.default_rng(seed)
    lat = np.diag([5.0 + n[0], 6.0 + n[1], 7.0 + n[2]])
    v = rng.standard_normal(n) * rng.uniform(0.0, 3.0, n)
    sysm = S.System(name="box", lattice=lat, omega=float(np.linalg.det(lat)), n1=n[0], n2=n[1], n3=n[2],
                    v_loc=v.reshape(-1), species=[], atom_species=np.zeros(0, np.int32), atom_z=np.zeros(0, np.int32),
                    atom_tau=np.zeros((0, 3)), ecut=1.0)
    # an ellipsoid of G-vectors (half of each axis), in random order
    ax = [np.arange(-(m // 4), m // 4 + 1) if m > 2 else np.array([0]) for m in n]
    g = np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    r = (g / np.maximum(1.0, np.array(n) / 4.0)) ** 2
    g = g[r.sum(1) <= 1.5]
    g = g[rng.permutation(len(g))]
    kin = rng.uniform(0.0, 2.0, len(g))
    kp = S.KPoint(npw=len(g), k_frac=np.zeros(3), g_idx=np.ascontiguousarray(g, dtype=np.int32),
                  kvec=np.ascontiguousarray(g, dtype=np.float64), kinetic=kin)
    psi = rng.standard_normal((nb, len(g))) + 1j * rng.standard_normal((nb, len(g)))
    psi *= np.exp(-rng.uniform(0.0, 30.0, nb)[:, None] * (g / (1.0 + np.array(n))).__pow__(2).sum(1)[None, :])
    return sysm, kp, v, psi


def _grid(n, kp, c):
    G = np.zeros(n, complex)
    G[tuple((kp.g_idx[:, d] % n[d]) for d in range(3))] = c
    return np.fft.ifftn(G) * np.prod(n)


def _apply(n, kp, v, psi):
    at = tuple((kp.g_idx[:, d] % n[d]) for d in range(3))
    return np.stack([kp.kinetic * c + (np.fft.fftn(v * _grid(n, kp, c)) / np.prod(n))[at] for c in psi])


@pytest.mark.parametrize("n", GRIDS)
def test_fp64_local_term(n):
    from effmass_gb300 import build
    from effmass_gb300.hamiltonian import Hamiltonian
    build.build()
    sysm, kp, v, psi = _case(n)
    scale = 2.0 ** np.array([0, 200, -300, 17, -5])[:, None]
    with Hamiltonian(sysm) as H:
        H.set_kpoint(0, kp)
        ref = _apply(n, kp, v, psi)
        for nb in (5, 1):
            out = np.zeros_like(psi[:nb])
            H.at_k(0)(nb, psi[:nb] * scale[:nb], out)
            err = np.linalg.norm(out / scale[:nb] - ref[:nb], axis=1) / np.linalg.norm(ref[:nb], axis=1)
            assert err.max() <= TOL, (nb, err)
        out2 = np.zeros_like(psi)
        e = H.apply_energies(0, 5, psi * scale[::-1], out2)
        plain = np.zeros_like(psi)
        H.at_k(0)(5, psi * scale[::-1], plain)
        assert np.array_equal(out2, plain)
        want = np.einsum("bg,bg->b", psi.conj(), ref).real * scale[::-1, 0] ** 2
        size = np.linalg.norm(psi, axis=1) * np.linalg.norm(ref, axis=1) * scale[::-1, 0] ** 2
        assert (np.abs(e - want) <= TOL * size).all()
        occ = np.array([2.0, 1.5, 0.0, 0.3, 1.0])
        rho = H.density(0, 5, psi, occ)
        want = sum(o * np.abs(_grid(n, kp, c)) ** 2 for o, c in zip(occ, psi))
        assert np.linalg.norm(rho - want) <= TOL * np.linalg.norm(want)


def test_fp64_local_nonfinite_and_zero_bands():
    from effmass_gb300 import build
    from effmass_gb300.hamiltonian import Hamiltonian
    build.build()
    n = (12, 15, 16)
    sysm, kp, v, psi = _case(n)
    ref = _apply(n, kp, v, psi)
    psi = psi.copy()
    psi[0] = 0
    psi[2, 7] = np.nan
    psi[4, 3] = 1j * np.inf
    with Hamiltonian(sysm) as H:
        H.set_kpoint(0, kp)
        out = np.zeros_like(psi)
        H.at_k(0)(5, psi, out)
    assert not out[0].any()
    assert np.isnan(out[2]).all() and not np.isfinite(out[4]).any()
    for b in (1, 3):
        assert np.linalg.norm(out[b] - ref[b]) <= TOL * np.linalg.norm(ref[b])
