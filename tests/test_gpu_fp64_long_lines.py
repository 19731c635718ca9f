"""FP64 local term on grids with an axis of hundreds of points: bands whose lines
are flat, decay, or have one large coefficient, against long double transforms.

Tolerance: complex128 transforms of n points carry about 2^-53 log2(n), 1e-15 for the
longest axis here.
"""
import numpy as np
import pytest

from effmass_gb300 import system as S

pytestmark = pytest.mark.gpu
TOL = 1e-15
GRIDS = [(182, 4, 3), (500, 2, 3), (512, 3, 2), (2, 500, 8), (2, 8, 500), (4, 363, 6), (3, 6, 400), (1, 1, 490)]


def _case(n):
    rng = np.random.default_rng(sum(n))
    g = np.stack(np.meshgrid(*[np.arange(-(m // 4), m // 4 + 1) if m > 2 else np.array([0]) for m in n], indexing="ij"),
                 -1).reshape(-1, 3)
    big = int(np.argmax(n))
    rnd = rng.standard_normal(len(g)) + 1j * rng.standard_normal(len(g))
    psi = np.stack([rnd, rnd * np.where((g == 0).all(1), 1.0, 1e-9), rnd * np.exp(-0.5 * np.abs(g[:, big])),
                    rnd / np.abs(rnd)])
    v = rng.standard_normal(n)
    sysm = S.System(name="long", lattice=np.diag([5.0 + m for m in n]), omega=float(np.prod([5.0 + m for m in n])),
                    n1=n[0], n2=n[1], n3=n[2], v_loc=v.reshape(-1), species=[], atom_species=np.zeros(0, np.int32),
                    atom_z=np.zeros(0, np.int32), atom_tau=np.zeros((0, 3)), ecut=1.0)
    kp = S.KPoint(npw=len(g), k_frac=np.zeros(3), g_idx=np.ascontiguousarray(g, dtype=np.int32),
                  kvec=np.ascontiguousarray(g, dtype=np.float64), kinetic=np.zeros(len(g)))
    return sysm, kp, v, psi


@pytest.mark.parametrize("n", GRIDS)
def test_fp64_local_term_of_long_lines(n):
    from effmass_gb300 import build
    from effmass_gb300.hamiltonian import Hamiltonian
    build.build()
    sysm, kp, v, psi = _case(n)
    at = tuple(kp.g_idx[:, d] % n[d] for d in range(3))
    with Hamiltonian(sysm) as H:
        H.set_kpoint(0, kp)
        out, again = np.zeros_like(psi), np.zeros_like(psi)
        H.apply(0, len(psi), psi, out, "fp64")
        H.apply(0, len(psi), psi, again, "fp64")
        rho = H.density(0, 1, psi[1:2], np.ones(1))
    assert np.array_equal(out, again)
    for b, c in enumerate(psi):
        grid = np.zeros(n, np.clongdouble)
        grid[at] = c
        r = np.fft.ifftn(grid)
        want = np.fft.fftn(v.astype(np.longdouble) * r)[at]
        err = np.sqrt((np.abs(out[b] - want) ** 2).sum() / (np.abs(want) ** 2).sum())
        assert err <= TOL, (b, float(err))
        if b == 1:
            want = np.abs(r * np.longdouble(np.prod(n))) ** 2
            assert np.sqrt(((rho - want) ** 2).sum() / (want ** 2).sum()) <= 2 * TOL


@pytest.mark.parametrize("n", [(128, 4, 4), (4, 128, 4), (4, 4, 128), (160, 3, 4), (4, 176, 4), (180, 4, 4), (4, 4, 144)])
def test_fp64_local_term_of_middling_lines(n):
    """Three axes, each rounded to about 2^-53 of its lines' norm: 4e-16."""
    from effmass_gb300 import build
    from effmass_gb300.hamiltonian import Hamiltonian
    build.build()
    sysm, kp, v, psi = _case(n)
    at = tuple(kp.g_idx[:, d] % n[d] for d in range(3))
    out = np.zeros_like(psi)
    with Hamiltonian(sysm) as H:
        H.set_kpoint(0, kp)
        H.apply(0, len(psi), psi, out, "fp64")
    for b, c in enumerate(psi):
        grid = np.zeros(n, np.clongdouble)
        grid[at] = c
        want = np.fft.fftn(v.astype(np.longdouble) * np.fft.ifftn(grid))[at]
        err = np.sqrt((np.abs(out[b] - want) ** 2).sum() / (np.abs(want) ** 2).sum())
        assert err <= 4e-16, (b, float(err))
