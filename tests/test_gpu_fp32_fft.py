"""FP32 local term (csrc/local.cu) against numpy's complex128 transforms on grids
that mix compile-time plans of two and three stages, with lengths that the x
pass's column tiles do not divide, and with planes whose rows are all in use.

Tolerance: complex64 transforms of N points carry about eps log2(N) with eps =
2^-24, the 3-D round trip of V psi three times that: 19 x 3 x 6e-8 = 3.4e-6 for
the largest grid here; 5e-6 of the band's norm.
"""
import numpy as np
import pytest

from effmass_gb300 import system as S

pytestmark = pytest.mark.gpu
TOL = 5e-6
GRIDS = [(36, 64, 64), (64, 36, 36), (24, 32, 32), (32, 32, 64), (40, 40, 40), (30, 30, 30), (30, 60, 60), (60, 30, 30),
         (48, 48, 48), (72, 60, 60), (60, 72, 72), (7, 48, 48), (20, 24, 24), (30, 30, 60), (36, 36, 72), (24, 24, 48)]


@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("n", GRIDS)
def test_fp32_local_term(n, full):
    from effmass_gb300 import build
    from effmass_gb300.hamiltonian import Hamiltonian
    build.build()
    rng = np.random.default_rng(7)
    lat = np.diag([5.0 + m for m in n])
    v = rng.standard_normal(n)
    sysm = S.System(name="box", lattice=lat, omega=float(np.linalg.det(lat)), n1=n[0], n2=n[1], n3=n[2],
                    v_loc=v.reshape(-1), species=[], atom_species=np.zeros(0, np.int32), atom_z=np.zeros(0, np.int32),
                    atom_tau=np.zeros((0, 3)), ecut=1.0)
    reach = [m // 2 - 1 if full else m // 4 for m in n]
    g = np.stack(np.meshgrid(*[np.arange(-r, r + 1) for r in reach], indexing="ij"), -1).reshape(-1, 3)
    g = g[rng.permutation(len(g))[:6000]]
    kp = S.KPoint(npw=len(g), k_frac=np.zeros(3), g_idx=np.ascontiguousarray(g, dtype=np.int32),
                  kvec=np.ascontiguousarray(g, dtype=np.float64), kinetic=rng.uniform(0.0, 2.0, len(g)))
    psi = rng.standard_normal((5, len(g))) + 1j * rng.standard_normal((5, len(g)))
    at = tuple(g[:, d] % n[d] for d in range(3))
    ref = []
    for c in psi:
        G = np.zeros(n, complex)
        G[at] = c
        ref.append(kp.kinetic * c + np.fft.fftn(v * np.fft.ifftn(G))[at])
    ref = np.stack(ref)
    with Hamiltonian(sysm) as H:
        H.set_kpoint(0, kp)
        for call in (lambda o: H.apply(0, 5, psi, o, "fp32"), lambda o: H.apply_energies(0, 5, psi, o, "fp32")):
            out = np.zeros_like(psi)
            call(out)
            err = np.linalg.norm(out - ref, axis=1) / np.linalg.norm(ref, axis=1)
            assert err.max() <= TOL, err
