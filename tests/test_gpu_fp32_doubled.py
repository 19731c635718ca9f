"""FP32 local term (csrc/local.cu) of cells doubled along y, z or both, whose plane passes
take a compile-time plan per axis, against numpy's complex128 transforms.

Tolerance as in test_gpu_fp32_fft.py: three transforms of at most 2^18 points in
complex64, 3 x 18 x 6e-8 = 3.2e-6; 5e-6 of the band's norm.
"""
import numpy as np
import pytest

from effmass_gb300 import system as S

pytestmark = pytest.mark.gpu
TOL = 5e-6
GRIDS = [(36, 72, 36), (24, 48, 24), (32, 64, 32), (30, 60, 30), (20, 72, 36), (7, 36, 72), (60, 30, 60), (48, 64, 32),
         (36, 48, 72), (24, 24, 72)]


@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("n", GRIDS)
def test_fp32_local_term_of_doubled_cells(n, full):
    from effmass_gb300 import build
    from effmass_gb300.hamiltonian import Hamiltonian
    build.build()
    rng = np.random.default_rng(sum(n))
    v = rng.standard_normal(n)
    sysm = S.System(name="box", lattice=np.diag([5.0 + m for m in n]), omega=float(np.prod([5.0 + m for m in n])),
                    n1=n[0], n2=n[1], n3=n[2], v_loc=v.reshape(-1), species=[], atom_species=np.zeros(0, np.int32),
                    atom_z=np.zeros(0, np.int32), atom_tau=np.zeros((0, 3)), ecut=1.0)
    reach = [m // 2 - 1 if full else m // 4 for m in n]
    g = np.stack(np.meshgrid(*[np.arange(-r, r + 1) for r in reach], indexing="ij"), -1).reshape(-1, 3)
    g = g[rng.permutation(len(g))[:6000]]
    kp = S.KPoint(npw=len(g), k_frac=np.zeros(3), g_idx=np.ascontiguousarray(g, dtype=np.int32),
                  kvec=np.ascontiguousarray(g, dtype=np.float64), kinetic=rng.uniform(0.0, 2.0, len(g)))
    psi = rng.standard_normal((3, len(g))) + 1j * rng.standard_normal((3, len(g)))
    at = tuple(g[:, d] % n[d] for d in range(3))
    out = np.zeros_like(psi)
    with Hamiltonian(sysm) as H:
        H.set_kpoint(0, kp)
        H.apply(0, 3, psi, out, "fp32")
    for b, c in enumerate(psi):
        grid = np.zeros(n, complex)
        grid[at] = c
        want = kp.kinetic * c + np.fft.fftn(v * np.fft.ifftn(grid))[at]
        assert np.linalg.norm(out[b] - want) <= TOL * np.linalg.norm(want)
