"""FP32 projector sums below the normal float range."""
import numpy as np
import pytest

from effmass_gb300 import system as S

pytestmark = pytest.mark.gpu


def test_fp32_nonlocal_term_of_tiny_bands():
    """Contributions below the normal float range reach H|psi>.  Coefficients under 2^-14
    of one are rounded to zero with the bands on the way in, and sums near 2^-130 to
    2^-149: together far below the hundredth that is allowed."""
    from effmass_gb300 import build
    from effmass_gb300.hamiltonian import Hamiltonian
    build.build()
    sysm = S.make_system("tinyd")
    kp = S.g_sphere(sysm.lattice, (0.1, -0.2, 0.3), sysm.ecut)
    kp.kinetic[:] = 0.0
    sysm.v_loc[:] = 0.0
    sysm.species[0].lam = sysm.species[0].lam * 2.0 ** -12
    psi = S.make_bands(kp, 3)
    with Hamiltonian(sysm) as H:
        H.set_kpoint(0, kp)
        want, out = np.zeros_like(psi), np.zeros_like(psi)
        H.apply(0, 3, psi, want, "fp32")
        H.apply(0, 3, psi * 2.0 ** -112, out, "fp32")
    assert np.abs(want).max() < 2.0 ** -14  # so that the scaled result is below 2^-126
    assert np.linalg.norm(out * 2.0 ** 112 - want) <= 1e-2 * np.linalg.norm(want)
