"""A server lane runs its calls on one stream, so a job needs the larger of the
local and the nonlocal workspace, not both: an FP32 job whose budget is its bands
and its transforms is admitted."""
import numpy as np
import pytest

from conftest import rel_err
from effmass_gb300 import system as S

pytestmark = pytest.mark.gpu


def test_fp32_job_fits_bands_and_transforms():
    from effmass_gb300 import build
    from effmass_gb300.hamiltonian import Hamiltonian
    from effmass_gb300.serving import Job, Server
    build.build()
    sysm = S.make_system("sc8")
    kp = S.g_sphere(sysm.lattice, (0.1, -0.2, 0.3), sysm.ecut)
    nb = 48
    psi = S.make_bands(kp, nb)
    planes = len(np.unique(kp.g_idx[:, 0] % sysm.n1))
    up = lambda b: -(-b // 256) * 256  # noqa: E731
    need = 2 * up(16 * nb * kp.npw) + up(8 * nb * planes * sysm.n2 * sysm.n3)
    with Hamiltonian(sysm) as H:
        H.set_kpoint(0, kp)
        want = np.zeros_like(psi)
        H.apply(0, nb, psi, want, "fp64")
        with Server([H], lanes=1, budget_gb=need / 2 ** 30, precision="fp32") as srv:
            out = np.zeros_like(psi)
            srv.wait(srv.submit([Job(0, 0, psi, out, None)]))
            assert srv.stats()["peak_bytes"] == need
    assert rel_err(out, want) <= 1e-6
