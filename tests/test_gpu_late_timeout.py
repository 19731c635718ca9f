"""A bounded wait that gives up in a call that does not synchronise is reported by
the next call that does, whichever it is, and once.  The wait runs out by the test
hook of test_gpu_timeout.py: nothing is faulted."""
import numpy as np
import pytest

from effmass_gb300 import abi
from effmass_gb300 import system as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("reporter", ["density", "hessian", "apply"])
def test_timeout_of_an_asynchronous_fp64_call(reporter):
    torch = pytest.importorskip("torch")
    from effmass_gb300 import build
    from effmass_gb300._lib import HpsiError, load
    from effmass_gb300.hamiltonian import Hamiltonian
    build.build()
    sysm = S.make_system("sc8")
    kp = S.g_sphere(sysm.lattice, (0.1, -0.2, 0.3), sysm.ecut)
    psi = S.make_bands(kp, 4)
    dev = torch.from_numpy(psi).cuda()
    with Hamiltonian(sysm) as H:
        H.set_kpoint(0, kp)
        hess = np.zeros_like(psi)
        if reporter == "hessian":
            sp = sysm.species[0]
            q = np.arange(sp.beta_q.shape[1])
            H.set_hessian_tables(0, np.zeros((3, sp.beta_q.shape[0], len(q))), sp.dq)

        def report():
            if reporter == "density":
                H.density(0, 4, psi, np.ones(4), precision="fp32")
            elif reporter == "hessian":
                H.hess_apply(0, 4, psi, {"xx": hess}, "fp32")
            else:
                H.apply(0, 4, psi, np.zeros_like(psi), "fp32")

        report()
        try:
            assert load().hpsi_selftest_wait_limit(0) == abi.HPSI_OK
            H.apply(0, 4, dev, torch.zeros_like(dev), "fp64")
            torch.cuda.synchronize()
        finally:
            assert load().hpsi_selftest_wait_limit(-1) == abi.HPSI_OK
        with pytest.raises(HpsiError) as ei:
            report()
        assert ei.value.status == abi.HPSI_ERR_TIMEOUT
        report()
