"""FP32 projector GEMMs (csrc/gemm.cu) at the edges of their tiles, and the side stream of FP32 calls.

H|psi> in FP32 is compared with FP64 per band.  Tolerance: sums of K <= 3000
terms, each rounded to 24 bits, are off by sqrt(K) 2^-24 = 3e-6 of their
2-norm; ten times that, 3e-5, allows for cancellation in the expansion.  The
projection chain on the side stream adds the same terms in the same order as
on the caller's, so both give the same bits.
"""
import numpy as np
import pytest

from effmass_gb300 import system as S

pytestmark = pytest.mark.gpu
TOL = 3e-5


@pytest.mark.parametrize("name,nb", [("tiny", 1), ("tiny", 33), ("tinyd", 16), ("tinyd", 17), ("fcc2", 16), ("fcc2", 17),
                                     ("fcc2", 33), ("fcc2", 58), ("fcc2", 59), ("fcc2", 257), ("sc8", 4), ("sc8", 31),
                                     ("sc8", 48), ("sc8", 129)])
def test_fp32_apply(name, nb):
    torch = pytest.importorskip("torch")
    from effmass_gb300 import build
    from effmass_gb300.hamiltonian import Hamiltonian
    build.build()
    sysm = S.make_system(name)
    kp = S.g_sphere(sysm.lattice, (0.1, -0.2, 0.3), sysm.ecut)
    H = Hamiltonian(sysm)
    H.set_kpoint(0, kp)
    rng = np.random.default_rng(nb)
    psi = rng.standard_normal((nb, kp.npw)) + 1j * rng.standard_normal((nb, kp.npw))
    psi = torch.from_numpy(psi / (1.0 + kp.kinetic)).cuda()
    outs = []
    for prec, one in (("fp64", False), ("fp32", False), ("fp32", True)):
        out = torch.zeros_like(psi)
        H.apply(0, nb, psi, out, prec, one_stream=one)
        torch.cuda.synchronize()
        outs.append(out)
    ref, side, one = outs
    assert float((torch.linalg.norm(side - ref, dim=1) / torch.linalg.norm(ref, dim=1)).max()) <= TOL
    assert torch.equal(side, one)
    H.close()
