"""FP64 calls with the projection chain on the side stream (default) and on the caller's
(HPSI_ONE_STREAM): the same kernels on the same inputs, so the same bits.  With
HPSI_ONE_STREAM nothing is queued on another stream, also where two G share a grid
point and the energies come from a second product: a captured call is one chain."""
import ctypes as C

import numpy as np
import pytest

from conftest import load_case
from effmass_gb300 import abi

pytestmark = pytest.mark.gpu


def _calls(H, psi, prec, one):
    import torch
    from effmass_gb300._lib import load
    h, e = torch.zeros_like(psi), torch.zeros(psi.shape[0], dtype=torch.float64, device="cuda")
    f = abi.PRECISIONS[prec] | abi.HPSI_DEVICE_PTRS | (abi.HPSI_ONE_STREAM if one else 0)
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    nb = psi.shape[0]
    assert load().hpsi_apply(H.ctx, 0, nb, psi.data_ptr(), h.data_ptr(), f, st) == 0
    assert load().hpsi_apply_energies(H.ctx, 0, nb, psi.data_ptr(), h.data_ptr(), e.data_ptr(), f, st) == 0
    return h, e


@pytest.mark.parametrize("name", ["tinyd", "sc8", "alias"])
def test_side_stream_equals_one_stream(name):
    torch = pytest.importorskip("torch")
    from effmass_gb300 import build
    from effmass_gb300.hamiltonian import Hamiltonian
    build.build()
    sysm, kp, psi, _, _ = load_case(name)
    with Hamiltonian(sysm) as H:
        H.set_kpoint(0, kp)
        p = torch.from_numpy(np.ascontiguousarray(psi)).cuda()
        for prec in ("fp64", "fp32", "tc"):
            a, b = _calls(H, p, prec, False), _calls(H, p, prec, True)
            torch.cuda.synchronize()
            assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
            assert torch.any(a[0])


@pytest.mark.parametrize("name", ["sc8", "alias"])
@pytest.mark.parametrize("prec", ["fp64", "fp32", "tc"])
def test_one_stream_is_one_chain(name, prec):
    torch = pytest.importorskip("torch")
    from effmass_gb300 import build
    from effmass_gb300._lib import load
    from effmass_gb300.hamiltonian import Hamiltonian
    build.build()
    cuda = C.CDLL("libcuda.so.1")
    sysm, kp, psi, _, _ = load_case(name)
    with Hamiltonian(sysm) as H:
        H.set_kpoint(0, kp)
        p = torch.from_numpy(np.ascontiguousarray(psi)).cuda()
        h, e = _calls(H, p, prec, True)
        torch.cuda.synchronize()
        st = C.c_void_p(torch.cuda.Stream().cuda_stream)
        flags = abi.PRECISIONS[prec] | abi.HPSI_DEVICE_PTRS | abi.HPSI_ONE_STREAM
        graph, nodes, edges = C.c_void_p(), C.c_size_t(), C.c_size_t()
        assert cuda.cuStreamBeginCapture_v2(st, 1) == 0  # thread-local
        rc = load().hpsi_apply_energies(H.ctx, 0, p.shape[0], p.data_ptr(), h.data_ptr(), e.data_ptr(), flags, st)
        assert cuda.cuStreamEndCapture(st, C.byref(graph)) == 0 and rc == 0
        assert cuda.cuGraphGetNodes(graph, None, C.byref(nodes)) == 0
        # a work node has its predecessor in the chain; events add none on one stream
        assert cuda.cuGraphGetEdges_v2(graph, None, None, None, C.byref(edges)) == 0
        assert nodes.value > 3 and edges.value == nodes.value - 1
        assert cuda.cuGraphDestroy(graph) == 0
