"""Calls captured into a CUDA graph before the projector rows they need are built.

What a capture records has not run when the capture ends, so the next eager call
must build for itself, and a replay must give the same.  Every result is compared
bit for bit with a context that makes only eager calls (the same kernels on the
same inputs).
"""
import numpy as np
import pytest

from effmass_gb300 import abi
from effmass_gb300 import system as S

pytestmark = pytest.mark.gpu
K = ((0.1, -0.2, 0.3), (0.2, 0.1, -0.4))


def _context():
    from effmass_gb300 import build
    from effmass_gb300.hamiltonian import Hamiltonian
    build.build()
    sysm = S.make_system("tinyd")
    kps = [S.g_sphere(sysm.lattice, k, sysm.ecut) for k in K]
    H = Hamiltonian(sysm)
    for i, kp in enumerate(kps):
        H.set_kpoint(i, kp)
    return H, kps


def _bands(kps):
    import torch
    return [torch.from_numpy(S.make_bands(kp, 6, seed=3)).cuda() for kp in kps]


def _grad(H, kid, psi, prec):
    import torch
    from effmass_gb300.hamiltonian import GradHPsi
    g = torch.zeros((3,) + tuple(psi.shape), dtype=psi.dtype, device=psi.device)
    return g, lambda: H.grad_apply(kid, psi.shape[0], psi, GradHPsi(g[0], g[1], g[2]), prec)


def _apply(H, kid, psi, prec):
    import torch
    h = torch.zeros_like(psi)
    return h, lambda: H.apply(kid, psi.shape[0], psi, h, prec)


def _capture(call):
    import torch
    st, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        graph.capture_begin(capture_error_mode="thread_local")
        call()
        graph.capture_end()
    return graph


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("first,captured", [(_apply, _grad), (_grad, _apply)])
def test_first_use_captured(prec, first, captured):
    torch = pytest.importorskip("torch")
    F, kps = _context()
    psi = _bands(kps)
    want = []
    for op in (_apply, _grad):
        out, call = op(F, 0, psi[0], prec)
        call()
        want.append(out)
    torch.cuda.synchronize()
    F.close()
    expected = want[0 if captured is _apply else 1]

    H, _ = _context()
    H.set_kpoint(0, kps[1])  # an earlier binding of slot 0 that built everything
    for op in (_grad, _apply):
        for kid in (0, 1):
            op(H, kid, psi[1], prec)[1]()
    H.set_kpoint(0, kps[0])
    first(H, 0, psi[0], prec)[1]()
    out, call = captured(H, 0, psi[0], prec)
    graph = _capture(call)
    assert not torch.any(out)
    eager, call = captured(H, 0, psi[0], prec)
    call()
    torch.cuda.synchronize()
    assert torch.equal(eager, expected)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, expected)
    H.close()


def test_tensor_core_tables_are_not_built_inside_a_capture():
    """Their build reads host tables of the call: refused, and the capture goes on."""
    torch = pytest.importorskip("torch")
    from effmass_gb300._lib import HpsiError
    H, kps = _context()
    psi = _bands(kps)
    for kid in (0, 1):
        _apply(H, kid, psi[kid], "tc")[1]()
    H.set_kpoint(0, kps[0])  # the tables' buffer is free for the next binding
    out, call = _apply(H, 0, psi[0], "tc")
    mark = torch.zeros(4, device="cuda")

    def refused():
        mark.add_(1.0)
        with pytest.raises(HpsiError) as ei:
            call()
        assert ei.value.status == abi.HPSI_ERR_STATE

    graph = _capture(refused)
    graph.replay()
    call()
    eager, again = _apply(H, 0, psi[0], "tc")
    again()
    torch.cuda.synchronize()
    assert torch.all(mark == 1.0) and torch.any(out) and torch.equal(out, eager)
    assert np.isfinite(out.cpu().numpy()).all()
    H.close()
