"""FP64 calls where the device has no room for the digit slices of the tensor-core
GEMMs (csrc/d64_gemm.cu): they run the SIMT GEMMs, ask for the room once, keep
their workspace and stay capturable; and what is held for the slices goes back
when anything else finds no room.  Memory is short by a test hook of the context.

Tolerance between the two kinds of GEMM: 1e-13 of the result's norm, as derived
in test_gpu_fp64_tc.py.
"""
import ctypes as C

import numpy as np
import pytest

from effmass_gb300 import system as S

pytestmark = pytest.mark.gpu
TOL = 1e-13
NB = 48


class Case:
    def __init__(self):
        import torch
        from effmass_gb300 import build
        from effmass_gb300._lib import load
        from effmass_gb300.hamiltonian import Hamiltonian
        build.build()
        self.lib = load()
        self.sysm = S.make_system("sc8")
        self.kp = S.g_sphere(self.sysm.lattice, (0.1, -0.2, 0.3), self.sysm.ecut)
        self.H = Hamiltonian(self.sysm)
        self.H.set_kpoint(0, self.kp)
        self.psi = torch.from_numpy(S.make_bands(self.kp, NB)).cuda()

    def memory(self, room=-1, oom=0):
        assert self.lib.hpsi_selftest_memory(self.H.ctx, room, oom) == 0

    def state(self):
        out = (C.c_longlong * 5)()
        assert self.lib.hpsi_selftest_memory_state(self.H.ctx, out) == 0
        return list(out)

    def call(self, op):
        import torch
        from effmass_gb300.hamiltonian import GradHPsi
        H, psi = self.H, self.psi
        if op == "apply":
            out = torch.zeros_like(psi)
            return out, lambda: H.apply(0, NB, psi, out, "fp64")
        if op == "energies":
            out, e = torch.zeros_like(psi), torch.zeros(NB, dtype=torch.float64, device="cuda")
            return e, lambda: H.apply_energies(0, NB, psi, out, "fp64", e=e)
        if op == "grad":
            out = torch.zeros((3,) + tuple(psi.shape), dtype=psi.dtype, device="cuda")
            return out, lambda: H.grad_apply(0, NB, psi, GradHPsi(out[0], out[1], out[2]), "fp64")
        out = torch.zeros((3, NB, NB), dtype=psi.dtype, device="cuda")
        return out, lambda: H.velocity_matrix(0, NB, psi, out=out, precision="fp64")


def _near(a, b):
    import torch
    return float(torch.linalg.vector_norm(a - b)) <= TOL * float(torch.linalg.vector_norm(b))


@pytest.mark.parametrize("op", ["apply", "energies", "grad", "velocity"])
def test_no_room_for_the_slices(op):
    torch = pytest.importorskip("torch")
    c = Case()
    want, run = c.call(op)
    run()
    c.memory(room=0)
    outs, states = [], []
    for _ in range(3):
        out, run = c.call(op)
        run()
        torch.cuda.synchronize()
        outs.append(out)
        states.append(c.state())
    assert _near(outs[0], want)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    assert states[0][2] == 0 and states[0] == states[1] == states[2]  # one attempt, the workspace stays
    c.memory()
    out, run = c.call(op)
    run()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    c.H.close()


@pytest.mark.parametrize("op", ["apply", "grad"])
def test_warm_call_is_captured_without_the_slices(op):
    torch = pytest.importorskip("torch")
    c = Case()
    c.memory(room=0)
    want, run = c.call(op)
    run()
    for room in (0, -1):  # still no room; room again, which a capture cannot take
        c.memory(room=room)
        out, run = c.call(op)
        st, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.stream(st):
            graph.capture_begin(capture_error_mode="thread_local")
            run()
            graph.capture_end()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    c.H.close()


def test_slices_go_back_when_room_is_short():
    torch = pytest.importorskip("torch")
    c = Case()
    want, run = c.call("grad")
    run()
    torch.cuda.synchronize()
    assert c.state()[2] > 0
    c.memory(oom=1)
    c.H.set_kpoint(1, c.kp)  # its tables find no room at first
    assert c.state()[2] == 0
    out, run = c.call("grad")
    run()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    # in the middle of a call: the projector matrix of slot 1
    assert c.state()[2] > 0
    c.memory(oom=1)
    out = torch.zeros_like(c.psi)
    c.H.apply(1, NB, c.psi, out, "fp64")
    ref, run = c.call("apply")
    run()
    torch.cuda.synchronize()
    assert _near(out, ref) and np.isfinite(out.cpu().numpy()).all()
    c.H.close()
