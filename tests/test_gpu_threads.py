"""GPU test of calls from several host threads at once, each with its own stream, workspace and molecule, so
that their kernels' shared-memory sizes differ: every call succeeds and gives what it gives alone."""
import ctypes
import threading

import pytest
import torch

from deeperwin_gb300 import _lib, api, arch as A, params as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("energy", [False, True])
def test_threads_with_different_shapes(cuda, prec, energy):
    L = _lib.lib()
    states = []
    for mol, B in ((A.lih(), 1), (A.h_chain(10), 3), (A.c2h4_shaped(), 2), (A.scale_molecule(5), 1)):
        a = A.arch_for(mol, 4)
        params = api.Params.from_dict(a, P.init_params(a, 0, bias_std=0.1), prec)
        r = torch.as_tensor(A.init_walkers(mol, B, seed=3).astype("float32"), device="cuda")
        R, Z = api._geometry(mol.R, mol.Z, torch.device("cuda"))
        nb = L.dw_workspace_bytes(ctypes.byref(params.c_arch), params.prec, B, int(energy))
        ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
        states.append((params, r, R, Z, ws, torch.empty(B, device="cuda"), torch.empty(B, device="cuda"), torch.cuda.Stream()))

    def call(state):
        params, r, R, Z, ws, lp, E, stream = state
        args = (ctypes.byref(params.c_arch), params.prec, api._ptr(params.flat), api._ptr(params.prepared), api._ptr(r),
                len(r), api._ptr(R), api._ptr(Z))
        tail = (api._ptr(ws), ws.numel(), ctypes.c_void_p(stream.cuda_stream))
        if energy:
            return L.dw_local_energy(*args, api._ptr(E), api._ptr(lp), None, *tail)
        return L.dw_log_psi_sqr(*args, api._ptr(lp), None, *tail)

    alone = []
    for s in states:
        torch.cuda.synchronize()
        assert call(s) == 0
        torch.cuda.synchronize()
        alone.append((s[5].cpu(), s[6].cpu()))
    failed, different = [0] * len(states), [0] * len(states)

    def work(k):
        s = states[k]
        for _ in range(400 if prec != "fp64" else 60):
            failed[k] += call(s) != 0
            s[7].synchronize()
            different[k] += not torch.equal(s[5].cpu(), alone[k][0])
            if energy:
                different[k] += not torch.equal(s[6].cpu(), alone[k][1])

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(states))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert failed == [0] * len(states) and different == [0] * len(states), (failed, different)


def test_fp64_inverse_under_contention(cuda):
    """Inverses and log|det| of the FP64 determinant algebra while other streams' blocks share the SMs, so that the
    warps of a block run far apart: the same bits on every call."""
    L = _lib.lib()
    mol = A.scale_molecule(5)
    a = A.arch_for(mol, 4)
    params = api.Params.from_dict(a, P.init_params(a, 0, bias_std=0.1), "fp32_det64")
    r = torch.as_tensor(A.init_walkers(mol, 1, seed=3).astype("float32"), device="cuda")
    R, Z = api._geometry(mol.R, mol.Z, torch.device("cuda"))
    nb = L.dw_workspace_bytes(ctypes.byref(params.c_arch), params.prec, 1, 1)
    states = [(torch.empty(nb, dtype=torch.uint8, device="cuda"), torch.empty(1, device="cuda"), torch.empty(1, device="cuda"),
               torch.cuda.Stream()) for _ in range(4)]
    torch.cuda.synchronize()

    def call(s):
        return L.dw_local_energy(ctypes.byref(params.c_arch), params.prec, api._ptr(params.flat), api._ptr(params.prepared),
                                 api._ptr(r), 1, api._ptr(R), api._ptr(Z), api._ptr(s[1]), api._ptr(s[2]), None, api._ptr(s[0]),
                                 nb, ctypes.c_void_p(s[3].cuda_stream))

    assert call(states[0]) == 0
    torch.cuda.synchronize()
    alone = [states[0][1].item(), states[0][2].item()]
    wrong = []

    def work(s):
        for _ in range(2000):
            status = call(s)
            s[3].synchronize()
            got = [s[1].item(), s[2].item()]
            if status or got != alone:
                wrong.append((status, got))

    threads = [threading.Thread(target=work, args=(s,)) for s in states]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, (len(wrong), wrong[:4], alone)


def test_refused_launch_is_reported(cuda):
    """A launch that fails is an error of the call that made it, whatever the call does next, and of no later call."""
    L = _lib.lib()
    E = torch.zeros(8, device="cuda")
    out = torch.empty(3, dtype=torch.float64, device="cuda")
    for _ in range(2):
        assert L.dw_debug_refused_launch(None) == 4          # DW_ERR_CUDA
        assert L.dw_energy_stats(api._ptr(E), 8, api._ptr(out), None) == 0
    torch.cuda.synchronize()
