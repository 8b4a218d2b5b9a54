"""GPU test of workspaces between the least that the entry points take and what dw_workspace_bytes asks for: the
same energies from fewer walkers per chunk, without digit planes or without scratch for the digit tangents."""
import ctypes

import numpy as np
import pytest
import torch

from deeperwin_gb300 import _lib, api, arch as A, params as P

pytestmark = pytest.mark.gpu

DIGITS_RTOL = 2.4e-7       # outputs rounded to float32, of FP64 sums that round differently in their last bits


def _call(params, r, R, Z, nbytes, offset=0, mode=1):
    L = _lib.lib()
    B = len(r)
    room = torch.full((nbytes + 256,), 0xff, dtype=torch.uint8, device="cuda")
    ws = ctypes.c_void_p((room.data_ptr() + 255) // 256 * 256 + offset)
    E, lp = torch.full((B,), -7.0, device="cuda"), torch.full((B,), -7.0, device="cuda")
    g = torch.zeros(B, 3 * params.arch.n_el, device="cuda")
    args = (ctypes.byref(params.c_arch), params.prec, api._ptr(params.flat), api._ptr(params.prepared), api._ptr(r), B,
            api._ptr(R), api._ptr(Z))
    if mode:
        st = L.dw_local_energy(*args, api._ptr(E), api._ptr(lp), api._ptr(g), ws, nbytes, None)
    else:
        st = L.dw_log_psi_sqr(*args, api._ptr(lp), None, ws, nbytes, None)
    launches = L.dw_last_launch_count()
    torch.cuda.synchronize()
    assert L.dw_debug_tc_error_flag() == 0
    return st, E.double().cpu().numpy(), lp.double().cpu().numpy(), g.double().cpu().numpy(), launches


def _sizes(params, B, mode):
    L = _lib.lib()
    a = ctypes.byref(params.c_arch)
    return L.dw_workspace_bytes(a, params.prec, B, mode), L.dw_debug_workspace_least_bytes(a, params.prec, B, mode)


def _setup(mol, K, prec, B, seed=3):
    a = A.arch_for(mol, K)
    params = api.Params.from_dict(a, P.init_params(a, 5, bias_std=0.1, envelope_jitter=0.2), prec)
    r = torch.as_tensor(A.init_walkers(mol, B, seed=seed).astype(np.float32), device="cuda")
    R, Z = api._geometry(mol.R, mol.Z, torch.device("cuda"))
    return params, r, R, Z


@pytest.mark.parametrize("name,K,B", [("lih", 8, 1), ("lih", 8, 37), ("c2h4", 4, 21), ("s40", 3, 3)])
@pytest.mark.parametrize("mode", [0, 1])
def test_fp64_form(cuda, name, K, B, mode):
    mol = {"lih": A.lih, "c2h4": A.c2h4_shaped, "s40": A.scale_molecule}[name]()
    params, r, R, Z = _setup(mol, K, "fp64", B)
    full, least = _sizes(params, B, mode)
    st, E, lp, g, _ = _call(params, r, R, Z, full, 0, mode)
    assert st == 0 and np.all(np.isfinite(lp))
    S = (g ** 2).sum(1) + np.abs(E) + 1e3                      # magnitude of the terms of E_L
    # smaller chunks, planes with a base that TMA does not take as it is, no planes at all
    for nbytes, offset in ((full, 8), ((full + least) // 2, 0), (least + (full - least) // 8, 0), (least, 0), (least, 8)):
        st, E2, lp2, g2, _ = _call(params, r, R, Z, nbytes, offset, mode)
        assert st == 0
        assert np.all(np.abs(lp2 - lp) <= DIGITS_RTOL * np.abs(lp))
        if mode:
            assert np.all(np.abs(E2 - E) <= DIGITS_RTOL * np.abs(E) + 1e-10 * S)
            assert np.all(np.abs(g2 - g) <= DIGITS_RTOL * np.abs(g) + 1e-10 * np.abs(g).max())
    st, E2, lp2, g2, _ = _call(params, r, R, Z, least - 4096 - 4 * B - 512, 0, mode)
    assert st == 3 and np.all(lp2 == -7.0)


@pytest.mark.parametrize("prec", ["fp32_det64", "mixed_det64"])
def test_fp64_determinant_forms_take_the_digit_tangents(cuda, prec):
    mol = A.scale_molecule()
    params, r, R, Z = _setup(mol, 4, prec, 5)
    full, least = _sizes(params, 5, 1)
    st, E, lp, g, launches = _call(params, r, R, Z, full)
    assert st == 0
    st, E2, lp2, g2, fewer = _call(params, r, R, Z, least)
    assert st == 0 and launches > fewer                        # one launch of the FP64 loop in their place
    S = (g ** 2).sum(1) + np.abs(E) + 1e3
    assert np.array_equal(lp, lp2) and np.all(np.abs(E2 - E) <= DIGITS_RTOL * np.abs(E) + 1e-10 * S)
    # the same form on the same walkers in a workspace of more than is asked for: the same route, the same bits
    st, E3, lp3, g3, same = _call(params, r, R, Z, full + (64 << 20))
    assert st == 0 and same == launches and np.array_equal(E, E3) and np.array_equal(g, g3)


@pytest.mark.parametrize("name,K,B", [("c2h4", 8, 48), ("s40", 4, 40)])
def test_mixed_form_with_re_evaluated_walkers(cuda, name, K, B):
    """The re-evaluation's two tiers in a smaller region: FP64 walkers in several chunks of the valid count, and
    without planes."""
    L = _lib.lib()
    mol = {"c2h4": A.c2h4_shaped, "s40": A.scale_molecule}[name]()
    params, r, R, Z = _setup(mol, K, "mixed", B)
    for k in (0, 3, 5, 9, 11, 30):           # two up electrons close to one another: near a node
        r[k, 1] = r[k, 0] + (1e-4 if k % 2 else 2e-3)
    full, least = _sizes(params, B, 1)
    count = [ctypes.c_int64() for _ in range(3)]
    L.dw_guard_stats(None, None, None, 1)
    st, E, lp, g, _ = _call(params, r, R, Z, full)
    assert st == 0
    L.dw_guard_tier_stats(1, *[ctypes.byref(c) for c in count], 0)
    assert count[1].value >= 3                                  # walkers of the FP64 tier
    S = (g ** 2).sum(1) + np.abs(E) + 1e3
    for share in (0.75, 0.5, 0.25, 0.0):
        st, E2, lp2, g2, _ = _call(params, r, R, Z, int(least + share * (full - least)))
        assert st == 0
        assert np.all(np.abs(lp2 - lp) <= DIGITS_RTOL * np.abs(lp))
        assert np.all(np.abs(E2 - E) <= DIGITS_RTOL * np.abs(E) + 1e-9 * S), np.abs(E2 - E).max()


@pytest.mark.parametrize("prec", ["fp32", "mixed", "bf16", "fp32_det64", "mixed_det64"])
def test_misaligned_workspace_is_refused(cuda, prec):
    """Below 16 bytes (the FP64 form takes 8) nothing is launched on a workspace that vector stores would fault on."""
    L = _lib.lib()
    params, r, R, Z = _setup(A.lih(), 2, prec, 3)
    for mode in (0, 1):
        full = _sizes(params, 3, mode)[0]
        for offset in (4, 8):
            st, E, lp, _, launches = _call(params, r, R, Z, full, offset, mode)
            assert st == 3 and launches == 0 and np.all(lp == -7.0)
        assert _call(params, r, R, Z, full, 16, mode)[0] == 0
    if prec in ("fp32", "mixed"):
        nb = L.dw_workspace_bytes(ctypes.byref(params.c_arch), params.prec, 3, 3)
        ws, grad = torch.empty(nb + 256, dtype=torch.uint8, device="cuda"), torch.zeros_like(params.flat)
        base = (ws.data_ptr() + 255) // 256 * 256
        for offset, status in ((4, 3), (8, 3), (16, 0)):
            assert L.dw_log_psi_sqr_backward(ctypes.byref(params.c_arch), params.prec, api._ptr(params.flat),
                                             api._ptr(params.prepared), api._ptr(r), 3, api._ptr(R), api._ptr(Z),
                                             api._ptr(torch.ones(3, device="cuda")), api._ptr(grad),
                                             ctypes.c_void_p(base + offset), nb, None) == status
        torch.cuda.synchronize()
