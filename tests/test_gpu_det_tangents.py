"""GPU test of the determinant tangents with 8 x 8 patches (k_det_tangents_t8) against the 4 x 4 tile
kernel: the same FP32 products and sums in the same order, so the local energies are the same bits."""
import ctypes

import numpy as np
import pytest
import torch

from deeperwin_gb300 import _lib, api, arch as A, params as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_el", [13, 14, 16, 17, 24, 25, 27, 31, 32])
def test_patch_sizes_agree_bit_for_bit(cuda, n_el):
    L = _lib.lib()
    mol = A.Molecule(R=np.arange(12.0).reshape(4, 3) ** 1.3, Z=np.array([8, 8, 8, 8]), n_el=n_el, n_up=(n_el + 1) // 2)
    a = A.arch_for(mol, 3)
    params = api.Params.from_dict(a, P.init_params(a, 6, bias_std=0.1, envelope_jitter=0.2), "mixed")
    rt = torch.as_tensor(A.init_walkers(mol, 7, seed=4).astype(np.float32), device="cuda")
    Rt, Zt = api._geometry(mol.R, mol.Z, "cuda")
    nb = L.dw_workspace_bytes(ctypes.byref(params.c_arch), params.prec, 7, 1)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    out = {}
    for tile in (0, 1):
        E, lp, sc = torch.empty(7, device="cuda"), torch.empty(7, device="cuda"), torch.empty(7, 3, device="cuda")
        prev = L.dw_debug_set_det_tangents_kernel(tile)
        try:
            _lib.check(L.dw_debug_local_energy_scales(
                ctypes.byref(params.c_arch), params.prec, api._ptr(params.flat), api._ptr(params.prepared), api._ptr(rt), 7,
                api._ptr(Rt), api._ptr(Zt), api._ptr(E), api._ptr(lp), api._ptr(sc), api._ptr(ws), nb, api._stream()), "scales")
        finally:
            L.dw_debug_set_det_tangents_kernel(prev)
        out[tile] = (E, sc)
    if n_el != 16:       # 16: the pipelined kernel, which adds the tiles' traces in another order
        assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert bool(torch.isfinite(out[0][0]).all())
