"""GPU test of the FP64 GEMM by exact digit products (fp64_gemm.cu) against extended precision.

The result is rounded to FP64 once (2^-53 relative); rounding the operands to 62 bits below their row's
or column's maximum and dropping the digit products beyond the ninth diagonal adds at most
K 2^-57 max|a_row| max|w_col|.
"""
import ctypes

import numpy as np
import pytest
import torch

from deeperwin_gb300 import _lib

pytestmark = pytest.mark.gpu


def _product(A, W):
    L = _lib.lib()
    M, K = A.shape
    N = W.shape[1]
    a, w = torch.as_tensor(A, device="cuda"), torch.as_tensor(W, device="cuda")
    c = torch.full((M, N), float("nan"), dtype=torch.float64, device="cuda")
    ws = torch.empty(L.dw_debug_gemm_fp64_bytes(M, N, K), dtype=torch.uint8, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())   # noqa: E731
    _lib.check(L.dw_debug_gemm_fp64(p(a), K, p(w), N, p(c), M, N, K, p(ws), None), "dw_debug_gemm_fp64")
    torch.cuda.synchronize()
    assert L.dw_debug_tc_error_flag() == 0
    return c.cpu().numpy()


@pytest.mark.parametrize("M,N,K", [(1, 32, 24), (5, 1, 1), (128, 48, 32), (129, 49, 33), (127, 47, 31), (300, 256, 320),
                                   (77, 64, 64), (200, 45, 256), (640, 256, 512), (24000, 256, 100)])
@pytest.mark.parametrize("spread", [0, 12])
def test_digit_products_match_extended_precision(cuda, M, N, K, spread):
    rng = np.random.default_rng(M + N + K + spread)
    # rows and columns of very different magnitudes, and entries of one row that span many binades
    A = rng.standard_normal((M, K)) * np.exp2(rng.integers(-spread, spread + 1, (M, K))) * np.exp2(rng.integers(-40, 40, (M, 1)))
    W = (rng.standard_normal((K, N)) * np.exp2(rng.integers(-spread, spread + 1, (K, N)))).astype(np.float32)
    A[rng.integers(0, M)] = 0.0
    c = _product(A, W)
    take = np.unique(np.concatenate([np.arange(min(M, 64)), rng.integers(0, M, 64), [M - 1]]))
    ref = A[take].astype(np.longdouble) @ W.astype(np.longdouble)
    bound = 2.0 ** -53 * np.abs(ref) + K * 2.0 ** -57 * np.abs(A[take]).max(1)[:, None] * np.abs(W).max(0)[None]
    err = np.abs(c[take].astype(np.longdouble) - ref)
    assert np.all(err <= bound), float((err / np.maximum(bound, 1e-300)).max())


def test_rows_and_columns_outside_the_digits_range(cuda):
    """Infinities, NaN, subnormal and extreme rows give what FP64 arithmetic gives."""
    rng = np.random.default_rng(0)
    A = rng.standard_normal((140, 40))
    W = rng.standard_normal((40, 50)).astype(np.float32)
    A[0, 3], A[1, 4], A[2, 5] = np.inf, np.nan, -np.inf
    A[3] *= 1e-310
    A[4] *= 1e-305
    A[5] *= 1e300
    A[6, 1:] *= 1e-200
    A[139, 39] = np.nan
    W[7, 3], W[8, 4] = np.inf, np.nan
    W[:, 5] = 0.0
    W[:, 6] = 1e-42
    c = _product(A, W)
    with np.errstate(all="ignore"):
        ref = (A.astype(np.longdouble) @ W.astype(np.longdouble)).astype(np.float64)
    np.testing.assert_array_equal(np.isnan(c), np.isnan(ref))
    np.testing.assert_array_equal(np.isinf(c), np.isinf(ref))
    ok = np.isfinite(ref)
    scale = (np.abs(np.where(np.isfinite(A), A, 0)).max(1)[:, None] * np.abs(np.where(np.isfinite(W), W, 0)).max(0)[None])
    # sequential FP64 sums of 40 terms, and the subnormal spacing
    bound = 40 * 2.0 ** -53 * np.abs(ref) + 40 * 40 * 2.0 ** -53 * scale + 40 * 5e-324
    assert np.all(np.abs(c[ok] - ref[ok]) <= bound[ok])


@pytest.mark.parametrize("n_el", [23, 24, 27, 33, 40, 48, 49])
def test_determinant_tangents_by_digits(cuda, n_el):
    """The FP64 form's local energy across the electron counts where the determinant tangents change from the
    FP64 loop to digit products and back: E_L and the gradient of walkers and nuclei translated together (an exact
    symmetry; the coordinates are multiples of 2^-12, so nothing is rounded) agree to the FP32 rounding of the outputs
    plus 1e-10 of the magnitudes summed. (Their values are pinned to the oracle in test_gpu_fp64.py, n = 34 and 40.)"""
    from deeperwin_gb300 import api, arch as A, params as P
    n_ions = 8
    Z = np.array([8] * n_ions)
    mol = A.Molecule(R=np.stack([np.arange(n_ions) * 2.0, np.arange(n_ions) % 2 * 1.5, np.zeros(n_ions)], 1), Z=Z, n_el=n_el,
                     n_up=(n_el + 1) // 2)
    a = A.arch_for(mol, 2)
    p = P.init_params(a, 3, bias_std=0.1, envelope_jitter=0.2)
    r = A.init_walkers(mol, 5, seed=9).astype(np.float32)
    params = api.Params.from_dict(a, p, "fp64")
    E, lp, g = api.local_energy(params, (a.n_up, a.n_dn), r, mol.R, mol.Z, return_grad=True)
    assert bool(torch.isfinite(E).all())
    r = np.round(r * 4096) / 4096
    E0, lp0, g0 = api.local_energy(params, (a.n_up, a.n_dn), r, mol.R, mol.Z, return_grad=True)
    E1, lp1, g1 = api.local_energy(params, (a.n_up, a.n_dn), r + 4.0, mol.R + 4.0, mol.Z, return_grad=True)
    S = (g0.double() ** 2).sum(1) + E0.double().abs() + 1e3
    assert bool(((E0.double() - E1.double()).abs() <= 2.4e-7 * E0.double().abs() + 1e-10 * S).all())
    assert bool(((g0 - g1).abs() <= 2.4e-7 * g0.abs() + 1e-10 * g0.abs().max()).all())
    assert L_flag() == 0


def L_flag():
    return _lib.lib().dw_debug_tc_error_flag()
