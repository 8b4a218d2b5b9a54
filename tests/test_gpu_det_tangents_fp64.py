"""GPU test of the FP64 determinant tangents: g_t = tr(A^-1 dA_t) and lapdet = tr(A^-1 Lap A) - sum_t
tr((A^-1 dA_t)^2) by digit products (24 <= n <= 48) and by the FP64 loop, against extended precision on the
same matrices and inverses, with rows and columns of very different magnitudes.

Bound, u = 2^-53: an FP64 sum E_ij = sum_o dA_io A^-1_oj of n terms is off by n u S_ij, S = |dA| |A^-1|. Digits
are rounded at 2^-63 of a row's (column's) scale and the dropped products are below 2^-59.5 n of both scales;
the scales are powers of two, up to twice the largest entry, after the orbital index is scaled by r_o, the
power of two below the largest entry of row o of A^-1: together below n 2^-57 max_o |dA_io| r_o max_o |A^-1_oj| / r_o.
The traces add n or n^2 terms, lapdet 3 n channels.
"""
import ctypes

import numpy as np
import pytest
import torch

from deeperwin_gb300 import _lib

pytestmark = pytest.mark.gpu


def _matrices(n, nmat, kind, seed):
    """Slater channels [nmat, 3 n + 2, n, n] and inverses."""
    rng = np.random.default_rng(seed)
    MO = rng.standard_normal((nmat, 3 * n + 2, n, n))
    if kind == "columns":            # orbitals spread over 2^40
        MO *= np.exp2(rng.uniform(-40, 0, (nmat, 1, 1, n)))
    elif kind == "both":
        MO *= np.exp2(rng.uniform(-30, 0, (nmat, 1, n, 1))) * np.exp2(rng.uniform(-40, 0, (nmat, 1, 1, n)))
    elif kind == "envelopes":        # exponential envelopes: entries of a row span hundreds of binades
        a, d = rng.uniform(0.3, 8, (nmat, 1, 1, n)), rng.uniform(0, 12, (nmat, 1, n, 1))
        MO *= np.exp(-a * d)
    elif kind == "range":            # a few columns far from the others
        c = np.zeros(n)
        c[:3] = [-500, -250, 150]
        MO *= np.exp2(c)
    inv = np.linalg.inv(MO[:, 0] / _pow2(MO[:, 0])) / np.swapaxes(_pow2(MO[:, 0]), 1, 2)
    return MO, np.ascontiguousarray(inv)


def _pow2(A):
    """Powers of two by columns, so that the inverse is formed of ordinary numbers."""
    return np.exp2(np.floor(np.log2(np.abs(A).max(1, keepdims=True))))


def _tangents(MO, inv, sign=None, K=1, nvalid=None, scratch=None):
    L = _lib.lib()
    nmat, T, n, _ = MO.shape
    p = lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else 0)   # noqa: E731
    mo, ai = torch.as_tensor(MO, device="cuda"), torch.as_tensor(inv, device="cuda")
    sg = torch.ones(nmat, dtype=torch.float64, device="cuda") if sign is None else torch.as_tensor(sign, device="cuda")
    g = torch.full((nmat, 3 * n), -7.0, dtype=torch.float64, device="cuda")
    lap = torch.full((nmat,), -7.0, dtype=torch.float64, device="cuda")
    nb = L.dw_debug_det_tangents_fp64_bytes(n, nmat) if scratch is None else scratch
    ws = torch.empty(max(nb, 1), dtype=torch.uint8, device="cuda")
    nv = None if nvalid is None else torch.tensor([nvalid], dtype=torch.int32, device="cuda")
    _lib.check(L.dw_debug_det_tangents_fp64(p(mo), p(ai), p(sg), n, K, nmat, p(nv), p(g), p(lap), p(ws), nb, None), "dets")
    launches = L.dw_last_launch_count()
    torch.cuda.synchronize()
    assert L.dw_debug_tc_error_flag() == 0
    return g.cpu().numpy(), lap.cpu().numpy(), launches


def _reference(MO, inv):
    """g, lapdet in extended precision, and the bounds of the FP64 results."""
    n = MO.shape[-1]
    u = 2.0 ** -53
    dA, W = MO[1:].astype(np.longdouble), inv.astype(np.longdouble)
    E, S = np.matmul(dA, W), np.matmul(np.abs(dA), np.abs(W))
    r = np.exp2(np.floor(np.log2(np.abs(W).max(1))))
    dE = n * u * S + n * 2.0 ** -57 * (np.abs(dA) * r).max(2)[:, :, None] * (np.abs(W) / r[:, None]).max(0)
    tr, dtr = np.trace(E, axis1=1, axis2=2), np.trace(dE + n * u * S, axis1=1, axis2=2)
    Et, dEt = np.swapaxes(E, 1, 2), np.swapaxes(dE, 1, 2)
    tr2 = (E * Et).sum((1, 2))[:-1]
    d2 = (np.abs(E) * dEt + np.abs(Et) * dE + dE * dEt + (n * n + 3 * n) * u * np.abs(E * Et)).sum((1, 2))[:-1]
    return tr[:-1], dtr[:-1], tr[-1] - tr2.sum(), dtr[-1] + d2.sum() + u * abs(tr[-1])


@pytest.mark.parametrize("n", [23, 24, 27, 40, 47, 48, 49])
@pytest.mark.parametrize("kind", ["even", "columns", "both", "envelopes", "range"])
def test_tangents_match_extended_precision(cuda, n, kind):
    MO, inv = _matrices(n, 2, kind, n)
    for scratch in (None, 0):                # digit products where they serve, and the FP64 loop
        g, lap, launches = _tangents(MO, inv, scratch=scratch)
        assert (launches > 1) == (scratch is None and 24 <= n <= 48)
        tr, dtr, ld, dld = _reference(MO[1], inv[1])
        assert np.all(np.abs(g[1] - tr) <= dtr), float((np.abs(g[1] - tr) / dtr).max())
        assert abs(lap[1] - ld) <= dld, float(abs(lap[1] - ld) / dld)


def test_groups_of_matrices_and_valid_counts(cuda):
    """Scratch for fewer matrices at a time, and a device-side count, leave every valid matrix the same bits."""
    n, K, nmat = 25, 3, 81
    MO, inv = _matrices(n, nmat, "columns", 1)
    g0, l0, full = _tangents(MO, inv, K=K)
    nb = _lib.lib().dw_debug_det_tangents_fp64_bytes(n, nmat)
    for share, nvalid in ((1.0, 20), (0.5, None), (0.5, 13), (0.5, 0)):
        g, lap, launches = _tangents(MO, inv, K=K, nvalid=nvalid, scratch=int(nb * share))
        assert launches > full if share < 1 else launches == full
        k = nmat if nvalid is None else nvalid * K
        assert np.array_equal(g[:k], g0[:k]) and np.array_equal(lap[:k], l0[:k])
        assert np.all(g[k:] == -7.0) and np.all(lap[k:] == -7.0)
    g, lap, launches = _tangents(MO, inv, K=K, scratch=nb // 3)      # fewer than 32 matrices: the loop
    assert launches == 1
    gl, ll, _ = _tangents(MO, inv, K=K, scratch=0)
    assert np.array_equal(g, gl) and np.array_equal(lap, ll)


def test_singular_and_non_finite_matrices(cuda):
    n = 26
    MO, inv = _matrices(n, 5, "even", 3)
    sign = np.array([1.0, 0.0, -1.0, 1.0, 1.0])
    inv[1] = 0.0                                       # a singular matrix: its tangents are zeros
    MO[2, 5, 3, 4] = np.nan
    MO[3, 7, 2, 2] = np.inf
    MO[4, :, :, 6] *= 2.0 ** -1055                     # subnormal orbital
    inv[4, 6] *= 2.0 ** 1000
    g, lap, _ = _tangents(MO, inv, sign=sign)
    gl, ll, _ = _tangents(MO, inv, sign=sign, scratch=0)
    assert np.all(g[1] == 0.0) and lap[1] == 0.0
    np.testing.assert_array_equal(np.isfinite(g), np.isfinite(gl))
    np.testing.assert_array_equal(np.isfinite(lap), np.isfinite(ll))
    ok = np.isfinite(gl)
    g, gl = np.where(ok, g, 0), np.where(ok, gl, 0)
    S = np.einsum("mtio,moi->mt", np.abs(MO[:, 1:-1]), np.abs(inv))
    assert np.all((np.abs(g - gl) <= n * 2.0 ** -51 * S)[ok])
