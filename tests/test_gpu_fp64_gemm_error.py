"""GPU test of the FP64 GEMM by digit products where the large entries of a row meet small entries of a column,
against extended precision: the error stays that of an FP64 sum, relative to S = sum |a| |w|.

Bound: an FP64 sum of K terms is off by K 2^-53 S. Digits are off by 2^-53 |c| and K 2^-59.5 of the row's and
column's scales, and are taken where S is at least 2^-6 of both (to 2 %): K 2^-53.4 S.
"""
import ctypes

import numpy as np
import pytest
import torch

from deeperwin_gb300 import _lib, api, arch as A, params as P
from .test_gpu_fp64_gemm import _product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(130, 50, 36), (200, 100, 320), (40, 64, 512), (300, 32, 24)])
@pytest.mark.parametrize("kind", ["even", "inner", "disjoint", "outliers", "zeros"])
def test_error_is_relative_to_the_sum_of_magnitudes(cuda, M, N, K, kind):
    rng = np.random.default_rng(M + K)
    A, W = rng.standard_normal((M, K)), rng.standard_normal((K, N))
    if kind == "inner":              # the inner index scaled by powers of two
        s = rng.uniform(-50, 50, K)
        A, W = A * np.exp2(s), W * np.exp2(-s)[:, None]
    elif kind == "disjoint":         # large entries of the rows meet zeros or tiny entries of half of the columns
        A[:, : K // 2] *= 2.0 ** 45
        W[: K // 2, ::4] = 0.0
        W[: K // 2, 1::4] *= 2.0 ** -60
    elif kind == "outliers":
        A[rng.random((M, K)) < 0.02] *= 2.0 ** 30
        W[rng.random((K, N)) < 0.02] *= 2.0 ** 30
    elif kind == "zeros":            # rows and columns of zeros, and rows and columns with few entries
        A[rng.random((M, K)) < 0.97] = 0.0
        W[rng.random((K, N)) < 0.9] = 0.0
        A[3], W[:, 5] = 0.0, 0.0
    W = W.astype(np.float32)
    c = _product(A, W)
    ref = A.astype(np.longdouble) @ W.astype(np.longdouble)
    S = np.abs(A).astype(np.longdouble) @ np.abs(W).astype(np.longdouble)
    err = np.abs(c - ref)
    assert np.all(err <= (K + 2) * 2.0 ** -53 * S), float((err / np.maximum(S, 1e-300)).max() * 2.0 ** 53 / K)


def test_timer_reports_the_multiply_adds(cuda):
    """The fp64_gemm timer's operations are those of the 16 products of a local energy."""
    L = _lib.lib()
    mol, B = A.lih(), 3
    a = A.arch_for(mol, 8)
    params = api.Params.from_dict(a, P.init_params(a, 0), "fp64")
    r = A.init_walkers(mol, B, seed=1)
    api.local_energy(params, (a.n_up, a.n_dn), r, mol.R, mol.Z)
    L.dw_timer_enable(1)
    try:
        api.local_energy(params, (a.n_up, a.n_dn), r, mol.R, mol.Z)
        torch.cuda.synchronize()
        ms, flops, by, count = ctypes.c_double(), ctypes.c_double(), ctypes.c_double(), ctypes.c_int64()
        L.dw_timer_read(b"fp64_gemm", ctypes.byref(ms), ctypes.byref(count), ctypes.byref(flops), ctypes.byref(by))
    finally:
        L.dw_timer_enable(0)
    C = 3 * a.n_el + 2
    h = [a.h_width(layer) for layer in range(4)]
    e = [4, 32, 32, 32]
    per_row = sum(h) * 32 + sum(x + 32 + y for x, y in zip(h, e)) * 256 + 256 * a.n_dets * a.n_el + 256 * 64 + 64 * 64
    assert count.value == 16 and flops.value == 2.0 * B * C * (a.n_el * per_row + sum(2 * x for x in h) * 256)
