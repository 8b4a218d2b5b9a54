"""GPU test of the tangent passes' GEMM (gemm_jet.cu): channel rows of electrons times split-BF16 weights
with the forward-Laplacian tanh, against FP64. (Its envelope epilogue is covered by the local-energy
tests over electron and determinant counts.)

Operands are given as their BF16 parts (x = hi + lo exactly), so the product is off by the dropped
lo lo term (below 2^-16 |a| |w| per product) and the FP32 accumulation (K 2^-23): z is within
dz = (2^-16 + K 2^-23) sum |a| |w|. The jet y = (tanh z0, d1 z_t, d1 z_L - 2 y0 d1 sum z_t^2) adds the
tanh and its derivative at a shifted z0 (|d y0| <= dz0, |d d1| <= 2 dz0) and FP32 rounding, and a
split-BF16 result is rounded by 2^-16.
"""
import ctypes

import pytest
import torch

from deeperwin_gb300 import _lib

pytestmark = pytest.mark.gpu


def _split(x):
    hi = x.bfloat16()
    return hi, (x - hi.float()).bfloat16()


@pytest.mark.parametrize("T,n,ns,i0", [(8, 2, 2, 0), (14, 4, 4, 0), (17, 5, 2, 3), (32, 10, 10, 0), (50, 16, 8, 8),
                                       (83, 27, 27, 0), (122, 40, 20, 0), (128, 42, 42, 0)])
@pytest.mark.parametrize("nw,NF,K,out,ldc", [(3, 256, 320, 2, 320), (1, 64, 64, 2, 64), (7, 32, 24, 0, 32), (5, 160, 256, 2, 320),
                                            (9, 128, 100, 2, 320), (6, 128, 256, 2, 320), (5, 64, 256, 2, 64)])
def test_jet_gemm(cuda, T, n, ns, i0, nw, NF, K, out, ldc):
    g = torch.Generator(device="cuda").manual_seed(T * 1000 + NF + K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)          # noqa: E731
    lda, Kp, rows = (K + 63) // 64 * 64, (K + 63) // 64 * 64, nw * n * T
    a, w = rnd(rows, K), rnd(NF, K) / K ** 0.5
    ah, al = _split(a)
    A = torch.full((rows, 2 * lda), float("nan"), device="cuda", dtype=torch.bfloat16)
    A[:, :K], A[:, lda:lda + K] = ah, al
    wh, wl = _split(w)
    W = torch.zeros(2, NF, Kp, device="cuda", dtype=torch.bfloat16)
    W[0, :, :K], W[1, :, :K] = wh, wl
    a, w = (ah.float() + al.float()).double(), (wh.float() + wl.float()).double()
    bias = rnd(NF)
    rb = rnd(nw * T, 256) if NF == 256 else None
    C = torch.full((rows, 2 * ldc if out == 2 else ldc), 7.0, device="cuda",
                   dtype=torch.bfloat16 if out == 2 else torch.float32)
    L = _lib.lib()
    p = lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else 0)   # noqa: E731
    _lib.check(L.dw_debug_gemm_jet(out, p(A), lda, p(W[0]), p(W[1]), p(C), ldc, nw, n, T, ns, i0, NF, K, p(bias),
                                   p(rb), None), "dw_debug_gemm_jet")
    torch.cuda.synchronize()
    assert L.dw_debug_tc_error_flag() == 0
    got = (C[:, :NF].double() + C[:, ldc:ldc + NF].double()) if out == 2 else C[:, :NF].double()
    got, rest = got.view(nw, n, T, NF)[:, i0:i0 + ns], C.view(nw, n, T, -1)
    # rows of other electrons and columns beyond the features stay as they were
    assert bool((rest[:, :i0] == 7).all()) and bool((rest[:, i0 + ns:] == 7).all()) and bool((C[:, NF:ldc] == 7).all())
    z = (a @ w.T).view(nw, n, T, NF)[:, i0:i0 + ns]
    dz = ((2.0 ** -16 + K * 2.0 ** -23) * (a.abs() @ w.abs().T)).view(nw, n, T, NF)[:, i0:i0 + ns]
    if rb is not None:
        z = z + rb.double().view(nw, 1, T, 256)
    z[:, :, 0] += bias.double()
    dz = dz + 2.0 ** -23 * z.abs()
    y0, d0 = torch.tanh(z[:, :, :1]), dz[:, :, :1]
    d1, zt, dzt = 1 - y0 * y0, z[:, :, 1:T - 1], dz[:, :, 1:T - 1]
    s, ds = (zt ** 2).sum(2, keepdim=True), (2 * zt.abs() * dzt + dzt ** 2).sum(2, keepdim=True)
    ref = torch.cat([y0, d1 * zt, d1 * z[:, :, T - 1:] - 2 * y0 * d1 * s], 2)
    r = 2.0 ** -20 * s                                    # FP32 sums of up to 126 squares
    tol = torch.cat([d0, dzt + 2 * d0 * zt.abs(), dz[:, :, T - 1:] + 2 * d0 * z[:, :, T - 1:].abs()
                     + 2 * (ds + r) + 6 * d0 * (s + ds)], 2) + 2.0 ** -20 * (ref.abs() + 1)
    if out == 2:
        tol = tol + 2.0 ** -16 * ref.abs()
    assert bool(((got - ref).abs() <= tol).all()), float(((got - ref).abs() / tol).max())
