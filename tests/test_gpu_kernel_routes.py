"""GPU tests of single kernels at the sizes where their dispatch changes: the determinant tangents in 8 x 8 patches, the
FP32 GEMM's tiles, and the tangent GEMM with one BF16 part and with the envelope epilogue."""
import ctypes

import numpy as np
import pytest
import torch

from deeperwin_gb300 import _lib, api, arch as A, params as P

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr() if t is not None else 0)


def _energies(params, rt, Rt, Zt, which):
    L = _lib.lib()
    B = len(rt)
    nb = L.dw_workspace_bytes(ctypes.byref(params.c_arch), params.prec, B, 1)
    ws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    E, lp, sc = torch.empty(B, device="cuda"), torch.empty(B, device="cuda"), torch.empty(B, 3, device="cuda")
    prev = L.dw_debug_set_det_tangents_kernel(which)
    try:
        _lib.check(L.dw_debug_local_energy_scales(
            ctypes.byref(params.c_arch), params.prec, api._ptr(params.flat), api._ptr(params.prepared), api._ptr(rt), B,
            api._ptr(Rt), api._ptr(Zt), api._ptr(E), api._ptr(lp), api._ptr(sc), api._ptr(ws), nb, api._stream()), "scales")
    finally:
        L.dw_debug_set_det_tangents_kernel(prev)
    return E, sc


@pytest.mark.parametrize("n_el", [20, 28])
def test_tangent_patches_with_padded_planes(cuda, n_el):
    """n a multiple of 4 with padding takes 16-byte copies into padded planes: the same bits as the 4 x 4 tiles."""
    mol = A.Molecule(R=np.arange(15.0).reshape(5, 3) ** 1.3, Z=np.array([8] * 5), n_el=n_el, n_up=(n_el + 1) // 2)
    a = A.arch_for(mol, 3)
    params = api.Params.from_dict(a, P.init_params(a, 6, bias_std=0.1, envelope_jitter=0.2), "mixed")
    rt = torch.as_tensor(A.init_walkers(mol, 7, seed=4).astype(np.float32), device="cuda")
    Rt, Zt = api._geometry(mol.R, mol.Z, "cuda")
    E0, s0 = _energies(params, rt, Rt, Zt, 0)
    E1, s1 = _energies(params, rt, Rt, Zt, 1)
    assert bool(torch.isfinite(E0).all())
    assert torch.equal(E0, E1) and torch.equal(s0, s1)


@pytest.mark.parametrize("n", [2, 4, 7, 8, 12, 13, 15, 16, 17, 20, 24, 25, 28, 32, 33, 36, 39, 40, 41, 50, 63, 64])
def test_fp32_tangents_match_fp64(cuda, n):
    """g_t = tr C_t and lapdet = tr C_lap - sum_t tr(C_t^2), C = A^-1 D, against FP64 on the same FP32 matrices. With u =
    2^-24 an entry of C is off by n u S, S = |A^-1| |D|; a trace adds up to 16 and 100 terms in FP32 (a tile, its tiles)."""
    rng = np.random.default_rng(n)
    nmat, u = 5, 2.0 ** -24
    MO = (rng.standard_normal((nmat, 3 * n + 2, n, n)) * np.exp2(rng.uniform(-6, 0, (nmat, 1, 1, n)))).astype(np.float32)
    inv = np.linalg.inv(MO[:, 0].astype(np.float64)).astype(np.float32)
    sign = np.array([1.0, -1.0, 0.0, 1.0, 1.0])
    t = [torch.as_tensor(x, device="cuda") for x in (MO, inv, sign)]
    g, lap = torch.empty(nmat, 3 * n, dtype=torch.float64, device="cuda"), torch.empty(nmat, dtype=torch.float64, device="cuda")
    _lib.check(_lib.lib().dw_debug_det_tangents(_p(t[0]), _p(t[1]), _p(t[2]), n, nmat, _p(g), _p(lap), None), "det_tangents")
    g, lap = g.cpu().numpy(), lap.cpu().numpy()
    for m in range(nmat):
        if sign[m] == 0:
            assert np.all(g[m] == 0) and lap[m] == 0
            continue
        C = inv[m].astype(np.float64) @ MO[m, 1:].astype(np.float64)
        d = n * u * (np.abs(inv[m]).astype(np.float64) @ np.abs(MO[m, 1:]).astype(np.float64))
        tr, Ct, dt = np.trace(C, axis1=1, axis2=2), np.swapaxes(C, 1, 2), np.swapaxes(d, 1, 2)
        dtr = np.trace(d, axis1=1, axis2=2) + 116 * u * np.abs(np.diagonal(C, axis1=1, axis2=2)).sum(1)
        tr2 = (C * Ct).sum((1, 2))[:-1]
        d2 = (np.abs(C) * dt + np.abs(Ct) * d + d * dt + 118 * u * np.abs(C * Ct)).sum((1, 2))[:-1]
        assert np.all(np.abs(g[m] - tr[:-1]) <= dtr[:-1]), float((np.abs(g[m] - tr[:-1]) / dtr[:-1]).max())
        assert abs(lap[m] - (tr[-1] - tr2.sum())) <= dtr[-1] + d2.sum()


@pytest.mark.parametrize("N,K", [(32, 32), (64, 256), (256, 320), (256, 512), (40, 100), (300, 64), (7, 5)])
@pytest.mark.parametrize("act", [0, 1])
def test_fp32_gemm_tiles_give_the_same_bits(cuda, N, K, act):
    """Every tile forms an output as one FMA chain over k, so the first rows do not depend on how many follow."""
    L = _lib.lib()
    M = 128 * 2 * 160 + 77                   # beyond two blocks of 128 rows per SM
    g = torch.Generator(device="cuda").manual_seed(N + K)
    a = torch.randn(M, K, device="cuda", generator=g)
    w = torch.randn(K, N, device="cuda", generator=g) / K ** 0.5
    bias, rpw = torch.randn(N, device="cuda", generator=g), 5
    rb = torch.randn((M + rpw - 1) // rpw, N, device="cuda", generator=g)
    out = {}
    for m in (1, 7, 8, 64, 65, 127, 129, 2048, 8192, 128 * 152 + 1, M):
        c = torch.full((m, N), float("nan"), device="cuda")
        _lib.check(L.dw_debug_gemm_f32(_p(a), K, _p(w), N, _p(c), N, m, N, K, _p(bias), _p(rb), rpw, act, None), "gemm_f32")
        torch.cuda.synchronize()
        out[m] = c
    z = a.double() @ w.double() + bias.double() + rb.double().repeat_interleave(rpw, 0)[:M]
    S = a.double().abs() @ w.double().abs() + bias.double().abs() + rb.double().abs().repeat_interleave(rpw, 0)[:M]
    ref = torch.tanh(z) if act else z
    assert bool(((out[M].double() - ref).abs() <= (K + 4) * 2.0 ** -24 * S + 2.0 ** -21).all())
    for m, c in out.items():
        assert torch.equal(c, out[M][:m]), m


@pytest.mark.parametrize("T,n,ns,i0", [(8, 2, 2, 0), (17, 5, 2, 3), (50, 16, 8, 8), (83, 27, 27, 0), (128, 42, 42, 0)])
@pytest.mark.parametrize("nw,NF,K,out,ldc", [(3, 256, 320, 1, 320), (1, 64, 64, 1, 64), (7, 32, 24, 0, 32), (5, 64, 256, 1, 64)])
def test_jet_gemm_with_one_part(cuda, T, n, ns, i0, nw, NF, K, out, ldc):
    """BF16 operands: products are exact, the FP32 sums are off by K 2^-23 sum |a| |w|; the jet and the rounding of a
    BF16 result (2^-8) as in the split form's test."""
    g = torch.Generator(device="cuda").manual_seed(T * 1000 + NF + K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)          # noqa: E731
    lda, rows = (K + 63) // 64 * 64, nw * n * T
    a, w = rnd(rows, K).bfloat16(), (rnd(NF, K) / K ** 0.5).bfloat16()
    X = torch.full((rows, lda), float("nan"), device="cuda", dtype=torch.bfloat16)
    X[:, :K] = a
    W = torch.zeros(NF, lda, device="cuda", dtype=torch.bfloat16)
    W[:, :K] = w
    a, w = a.double(), w.double()
    bias, rb = rnd(NF), rnd(nw * T, 256) if NF == 256 else None
    C = torch.full((rows, ldc), 7.0, device="cuda", dtype=torch.bfloat16 if out else torch.float32)
    L = _lib.lib()
    _lib.check(L.dw_debug_gemm_jet_bf16(out, _p(X), lda, _p(W), _p(C), ldc, nw, n, T, ns, i0, NF, K, _p(bias), _p(rb), None), "jet")
    torch.cuda.synchronize()
    assert L.dw_debug_tc_error_flag() == 0
    got, rest = C[:, :NF].double().view(nw, n, T, NF)[:, i0:i0 + ns], C.view(nw, n, T, -1)
    assert bool((rest[:, :i0] == 7).all()) and bool((rest[:, i0 + ns:] == 7).all()) and bool((C[:, NF:] == 7).all())
    z = (a @ w.T).view(nw, n, T, NF)[:, i0:i0 + ns]
    dz = (K * 2.0 ** -23 * (a.abs() @ w.abs().T)).view(nw, n, T, NF)[:, i0:i0 + ns]
    if rb is not None:
        z = z + rb.double().view(nw, 1, T, 256)
    z[:, :, 0] += bias.double()
    dz = dz + 2.0 ** -23 * z.abs()
    y0, d0 = torch.tanh(z[:, :, :1]), dz[:, :, :1]
    d1, zt, dzt = 1 - y0 * y0, z[:, :, 1:T - 1], dz[:, :, 1:T - 1]
    s, ds = (zt ** 2).sum(2, keepdim=True), (2 * zt.abs() * dzt + dzt ** 2).sum(2, keepdim=True)
    ref = torch.cat([y0, d1 * zt, d1 * z[:, :, T - 1:] - 2 * y0 * d1 * s], 2)
    tol = torch.cat([d0, dzt + 2 * d0 * zt.abs(), dz[:, :, T - 1:] + 2 * d0 * z[:, :, T - 1:].abs()
                     + 2 * (ds + 2.0 ** -20 * s) + 6 * d0 * (s + ds)], 2) + 2.0 ** -20 * (ref.abs() + 1)
    if out:
        tol = tol + 2.0 ** -8 * ref.abs()
    assert bool(((got - ref).abs() <= tol).all()), float(((got - ref).abs() / tol).max())


@pytest.mark.parametrize("np_", [1, 2])
@pytest.mark.parametrize("n,N,dets,ns,i0,nw,packed", [(2, 1, 3, 1, 1, 4, False), (5, 3, 11, 3, 0, 5, True), (10, 10, 16, 5, 5, 3, False),
                                                     (16, 6, 32, 8, 8, 4, True), (27, 5, 8, 13, 14, 2, False),
                                                     (40, 12, 4, 20, 0, 1, True), (42, 16, 2, 21, 21, 2, False)])
def test_jet_gemm_with_envelopes(cuda, np_, n, N, dets, ns, i0, nw, packed):
    """Slater channels MO[b][k][t][i][o] = envelope x backflow with the product rule, against FP64. The backflow rows
    are off by dz as in the tests of the tanh epilogue; an envelope's terms w exp(-a d) by 2^-20 (1 + a d) of their
    magnitude (FP32 distance, product and exponential), their derivatives' factors a / d, a^2, 2 a / d included."""
    g = torch.Generator(device="cuda").manual_seed(n * 100 + dets + np_)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)          # noqa: E731
    K, lda, T, KN = 256, 320, 3 * n + 2, dets * n
    rows = nw * n * T
    a, w = rnd(rows, K), rnd(KN, K) / K ** 0.5
    ah, wh = a.bfloat16(), w.bfloat16()
    al, wl = (a - ah.float()).bfloat16(), (w - wh.float()).bfloat16()
    X = torch.full((rows, np_ * lda), float("nan"), device="cuda", dtype=torch.bfloat16)
    X[:, :K] = ah
    if np_ == 2:
        X[:, lda:lda + K] = al
        a, w = ah.double() + al.double(), wh.double() + wl.double()
        unit = 2.0 ** -16 + K * 2.0 ** -23
    else:
        a, w = ah.double(), wh.double()
        unit = K * 2.0 ** -23
    nseg = 2 if packed else 1
    r, R = 1.5 * rnd(nw, n, 3), 1.5 * rnd(nseg, N, 3)
    Z = torch.full((nseg, N), 3, dtype=torch.int32, device="cuda")
    if packed:
        Z[1, N // 2:] = 0                                                   # padding of a smaller molecule
    seg = torch.arange(nw, device="cuda", dtype=torch.int32) % 2 if packed else None
    alpha, wts = 0.3 + 2 * torch.rand(N, KN, device="cuda", generator=g), rnd(N, KN)
    MO = torch.full((nw, dets, T, n, n), 7.0, device="cuda")
    L = _lib.lib()
    _lib.check(L.dw_debug_gemm_jet_env(np_, _p(X), lda, _p(wh), _p(wl if np_ == 2 else None), _p(r), _p(R), _p(Z), _p(seg), nseg,
                                       _p(alpha), _p(wts), _p(MO), nw, n, N, dets, ns, i0, K, None), "env")
    torch.cuda.synchronize()
    assert L.dw_debug_tc_error_flag() == 0
    assert bool((MO[:, :, :, :i0] == 7).all()) and bool((MO[:, :, :, i0 + ns:] == 7).all())
    got = MO[:, :, :, i0:i0 + ns].double().permute(0, 3, 2, 1, 4).reshape(nw, ns, T, KN)       # [b, i, t, (k, o)]
    bf = (a @ w.T).view(nw, n, T, KN)[:, i0:i0 + ns]
    dz = (unit * (a.abs() @ w.abs().T)).view(nw, n, T, KN)[:, i0:i0 + ns] + 2.0 ** -23 * bf.abs()
    geo = seg.long() if packed else torch.zeros(nw, dtype=torch.long, device="cuda")
    diff = r.double()[:, i0:i0 + ns, None] - R.double()[geo][:, None]                          # [b, i, I, 3]
    d = diff.norm(dim=-1)
    on = (Z[geo] > 0).double()[:, None, :, None]
    al64, e = alpha.double(), None
    e = on * wts.double() * torch.exp(-al64 * d[..., None])                                    # [b, i, I, KN]
    rel = 2.0 ** -20 * (1 + al64 * d[..., None])
    env, denv = e.sum(2), (e.abs() * rel).sum(2)
    gt = [(-al64 * e / d[..., None] * diff[..., c:c + 1]) for c in range(3)]
    gr, dgr = [x.sum(2) for x in gt], [(x.abs() * rel * 2).sum(2) for x in gt]
    lap = (e * (al64 ** 2 - 2 * al64 / d[..., None])).sum(2)
    dlap = (e.abs() * (al64 ** 2 + 2 * al64 / d[..., None]) * rel * 2).sum(2)
    ref, tol = env[:, :, None] * bf, env.abs()[:, :, None] * dz + denv[:, :, None] * (bf.abs() + dz)
    mag = (env.abs()[:, :, None] * bf.abs()).clone()
    for i in range(ns):
        for c in range(3):
            t = 1 + 3 * (i0 + i) + c
            ref[:, i, t] += gr[c][:, i] * bf[:, i, 0]
            tol[:, i, t] += gr[c][:, i].abs() * dz[:, i, 0] + dgr[c][:, i] * (bf[:, i, 0].abs() + dz[:, i, 0])
            mag[:, i, t] += gr[c][:, i].abs() * bf[:, i, 0].abs()
            ref[:, i, T - 1] += 2 * gr[c][:, i] * bf[:, i, t]
            tol[:, i, T - 1] += 2 * (gr[c][:, i].abs() * dz[:, i, t] + dgr[c][:, i] * (bf[:, i, t].abs() + dz[:, i, t]))
            mag[:, i, T - 1] += 2 * gr[c][:, i].abs() * bf[:, i, t].abs()
    ref[:, :, T - 1] += lap * bf[:, :, 0]
    tol[:, :, T - 1] += lap.abs() * dz[:, :, 0] + dlap * (bf[:, :, 0].abs() + dz[:, :, 0])
    mag[:, :, T - 1] += lap.abs() * bf[:, :, 0].abs()
    tol = tol + 2.0 ** -20 * mag + 1e-30
    assert bool(((got - ref).abs() <= tol).all()), float(((got - ref).abs() / tol).max())
