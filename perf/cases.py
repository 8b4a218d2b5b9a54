"""Performance cases of the variational Monte Carlo inner loop: the calls a user's program makes
through ``deeperwin_gb300.api`` and ``deeperwin_gb300.vmc``, over the range of molecules and walker
counts of the repository's workloads (2 to 40 electrons, 4 to 64 determinants, 1 to 8192 walkers).

A case names an operation and its sizes:

* ``op``: "logpsi" (log psi^2 of all walkers), "energy" (local energies by the forward Laplacian),
  "mcmc" (re-evaluation and Metropolis-Hastings steps), "gradient" (the parameter gradient of
  sum_b coeff_b log psi^2_b) or "step" (local energies, clipping and the VMC gradient in one call);
* ``mol``: a molecule of ``deeperwin_gb300.arch`` by name, or "random" (neutral, nuclei with charges
  1, 6, 7, 8 in a box, ``n_el`` electrons);
* ``precision``: "mixed" (the production form), "fp32" (the plain form), "fp64" (the anchor form).

Weights are a seeded random initialisation with non-zero biases and jittered envelopes, as some
optimisation steps leave them; walkers start Gaussian around the nuclei and have made some
Metropolis-Hastings steps towards |psi|^2 (in plain torch, so that every build sees the same ones).
"""
import math

import numpy as np
import torch

from deeperwin_gb300 import api, vmc
from deeperwin_gb300 import arch as A
from deeperwin_gb300 import params as P

MOLECULES = {"lih": A.lih, "h10": A.h_chain, "c2h4": A.c2h4_shaped, "scale40": A.scale_molecule}


def listed():
    return [
        # one configuration of a small molecule, as a program that scans or plots psi asks for it
        dict(name="logpsi_lih_one", op="logpsi", mol="lih", n_dets=8, walkers=1, precision="fp32"),
        # the chain of the smallest workload between two optimisation steps (20 inter-steps, 2048 walkers)
        dict(name="mcmc_lih_fp32", op="mcmc", mol="lih", n_dets=8, walkers=2048, precision="fp32", steps=20),
        # the same workload's local energies, in the plain form
        dict(name="energy_lih_fp32", op="energy", mol="lih", n_dets=8, walkers=2048, precision="fp32"),
        # log psi^2 of a large batch: hydrogen chain, 8192 walkers (a forward of the chain, or a density estimate)
        dict(name="logpsi_h10", op="logpsi", mol="h10", n_dets=16, walkers=8192, precision="mixed"),
        # the hydrogen chain's local energies
        dict(name="energy_h10", op="energy", mol="h10", n_dets=16, walkers=8192, precision="mixed"),
        # the three parts of an optimisation step of the benchmark's workload: chain, energies, gradient
        dict(name="mcmc_c2h4", op="mcmc", mol="c2h4", n_dets=32, walkers=4096, precision="mixed", steps=10),
        dict(name="energy_c2h4", op="energy", mol="c2h4", n_dets=32, walkers=4096, precision="mixed"),
        dict(name="gradient_c2h4", op="gradient", mol="c2h4", n_dets=32, walkers=4096, precision="mixed"),
        # the energies and gradient of one small served molecule, odd electron and walker counts
        dict(name="step_13el", op="step", mol="random", n_el=13, n_dets=8, walkers=1111, precision="mixed"),
        # an energy request near the upper end of the served range, odd sizes
        dict(name="energy_27el", op="energy", mol="random", n_el=27, n_dets=8, walkers=1500, precision="mixed"),
        # the largest molecule: 40 electrons, 64 determinants
        dict(name="energy_scale40", op="energy", mol="scale40", n_dets=64, walkers=512, precision="mixed"),
        # reference energies of a few walkers in the FP64 form
        dict(name="energy_c2h4_fp64", op="energy", mol="c2h4", n_dets=32, walkers=64, precision="fp64"),
    ]


# passes over the network that one walker costs, relative to a value forward
def _passes(case, n_el):
    return {"logpsi": 1, "mcmc": case.get("steps", 0) + 1, "energy": 3 * n_el + 2, "gradient": 3,
            "step": 3 * n_el + 5}[case["op"]]


def draw(rng):
    while True:
        op = rng.choice(["logpsi", "mcmc", "energy", "energy", "gradient", "step"])
        precision = rng.choice(["mixed", "mixed", "mixed", "fp32"] + (["fp64"] if op == "energy" else []))
        n_el = round(math.exp(rng.uniform(math.log(2), math.log(40))))
        n_dets = rng.choice([4, 8, 11, 16, 24, 32, 64])
        # bounded by the work of the largest listed case, and the plain and FP64 forms by their slower arithmetic
        walkers = round(math.exp(rng.uniform(0.0, math.log(8192))))
        case = dict(op=op, mol="random", n_el=n_el, n_dets=n_dets, walkers=walkers, precision=precision)
        if op == "mcmc":
            case["steps"] = rng.choice([1, 5, 10, 20])
        top = work(next(c for c in listed() if c["name"] == "energy_scale40"))["flops"]
        if work(case)["flops"] * {"mixed": 1, "fp32": 2, "fp64": 40}[precision] <= top:
            return case


def _molecule(case):
    if case["mol"] != "random":
        return MOLECULES[case["mol"]]()
    n = case["n_el"]
    rng = np.random.default_rng(1000 + n)
    Z = []
    while n - sum(Z) >= 10 and len(Z) < 5:
        Z.append(int(rng.choice([6, 7, 8])))
    rest = n - sum(Z)
    while rest > 11:                    # at most 16 nuclei
        Z.append(8)
        rest -= 8
    Z += [1] * rest
    box = 6.0
    for attempt in range(100000):
        R = rng.uniform(0.0, box, size=(len(Z), 3))
        if (np.linalg.norm(R[:, None] - R[None], axis=-1) + 1e9 * np.eye(len(Z))).min() >= 1.5:
            break
        box += 1e-3
    return A.Molecule(R=R - R.mean(axis=0), Z=np.array(Z, np.int64), n_el=n, n_up=(n + 1) // 2, name=f"random{n}")


def _equilibrated(weights, a, r, R, Z, rng, steps=10, stepsize=0.2):
    """Metropolis-Hastings steps of the walkers r in float32, by the plain torch forward below."""
    p = {k: torch.as_tensor(v.astype(np.float32), device=r.device) for k, v in weights.items()}

    def log_psi_sqr(x):
        return torch.cat([_log_psi_sqr_jets(p, a, y, R, Z, False)[1][0] for y in x.split(_chunk(a, 1))])

    lp = log_psi_sqr(r)
    for _ in range(steps):
        move = torch.as_tensor(rng.standard_normal(r.shape, np.float32), device=r.device)
        u = torch.as_tensor(rng.random(len(r), np.float32), device=r.device)
        new = r + stepsize * move
        lp_new = log_psi_sqr(new)
        accept = torch.log(u) < lp_new - lp
        r, lp = torch.where(accept[:, None, None], new, r), torch.where(accept, lp_new, lp)
    return r.contiguous()


@torch.no_grad()
def _inputs(case, seed):
    """Molecule, model shape, weights by name (float32 values), walkers, nuclei: all from the seed alone."""
    mol = _molecule(case)
    arch = A.arch_for(mol, case["n_dets"], z_max=8)
    weights = P.init_params(arch, seed, bias_std=0.1, envelope_jitter=0.1)
    rng = np.random.default_rng(seed + 1)
    r = torch.as_tensor(A.init_walkers(mol, case["walkers"], seed + 2).astype(np.float32), device="cuda")
    R = torch.as_tensor(mol.R.astype(np.float32), device="cuda")
    Z = torch.as_tensor(mol.Z.astype(np.int32), device="cuda")
    # the optimisation's coefficients (E_clip - mean) / B
    coeff = torch.as_tensor(rng.standard_normal(case["walkers"], np.float32) / case["walkers"], device="cuda")
    return mol, arch, weights, _equilibrated(weights, arch, r, R, Z, rng), R, Z, coeff


def prepare(case, seed):
    mol, arch, weights, r, R, Z, coeff = _inputs(case, seed)
    params = api.Params.from_dict(arch, weights, case["precision"])
    state = dict(op=case["op"], arch=arch, params=params, r=r, R=R, Z=Z)
    if case["op"] == "mcmc":
        state["chain"] = api.MCMCState(state["r"], mol.R, mol.Z, seed=seed, stepsize=0.1)
        state["mcmc"] = api.MetropolisHastingsMonteCarlo(api.MCMCConfig())
        state["steps"] = case["steps"]
    elif case["op"] == "gradient":
        state["coeff"] = coeff
    elif case["op"] == "step":
        state["value_and_grad"] = vmc.build_value_and_grad_func()
    return state


def run(state):
    op, a, params = state["op"], state["arch"], state["params"]
    r, R, Z = state["r"], state["R"], state["Z"]
    if op == "logpsi":
        phase, log_psi_sqr = api.log_psi_sqr(params, a.n_up, a.n_dn, r, R, Z)
        return {"phase": phase, "log_psi_sqr": log_psi_sqr}
    if op == "energy":
        E, log_psi_sqr, grad = api.local_energy(params, (a.n_up, a.n_dn), r, R, Z, return_grad=True)
        return {"E_loc": E, "log_psi_sqr": log_psi_sqr, "grad_r": grad}
    if op == "mcmc":
        chain = state["mcmc"].run_mcmc_steps(None, state["chain"], params, a.n_up, a.n_dn, n_steps=state["steps"])
        # the chain's scalars by their types: running and last acceptance, step size, step number
        s = chain.scalars
        return {"r": chain.r, "log_psi_sqr": chain.log_psi_sqr, "age": chain.walker_age,
                "acceptance": s[:16].view(torch.float64), "stepsize": s[16:20].view(torch.float32),
                "step_nr": s[20:24].view(torch.int32)}
    if op == "gradient":
        return {"grads": vmc.log_psi_sqr_backward(params, r, R, Z, state["coeff"])}
    (loss, (clipping, aux)), grads = state["value_and_grad"](params, vmc.init_clipping_state(), (a.n_up, a.n_dn),
                                                             (r, R, Z))
    return {"loss": loss, "E_loc": aux["E_loc"], "E_var": aux["E_var"], "clip_center": clipping[0],
            "clip_width": clipping[1], "grads": grads}


def work(case):
    """Multiply-adds (two operations each) of the network and the determinants once per pass over
    them, walkers and weights read once, outputs written once."""
    mol = _molecule(case)
    a = A.arch_for(mol, case["n_dets"], z_max=8)
    n, B, kn = a.n_el, case["walkers"], a.n_orb_cols
    # per electron: layer inputs (the spin means' share once per walker), orbitals, Jastrow; per pair and
    # electron-ion pair: the 32-wide streams
    per_el = sum((a.in_width(l) - 2 * a.h_width(l)) * 256 + a.h_width(l) * 32 for l in range(4)) + 256 * kn + 256 * 64 + 64 * 64
    per_walker = sum(2 * a.h_width(l) * 256 for l in range(4))
    streams = (n * n * 6 * 32 * 32 + n * a.n_ions * 3 * 32 * 32)
    network = 2.0 * (n * per_el + per_walker)
    dets = 2.0 * case["n_dets"] * n ** 3
    passes = _passes(case, n)
    flops = B * (passes * network + 2.0 * streams * min(passes, 3 if case["op"] == "energy" else passes))
    if case["op"] in ("energy", "step"):
        flops += B * dets * (1 + 3 * n)          # inverse, and A^-1 dA of every direction
    else:
        flops += B * dets / 3 * passes
    n_params = sum(int(np.prod(s)) for s in P.param_shapes(a).values())
    outputs = {"logpsi": 2 * B, "mcmc": B * (3 * n + 2), "energy": B * (3 * n + 2), "gradient": n_params,
               "step": B + n_params}[case["op"]]
    return {"bytes": 4.0 * (B * 3 * n + n_params + outputs), "flops": flops}


# ------------------------------------------------------------------- the same in 64 bits, in plain torch
# A jet is a tensor with a leading channel axis: [value, d/dr_1x, d/dr_1y, ..., d/dr_nz, Laplacian],
# or the value alone (one channel).

def _chunk(a, channels):
    """Walkers whose pair streams, layer rows and orbitals take a few GB in 64 bits."""
    n = a.n_el
    return max(1, int(4e9 / (8 * channels * (6 * n * n * 32 + n * (6 * 256 + 4 * a.n_orb_cols) + n * a.n_ions * 64))))


def _linear(x, w, b=None):
    y = x @ w
    if b is not None:
        y = torch.cat([y[:1] + b, y[1:]])
    return y


def _tanh(x):
    y = torch.tanh(x[:1])
    if len(x) == 1:
        return y
    d = 1 - y * y
    return torch.cat([y, d * x[1:-1], d * x[-1:] - 2 * y * d * (x[1:-1] ** 2).sum(0, keepdim=True)])


def _mul(x, y):
    if len(x) == 1:
        return x * y
    return torch.cat([x[:1] * y[:1], x[1:-1] * y[:1] + x[:1] * y[1:-1],
                      x[-1:] * y[:1] + x[:1] * y[-1:] + 2 * (x[1:-1] * y[1:-1]).sum(0, keepdim=True)])


def _dense(p, name, x):
    return _tanh(_linear(x, p[name + ".w"], p[name + ".b"]))


def _residual(new, old):
    return (new + old) / math.sqrt(2.0) if new.shape == old.shape else new


def _log_psi_sqr_jets(p, a, r, R, Z, jets):
    """(phase [B], log psi^2 as a jet [C, B]) of walkers r [B, n, 3]."""
    B, n, _ = r.shape
    N, K, nu, C = len(R), a.n_dets, a.n_up, 3 * n + 2 if jets else 1
    eye = torch.eye(n, dtype=r.dtype, device=r.device)
    diff = r[:, :, None] - R
    d = diff.norm(dim=-1)
    pair = r[:, None] - r[:, :, None] + eye[:, :, None]
    d_ee = pair.norm(dim=-1) * (1 - eye)
    h_ei = r.new_zeros(C, B, n, N, 4)
    h_ei[0, ..., 0], h_ei[0, ..., 1:] = d, diff
    h_ee = r.new_zeros(C, B, n, n, 1)
    h_ee[0, ..., 0] = d_ee
    if jets:
        unit = pair / (d_ee + eye)[..., None] * (1 - eye)[..., None]        # d |r_j - r_i| / d r_j
        for i in range(n):
            for c in range(3):
                t = 1 + 3 * i + c
                h_ei[t, :, i, :, 0] = diff[:, i, :, c] / d[:, i]
                h_ei[t, :, i, :, 1 + c] = 1.0
                h_ee[t, :, :, i, 0] += unit[:, :, i, c]
                h_ee[t, :, i, :, 0] -= unit[:, i, :, c]
        h_ei[-1, ..., 0] = 2 / d
        h_ee[-1, ..., 0] = 4 / (d_ee + eye) * (1 - eye)
    dist = h_ei[..., :1]
    h = h_ei.reshape(C, B, n, 4 * N)
    ion = p["ion_embed"][(Z - a.z_min).long()]
    # same-spin pairs through h_same / w_same, opposite-spin pairs through h_diff / w_diff
    up = torch.arange(n, device=r.device) < nu
    same = (up[:, None] == up[None])[:, :, None]

    def two(name_same, name_diff, x):
        return torch.where(same, _dense(p, name_same, x), _dense(p, name_diff, x))

    for l in range(a.n_iter):
        s = f"symm{l}"
        hm = _dense(p, f"{s}.h_map", h)
        conv_ee = _mul(two(f"{s}.w_same", f"{s}.w_diff", h_ee), hm[:, :, None]).sum(3)
        him = torch.tanh(ion @ p[f"{s}.h_ion_map.w"] + p[f"{s}.h_ion_map.b"])
        conv_ei = (h_ei * him).sum(3)
        mean = [x.mean(2, keepdim=True).expand(h.shape) for x in (h[:, :, :nu], h[:, :, nu:])]
        h = _dense(p, f"h_el{l}", torch.cat([h] + mean + [conv_ee, conv_ei], -1))
        if l < a.n_iter - 1:
            h_ee = _residual(two(f"h_same{l}", f"h_diff{l}", h_ee), h_ee)
            h_ei = _residual(_dense(p, f"h_ei{l}", h_ei), h_ei)

    def orbitals(x, x_dist, spin):
        bf = _linear(x, p[f"bf_{spin}.w"])
        al = torch.nn.functional.softplus(p[f"alpha_{spin}"])               # [N, K n]
        e = p[f"weights_{spin}"] * torch.exp(-al * x_dist[:1])              # [1, B, ns, N, K n]
        env = [e.sum(-2)]
        if jets:
            env.append(torch.stack([(-al * e[0] * x_dist[t]).sum(-2) for t in range(1, C - 1)]))
            # the electron's own three directions have |grad d| = 1 and Laplacian 2 / d
            env.append(((al * al - al * x_dist[-1:]) * e).sum(-2))
        return _mul(torch.cat(env), bf)

    mo = torch.cat([orbitals(h[:, :, :nu], dist[:, :, :nu], "up"), orbitals(h[:, :, nu:], dist[:, :, nu:], "dn")], 2)
    mo = mo.reshape(C, B, n, K, n).transpose(2, 3)                          # [C, B, K, n, n]
    sign, logdet = torch.linalg.slogdet(mo[0])
    shift, top = logdet.max(-1)
    w = torch.exp(logdet - shift[:, None]) * sign
    psi = w.sum(-1)
    den = psi.abs() + 1e-8
    out = [torch.log(den) + shift]
    if jets:
        inv = torch.linalg.inv(mo[0])
        g = r.new_empty(C - 2, B, K)
        lap = torch.einsum("bkij,bkji->bk", inv, mo[-1])
        for t in range(C - 2):
            m = inv @ mo[1 + t]
            g[t] = torch.einsum("bkii->bk", m)
            lap = lap - torch.einsum("bkij,bkji->bk", m, m)
        g_top = g.gather(2, top[None, :, None].expand(C - 2, B, 1))
        lap_top = lap.gather(1, top[:, None])
        u = g - g_top
        s1 = (w * u).sum(-1) * psi.sign() / den                             # gradient of log(|psi| + eps)
        s2 = (w * (lap - lap_top + (u * u).sum(0))).sum(-1) * psi.sign() / den - (s1 * s1).sum(0)
        out += list(s1 + g_top[..., 0]) + [s2 + lap_top[:, 0]]
    x = h
    for l in range(2):
        x = _dense(p, f"jas{l}", x)
    jastrow = (x @ p["jas2.w"]).sum((-2, -1))
    return torch.where(psi < 0, math.pi, 0.0), 2 * torch.stack(out) + jastrow


def _potential(r, R, Z):
    n, N = r.shape[1], len(R)
    iu, ju = torch.triu_indices(n, n, 1, device=r.device)
    I, J = torch.triu_indices(N, N, 1, device=r.device)
    Zd = Z.to(r.dtype)
    return (1 / (r[:, iu] - r[:, ju]).norm(dim=-1)).sum(-1) - (Zd / (r[:, :, None] - R).norm(dim=-1)).sum((-2, -1)) \
        + (Zd[I] * Zd[J] / (R[I] - R[J]).norm(dim=-1)).sum()


def exact(case, seed):
    # a chain's accept decisions amplify the last bit; the largest batches take too long in 64 bits
    if case["op"] == "mcmc" or work(case)["flops"] > 8e12:
        return None
    mol, a, weights, r, R, Z, coeff = _inputs(case, seed)
    double = dict(dtype=torch.float64, device="cuda")
    p = {k: torch.as_tensor(v.astype(np.float32), **double) for k, v in weights.items()}
    r, R, B, chunk = r.double(), R.double(), len(r), _chunk(a, 1)

    def energies():
        E, lps, gs = [], [], []
        for x in r.split(_chunk(a, 3 * a.n_el + 2)):
            _, j = _log_psi_sqr_jets(p, a, x, R, Z, True)
            E.append(-0.25 * j[-1] - 0.125 * (j[1:-1] ** 2).sum(0) + _potential(x, R, Z))
            lps.append(j[0])
            gs.append(j[1:-1].T)
        return torch.cat(E), torch.cat(lps), torch.cat(gs)

    def gradient(c):
        q = {k: v.clone().requires_grad_(True) for k, v in p.items()}
        for x, cx in zip(r.split(chunk), c.split(chunk)):
            (_log_psi_sqr_jets(q, a, x, R, Z, False)[1][0] * cx).sum().backward()
        offsets, total = P.layout(a)
        flat = torch.zeros(total, **double)
        for k, (o, size) in offsets.items():
            if q[k].grad is not None:
                flat[o:o + size] = q[k].grad.reshape(-1)
        return flat

    if case["op"] == "logpsi":
        got = [_log_psi_sqr_jets(p, a, x, R, Z, False) for x in r.split(chunk)]
        # the phase is 0 or pi by the sign of psi, which is not a rounded number
        return {"phase": None, "log_psi_sqr": torch.cat([j[0] for _, j in got])}
    if case["op"] == "gradient":
        return {"grads": gradient(coeff.double())}
    E, lp, g = energies()
    if case["op"] == "energy":
        return {"E_loc": E, "log_psi_sqr": lp, "grad_r": g}
    # one step from the empty clipping state (center 0, width 1e12)
    clipped = torch.tanh(E / 1e12) * 1e12
    center = clipped.mean()
    width = ((clipped - center) ** 2).mean().sqrt() * 5.0
    return {"loss": center, "E_loc": E, "E_var": ((E - E.mean()) ** 2).mean(), "clip_center": float(center),
            "clip_width": float(width), "grads": gradient((clipped - center) / B)}
