"""Performance cases of the phaseless-AFQMC framework.

Each case is one call (or one short chain of calls) that a user's program makes through the public entry
points: a phaseless step with the local energy of the incoming walkers, a whole block, a local-energy
measurement, the walker tail of a block (QR, resampling), an energy gradient.  The systems follow the seeded
synthetic recipe of ``trot_gb300.synthetic`` (symmetric Cholesky vectors with an exponential decay, trial
orbitals, walkers near the trial), made on the GPU; the Cholesky vectors carry the 0.1 factor under which the
population of the recipe stays alive.

``exact`` restates the same formulas in plain torch complex128.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import trot_gb300 as tg
from trot_gb300 import adjoint, blocks, mixed, walkers

DEV = "cuda"


def listed():
    return [
        # the smallest calls, where launches and latency count: one whole block (5 steps, QR, energy, SR) of a
        # small molecule in the default precision, and one mixed-precision step of the same system
        dict(name="block_fp64_n24_w64", op="block", kind="rhf_r", precision="fp64", norb=24, na=5, nb=5, nchol=120,
             decay=30.0, nwalk=64, dt=0.005, steps=5),
        dict(name="step_mixed_n24_w64", op="step", kind="rhf_r", precision="mixed", norb=24, na=5, nb=5, nchol=120,
             decay=30.0, nwalk=64, dt=0.005),
        # production propagation, UHF trial: default precision and the tensor-core path
        dict(name="step_fp64_uhf_n120_w1024", op="step", kind="uhf_u", precision="fp64", norb=120, na=12, nb=10,
             nchol=600, decay=150.0, nwalk=1024, dt=0.005),
        dict(name="step_mixed_uhf_n120_w1024", op="step", kind="uhf_u", precision="mixed", norb=120, na=12, nb=10,
             nchol=600, decay=150.0, nwalk=1024, dt=0.005),
        # a medium closed-shell system in the default precision
        dict(name="step_fp64_n80_w512", op="step", kind="rhf_r", precision="fp64", norb=80, na=10, nb=10, nchol=400,
             decay=30.0, nwalk=512, dt=0.01),
        # fragments of a local-correlation batch: ragged sizes, few walkers each
        dict(name="step_fp64_n135_w128", op="step", kind="rhf_r", precision="fp64", norb=135, na=16, nb=16, nchol=540,
             decay=30.0, nwalk=128, dt=0.005),
        dict(name="step_mixed_n97_w128", op="step", kind="rhf_r", precision="mixed", norb=97, na=12, nb=12, nchol=388,
             decay=30.0, nwalk=128, dt=0.005),
        # a measurement on a default-sized population: local energy and force bias, RHF trial, unrestricted walkers
        dict(name="energy_fp64_n67_w200", op="energy", kind="rhf_u", precision="fp64", norb=67, na=9, nb=9, nchol=270,
             decay=30.0, nwalk=200, dt=0.005),
        # CISD trial: one step at the trial's default precision, and a float64 (testing=True) local energy
        dict(name="step_cisd_n60_w256", op="step", kind="cisd", precision="mixed", norb=60, na=8, nb=8, nchol=300,
             decay=30.0, nwalk=256, dt=0.005),
        dict(name="energy_cisd_fp64_n41_w96", op="energy", kind="cisd", precision="fp64", norb=41, na=6, nb=6,
             nchol=164, decay=30.0, nwalk=96, dt=0.005),
        # backward: energy and its gradient through a block of two steps (forward, recompute, adjoint)
        dict(name="grad_n80_w512", op="grad", kind="rhf_r", precision="fp64", norb=80, na=10, nb=10, nchol=400,
             decay=30.0, nwalk=512, dt=0.01, steps=2),
        # the walker tail of a block: QR with norms, overlaps, comb resampling
        dict(name="tail_uhf_n120_w1024", op="tail", kind="uhf_u", precision="fp64", norb=120, na=12, nb=10, nchol=8,
             decay=150.0, nwalk=1024, dt=0.005),
    ]


def _loguni(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        op, kind, precision = rng.choice([
            ("step", "rhf_r", "fp64"), ("step", "uhf_u", "fp64"), ("step", "rhf_u", "fp64"), ("step", "rhf_r", "mixed"),
            ("step", "uhf_u", "mixed"), ("block", "rhf_r", "fp64"), ("block", "uhf_u", "mixed"),
            ("energy", "rhf_r", "fp64"), ("energy", "uhf_u", "fp64"), ("energy", "rhf_u", "mixed"),
            ("step", "cisd", "mixed"), ("energy", "cisd", "fp64"), ("grad", "rhf_r", "fp64"), ("tail", "uhf_u", "fp64")])
        top = 128 if precision == "mixed" else 160
        if kind == "uhf_u":
            top = 128
        if kind == "rhf_u":
            top = 120
        if kind == "cisd":
            top = 60
        if op == "grad":
            top = 96
        norb = _loguni(rng, 20, top)
        na = max(2, min(16, int(round(norb * rng.uniform(0.08, 0.2)))))
        if kind == "cisd":
            na = max(2, min(8, na))
        nb = na if kind != "uhf_u" else max(1, na - rng.randrange(0, 3))
        nchol = max(10, int(round(norb * rng.uniform(2.5, 5.0))))
        nwalk = _loguni(rng, 24, 256 if kind == "cisd" else 1024)
        case = dict(op=op, kind=kind, precision=precision, norb=norb, na=na, nb=nb, nchol=8 if op == "tail" else nchol,
                    decay=rng.choice([30.0, 150.0]), nwalk=nwalk, dt=rng.choice([0.005, 0.01]))
        if op == "block":
            case["steps"] = rng.randrange(2, 6)
        if op == "grad":
            case["steps"] = rng.randrange(1, 4)
        if _cost(case) <= most:
            return case


def _rand(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return lambda *s: torch.randn(*s, generator=g, device=DEV, dtype=torch.float64)


def _inputs(case, seed):
    """The arrays of one case, from the seed alone (plain torch)."""
    N, na, nb, G, W = case["norb"], case["na"], case["nb"], case["nchol"], case["nwalk"]
    rnd = _rand(seed)
    h1 = 0.05 * rnd(N, N)
    h1 = torch.triu(h1, 1)
    h1 = h1 + h1.T + torch.diag(-2.0 * torch.special.ndtr(rnd(N)))
    chol = rnd(G, N, N)
    chol = 0.5 * (chol + chol.transpose(1, 2))
    chol = chol * (0.03 * torch.exp(-torch.arange(G, device=DEV, dtype=torch.float64) / case["decay"]))[:, None, None]
    eps, c = torch.linalg.eigh(h1)
    d = dict(h0=0.0)
    if case["kind"] == "cisd":  # molecular-orbital basis, singles and doubles amplitudes
        h1 = c.T @ h1 @ c
        chol = torch.einsum("gpj,pi->gij", chol @ c, c).contiguous()
        v = N - na
        den = eps[None, None, na:, None] + eps[None, None, None, na:] - eps[:na, None, None, None] - \
            eps[None, :na, None, None] + 0.5
        c2 = (rnd(na, na, v, v) / den).permute(0, 2, 1, 3)
        c2 = 0.5 * (c2 + c2.permute(2, 3, 0, 1))
        d["ci1"] = 0.02 * rnd(na, v)
        d["ci2"] = (c2 * (0.2 / c2.norm())).contiguous()
        ca = torch.eye(N, device=DEV, dtype=torch.float64)[:, :na].contiguous()
        cb = ca
    else:
        # UHF: the beta orbitals of a slightly different core
        ca = c[:, :na].contiguous()
        cb = ca
        if case["kind"] == "uhf_u":
            t = 0.05 * rnd(N, N)
            cb = torch.linalg.eigh(h1 + 0.5 * (t + t.T))[1][:, :nb].contiguous()
    noise = 0.05 if case["kind"] == "cisd" else 0.1

    def near(mo):
        return (mo[None] + noise * torch.complex(rnd(W, N, mo.shape[1]), rnd(W, N, mo.shape[1]))).contiguous()

    w = near(ca) if case["kind"] in ("rhf_r", "cisd") else (near(ca), near(cb))
    steps = case.get("steps", 1)
    x = rnd(steps, W, G)
    weights = 0.5 + torch.special.ndtr(rnd(W))
    zeta = float(torch.special.ndtr(rnd(1))[0]) * 0.999
    d.update(h1=h1.contiguous(), chol=chol.contiguous(), ca=ca, cb=cb, w=w, x=x, weights=weights, zeta=zeta)
    # the running energy estimate a chain has in hand: the first walker's local energy
    one = tuple(t[:1] for t in w) if isinstance(w, tuple) else w[:1]
    d["e0"] = float(_energy(case, d, one).real[0])
    return d


def _wkind(case):
    return "restricted" if case["kind"] in ("rhf_r", "cisd") else "unrestricted"


def prepare(case, seed):
    d = _inputs(case, seed)
    N, na, nb, W = case["norb"], case["na"], case["nb"], case["nwalk"]
    mx = case["precision"] == "mixed"
    sysm = tg.System(norb=N, nelec=(na, nb), walker_kind=_wkind(case))
    ham = tg.HamChol(h0=d["h0"], h1=d["h1"], chol=d["chol"])
    params = tg.QmcParams(dt=case["dt"], n_walkers=W, n_prop_steps=case.get("steps", 1), seed=1)
    if case["kind"] == "cisd":
        trial = tg.cisd.CisdTrial(ci1=d["ci1"], ci2=d["ci2"])
        trial_ops = tg.cisd.make_cisd_trial_ops(sysm)
        meas_ops = tg.cisd.make_cisd_meas_ops(sysm) if mx else tg.cisd.make_cisd_meas_ops(sysm, testing=True,
                                                                                         mixed_precision=False)
    elif case["kind"] == "uhf_u":
        trial = tg.UhfTrial(d["ca"], d["cb"])
        trial_ops = tg.make_uhf_trial_ops(sysm)
        meas_ops = tg.make_uhf_meas_ops(sysm, mixed_precision=mx)
    else:
        trial = tg.RhfTrial(d["ca"])
        trial_ops = tg.make_rhf_trial_ops(sysm)
        meas_ops = tg.make_rhf_meas_ops(sysm, mixed_precision=mx)
    s = dict(case=case, sys=sysm, ham=ham, trial=trial, trial_ops=trial_ops, meas_ops=meas_ops, params=params,
             w=d["w"], x=d["x"], weights=d["weights"], zeta=d["zeta"], h1=d["h1"])
    if case["op"] == "grad":
        s["prob"] = adjoint.as_problem(d["h0"], d["chol"], trial, params, d["x"], walkers0=d["w"], e_estimate0=d["e0"],
                                       steps_per_block=case["steps"])
        return s
    if case["op"] == "tail":
        return s
    s["meas_ctx"] = meas_ops.build_meas_ctx(ham, trial)
    if case["op"] == "energy":
        if mx and case["kind"] != "cisd":
            mixed.context(s["meas_ctx"], None)
        return s
    prop_ops = tg.make_prop_ops("restricted", _wkind(case), mixed_precision=mx)
    s["prop_ops"] = prop_ops
    s["prop_ctx"] = prop_ops.build_prop_ctx(ham, trial_ops.get_rdm1(trial), params)
    if mx:  # the operands a program keeps for its run
        mixed.context(None if case["kind"] == "cisd" else s["meas_ctx"], s["prop_ctx"])
        if case["op"] == "block":
            mixed.context(s["meas_ctx"], None)
    st = prop_ops.init_prop_state(sys=sysm, ham_data=ham, trial_ops=trial_ops, trial_data=trial, meas_ops=meas_ops,
                                  params=params, initial_walkers=d["w"], initial_e_estimate=d["e0"])
    s["st"] = st._replace(weights=d["weights"].clone())
    s["e_out"] = torch.empty(W, dtype=torch.complex128, device=DEV)
    return s


def _state_out(st):
    return {"walkers": st.walkers, "weights": st.weights, "overlaps": st.overlaps, "scalars": st.scalars,
            "nodes": st.node_encounters}


def run(s):
    op = s["case"]["op"]
    if op == "step":
        st = s["prop_ops"].step(s["st"], params=s["params"], ham_data=s["ham"], trial_data=s["trial"],
                                trial_ops=s["trial_ops"], meas_ops=s["meas_ops"], meas_ctx=s["meas_ctx"],
                                prop_ctx=s["prop_ctx"], fields=s["x"][0], energy_out=s["e_out"])
        return {**_state_out(st), "energy": s["e_out"]}
    if op == "block":
        st, obs = blocks.block(s["st"], sys=s["sys"], params=s["params"], ham_data=s["ham"], trial_data=s["trial"],
                               trial_ops=s["trial_ops"], meas_ops=s["meas_ops"], meas_ctx=s["meas_ctx"],
                               prop_ops=s["prop_ops"], prop_ctx=s["prop_ctx"], fields_seq=s["x"], zeta=s["zeta"])
        s["st"] = st  # the chain goes on from here
        return {**_state_out(st), "block_energy": obs.scalars["energy"], "block_weight": obs.scalars["weight"]}
    if op == "energy":
        a = (s["w"], s["ham"], s["meas_ctx"], s["trial"])
        return {"energy": s["meas_ops"].require_kernel("energy")(*a),
                "force_bias": s["meas_ops"].require_kernel("force_bias")(*a)}
    if op == "grad":
        J, g = adjoint.energy_and_grad(s["h1"], s["prob"])
        return {"J": J, "grad": g}
    q, norm = walkers.orthogonalize(s["w"], s["sys"].walker_kind)
    ov = s["trial_ops"].overlap(q, s["trial"])
    w2, wt, idx = walkers.stochastic_reconfiguration(q, s["weights"], s["zeta"], s["sys"].walker_kind,
                                                     return_indices=True)
    return {"norm": norm, "overlaps": ov, "walkers": w2, "weights": wt, "indices": idx}


# ------------------------------------------------------------------ work of one pass
def _flops(case):
    N, G, W = case["norb"], case["nchol"], case["nwalk"]
    ns = [case["na"]] if _wkind(case) == "restricted" else [case["na"], case["nb"]]
    nt, n2 = sum(ns), sum(n * n for n in ns)
    if case["op"] == "tail":
        return W * sum(8 * N * n * n for n in ns)
    green = W * (4 * N * n2 + 8 * N * n2)
    energy = green + W * 4 * G * n2 * N
    prop = W * (4 * G * N * (N + 1) // 2 + 6 * 8 * N * N * nt + 2 * 4 * N * N * nt + 4 * N * n2)
    if case["kind"] == "cisd":
        n, v = case["na"], N - case["na"]
        nv = n * v
        fb = green + W * (4 * nv * nv + 16 * N * N * n + 4 * G * n * N + 4 * G * N * (N + 1) // 2)
        # gl, glgp and the l2ci2 quadratic form, the n x n products
        energy = fb + W * G * (4 * n * N * N + 8 * n * n * v + 4 * nv * nv + 4 * n * n * N * 2 + 8 * n * N * n)
        prop += W * 4 * nv * nv
    if case["op"] == "energy":
        return energy + (0 if case["kind"] != "cisd" else fb)
    if case["op"] == "step":
        return energy + prop
    fbias = green + W * 4 * G * nt * N
    if case["op"] == "block":
        return case["steps"] * (fbias + prop) + energy + W * sum(8 * N * n * n for n in ns)
    # gradient: a step forward, and backward twice its products; the energy and its adjoint
    return case["steps"] * (3 * (fbias + prop)) + 3 * energy


def _bytes(case):
    N, G, W = case["norb"], case["nchol"], case["nwalk"]
    nt = case["na"] if _wkind(case) == "restricted" else case["na"] + case["nb"]
    wb = 16 * W * N * nt
    if case["op"] == "tail":
        return 2 * wb + 8 * W * 6
    rot = 8 * G * N * (nt if case["kind"] == "uhf_u" else case["na"])
    ci = 8 * (case["na"] * (N - case["na"])) ** 2 if case["kind"] == "cisd" else 0
    chol = 8 * G * N * (N + 1) // 2
    if case["op"] == "energy":
        return wb + rot + ci + (chol if case["kind"] == "cisd" else 0) + 16 * W + 16 * W * G
    steps = case.get("steps", 1)
    return 2 * wb + rot + ci + chol + 8 * N * N + steps * 8 * W * G + 64 * W


def work(case):
    return {"bytes": _bytes(case), "flops": _flops(case)}


def _cost(case):
    """Relative cost for draw(): products, with the float64 ones weighted by their slower rate."""
    return _flops(case) * (1.0 if case["precision"] == "fp64" else 0.1)


# ------------------------------------------------------------------ the same in plain torch, 64 bits
def _c(a):
    return a.to(torch.complex128)


def _half_green(w, mo):
    m = torch.einsum("pi,bpj->bij", _c(mo), w)
    return torch.linalg.solve(m.transpose(-1, -2), w.transpose(-1, -2))


def _det(w, mo):
    return torch.linalg.det(torch.einsum("pi,bpj->bij", _c(mo), w))


def _spins(case, d, w):
    if case["kind"] in ("rhf_r", "cisd"):
        return [(w, d["ca"], 2.0)]
    return [(w[0], d["ca"], 1.0), (w[1], d["cb"], 1.0)]


def _rmul(a, b):
    """complex a @ real b"""
    return torch.complex(a.real @ b, a.imag @ b)


def _x_of(case, d, g):
    return g[:, :, case["na"]:]


def _cisd_ov(case, d, g):
    x = _x_of(case, d, g)
    o1 = torch.einsum("ia,zia->z", _c(d["ci1"]), x)
    m = (2.0 * d["ci2"] - d["ci2"].permute(0, 3, 2, 1)).reshape(x[0].numel(), -1)
    cg = _rmul(x.reshape(x.shape[0], -1), m).reshape(x.shape)
    return 1.0 + 2.0 * o1 + (cg * x).sum((1, 2)), o1, cg


def _overlap(case, d, w):
    if case["kind"] == "cisd":
        return _cisd_ov(case, d, _half_green(w, d["ca"]))[0] * _det(w, d["ca"]) ** 2
    out = 1.0
    for ws, mo, m in _spins(case, d, w):
        out = out * (_det(ws, mo) ** 2 if m == 2.0 else _det(ws, mo))
    return out


def _force_bias(case, d, w):
    G, N = d["chol"].shape[:2]
    if case["kind"] == "cisd":
        return _cisd(case, d, w, energy=False)
    fb = 0.0
    for ws, mo, m in _spins(case, d, w):
        rot = torch.matmul(mo.T, d["chol"]).reshape(G, -1)
        g = _half_green(ws, mo)
        fb = fb + m * _rmul(g.reshape(g.shape[0], -1), rot.T)
    return fb


def _energy(case, d, w, chunk=64):
    if case["kind"] == "cisd":
        W = w.shape[0]
        return torch.cat([_cisd(case, d, w[i:i + chunk], energy=True) for i in range(0, W, chunk)])
    G, N = d["chol"].shape[:2]
    W = (w[0] if isinstance(w, tuple) else w).shape[0]
    e1, coul, exc = 0.0, 0.0, 0.0
    for ws, mo, m in _spins(case, d, w):
        n = mo.shape[1]
        g = _half_green(ws, mo)
        e1 = e1 + m * torch.einsum("bij,ij->b", g, _c(mo.T @ d["h1"]))
        rot = torch.matmul(mo.T, d["chol"]).reshape(G * n, N).T
        cs, xs = [], []
        for i in range(0, W, chunk):
            gc = g[i:i + chunk]
            f = _rmul(gc.reshape(-1, N), rot).reshape(gc.shape[0], n, G, n).permute(0, 2, 3, 1)
            cs.append(torch.einsum("bgii->bg", f))
            xs.append((f * f.transpose(-1, -2)).sum((1, 2, 3)))
        coul = coul + m * torch.cat(cs)
        exc = exc + m * torch.cat(xs)
    return d["h0"] + e1 + 0.5 * (coul * coul).sum(1) - 0.5 * exc


def _cisd(case, d, w, energy):
    """Force bias, or local energy, of the CISD trial (molecular-orbital basis, all orbitals active)."""
    n, (G, N) = case["na"], d["chol"].shape[:2]
    W, v = w.shape[0], N - n
    g = _half_green(w, d["ca"])
    ov, ci1g, cg = _cisd_ov(case, d, g)
    x = _x_of(case, d, g)
    gci2g = (cg * x).sum((1, 2))
    gp = torch.zeros(W, N, v, dtype=torch.complex128, device=w.device)
    gp[:, :n] = x
    gp[:, n:] = -torch.eye(v, dtype=torch.complex128, device=w.device)
    m1 = torch.matmul(torch.matmul(gp, _c(d["ci1"].T)), g)
    m2 = torch.matmul(torch.matmul(gp, cg.transpose(1, 2)), g)
    cflat = d["chol"].reshape(G, N * N)
    lg = _rmul(g.reshape(W, -1), d["chol"][:, :n].reshape(G, -1).T)
    l1 = _rmul(m1.reshape(W, -1), cflat.T)
    l2 = _rmul(m2.reshape(W, -1), cflat.T)
    if not energy:
        return (2.0 * lg * ov[:, None] - 2.0 * (l1 + l2)) / ov[:, None]
    hg = torch.einsum("pj,bpj->b", _c(d["h1"][:n]), g)
    h1c = _c(d["h1"])
    e1 = 2.0 * hg * ov - 2.0 * torch.einsum("ij,bij->b", h1c, m1 + m2)
    f = _rmul(g.reshape(W * n, N), d["chol"][:, :n].reshape(G * n, N).T).reshape(W, n, G, n).permute(0, 2, 3, 1)
    e20 = 2.0 * (lg * lg).sum(1) - (f * f.transpose(-1, -2)).sum((1, 2, 3))
    c1g = torch.einsum("pt,bqt->bpq", _c(d["ci1"]), x)
    t1 = torch.einsum("bgpa,bap->b", torch.matmul(f, f), c1g)
    lci1 = torch.matmul(d["chol"][:, :, n:], d["ci1"].T)  # (G, N, n)
    bm = _rmul(g.reshape(W * n, N), lci1.permute(1, 0, 2).reshape(N, G * n)).reshape(W, n, G, n).permute(0, 2, 1, 3)
    t2 = (bm * f).sum((1, 2, 3))
    e21 = 2.0 * e20 * ci1g + 2.0 * (-2.0 * (l1 * lg).sum(1) + t1 - t2)
    gl = _rmul(g.reshape(W * n, N), d["chol"].permute(1, 0, 2).reshape(N, G * N)).reshape(W, n, G, N).permute(0, 2, 1, 3)
    lm = torch.matmul(_c(d["chol"][:, :n].reshape(G * n, N)), m2.transpose(1, 2)).reshape(W, G, n, N)
    t3 = (gl * lm).sum((1, 2, 3))
    y = torch.matmul(gl.reshape(W, G * n, N), gp).reshape(W * G, n * v)
    ci2m = (2.0 * d["ci2"] - d["ci2"].permute(0, 3, 2, 1)).reshape(n * v, n * v)
    t4 = (_rmul(y, ci2m) * y).sum(1).reshape(W, G).sum(1)
    e22 = e20 * gci2g + 4.0 * (-(l2 * lg).sum(1) + 0.5 * t3) + t4
    return (e1 + e20 + e21 + e22) / ov + d["h0"]


def _consts(case, d, h1):
    rd = sum(m * mo @ mo.T for mo, m in ([(d["ca"], 2.0)] if _wkind(case) == "restricted"
                                          else [(d["ca"], 1.0), (d["cb"], 1.0)]))
    t = torch.einsum("gij,ji->g", d["chol"], rd)
    v0 = 0.5 * torch.einsum("gik,gkj->ij", d["chol"], d["chol"])
    h1e = h1 - v0 + torch.einsum("g,gik->ik", t, d["chol"])
    return t, -d["h0"] + 0.5 * (t * t).sum(), torch.linalg.matrix_exp(-0.5 * case["dt"] * h1e)


def _step(case, d, k, w, wt, ov, es, ee, x):
    t, h0p, eh = k
    s, dt = math.sqrt(case["dt"]), case["dt"]
    G, N = d["chol"].shape[:2]
    fb = _force_bias(case, d, w)
    mf = 1j * _c(t)
    fs = -s * (1j * fb - mf)
    xs = _c(x) - fs
    sh = (xs * mf).sum(1)
    ft = (x * fs - 0.5 * fs * fs).sum(1)
    V = _rmul(xs, d["chol"].reshape(G, N * N)).reshape(-1, N, N)

    def prop(u):
        u = torch.matmul(_c(eh), u)
        out, term = u, u
        for j in range(1, 7):
            term = (1j * s / j) * torch.matmul(V, term)
            out = out + term
        return torch.matmul(_c(eh), out)

    w = tuple(prop(u) for u in w) if isinstance(w, tuple) else prop(w)
    ovn = _overlap(case, d, w)
    r = ovn / ov
    imp = torch.exp(-s * sh + ft + dt * (es + h0p)) * r
    ph = torch.abs(imp) * torch.cos(torch.angle(torch.exp(-s * sh) * r))
    ph = torch.where(~torch.isfinite(ph) | (ph < 1e-3), torch.zeros_like(ph), ph)
    nodes = int((ph <= 0).sum())
    ph = torch.where(ph > 100.0, torch.zeros_like(ph), ph)
    wt = wt * ph
    wt = torch.where(wt > 100.0, torch.zeros_like(wt), wt)
    es = ee - 0.1 * torch.log(torch.clamp(wt.mean(), min=1e-300)) / dt
    return w, wt, ovn, es, nodes


def _qr(w):
    q, r = torch.linalg.qr(w)
    dg = torch.diagonal(r, dim1=-2, dim2=-1)
    ph = torch.where(dg.abs() > 0, dg / dg.abs(), torch.ones_like(dg))
    return q * ph[:, None, :], dg.abs().prod(-1)


def _sr(wt, zeta):
    a = np.abs(wt.detach().cpu().numpy())
    cw = np.cumsum(a)
    W = len(a)
    idx = np.searchsorted(cw, cw[-1] * (np.arange(W) + zeta) / W, side="left").clip(max=W - 1)
    return torch.as_tensor(idx, device=DEV), torch.full((W,), cw[-1] / W, dtype=torch.float64, device=DEV)


def exact(case, seed):
    d = _inputs(case, seed)
    w, op = d["w"], case["op"]
    if op == "energy":
        return {"energy": _energy(case, d, w), "force_bias": _force_bias(case, d, w)}
    if op == "tail":
        qa, na = _qr(w[0])
        qb, nb = _qr(w[1])
        idx, wt = _sr(d["weights"], d["zeta"])
        return {"norm": _c(na * nb), "overlaps": _overlap(case, d, (qa, qb)), "walkers": (qa[idx], qb[idx]),
                "weights": wt, "indices": idx}
    es = ee = torch.tensor(d["e0"], dtype=torch.float64, device=DEV)
    if op == "grad":
        h1 = d["h1"].clone().requires_grad_(True)
        dd = dict(d, h1=h1)
        k = _consts(case, d, h1)
        wt = torch.ones(case["nwalk"], dtype=torch.float64, device=DEV)
        ov = _overlap(case, d, w).detach()
        for x in d["x"]:
            w, wt, ov, es, _ = _step(case, d, k, w, wt, ov, es, ee, x)
        q, _ = _qr(w)
        e = _energy(case, dd, q, chunk=1 << 30).real
        e = torch.where((e - ee).abs() <= math.sqrt(2.0 / case["dt"]), e, ee.expand_as(e))
        J = (wt * e).sum() / wt.sum()
        (g,) = torch.autograd.grad(J, h1)
        return {"J": J.detach(), "grad": g}
    k = _consts(case, d, d["h1"])
    wt, ov, nodes = d["weights"], _overlap(case, d, w), 0
    energy = _energy(case, d, w) if op == "step" else None
    for x in d["x"]:
        w, wt, ov, es, nd = _step(case, d, k, w, wt, ov, es, ee, x)
        nodes += nd
    count = torch.tensor([nodes], device=DEV)
    out = {"walkers": w, "weights": wt, "overlaps": ov, "scalars": torch.stack([es, ee]), "nodes": count}
    if op == "step":
        return {**out, "energy": energy}
    w = tuple(_qr(u)[0] for u in w) if isinstance(w, tuple) else _qr(w)[0]
    e = _energy(case, d, w).real
    e = torch.where((e - ee).abs() > math.sqrt(2.0 / case["dt"]), ee.expand_as(e), e)
    eb = (wt * e).sum() / wt.sum()
    idx, wsr = _sr(wt, d["zeta"])
    w2 = tuple(u[idx] for u in w) if isinstance(w, tuple) else w[idx]
    return {"walkers": w2, "weights": wsr, "overlaps": _overlap(case, d, w2),
            "scalars": torch.stack([es, 0.9 * ee + 0.1 * eb]), "nodes": count, "block_energy": eb,
            "block_weight": wt.sum()}
