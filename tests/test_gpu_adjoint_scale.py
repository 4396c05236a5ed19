"""The field cotangents of the step adjoint where sqrt(dt) |V| is above one and where walker columns differ in size: the
terms of g_V = sum_l s_l u_l^H then differ by many orders, in opposite directions in the two factors."""
import ctypes

import numpy as np
import pytest
import torch

from trot_gb300 import _lib, adjoint, native, synthetic
from trot_gb300.core import QmcParams
from trot_gb300.trial import RhfTrial

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")]
TERMS = 6


def _solve_gj(m):
    """Inverses of (W, n, n) matrices by Gauss-Jordan with row pivoting, in the dtype of m (numpy.linalg has no long double)."""
    W, n, _ = m.shape
    a = np.concatenate([m, np.broadcast_to(np.eye(n, dtype=m.dtype), m.shape)], 2)
    for b in range(W):
        for k in range(n):
            p = k + int(np.argmax(np.abs(a[b, k:, k])))
            a[b, [k, p]] = a[b, [p, k]]
            a[b, k] = a[b, k] / a[b, k, k]
            for i in range(n):
                if i != k:
                    a[b, i] = a[b, i] - a[b, i, k] * a[b, k]
    return a[:, :, n:]


def _vjp(real, w, C, chol, mf, E, x, gw, dt, mult):
    """Cotangent of the walkers for the cotangent gw of the propagated ones (weights and overlaps with cotangent 0):
    g_w = E^T g_w1 + the force bias's part.  Returns (g_w, force-bias part), every sum in `real` precision."""
    c = np.clongdouble if real is np.longdouble else np.complex128
    w, gw, x = w.astype(c), gw.astype(c), x.astype(real)
    C, chol, mf, E = C.astype(real), chol.astype(real), mf.astype(real), E.astype(real)
    sq = np.sqrt(real(dt))
    N, n = C.shape
    G = chol.shape[0]
    rmul = lambda a, b: (a.real @ b) + 1j * (a.imag @ b)  # complex a @ real b
    P = _solve_gj(np.stack([C.T @ v.real + 1j * (C.T @ v.imag) for v in w]))
    Gt = np.stack([v @ p for v, p in zip(w, P)])  # (W, N, n)
    R = np.stack([C.T @ L for L in chol])  # (G, n, N)
    fb = real(mult) * rmul(Gt.transpose(0, 2, 1).reshape(len(w), -1), R.reshape(G, -1).T)
    xs = x + 1j * sq * (fb - mf)
    V = rmul(xs, chol.reshape(G, -1)).reshape(len(w), N, N)
    ck = [c(1)]
    for k in range(1, TERMS + 1):
        ck.append(ck[-1] * (1j * sq) / real(k))
    out, part = [], []
    for b in range(len(w)):
        u = [E @ w[b].real + 1j * (E @ w[b].imag)]
        for _ in range(TERMS - 1):
            u.append(V[b] @ u[-1])
        v = [E.T @ gw[b].real + 1j * (E.T @ gw[b].imag)]
        for _ in range(TERMS):
            v.append(V[b].conj().T @ v[-1])
        g1 = sum(np.conj(ck[k]) * v[k] for k in range(TERMS + 1))
        gV = sum(sum(np.conj(ck[j + l + 1]) * v[j] for j in range(TERMS - l)) @ u[l].conj().T for l in range(TERMS))
        gxs = chol.reshape(G, -1) @ gV.real.reshape(-1) + 1j * (chol.reshape(G, -1) @ gV.imag.reshape(-1))
        gfb = -1j * sq * gxs  # xs = x + i sqrt(dt) (fb - mf)
        gG = real(mult) * rmul(gfb[None], R.reshape(G, -1)).reshape(n, N).T  # of Gt
        p = (gG - C @ (Gt[b].conj().T @ gG).astype(c)) @ P[b].conj().T
        part.append(p)
        out.append(E.T @ g1.real + 1j * (E.T @ g1.imag) + p)
    return np.stack(out), np.stack(part)


@pytest.mark.parametrize("N,n,G,dt,factor,spread", [
    (80, 10, 120, 0.01, 1.0, 0), (120, 16, 150, 0.005, 1.0, 0), (33, 7, 60, 0.01, 1.0, 3), (24, 17, 40, 0.005, 0.1, 4)])
def test_field_cotangents(N, n, G, dt, factor, spread):
    """Error against long double, per walker relative to the force-bias part (the one that depends on g_V): no more than
    20 times that of the same formulas in plain float64.  factor 1: the synthetic recipe as it is, sqrt(dt) |V| from 0.9
    to 2.8; spread: the walker's columns (and, inversely, their cotangents) spread over 10^spread."""
    W = 2
    ss = synthetic.make_system(N, (n, n), G, seed=N)
    chol = factor * ss.chol
    w = synthetic.perturbed_walkers(ss.mo_a, W, 0.1, 5)
    rng = np.random.default_rng(N)
    gw = rng.standard_normal(w.shape) + 1j * rng.standard_normal(w.shape)
    scale = 10.0 ** np.linspace(-spread / 2, spread / 2, n)
    w, gw = w * scale, gw / scale
    x = rng.standard_normal((W, G))
    prob = adjoint.as_problem(0.0, chol, RhfTrial(ss.mo_a), QmcParams(dt=dt, n_walkers=W, weight_floor=0.0, weight_cap=1e300),
                              x[None], walkers0=w, e_estimate0=0.0, steps_per_block=1)
    E = adjoint.ExpH1Half.apply(torch.as_tensor(ss.h1).cuda(), prob).detach()
    # overlaps and shift terms under which the walkers stay live: the old overlaps take the propagated ones' phase
    s = prob.system(exp_h1_half=E)
    wd = torch.as_tensor(w).cuda()
    st = _lib.TrotState()
    ov = torch.full((W,), 1.0, dtype=torch.complex128, device="cuda")
    wt = torch.ones(W, dtype=torch.float64, device="cuda")
    scal = torch.zeros(2, dtype=torch.float64, device="cuda")
    nodes = torch.zeros(1, dtype=torch.int64, device="cuda")
    probe = [t.clone() for t in (wd, wt, ov, scal)]
    st.walkers_a, st.weights, st.overlaps, st.scalars = (t.data_ptr() for t in probe)
    st.node_encounters = nodes.data_ptr()
    xd = torch.as_tensor(x).cuda()
    ws, nws = native.ws_for(s, _lib.OP_PROP_STEP)
    _lib.call("trot_prop_step", ctypes.byref(s), ctypes.byref(st), xd.data_ptr(), 0, ws, nws, native.stream_ptr())
    mf = prob.mf_im.cpu().numpy()
    fb = np.stack([np.asarray(v) for v in (2 * np.einsum("gij,wji->wg", np.stack([ss.mo_a.T @ L for L in chol]), np.stack(
        [v @ np.linalg.inv(ss.mo_a.T @ v) for v in w])))])
    xs = x + 1j * np.sqrt(dt) * (fb - mf)
    c = -np.sqrt(dt) * (1j * (xs @ mf)).imag  # imp_ph = E Re(ov_new / ov_old e^{ic})
    new = probe[2].cpu().numpy()
    ov = torch.as_tensor(new * np.exp(1j * c)).cuda()
    st.walkers_a, st.weights, st.overlaps, st.scalars = wd.data_ptr(), wt.data_ptr(), ov.data_ptr(), scal.data_ptr()
    gd = torch.as_tensor(gw).cuda()
    zero_s = torch.zeros(2, dtype=torch.float64, device="cuda")
    out = [torch.empty_like(wd), torch.empty_like(wt), torch.empty_like(ov), torch.empty_like(scal), torch.zeros_like(E)]
    nb = _lib.load().trot_vjp_workspace_size(ctypes.byref(s), _lib.OP_PROP_STEP)
    vws = torch.zeros(nb, dtype=torch.uint8, device="cuda")
    _lib.call("trot_prop_step_vjp", ctypes.byref(s), ctypes.byref(st), xd.data_ptr(), gd.data_ptr(), 0, 0, 0,
              zero_s.data_ptr(), out[0].data_ptr(), 0, out[1].data_ptr(), out[2].data_ptr(), out[3].data_ptr(),
              out[4].data_ptr(), vws.data_ptr(), nb, native.stream_ptr())
    got = out[0].cpu().numpy()
    args = (w, ss.mo_a, chol, mf, E.cpu().numpy(), x, gw, dt, 2.0)
    ref, part = _vjp(np.longdouble, *args)
    f64 = _vjp(np.float64, *args)[0]
    # column by column (their sizes differ), largest over the walkers and columns
    size = np.abs(part).max(1)
    err = lambda y: float((np.abs(y - ref).max(1) / size).max())
    assert np.all(np.abs(got).max((1, 2)) > 0)  # the walkers are live
    print(f"N={N} n={n} spread={spread}: |ref|/|part| {float((np.abs(ref).max(1) / size).max()):.1f}, "
          f"float64 {err(f64):.1e}, library {err(got):.1e}")
    assert err(got) <= 20 * err(f64)
