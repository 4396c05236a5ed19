"""Step adjoint with its Taylor chains as digit products (20 orbitals and more) against torch autograd of the CPU twin:
restricted and unrestricted columns, with and without symmetric Cholesky vectors, off the tiles, and with a dead walker."""
import numpy as np
import pytest
import torch

from oracle import afqmc_torch_twin as twin
from tests.gpu_helpers import rel
from tests.test_gpu_adjoint import _c, _problem, _rand_like

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")]


@pytest.mark.parametrize("kind,N,n,nb,symmetric,dead", [
    ("rhf_r", 20, 3, None, True, False), ("rhf_r", 24, 17, None, False, False), ("uhf_u", 33, 5, 4, True, True),
    ("rhf_u", 40, 16, None, False, True), ("uhf_u", 65, 2, 1, True, False), ("rhf_r", 129, 4, None, True, True),
    ("rhf_u", 41, 4, None, False, True)])
def test_step_vjp_chain(kind, N, n, nb, symmetric, dead):
    from trot_gb300 import adjoint

    W = 5
    ss, fields, w0, prob = _problem(N=N, n=n, nb=nb, G=22, W=W, kind=kind)
    if not symmetric:
        prob.chol_packed = None  # V is still symmetric, but the transposed operand is used
    two = kind != "rhf_r"
    ws = [w0[0].copy(), w0[1].copy()] if two else [w0.copy()]
    wts = np.linspace(0.5, 1.5, W)
    if dead:  # a walker of zero weight whose data is not finite
        ws[0][2] = np.nan
        wts[2] = 0.0
    keep = np.array([i for i in range(W) if not (dead and i == 2)])
    mo_k = (_c(ss.mo_a), _c(ss.mo_b)) if kind == "uhf_u" else _c(ss.mo_a)
    rot = lambda m: torch.einsum("pi,gpj->gij", m, _c(ss.chol))
    rc = (rot(mo_k[0]), rot(mo_k[1])) if kind == "uhf_u" else rot(mo_k)
    eh_d = adjoint.ExpH1Half.apply(torch.as_tensor(ss.h1).cuda(), prob).detach()
    es, ee = torch.tensor(-1.7, dtype=torch.float64), torch.tensor(-2.1, dtype=torch.float64)
    consts = dict(mo=mo_k, rot_chol=rc, chol=_c(ss.chol), mf_im=prob.mf_im.cpu(), h0_prop=prob.h0_prop,
                  dt=prob.params.dt, n_terms=6, kind=kind)
    # walkers whose weight the step's guards set to zero cannot influence an objective: their cotangents are zero by
    # definition, so the twin's are taken over the others
    cw0 = [_c(w[keep]) for w in ws]
    cw0 = tuple(cw0) if two else cw0[0]
    live = twin.step(cw0, _c(wts[keep]), twin._overlap_k(cw0, mo_k, kind), es, ee, _c(fields[0][keep]),
                     eh=eh_d.cpu(), **consts)[1] != 0
    keep = keep[live.numpy()]
    cw = [_c(w[keep]).requires_grad_(True) for w in ws]
    ov0 = twin._overlap_k(tuple(cw) if two else cw[0], mo_k, kind).detach()
    ov_all = torch.ones(W, dtype=torch.complex128)
    ov_all[keep] = ov0
    dev = lambda x: x.cuda().requires_grad_(True)
    wa = dev(_c(ws[0]))
    wb = dev(_c(ws[1])) if two else torch.empty(0, dtype=torch.complex128, device="cuda", requires_grad=True)
    wt, ov = dev(_c(wts)), dev(ov_all)
    scal = dev(torch.tensor([-1.7, -2.1], dtype=torch.float64))
    eh = eh_d.clone().requires_grad_(True)
    outs = adjoint.Step.apply(wa, wb, wt, ov, scal, eh, torch.as_tensor(fields[0]).cuda(), prob)
    gs = [_rand_like(o.detach().cpu(), 10 + i) for i, o in enumerate(outs)]
    gs[4][0] = 0.0  # the population shift couples all weights through their mean
    ins = (wa, wb, wt, ov, eh) if two else (wa, wt, ov, eh)
    grads = torch.autograd.grad([o for o in outs if o.numel()], ins,
                                [g.cuda() for g, o in zip(gs, outs) if o.numel()])
    out = np.setdiff1d(np.arange(W), keep)
    for g in grads[:-1]:
        assert torch.all(torch.isfinite(torch.view_as_real(g) if g.is_complex() else g))
        assert torch.all(g[torch.as_tensor(out).cuda()] == 0)
    if not keep.size:
        return
    cwt, cov = _c(wts[keep]).requires_grad_(True), ov0.clone().requires_grad_(True)
    ceh = eh.detach().cpu().requires_grad_(True)
    wn, wtn, ovn, _ = twin.step(tuple(cw) if two else cw[0], cwt, cov, es, ee, _c(fields[0][keep]), eh=ceh, **consts)
    wn = list(wn) if two else [wn]
    cg = [g[keep] for g in gs[:2] if g.numel()] + [gs[2][keep], gs[3][keep]]
    loss = sum(torch.sum((g.conj() * o).real) if o.is_complex() else torch.sum(g * o)
               for g, o in zip(cg, wn + [wtn, ovn]))
    ref = torch.autograd.grad(loss, cw + [cwt, cov, ceh])
    for g, r in zip(grads[:-1], ref[:-1]):
        assert rel(g.cpu().numpy()[keep], r.numpy()) < 1e-9
    assert rel(grads[-1].cpu().numpy(), ref[-1].numpy()) < 1e-9
