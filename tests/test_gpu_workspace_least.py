"""Ops in the least workspace the library names (no digit scratch) and in whatever memory there is, and the Trotter digit
products in passes over the walkers."""
import numpy as np
import pytest
import torch

from tests.gpu_helpers import Setup, cpu, dev
from trot_gb300 import _lib, adjoint, native, synthetic

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")]


def _system(kind, N, nelec, G, W):
    ss = synthetic.make_system(N, nelec, G, decay=30.0, seed=N, h0=0.3)
    F = Setup(kind, ss.h0, ss.h1, 0.1 * ss.chol, ss.mo_a, ss.mo_b, 0.005, W)
    wa = synthetic.perturbed_walkers(ss.mo_a, W, 0.1, 14)
    return F, wa if kind == "rhf_r" else (wa, synthetic.perturbed_walkers(ss.mo_b, W, 0.1, 15)), ss


def _step(F, walkers, W, x):
    e = torch.empty(W, dtype=torch.complex128, device="cuda")
    st = F.step(F.state(F.walkers(walkers), np.ones(W), cpu(F.overlap(F.walkers(walkers))), 0.0, -1.0), x, energy_out=e)
    w = st.walkers if isinstance(st.walkers, tuple) else (st.walkers,)
    return [cpu(t) for t in (*w, st.weights, st.overlaps, e)]


def _close(a, b, tol=1e-11):
    for x, y in zip(a, b):
        assert np.max(np.abs(x - y)) <= tol * np.max(np.abs(y))


def _all_ops():
    """every op that has digit scratch, on small systems"""
    W, G = 6, 60
    F, walkers, ss = _system("uhf_u", 40, (7, 6), G, W)
    w, x = F.walkers(walkers), dev(synthetic.fields(W, G, 2, seed=16))
    out = [cpu(F.energy(w)), cpu(F.force_bias(w)), *_step(F, walkers, W, x[0])]
    from trot_gb300.prop import make_trotter_ops
    from trot_gb300.prop_fp import make_prop_ops_fp

    out += [cpu(t) for t in make_trotter_ops("restricted", "unrestricted").apply_trotter(w, x[1].to(torch.complex128),
                                                                                         F.prop_ctx, 6)]
    fp = make_prop_ops_fp("restricted", "unrestricted", F.sys)
    import trot_gb300 as tg

    fpp = tg.QmcParamsFp(dt=0.005, n_walkers=W, ene0=-1.0, seed=1)
    fctx = fp.build_prop_ctx(F.ham, F.trial_ops.get_rdm1(F.trial), fpp)
    st = fp.step(F.state(F.walkers(walkers), np.ones(W), np.ones(W, complex), 0.0, -1.0), params=fpp, ham_data=F.ham,
                 trial_data=F.trial, trial_ops=F.trial_ops, meas_ops=F.meas_ops, meas_ctx=F.meas_ctx, prop_ctx=fctx,
                 fields=x[0], zeta=torch.tensor([0.4], dtype=torch.float64, device="cuda"))
    out += [cpu(st.walkers[0]), cpu(st.weights)]
    R, wr, ss = _system("rhf_r", 30, (5, 5), G, W)
    prob = adjoint.as_problem(ss.h0, 0.1 * ss.chol, R.trial, R.params, synthetic.fields(W, G, 2, seed=3), walkers0=wr,
                              e_estimate0=float(cpu(R.energy(R.walkers(wr))).real.mean()), steps_per_block=2)
    J, g = adjoint.energy_and_grad(ss.h1, prob)
    out += [np.asarray([float(J)]), cpu(g) if isinstance(g, torch.Tensor) else np.asarray(g)]
    from tests.test_gpu_cisd import CisdSetup, _synthetic

    cs, cw = _synthetic(31, 6, 70, W, 0.1)
    S = CisdSetup(cs.h0, cs.h1, cs.chol, cs.ci1, cs.ci2, W)
    cw = dev(cw)
    return out + [cpu(S.energy(cw)), cpu(S.force_bias(cw)), cpu(S.overlap(cw))]


def test_least_workspace_of_every_op(monkeypatch):
    ref = _all_ops()
    asked = []

    def least_only(nbytes, least=None):
        asked.append((nbytes, nbytes if least is None else least() if callable(least) else least))
        return torch.zeros(max(asked[-1][1], 256), dtype=torch.uint8, device="cuda")

    monkeypatch.setattr(native, "workspace", least_only)
    monkeypatch.setattr(native, "empty_or_least", least_only)
    _close(_all_ops(), ref, 1e-10)
    assert sum(l < n for n, l in asked) >= 10


def test_memory_runs_out():
    """A workspace that does not fit beside the rest of the program: the least one serves, and the full one once it fits."""
    W, G = 2000, 100
    F, walkers, _ = _system("rhf_r", 96, (12, 12), G, W)
    x = dev(synthetic.fields(W, G, 1, seed=16)[0])
    ref = _step(F, walkers, W, x)
    s = native.system(_lib.RHF_R, W, F.trial, F.meas_ctx, F.prop_ctx, params=F.params)
    import ctypes

    full = _lib.load().trot_workspace_size(ctypes.byref(s), _lib.OP_PROP_STEP)
    least = _lib.load().trot_workspace_size_least(ctypes.byref(s), _lib.OP_PROP_STEP)
    room = 128 << 20  # for the step's own tensors
    assert full - least > 2 * room
    stream = torch.cuda.Stream()  # its own workspace
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    with torch.cuda.stream(stream):
        try:
            torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + least + room) / total)
            got = [_step(F, walkers, W, x) for _ in range(2)]
            size = native.workspace(256).numel()
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0)
        assert least <= size < full
        again = _step(F, walkers, W, x)
        assert native.workspace(256).numel() >= full
    _close(got[0], ref)
    for a, b in zip(got[0], got[1]):
        assert np.array_equal(a, b)
    for a, b in zip(again, ref):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("kind,nelec", [("rhf_r", (5, 5)), ("uhf_u", (3, 2))])
def test_trotter_passes(kind, nelec):
    """More walkers than one pass of the Trotter digit products takes: the same bits as a few of them alone."""
    N, G, W = 64, 24, 9000
    F, walkers, _ = _system(kind, N, nelec, G, W)
    x = dev(synthetic.fields(W, G, 1, seed=16)[0])
    whole = _step(F, walkers, W, x)
    for a, b in ((0, 40), (4480, 4540), (W - 30, W)):
        part = tuple(w[a:b] for w in walkers) if isinstance(walkers, tuple) else walkers[a:b]
        for p, q in zip(_step(F, part, b - a, x[a:b].contiguous()), whole):
            assert np.array_equal(p, q[a:b])
