"""The device-timeout path of the FP64 digit products, without a fault: the test switch (as in test_gpu_timeouts.py) makes
the first bounded wait of every product run out.  Nothing computed from skipped products may look like a number, the status
words keep the record, and calls after it are untouched."""
import ctypes

import numpy as np
import pytest
import torch

from tests.gpu_helpers import Setup, cpu, dev
from tests.test_gpu_timeouts import _TimeoutSwitch
from trot_gb300 import _lib, adjoint, native, synthetic

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")]
N, G, W = 24, 120, 8


def _record():
    """(sticky word of this stream's workspace, cleared; status of its last call)"""
    torch.cuda.synchronize()
    buf = native.workspace(1)
    st = ctypes.c_int(-1)
    _lib.call("trot_workspace_status", buf.data_ptr(), ctypes.addressof(st))
    last = st.value
    _lib.call("trot_workspace_timeouts", buf.data_ptr(), 1, ctypes.addressof(st))
    return st.value, last


def _isnan(x):
    return np.isnan(x.real) & np.isnan(x.imag)


def _system(kind="uhf_u"):
    ss = synthetic.make_system(N, (5, 5) if kind == "rhf_r" else (5, 4), G, decay=30.0, seed=13, h0=0.3)
    wa = synthetic.perturbed_walkers(ss.mo_a, W, 0.1, 14)
    w = wa if kind == "rhf_r" else (wa, synthetic.perturbed_walkers(ss.mo_b, W, 0.1, 15))
    return ss, Setup(kind, ss.h0, ss.h1, ss.chol, ss.mo_a, ss.mo_b, 0.005, W), w


@pytest.mark.parametrize("kind", ["rhf_r", "uhf_u"])
def test_energy_force_bias_and_step(kind):
    ss, F, walkers = _system(kind)
    w = F.walkers(walkers)
    e, fb = cpu(F.energy(w)), cpu(F.force_bias(w))
    _record()
    with _TimeoutSwitch():
        et = cpu(F.energy(w))
        assert _record() == (6, 6)
        fbt = cpu(F.force_bias(w))
        assert _record() == (6, 6)
    assert np.all(_isnan(et)) and np.all(_isnan(fbt))
    assert np.array_equal(cpu(F.energy(w)), e) and np.array_equal(cpu(F.force_bias(w)), fb)
    assert _record() == (0, 0)
    ov = cpu(F.overlap(w))
    x = dev(synthetic.fields(W, G, 2, seed=16))
    st = F.state(F.walkers(walkers), np.ones(W), ov, 0.0, -1.0)
    with _TimeoutSwitch():
        st = F.step(st, x[0])
        torch.cuda.synchronize()
        assert np.all(np.isnan(cpu(st.weights))) and np.isnan(float(st.pop_control_ene_shift))
    with pytest.raises(_lib.TrotError) as ei:
        native.check_device_timeouts()
    assert ei.value.status == 6
    st = F.step(F.state(F.walkers(walkers), np.ones(W), ov, 0.0, -1.0), x[1])
    torch.cuda.synchronize()
    assert np.all(np.isfinite(cpu(st.weights))) and _record() == (0, 0)


def test_block_energy_of_a_timed_out_call():
    """NaN energies cost their walkers their weights; those of a timed-out call make the whole block NaN."""
    _, F, walkers = _system()
    w = F.walkers(walkers)
    e = F.energy(w)
    with _TimeoutSwitch():
        et = F.energy(w)
    _record()

    def tail(energy):
        wt = torch.ones(W, dtype=torch.float64, device="cuda")
        scal = torch.tensor([0.0, float(e.real.mean())], dtype=torch.float64, device="cuda")
        obs = torch.empty(2, dtype=torch.float64, device="cuda")
        _lib.call("trot_block_energy", W, energy.data_ptr(), wt.data_ptr(), scal.data_ptr(), 0.005, 0.1, obs.data_ptr(),
                  native.stream_ptr())
        return cpu(wt), cpu(scal), cpu(obs)

    bad = e.clone()
    bad[3] = float("nan")
    wt, scal, obs = tail(bad)
    assert wt.sum() == W - 1 and np.all(np.isfinite(scal)) and np.all(np.isfinite(obs))
    wt, scal, obs = tail(et)
    assert np.all(np.isnan(wt)) and np.isnan(scal[1]) and np.all(np.isnan(obs))


def test_trotter():
    """walkers propagated by skipped products are NaN"""
    _, F, walkers = _system()
    from trot_gb300.prop import make_trotter_ops

    w = F.walkers(walkers)
    x = dev(synthetic.fields(W, G, 1, seed=3)[0]).to(torch.complex128)
    ops = make_trotter_ops("restricted", "unrestricted")
    _record()
    with _TimeoutSwitch():
        out = ops.apply_trotter(w, x, F.prop_ctx, 6)
    assert _record() == (6, 6)
    assert all(np.all(_isnan(cpu(o))) for o in out)


@pytest.mark.parametrize("op", ["step", "energy"])
def test_vjp(op):
    """The gradients of a timed-out vector-Jacobian product are NaN, all of them."""
    ss, F, walkers = _system("rhf_r")
    w = F.walkers(walkers)
    s = native.system(_lib.RHF_R, W, F.trial, F.meas_ctx, F.prop_ctx, h0=ss.h0, params=F.params)
    code = _lib.OP_PROP_STEP if op == "step" else _lib.OP_LOCAL_ENERGY
    nb = _lib.load().trot_vjp_workspace_size(ctypes.byref(s), code)
    ws = torch.zeros(nb, dtype=torch.uint8, device="cuda")
    wt, ov = torch.ones(W, dtype=torch.float64, device="cuda"), F.overlap(w)
    scal = torch.zeros(2, dtype=torch.float64, device="cuda")
    x = dev(synthetic.fields(W, G, 1, seed=3)[0])
    g = torch.ones_like(w)

    def call():
        if op == "step":
            out = [torch.zeros_like(w), torch.zeros_like(wt), torch.zeros_like(ov), torch.zeros_like(scal),
                   torch.zeros((N, N), dtype=torch.float64, device="cuda")]
            st = _lib.TrotState()
            st.walkers_a, st.weights, st.overlaps, st.scalars = w.data_ptr(), wt.data_ptr(), ov.data_ptr(), scal.data_ptr()
            _lib.call("trot_prop_step_vjp", ctypes.byref(s), ctypes.byref(st), x.data_ptr(), g.data_ptr(), 0, 0, 0,
                      scal.data_ptr(), out[0].data_ptr(), 0, out[1].data_ptr(), out[2].data_ptr(), out[3].data_ptr(),
                      out[4].data_ptr(), ws.data_ptr(), nb, native.stream_ptr())
        else:
            out = [torch.zeros_like(w), torch.zeros((N, N), dtype=torch.float64, device="cuda")]
            _lib.call("trot_local_energy_vjp", ctypes.byref(s), w.data_ptr(), 0, wt.data_ptr(), out[0].data_ptr(), 0,
                      out[1].data_ptr(), ws.data_ptr(), nb, native.stream_ptr())
        torch.cuda.synchronize()
        return [cpu(torch.view_as_real(o) if o.is_complex() else o) for o in out]

    with _TimeoutSwitch():
        bad = call()
    assert all(np.all(np.isnan(o)) for o in bad)
    assert ws[:16].view(torch.int32).tolist()[0::3] == [6, 6]
    assert all(np.all(np.isfinite(o)) for o in call())
    assert ws[:16].view(torch.int32).tolist()[0::3] == [0, 6]


def test_cisd_and_context():
    """CISD energies are NaN and its overlap's record is its own; a context whose squares timed out says so."""
    from tests.test_gpu_cisd import CisdSetup, _synthetic

    cs, w = _synthetic(31, 6, 70, W, 0.1)
    c, w = CisdSetup(cs.h0, cs.h1, cs.chol, cs.ci1, cs.ci2, W), dev(w)
    _record()
    with _TimeoutSwitch():
        e = cpu(c.energy(w))
        assert np.all(_isnan(e)) and _record() == (6, 6)
    ov = cpu(c.overlap(w))
    assert np.all(np.isfinite(ov)) and _record() == (0, 0)
    ss, F, _ = _system()
    with _TimeoutSwitch():
        with pytest.raises(_lib.TrotError) as ei:
            F.prop_ops.build_prop_ctx(F.ham, F.trial_ops.get_rdm1(F.trial), F.params)
    assert ei.value.status == 6
