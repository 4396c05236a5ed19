"""A step moves its walkers by the same bits whether or not it also reports their energy, and the energy it reports is the
local-energy op's: FP64 steps of every kind, with digit products (20 orbitals and more), below them, and the CISD trial."""
import numpy as np
import pytest
import torch

from tests.gpu_helpers import Setup, cpu, dev
from trot_gb300 import synthetic

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")]


def _states(F, walkers, W, G, step):
    ov = cpu(F.overlap(F.walkers(walkers)))
    x = dev(synthetic.fields(W, G, 1, seed=16)[0])
    out, e = [], torch.empty(W, dtype=torch.complex128, device="cuda")
    for energy in (None, e):
        st = step(F.state(F.walkers(walkers), np.linspace(0.5, 1.5, W), ov, 0.1, -1.0), x, energy)
        w = st.walkers if isinstance(st.walkers, tuple) else (st.walkers,)
        out.append([cpu(t) for t in (*w, st.weights, st.overlaps, st.scalars)])
    return out, cpu(e)


@pytest.mark.parametrize("kind,N,nelec,G,W", [
    ("rhf_r", 12, (3, 3), 30, 9), ("rhf_r", 20, (1, 1), 40, 5), ("rhf_u", 24, (5, 5), 130, 33), ("uhf_u", 41, (9, 6), 127, 17),
    ("rhf_u", 65, (7, 7), 129, 40), ("uhf_u", 129, (12, 17), 260, 3),
    ("rhf_r", 24, (16, 16), 500, 2200), ("rhf_u", 20, (10, 10), 800, 1100)])  # two passes over the walkers
def test_step(kind, N, nelec, G, W):
    ss = synthetic.make_system(N, nelec, G, decay=30.0, seed=N, h0=0.3)
    wa = synthetic.perturbed_walkers(ss.mo_a, W, 0.1, 14)
    F = Setup(kind, ss.h0, ss.h1, 0.1 * ss.chol, ss.mo_a, ss.mo_b, 0.005, W)
    walkers = wa if kind == "rhf_r" else (wa, synthetic.perturbed_walkers(ss.mo_b, W, 0.1, 15))
    e0 = cpu(F.energy(F.walkers(walkers)))
    (a, b), e = _states(F, walkers, W, G, lambda st, x, eo: F.step(st, x, energy_out=eo))
    assert np.count_nonzero(a[-3]) > W // 2  # most walkers are live
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    assert np.array_equal(e, e0)


@pytest.mark.parametrize("N,n", [(14, 3), (24, 4)])
def test_cisd_step(N, n):
    from tests.test_gpu_cisd import CisdSetup, _synthetic

    G, W = 40, 6
    cs, w = _synthetic(N, n, G, W, 0.05)
    S = CisdSetup(cs.h0, cs.h1, 0.1 * cs.chol, 30.0 * cs.ci1, 5.0 * cs.ci2, W)  # amplitudes that count in the force bias
    S.walkers = dev
    S.state = lambda *a: Setup.state(S, *a)

    def step(st, x, eo):
        return S.prop_ops.step(st, params=S.params, ham_data=S.ham, trial_data=S.trial, trial_ops=S.trial_ops,
                               meas_ops=S.meas_ops, meas_ctx=S.meas_ctx, prop_ctx=S.prop_ctx, fields=x, energy_out=eo)

    e0 = cpu(S.energy(dev(w)))
    (a, b), e = _states(S, w, W, G, step)
    assert np.count_nonzero(a[-3]) > 0
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    assert np.array_equal(e, e0)
