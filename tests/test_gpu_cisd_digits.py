"""CISD energies and force biases in float64 with their contractions as digit products (20 orbitals and more) against
the oracle, off the tiles and chunks of the kernels, with symmetric and unsymmetric Cholesky vectors."""
import numpy as np
import pytest
import torch

import trot_gb300 as tg
from oracle import cisd_oracle as orc
from tests.gpu_helpers import cpu, dev
from trot_gb300 import synthetic

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")]


@pytest.mark.parametrize("N,n,G,W,sym", [(20, 1, 63, 3, True), (21, 5, 64, 2, False), (33, 16, 65, 3, True),
                                         (48, 17, 130, 1, True), (64, 3, 20, 17, False), (65, 8, 129, 2, True)])
def test_energy_and_force_bias(N, n, G, W, sym):
    cs = synthetic.make_cisd_system(N, n, G, seed=N, h0=0.4, scf_iters=5)
    chol = cs.chol
    if not sym:  # the formulas do not need symmetric vectors
        chol = chol + 0.05 * np.random.default_rng(1).standard_normal(chol.shape) * np.abs(chol).max(axis=(1, 2))[:, None, None]
    sysm = tg.System(norb=N, nelec=(n, n), walker_kind="restricted")
    ham = tg.HamChol(h0=cs.h0, h1=cs.h1, chol=chol)
    trial = tg.CisdTrial(ci1=cs.ci1, ci2=cs.ci2)
    ops = tg.make_cisd_meas_ops(sysm, testing=True, mixed_precision=False)
    ctx = ops.build_meas_ctx(ham, trial)
    assert ctx.chol_symmetric == sym
    w = synthetic.perturbed_walkers(np.eye(N)[:, :n], W, 0.05, 3)
    t = orc.CisdTrial(cs.ci1, cs.ci2)
    e_ref, f_ref = orc.energy(w, t, cs.h0, cs.h1, chol), orc.force_bias(w, t, chol)
    e = cpu(ops.kernels["energy"](dev(w), ham, ctx, trial))
    f = cpu(ops.kernels["force_bias"](dev(w), ham, ctx, trial))
    assert np.max(np.abs(e - e_ref)) <= 1e-11 * np.max(np.abs(e_ref))
    assert np.max(np.abs(f - f_ref)) <= 1e-11 * np.max(np.abs(f_ref))


@pytest.mark.parametrize("N,n,G,W", [(20, 1, 31, 3), (21, 7, 33, 2), (33, 9, 32, 5), (50, 17, 64, 2), (64, 3, 97, 1)])
def test_default_precision_energy(N, n, G, W):
    """The reference's float32 gl and l2ci2 with lg1 and G lci1 as digit products, off the chunks of 32 vectors, the
    tiles of 8 rows and the 64-column tiles of the split-BF16 products.  The bound is that of the default precision,
    1e-5 Hartree near the trial; the force bias stays in float64."""
    cs = synthetic.make_cisd_system(N, n, G, seed=N + 1, h0=0.4, scf_iters=5)
    sysm = tg.System(norb=N, nelec=(n, n), walker_kind="restricted")
    ham = tg.HamChol(h0=cs.h0, h1=cs.h1, chol=cs.chol)
    trial = tg.CisdTrial(ci1=cs.ci1, ci2=cs.ci2)
    ops = tg.make_cisd_meas_ops(sysm)
    ctx = ops.build_meas_ctx(ham, trial)
    w = synthetic.perturbed_walkers(np.eye(N)[:, :n], W, 0.05, 3)
    t = orc.CisdTrial(cs.ci1, cs.ci2)
    e = cpu(ops.kernels["energy"](dev(w), ham, ctx, trial))
    f = cpu(ops.kernels["force_bias"](dev(w), ham, ctx, trial))
    e_ref, f_ref = orc.energy(w, t, cs.h0, cs.h1, cs.chol), orc.force_bias(w, t, cs.chol)
    assert np.max(np.abs(e - e_ref)) <= 1e-5
    assert np.max(np.abs(f - f_ref)) <= 1e-11 * np.max(np.abs(f_ref))
