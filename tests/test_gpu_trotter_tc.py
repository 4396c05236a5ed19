"""The tensor-core Trotter kernel over its K chunks of 32 orbitals and over one or two walkers per CTA: a walker's bits do
not depend on the batch, and its values are those of the float64 action."""
import numpy as np
import pytest
import torch

from tests.gpu_helpers import Setup, cpu, dev, rel

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")]


@pytest.mark.parametrize("N,n", [(3, 1), (31, 3), (32, 8), (33, 4), (64, 5), (65, 2), (96, 9), (97, 16), (128, 12)])
def test_chunks_and_walkers_per_cta(N, n):
    """151 and 152 walkers take one per CTA, 153 to 304 two, 305 one again.  2e-5 is the tolerance of the path's other
    tests (float32 operands and sums)."""
    import trot_gb300 as tg
    from trot_gb300 import synthetic

    G, W = 40, 305
    ss = synthetic.make_system(N, (n, n), G, decay=30.0, seed=N, h0=0.2)
    S = Setup("rhf_r", ss.h0, ss.h1, ss.chol, ss.mo_a, ss.mo_b, 0.005, W, mixed=True)
    w = dev(synthetic.perturbed_walkers(ss.mo_a, W, 0.1, 3))
    rng = np.random.default_rng(5)
    xs = dev(rng.normal(size=(W, G)) + 0.3j * rng.normal(size=(W, G)))
    op = tg.make_trotter_ops("restricted", "restricted", mixed_precision=True).apply_trotter
    full = op(w, xs, S.prop_ctx, 6)
    ref = tg.make_trotter_ops("restricted", "restricted").apply_trotter(w, xs, S.prop_ctx, 6)
    assert rel(cpu(full), cpu(ref)) <= 2e-5
    for m in (1, 151, 153, 304):
        assert torch.equal(op(w[:m].contiguous(), xs[:m].contiguous(), S.prop_ctx, 6), full[:m])


@pytest.mark.parametrize("terms", [1, 31, 32, 33, 64])
def test_many_terms(terms):
    """The FP64 kernel's coefficients, 32 at a time, against the oracle (1e-10, the FP64 path's tolerance)."""
    import trot_gb300 as tg
    from oracle import afqmc_oracle as orc
    from trot_gb300 import synthetic

    N, n, G, W = 9, 2, 12, 3
    ss = synthetic.make_system(N, (n, n), G, decay=30.0, seed=2, h0=0.2)
    S = Setup("rhf_r", ss.h0, ss.h1, ss.chol, ss.mo_a, ss.mo_b, 0.01, W)
    w = synthetic.perturbed_walkers(ss.mo_a, W, 0.1, 3)
    rng = np.random.default_rng(5)
    xs = rng.normal(size=(W, G)) + 0.3j * rng.normal(size=(W, G))
    got = tg.make_trotter_ops("restricted", "restricted").apply_trotter(dev(w), dev(xs), S.prop_ctx, terms)
    ref = orc.apply_trotter_r(w, xs, orc.build_prop_ctx(ss.h0, ss.h1, ss.chol, ss.rdm1(), 0.01), terms)
    assert rel(cpu(got), ref) <= 1e-10
