"""The fused part of a default-precision step (force bias, shifted fields, operand image, local energy) and the
phaseless weight, off the kernel's tiles: more fields than a block has threads, a last chunk of one, padded rows."""
import numpy as np
import pytest
import torch

from tests.gpu_helpers import Setup, cpu, dev

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")]


def _setup(kind, N, nelec, G, W):
    from trot_gb300 import synthetic

    ss = synthetic.make_system(N, nelec, G, decay=30.0, seed=N, h0=0.2)
    w = [synthetic.perturbed_walkers(m, W, 0.05, 4 + i) for i, m in enumerate((ss.mo_a, ss.mo_b))]
    S = Setup(kind, ss.h0, ss.h1, ss.chol, ss.mo_a, ss.mo_b, 0.005, W, mixed=True)
    return S, (w[0] if kind == "rhf_r" else tuple(w))


@pytest.mark.parametrize("kind,N,nelec,G,W", [("rhf_r", 11, (2, 2), 1, 1), ("uhf_u", 12, (3, 2), 65, 63),
                                              ("rhf_r", 20, (4, 4), 256, 64), ("uhf_u", 23, (4, 5), 257, 65),
                                              ("rhf_u", 19, (3, 3), 521, 3)])
def test_step_is_the_sum_of_its_parts(kind, N, nelec, G, W):
    """Walkers of a step have the bits of the Trotter op on fields shifted on the host in the same roundings; its
    energies are those of the energy op up to the order of three sums of about G terms."""
    import trot_gb300 as tg

    S, w = _setup(kind, N, nelec, G, W)
    x = np.random.default_rng(G).standard_normal((W, G))
    wd = S.walkers(w)
    fb, e_ref = cpu(S.force_bias(wd)), cpu(S.energy(wd))
    mf = cpu(S.prop_ctx.mf_shifts_im)
    sq = S.prop_ctx.sqrt_dt
    xs = (x - fb.imag * sq) - 1j * (-sq * (fb.real - mf))
    want = tg.make_trotter_ops("restricted", S.walker_kind, mixed_precision=True).apply_trotter(
        S.walkers(w), dev(xs), S.prop_ctx, S.params.n_exp_terms)
    e = torch.empty(W, dtype=torch.complex128, device="cuda")
    st = S.state(S.walkers(w), np.ones(W), cpu(S.overlap(wd)), 0.0, 0.0)
    st = S.step(st, dev(x), energy_out=e)
    for a, b in zip(*((cpu(v) if isinstance(v, tuple) else (cpu(v),)) for v in (st.walkers, want))):
        assert np.array_equal(a, b)
    assert np.max(np.abs(cpu(e) - e_ref)) <= 1e-13 * max(1.0, np.max(np.abs(e_ref)))


@pytest.mark.parametrize("scale", [1.0, 1j, 1e25, 1e-25, 1e40, 1e-40, 1e200, 0.0])
@pytest.mark.parametrize("kind", ["rhf_r", "uhf_u"])
def test_phaseless_weight(kind, scale):
    """Weights for overlap ratios on both sides of the line to the general formula (2^100), and at its limits.  The
    exponent's rounding (about 1e-15) and a cosine near zero bound the error: 1e-12 of the factor's modulus."""
    S, w = _setup(kind, 16, (3, 3), 40, 9)
    x = np.random.default_rng(1).standard_normal((9, 40))
    wd = S.walkers(w)
    fb, ov = cpu(S.force_bias(wd)), cpu(S.overlap(wd))
    sq, dt, mf = S.prop_ctx.sqrt_dt, 0.005, 1j * cpu(S.prop_ctx.mf_shifts_im)
    shift = -sq * (1j * fb - mf)
    e_shift = -3.0 if abs(scale) == 0 else -3.0 - np.log(abs(scale)) / dt * (abs(np.log10(abs(scale))) < 200)
    old = ov * scale
    st = S.state(S.walkers(w), np.ones(9), old, e_shift, 0.0)
    st = S.step(st, dev(x))
    new, got = cpu(st.overlaps), cpu(st.weights)
    with np.errstate(all="ignore"):
        ratio = new / old
        v = -sq * ((x - shift) @ mf)
        u = v + (x * shift - 0.5 * shift ** 2).sum(1) + dt * (e_shift + S.prop_ctx.h0_prop)
        imp, ph = np.exp(u) * ratio, np.exp(v) * ratio
        fac = np.abs(imp) * np.cos(np.angle(ph))
        fac = np.where(np.isfinite(fac) & (fac >= 1e-3), fac, 0.0)
        fac = np.where(fac > 100.0, 0.0, fac)
    assert np.all(np.abs(got - fac) <= 1e-12 * np.where(np.isfinite(imp), np.abs(imp), 1.0))
