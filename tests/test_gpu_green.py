"""Standalone half-rotated Green's functions (trot_half_green) against the oracle's
``_half_green_from_overlap_matrix`` restatement, per spin, with the trial overlaps."""
import numpy as np
import pytest
import torch

from oracle import afqmc_oracle as orc
from tests.gpu_helpers import Setup, cpu, rel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("kind,N,nelec,W", [("rhf_r", 20, (4, 4), 9), ("rhf_u", 20, (4, 4), 7),
                                            ("uhf_u", 31, (6, 4), 11)])
def test_half_green_matches_oracle(kind, N, nelec, W):
    from trot_gb300 import synthetic
    from trot_gb300.trial import half_green_batched

    ss = synthetic.make_system(N, nelec, 3 * N, decay=30.0, seed=5, h0=0.2)
    mo_b = ss.mo_b if kind == "uhf_u" else ss.mo_a
    S = Setup(kind, ss.h0, ss.h1, ss.chol, ss.mo_a, mo_b, 0.01, W)
    wa = synthetic.perturbed_walkers(ss.mo_a, W, 0.1, 6)
    if kind == "rhf_r":
        walkers = S.walkers(wa)
        ref = orc.half_green(wa, ss.mo_a)
    else:
        wb = synthetic.perturbed_walkers(mo_b, W, 0.1, 7)
        walkers = S.walkers((wa, wb))
        ref = np.concatenate([orc.half_green(wa, ss.mo_a), orc.half_green(wb, mo_b)], axis=1)
    green, ov = half_green_batched(walkers, S.trial, S.walker_kind, with_overlaps=True)
    assert green.shape == ref.shape
    assert rel(cpu(green), ref) <= 1e-12
    assert rel(cpu(ov), cpu(S.trial_ops.overlap(walkers, S.trial))) <= 1e-14
    assert rel(cpu(half_green_batched(walkers, S.trial, S.walker_kind)), ref) <= 1e-12


@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")
@pytest.mark.parametrize("kind,N,na,nb,W", [("rhf_r", 3, 1, 1, 2), ("rhf_r", 90, 33, 33, 3), ("uhf_u", 64, 31, 64, 2),
                                            ("uhf_u", 130, 2, 17, 5), ("rhf_u", 41, 16, 16, 3), ("rhf_r", 1500, 4, 4, 2)])
def test_green_and_overlap_sizes(kind, N, na, nb, W):
    """Half Green's functions and overlaps at the edges of the kernel: one electron, more than a warp's lanes of
    electrons, tiles that only fit without row padding, walkers of extreme magnitude.  Condition numbers of order ten,
    so 1e-12 of the largest element."""
    import trot_gb300 as tg
    from oracle import afqmc_oracle as orc
    from tests.gpu_helpers import cpu, dev
    from trot_gb300 import synthetic
    from trot_gb300.trial import half_green_batched

    rng = np.random.default_rng(N + na)
    q = np.linalg.qr(rng.standard_normal((N, max(na, nb))))[0]
    ma, mb = np.ascontiguousarray(q[:, :na]), np.ascontiguousarray(q[:, :nb])
    wk = "restricted" if kind == "rhf_r" else "unrestricted"
    trial = tg.UhfTrial(ma, mb) if kind == "uhf_u" else tg.RhfTrial(ma)
    noise = 0.3 / np.sqrt(N)
    w = [synthetic.perturbed_walkers(ma, W, noise, 3), synthetic.perturbed_walkers(mb, W, noise, 4)]
    if na <= 2:
        w[0] = w[0] * np.array([1e150, 1e-150, 1, 1, 1])[:W, None, None]  # G does not depend on the scale
    wd = dev(w[0]) if wk == "restricted" else (dev(w[0]), dev(w[1]))
    g, ov = half_green_batched(wd, trial, wk, with_overlaps=True)
    ref = [orc.half_green(w[0], ma)] + ([] if wk == "restricted" else [orc.half_green(w[1], mb)])
    scale = [np.max(np.abs(r), axis=(1, 2), keepdims=True) for r in ref]
    ref = np.concatenate([r / s for r, s in zip(ref, scale)], axis=1)
    got = cpu(g)
    got = np.concatenate([got[:, :na] / scale[0]] + ([] if wk == "restricted" else [got[:, na:] / scale[1]]), axis=1)
    assert np.max(np.abs(got - ref)) <= 1e-12
    d = [np.linalg.det(orc._ovlp_mat(m, x)) for m, x in zip((ma, mb), w)]
    want = d[0] * d[0] if wk == "restricted" else d[0] * d[1]
    fin = np.isfinite(want) & (np.abs(want) > 1e-290)
    assert np.all(np.abs(cpu(ov) - want)[fin] <= (1e-11 * np.abs(want))[fin])


@pytest.mark.parametrize("n", [1, 2, 3, 5, 12, 13, 14, 15, 32, 33, 64])
def test_eliminations(n):
    """Inverses and determinants on both sides of the line between one and four warps, with walkers whose pivots are
    real, imaginary, or outside the range of the fast reciprocal (2^-300 to 2^300).  Same bounds as above."""
    N = min(2 * n + 1, 66)
    q = np.linalg.qr(np.random.default_rng(n).standard_normal((N, n)))[0]
    _check_scaled(N, n, q, np.array([1.0, 1j, -1j, 2.0 ** 310, 2.0 ** -310, 2.0 ** 299, 0.6 - 0.8j]))


def _check_scaled(N, n, q, scales):
    import trot_gb300 as tg
    from oracle import afqmc_oracle as orc
    from tests.gpu_helpers import cpu, dev
    from trot_gb300 import synthetic
    from trot_gb300.trial import half_green_batched

    base = synthetic.perturbed_walkers(q, len(scales), 0.3 / np.sqrt(N), 3)
    g, ov = half_green_batched(dev(base * scales[:, None, None]), tg.RhfTrial(np.ascontiguousarray(q)), "restricted",
                               with_overlaps=True)
    ref = orc.half_green(base, q)  # G does not depend on the scale
    assert np.max(np.abs(cpu(g) - ref)) <= 1e-12 * np.max(np.abs(ref))
    with np.errstate(all="ignore"):
        want = np.linalg.det(orc._ovlp_mat(q, base)) ** 2 * (scales ** n) ** 2
    fin = np.isfinite(want) & (np.abs(want) > 1e-290)
    assert np.all(np.abs(cpu(ov) - want)[fin] <= (1e-11 * np.abs(want))[fin])
