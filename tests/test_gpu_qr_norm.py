"""The norms det R that orthonormalisation returns, against extended precision: every walker's is a product over its columns,
so a bias of one rounding per column shows in the mean."""
import numpy as np
import pytest
import torch

from tests.gpu_helpers import cpu, dev

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")]


def _norm_ld(w):
    """prod_j R_jj by Gram-Schmidt, iterated three times, in long double; w (W, N, n)."""
    re, im = w.real.astype(np.longdouble), w.imag.astype(np.longdouble)
    out = np.ones(len(w), np.longdouble)
    for j in range(w.shape[2]):
        for _ in range(3):
            for i in range(j):
                a, b = re[:, :, i], im[:, :, i]
                cr = (a * re[:, :, j] + b * im[:, :, j]).sum(1)[:, None]
                ci = (a * im[:, :, j] - b * re[:, :, j]).sum(1)[:, None]
                re[:, :, j] -= a * cr - b * ci
                im[:, :, j] -= a * ci + b * cr
        d = np.sqrt((re[:, :, j] ** 2 + im[:, :, j] ** 2).sum(1))
        out *= d
        re[:, :, j] /= d[:, None]
        im[:, :, j] /= d[:, None]
    return out


@pytest.mark.parametrize("N,n,W", [(24, 5, 2000), (67, 9, 500), (120, 12, 300), (135, 16, 150), (160, 24, 80), (33, 1, 2000)])
def test_norm_roundings(N, n, W):
    """Relative error, RMS over the walkers: the columns' factors round independently, each by at most 2^-53 in its
    reciprocal, its correction and its product, i.e. sqrt(3 / 3) 2^-53 RMS for errors spread evenly; the restricted norm is
    the square of the product.  2 sqrt(n) 2^-53, and its sampling (1 / sqrt(2 W), four deviations)."""
    from trot_gb300 import walkers

    rng = np.random.default_rng(N)
    c = np.linalg.qr(rng.standard_normal((N, N)))[0][:, :n]
    w = c + 0.1 * (rng.standard_normal((W, N, n)) + 1j * rng.standard_normal((W, N, n)))
    _, norm = walkers.orthogonalize(dev(w), "restricted")
    ref = _norm_ld(w) ** 2
    err = ((cpu(norm).real - ref) / ref).astype(float)
    rms = np.sqrt(np.mean(err ** 2))
    print(f"N={N} n={n}: rms {rms:.2e}, mean {err.mean():.2e}, bound {2 * np.sqrt(n) * 2.0 ** -53:.2e}")
    assert rms <= 2 * np.sqrt(n) * 2.0 ** -53 * (1 + 4 / np.sqrt(2 * W))


@pytest.mark.parametrize("N,n", [(31, 30), (128, 7), (129, 7), (160, 9), (161, 2), (256, 5), (257, 33)])
def test_gram_schmidt_rows(N, n):
    """Walkers that only Gram-Schmidt orthogonalises, at the edges of the block sizes, beside one that it does not."""
    from tests.test_gpu_qr import check

    rng = np.random.default_rng(N + n)
    w = rng.standard_normal((3, N, n)) + 1j * rng.standard_normal((3, N, n))
    w[0, :, n - 1] = (1 - 2j) * w[0, :, 0] + 1e-5 * w[0, :, n - 1]
    w[2, :, 1] = w[2, :, 0] + 1e-3 * w[2, :, 1]
    check(w)
