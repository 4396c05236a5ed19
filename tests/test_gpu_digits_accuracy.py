"""The digit products' accuracy as such: their error against extended precision beside that of a float64 sum of the same
terms.  (The worst-case bound of test_gpu_digits.py would still hold with seven bits fewer.)"""
import numpy as np
import pytest
import torch

from tests.test_gpu_digits import LD, product

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")]


@pytest.mark.parametrize("M,N,K,nk,most", [
    (15, 127, 63, True, 1.0), (16, 128, 64, False, 1.0), (17, 129, 65, True, 1.0), (33, 257, 31, False, 1.0),
    (64, 300, 120, False, 1.0), (5, 640, 135, True, 1.0), (70, 70, 1830, True, 0.5), (200, 5, 601, False, 0.5),
    (200, 260, 33, True, 1.0)])
def test_error_beside_a_float64_sum(M, N, K, nk, most):
    """RMS over the outputs, each relative to its rows' maxima.  Rows cut to 54 bits below their maximum give 0.1 (K = 1830)
    to 0.4 (K = 31) of a float64 sum over k in order, 52 bits 0.4 to 1.6, five planes (45 bits) 50 and more, computed for
    these operands in long double."""
    rng = np.random.default_rng(M + N + K)
    a = rng.standard_normal((M, K)) + 1j * rng.standard_normal((M, K))
    a *= np.exp(3 * rng.standard_normal((M, 1)))
    b = rng.standard_normal((N, K)) * np.exp(-np.arange(K) / (0.3 * K))
    got = product(a, b if nk else np.ascontiguousarray(b.T), nk)
    for x, y in ((a.real, got.real), (a.imag, got.imag)):
        ref = x.astype(LD) @ b.astype(LD).T
        scale = np.abs(x).max(1)[:, None] * np.abs(b).max(1)[None]
        plain = np.zeros((M, N))
        for k in range(K):
            plain += x[:, k, None] * b[None, :, k]
        rms = lambda z: float(np.sqrt(np.mean((((z - ref) / scale).astype(float)) ** 2)))
        assert rms(y) <= most * rms(plain)


def test_rows_of_very_different_elements():
    """The error is relative to the maxima of the two rows, not to the terms: a large element that meets a zero costs the
    others their last bits (2^-54 of the maxima per term), as documented for trot_zgemm_digits."""
    rng = np.random.default_rng(8)
    M, N, K = 16, 130, 120
    a = (rng.standard_normal((M, K)) + 1j * rng.standard_normal((M, K))).copy()
    b = rng.standard_normal((N, K))
    a[:, 0], b[:, 0] = 2.0 ** 20, 0.0
    got = product(a, b, True)
    ref = a.real.astype(LD) @ b.astype(LD).T
    err = np.abs(got.real - ref).astype(float) / (2.0 ** 20 * np.abs(b).max(1)[None])
    assert err.max() <= 4 * np.sqrt(K) * 2.0 ** -54
