"""QR orthonormalisation (Cholesky factorisations with a Gram-Schmidt fallback) against numpy's Householder QR."""
import numpy as np
import pytest
import torch

from tests.gpu_helpers import cpu, dev
from trot_gb300 import walkers

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")]


def reference(w):
    q, r = np.linalg.qr(w)
    d = np.diagonal(r, axis1=-2, axis2=-1)
    ph = np.where(np.abs(d) > 0, d / np.abs(d), 1.0)
    return q * ph[:, None, :], np.prod(np.abs(d), axis=-1)


def check(w, factor=1.0):
    """|Q - Q_ref| <= 50 kappa eps (both are backward stable), Q^H Q = I to 50 eps, norms to n kappa eps."""
    q, norm = walkers.orthogonalize(dev(w), "restricted")
    q, norm = cpu(q), cpu(norm)
    n = w.shape[2]
    eps = 2.0 ** -53
    scale = np.max(np.abs(w), axis=1)  # column scaling does not change Q: the condition number of the scaled columns
    kappa = np.linalg.cond(w / scale[:, None, :])
    ref, rn = reference(w / scale[:, None, :])
    rn = rn * np.prod(scale, axis=1)
    err = np.max(np.abs(q - ref), axis=(1, 2))
    assert np.all(err <= 50 * factor * kappa * eps), err / (kappa * eps)
    g = np.swapaxes(q.conj(), 1, 2) @ q - np.eye(n)
    assert np.max(np.abs(g)) <= 50 * eps
    with np.errstate(over="ignore"):
        rn2 = rn ** 2
    fin = np.isfinite(rn2)  # a norm past the FP64 range is inf on both sides
    assert np.all(np.abs(norm.real - rn2)[fin] <= (50 * n * kappa * eps * rn2)[fin]) and np.all(norm.imag == 0)
    assert np.array_equal(norm.real[~fin], rn2[~fin])


@pytest.mark.parametrize("W,N,n", [(3, 5, 1), (2, 7, 2), (5, 24, 5), (4, 33, 32), (2, 64, 33), (2, 127, 12), (3, 129, 16),
                                   (2, 64, 64), (1, 300, 40), (2, 190, 64)])
def test_qr(W, N, n):
    rng = np.random.default_rng(N + n)
    w = rng.standard_normal((W, N, n)) + 1j * rng.standard_normal((W, N, n))
    check(w)
    if n > 1:  # columns of very different size
        check(w * np.exp(rng.uniform(-40, 40, (W, 1, n))))


@pytest.mark.parametrize("eps", [1e-1, 1e-2, 1e-4, 1e-7])
def test_nearly_dependent_columns(eps):
    """From well inside the Cholesky route to walkers that only Gram-Schmidt orthogonalises, side by side."""
    rng = np.random.default_rng(3)
    w = rng.standard_normal((4, 40, 6)) + 1j * rng.standard_normal((4, 40, 6))
    w[1, :, 4] = w[1, :, 2] + eps * w[1, :, 4]
    w[3, :, 1] = 2j * w[3, :, 0] + eps * w[3, :, 1]
    check(w)


def test_unrestricted_norms_and_non_finite_walkers():
    rng = np.random.default_rng(4)
    a = rng.standard_normal((5, 30, 4)) + 1j * rng.standard_normal((5, 30, 4))
    b = rng.standard_normal((5, 30, 3)) + 1j * rng.standard_normal((5, 30, 3))
    a[2, 3, 1] = np.nan
    b[4, 7, 2] = np.inf
    (qa, qb), norm = walkers.orthogonalize((dev(a), dev(b)), "unrestricted")
    qa, qb, norm = cpu(qa), cpu(qb), cpu(norm).real
    ok = [0, 1, 3]
    for q, w in ((qa, a), (qb, b)):
        assert np.max(np.abs(q[ok] - reference(w[ok])[0])) < 1e-13
    assert np.allclose(norm[ok], reference(a[ok])[1] * reference(b[ok])[1], rtol=1e-13)
    assert np.isnan(norm[2]) and not np.isfinite(norm[4])
    assert np.all(np.isfinite(qb[2])) and not np.all(np.isfinite(qa[2]))
