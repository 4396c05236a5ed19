"""The propagation context and its adjoint in workspaces without room for the squares' digit products: the sizes that the
FP64 squares need suffice, smaller ones are refused."""
import ctypes

import numpy as np
import pytest
import torch

from tests.gpu_helpers import cpu, dev
from trot_gb300 import _lib, native

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")]


def _need(N, G, vjp):
    """Bytes without digit products: status block, A, P0, P1 and the slices of the sum (adjoint: traces and four 2N x 2N
    matrices more), each at a multiple of 256 bytes."""
    tiles = ((N + 31) // 32) ** 2
    S = max(1, min(G, -(-304 // tiles)))
    S = -(-G // (-(-G // S)))
    sizes = [N * N, N * N, N * N, S * N * N] + ([G] + [4 * N * N] * 4 if vjp else [])
    used = 256
    for n in sizes:
        used = (used + 255) // 256 * 256 + 8 * n
    return used


@pytest.mark.parametrize("N,G", [(20, 30), (65, 40)])
@pytest.mark.parametrize("vjp", [False, True])
def test_small_workspace(N, G, vjp):
    rng = np.random.default_rng(N)
    h1, rho, gE = (dev(rng.standard_normal((N, N)) / N) for _ in range(3))
    chol = dev(rng.standard_normal((G, N, N)) / np.sqrt(N * G))
    lib = _lib.load()
    full = (lib.trot_prop_ctx_vjp_workspace_size_digits if vjp else lib.trot_prop_ctx_workspace_size_digits)(N, G)
    least = _need(N, G, vjp)
    assert least <= (lib.trot_prop_ctx_vjp_workspace_size if vjp else lib.trot_prop_ctx_workspace_size)(N, G) <= least + 256
    assert least < full // 4
    new = lambda *s: torch.zeros(s, dtype=torch.float64, device="cuda")

    def call(nbytes):
        ws = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
        if vjp:
            out = [new(N, N)]
            rc = lib.trot_prop_ctx_vjp(N, G, 0.05, h1.data_ptr(), chol.data_ptr(), rho.data_ptr(), gE.data_ptr(),
                                       out[0].data_ptr(), ws.data_ptr(), nbytes, native.stream_ptr())
        else:
            out = [new(G), new(1), new(N, N)]
            rc = lib.trot_build_prop_ctx(N, G, 0.3, 0.05, h1.data_ptr(), chol.data_ptr(), rho.data_ptr(), out[0].data_ptr(),
                                         out[1].data_ptr(), out[2].data_ptr(), ws.data_ptr(), nbytes, native.stream_ptr())
        st = ctypes.c_int(-1)
        _lib.call("trot_workspace_status", ws.data_ptr(), ctypes.addressof(st))
        return rc, st.value, [cpu(o) for o in out]

    ref = call(full)
    assert ref[:2] == (0, 0)
    for nbytes in (full - 512, least):
        rc, st, out = call(nbytes)
        assert (rc, st) == (0, 0)
        for a, b in zip(out, ref[2]):  # sums over N and G of elements of size one, both ways
            assert np.max(np.abs(a - b)) <= 1e-13 * max(1.0, np.max(np.abs(b)))
    assert call(least - 256)[0] == 4
