"""FP64-accurate digit products on the tensor cores (trot_zgemm_digits) against extended precision, at the edges
of the kernel's tiles (128 columns, 16 complex rows, K steps of 16, slabs of 64), and the FP64 ops with and
without the workspace the products need."""
import ctypes

import numpy as np
import pytest
import torch

from tests.gpu_helpers import Setup, cpu, dev
from trot_gb300 import _lib, native, synthetic

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")]
LD = np.longdouble


def product(a, b, nk, alpha=1.0, c0=None):
    """alpha a b(^T) (+ c0) by the library; a (M, K) complex, b (N, K) or (K, N) real."""
    M, K = a.shape
    N = b.shape[0] if nk else b.shape[1]
    A, B = dev(a), dev(b)
    C = torch.full((M, N), 7.0, dtype=torch.complex128, device="cuda") if c0 is None else dev(c0)
    ws = torch.zeros(_lib.load().trot_zgemm_digits_workspace(M, N, K), dtype=torch.uint8, device="cuda")
    _lib.call("trot_zgemm_digits", M, N, K, alpha, A.data_ptr(), K, B.data_ptr(), B.shape[1], int(nk), C.data_ptr(), N,
              int(c0 is not None), ws.data_ptr(), ws.numel(), native.stream_ptr())
    out = cpu(C)
    assert ws[:16].view(torch.int32).abs().sum().item() == 0  # no bounded wait ran out
    return out


def check(a, b, got):
    """a (M, K) complex, b (N, K) real.  Per output: both rows carry 54 bits below 2^e <= 4 max (e is raised by one for
    rows of large mean), the dropped digit products are smaller, each slab of 64 k rounds once in units of
    2^(e_a + e_b - 53 + max(0, log2 K - 10)), and the result is rounded to FP64."""
    K = a.shape[1]
    ma, mb = np.maximum(np.abs(a.real).max(1), np.abs(a.imag).max(1)), np.abs(b).max(1)
    unit = 2.0 ** (-53 + max(0, int(np.ceil(np.log2(K))) - 10))
    scale = 16.0 * ma[:, None] * mb[None]
    for x, y in ((a.real, got.real), (a.imag, got.imag)):
        ref = x.astype(LD) @ b.astype(LD).T
        tol = scale * (2.5 * K * 2.0 ** -54 + (K // 64 + 2) * unit) + 2.0 ** -52 * np.abs(ref).astype(float)
        assert np.all(np.abs((y - ref).astype(float)) <= tol)


@pytest.mark.parametrize("M,N,K,nk", [
    (1, 1, 20, True), (15, 127, 63, True), (16, 128, 64, False), (17, 129, 65, True), (33, 257, 31, False),
    (64, 300, 120, False), (5, 640, 135, True), (130, 70, 1830, True), (200, 5, 601, False), (2500, 260, 33, True)])
def test_product(M, N, K, nk):
    rng = np.random.default_rng(M + N + K)
    a = rng.standard_normal((M, K)) + 1j * rng.standard_normal((M, K))
    a *= np.exp(3 * rng.standard_normal((M, 1)))  # rows of different size
    b = rng.standard_normal((N, K)) * np.exp(-np.arange(K) / (0.3 * K))
    got = product(a, b if nk else np.ascontiguousarray(b.T), nk)
    check(a, b, got)
    c0 = rng.standard_normal((M, N)) + 1j * rng.standard_normal((M, N))
    acc = product(a, b if nk else np.ascontiguousarray(b.T), nk, alpha=-2.0, c0=c0)
    assert np.array_equal(acc, c0 - 2.0 * got)  # the product is scaled exactly and added once


def test_special_rows():
    """Equal elements (the largest digit sums), zero rows, extreme magnitudes, infinities and NaN."""
    M, N, K = 40, 140, 200
    rng = np.random.default_rng(5)
    a = rng.standard_normal((M, K)) + 1j * rng.standard_normal((M, K))
    b = rng.standard_normal((N, K))
    a[0] = 0.999 + 0.998j
    a[1] = 1.0 - 1.0j
    b[0], b[1], b[2] = 0.9990234, 1.0, -(1.0 - 2.0 ** -30)
    a[2] = 0
    b[3] = 0
    a[3] *= 1e-200
    b[4] *= 1e250
    a[4] *= 1e-290
    check(a, b, product(a, b, True))
    assert np.all(product(a, b, True)[2] == 0) and np.all(product(a, b, True)[:, 3] == 0)
    ref = product(a, b, True)
    a[7, 3] = np.nan
    a[8, 5] = complex(1.0, np.inf)
    b[130, 11] = np.inf
    got = product(a, b, True)
    assert np.all(np.isnan(got[7].real)) and np.all(np.isnan(got[:, 130]))
    assert np.all(np.isnan(got[8].imag))
    keep = np.ones((M, N), bool)
    keep[[7, 8]] = False
    keep[:, 130] = False
    assert np.array_equal(got[keep], ref[keep])


def test_rows_do_not_depend_on_the_batch():
    rng = np.random.default_rng(9)
    a = rng.standard_normal((300, 90)) + 1j * rng.standard_normal((300, 90))
    b = rng.standard_normal((200, 90))
    full = product(a, b, True)
    assert np.array_equal(product(a[37:52], b, True), full[37:52])
    assert np.array_equal(product(a, np.ascontiguousarray(b[100:171].T), False), full[:, 100:171])


@pytest.mark.parametrize("kind", ["rhf_r", "uhf_u"])
def test_small_workspace_runs_without_the_digit_products(kind):
    """A workspace that holds the op but not the products' scratch gives the same numbers on the FP64 pipe."""
    N, G, W = 26, 60, 9
    ss = synthetic.make_system(N, (4, 4) if kind == "rhf_r" else (4, 3), G, seed=2)
    S = Setup(kind, ss.h0, ss.h1, ss.chol, ss.mo_a, ss.mo_b, 0.01, W)
    wa = dev(synthetic.perturbed_walkers(ss.mo_a, W, 0.1, 3))
    wb = dev(synthetic.perturbed_walkers(ss.mo_b, W, 0.1, 4)) if kind == "uhf_u" else None
    s = native.system(native.kind_of(S.trial, S.sys.walker_kind), W, S.trial, S.meas_ctx, h0=ss.h0)
    need = _lib.load().trot_workspace_size(ctypes.byref(s), _lib.OP_LOCAL_ENERGY)
    out = []
    for frac in (1.0, 0.7, 0.5, 0.35, 0.25, 0.15):
        ws = torch.zeros(int(need * frac), dtype=torch.uint8, device="cuda")
        e = torch.zeros(W, dtype=torch.complex128, device="cuda")
        rc = _lib.load().trot_local_energy(ctypes.byref(s), wa.data_ptr(), native.ptr(wb), e.data_ptr(), ws.data_ptr(),
                                           ws.numel(), native.stream_ptr())
        assert rc in (0, 4)
        if rc == 0:
            out.append(cpu(e))
    assert len(out) >= 2
    for e in out[1:]:
        assert np.max(np.abs(e - out[0])) <= 1e-12 * np.max(np.abs(out[0]))


@pytest.mark.parametrize("kind,N,na,nb,G,W", [
    ("rhf_r", 20, 1, 1, 65, 3), ("rhf_r", 33, 2, 2, 64, 17), ("rhf_u", 40, 7, 7, 63, 5), ("uhf_u", 48, 16, 3, 130, 18),
    ("uhf_u", 37, 9, 17, 129, 33), ("rhf_r", 70, 33, 33, 71, 2), ("rhf_r", 129, 5, 5, 200, 20)])
def test_energy_from_digit_products(kind, N, na, nb, G, W):
    """Local energy (exchange sums and traces of f_g) and the step's force bias against the oracle: electrons per spin
    from 1 past 32, vectors and walkers off the kernel's chunks of 64 and 16.  FP64 sums over K <= 129 terms and G n^2
    products of a well-conditioned Green's function: 1e-11 of the largest energy."""
    from oracle import afqmc_oracle as orc

    rng = np.random.default_rng(N)
    h0, h1, chol = synthetic.hamiltonian(N, G, 30.0, seed=N, h0=0.3)
    mo = np.linalg.qr(rng.standard_normal((N, N)))[0]
    ma, mb = np.ascontiguousarray(mo[:, :na]), np.ascontiguousarray(mo[:, -nb:] if kind == "uhf_u" else mo[:, :nb])
    S = Setup(kind, h0, h1, chol, ma, mb, 0.005, W)
    w = synthetic.perturbed_walkers(ma, W, 0.05, 3)
    if kind != "rhf_r":
        w = (w, synthetic.perturbed_walkers(mb, W, 0.05, 4))
    if kind == "uhf_u":
        ctx, mo_o = orc.build_uhf_meas_ctx(h1, chol, ma, mb), (ma, mb)
    else:
        ctx, mo_o = orc.build_rhf_meas_ctx(h1, chol, ma), ma
    m = orc.Model(kind, h0, mo_o, ctx, orc.build_prop_ctx(h0, h1, chol, np.stack([ma @ ma.T, mb @ mb.T]), 0.005))
    e_ref, fb_ref = m.energy(w), m.force_bias(w)
    wd = S.walkers(w)
    e, fb = cpu(S.energy(wd)), cpu(S.force_bias(wd))
    assert np.max(np.abs(e - e_ref)) <= 1e-11 * np.max(np.abs(e_ref))
    assert np.max(np.abs(fb - fb_ref)) <= 1e-11 * np.max(np.abs(fb_ref))
    # the step takes its force bias from the traces of f_g when it also returns the energies, else from a product
    fields, outs = dev(rng.standard_normal((W, G))), []
    for with_energy in (True, False):
        wk = S.walkers(w)
        st = S.state(wk, np.ones(W), cpu(S.overlap(wk)), -1.0, -1.0)
        en = torch.zeros(W, dtype=torch.complex128, device="cuda") if with_energy else None
        S.step(st, fields, energy_out=en)
        if with_energy:
            assert np.array_equal(cpu(en), e)
        ws = st.walkers if isinstance(st.walkers, tuple) else (st.walkers,)
        outs.append([cpu(x) for x in ws])
    for x, y in zip(*outs):
        assert np.max(np.abs(x - y)) <= 1e-11 * np.max(np.abs(y))


@pytest.mark.parametrize("kind,N,na,nb,terms,W", [
    ("rhf_r", 50, 6, 6, 6, 3), ("rhf_r", 63, 16, 16, 1, 5), ("uhf_u", 64, 5, 12, 6, 2), ("uhf_u", 65, 17, 16, 10, 2),
    ("rhf_u", 96, 3, 3, 0, 4), ("rhf_r", 128, 1, 1, 6, 7), ("rhf_r", 129, 15, 15, 6, 2), ("rhf_r", 260, 3, 3, 3, 2)])
def test_trotter_from_digit_products(kind, N, na, nb, terms, W):
    """Trotter action and one step against the oracle: orbitals at the edges of the 128-row tiles of (re, im) rows and
    of K runs of 256, columns at the edges of the 32-row tiles, no and many Taylor terms.  FP64 sums over K <= 260
    terms: 1e-12 of the largest walker element."""
    from oracle import afqmc_oracle as orc

    G = 30
    rng = np.random.default_rng(N + na)
    h0, h1, chol = synthetic.hamiltonian(N, G, 30.0, seed=N)
    chol = 0.3 * chol
    mo = np.linalg.qr(rng.standard_normal((N, N)))[0]
    ma, mb = np.ascontiguousarray(mo[:, :na]), np.ascontiguousarray(mo[:, -nb:] if kind == "uhf_u" else mo[:, :nb])
    S = Setup(kind, h0, h1, chol, ma, mb, 0.01, W, n_exp_terms=terms)
    w = synthetic.perturbed_walkers(ma, W, 0.1, 3)
    if kind != "rhf_r":
        w = (w, synthetic.perturbed_walkers(mb, W, 0.1, 4))
    rho = np.stack([ma @ ma.T, mb @ mb.T])
    ctx = orc.build_prop_ctx(h0, h1, chol, rho, 0.01)
    xs = rng.standard_normal((W, G)) + 0.3j * rng.standard_normal((W, G))
    from trot_gb300.prop import make_trotter_ops

    got = make_trotter_ops("restricted", S.walker_kind).apply_trotter(S.walkers(w), dev(xs), S.prop_ctx, terms)
    ref = orc.apply_trotter_r(w, xs, ctx, terms) if kind == "rhf_r" else orc.apply_trotter_u(*w, xs, ctx, terms)
    for a, b in zip(*[(x if isinstance(x, tuple) else (x,)) for x in (got, ref)]):
        assert np.max(np.abs(cpu(a) - b)) <= 1e-12 * np.max(np.abs(b))
    mctx = orc.build_uhf_meas_ctx(h1, chol, ma, mb) if kind == "uhf_u" else orc.build_rhf_meas_ctx(h1, chol, ma)
    m = orc.Model(kind, h0, (ma, mb) if kind == "uhf_u" else ma, mctx, ctx)
    ov = m.overlap(w)
    x = rng.standard_normal((W, G))
    o = orc.afqmc_step(orc.State(w, np.ones(W), ov, -1.0, -1.0, 0), m, orc.Params(dt=0.01, n_exp_terms=terms), x)
    st = S.step(S.state(S.walkers(w), np.ones(W), ov, -1.0, -1.0), dev(x))
    assert np.max(np.abs(cpu(st.overlaps) - o.overlaps)) <= 1e-10 * np.max(np.abs(o.overlaps))
    assert np.allclose(cpu(st.weights), o.weights, rtol=1e-9, atol=1e-12)


def test_more_row_groups_than_a_grid_dimension_holds():
    """4100 walkers of 60 orbitals make 65600 groups of eight operand rows, past the 65535 of a grid's y and z; every
    walker keeps the bits of a run of its own."""
    from trot_gb300.prop import make_trotter_ops

    N, n, G, W = 60, 5, 24, 4100
    ss = synthetic.make_system(N, (n, n), G, seed=4)
    S = Setup("rhf_r", ss.h0, ss.h1, ss.chol, ss.mo_a, ss.mo_b, 0.01, W)
    w = dev(synthetic.perturbed_walkers(ss.mo_a, W, 0.1, 3))
    xs = dev(np.random.default_rng(2).standard_normal((W, G)) + 0j)
    op = make_trotter_ops("restricted", "restricted").apply_trotter
    full = op(w, xs, S.prop_ctx, 6)
    for a, b in ((0, 3), (2047, 2050), (4093, 4100)):
        assert torch.equal(full[a:b], op(w[a:b].contiguous(), xs[a:b].contiguous(), S.prop_ctx, 6))
