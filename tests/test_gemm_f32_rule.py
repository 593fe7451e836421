"""How fp32 products run as bf16 planes (ops/gemm.py): the rule on the CPU, its error on a GPU."""
import pytest
import torch

from gonn_b200 import lib as L
from gonn_b200.ops import gemm as G


@pytest.mark.parametrize("M,N,K,batch,chain", [
    (3000, 4096, 1024, 1, 1024), (4096, 4096, 4096, 1, 4096), (128, 4096, 4096, 1, 4096),
    (512, 512, 512, 1, 512), (128, 128, 128, 64, 128),
    # vocabulary heads and the largest squares: no less exact than the FMA kernel
    (4096, 50304, 4096, 1, 512), (50304, 4096, 4096, 1, 512), (16384, 16384, 16384, 1, 512), (13368, 13368, 13368, 1, 13368),
    (13384, 13384, 13384, 1, 512), (128, 43688, 4096, 1, 4096), (128, 43696, 4096, 1, 512), (1024, 1024, 1024, 170, 1024),
    (1024, 1024, 1024, 171, 256), (200, 10 ** 6, 200, 1, 128), (200, 10 ** 7, 100, 1, 100)])
def test_rule(M, N, K, batch, chain):
    assert G._plane_chain(M, N, K, batch) == chain


@pytest.mark.gpu
@pytest.mark.parametrize("draw", [torch.randn, torch.rand])
@pytest.mark.parametrize("M,N,K,ta,tb", [(128, 43696, 4096, False, True), (43700, 128, 4104, True, False), (136, 60000, 3000, False, False),
                                         (128, 176000, 1024, False, True), (300000, 130, 600, True, True)])
def test_the_largest_products_are_no_less_exact_than_fma(draw, M, N, K, ta, tb):
    assert 0 < G._plane_chain(M, N, K, 1) < K
    a, b = draw(*((K, M) if ta else (M, K)), device="cuda"), draw(*((N, K) if tb else (K, N)), device="cuda")
    want = (a.t() if ta else a).double() @ (b.t() if tb else b).double()
    err = {}
    for mode in ("bf16x3", "simt"):
        old = G.set_fp32_gemm_mode(mode)
        try:
            err[mode] = float((G.gemm(a, b, trans_a=ta, trans_b=tb).double() - want).norm() / want.norm())
        finally:
            G.set_fp32_gemm_mode(old)
    assert err["bf16x3"] <= err["simt"], err


@pytest.mark.gpu
@pytest.mark.parametrize("ta,tb", [(False, True), (False, False), (True, False), (True, True)])
@pytest.mark.parametrize("bias,beta,batch", [(True, False, 1), (False, True, 1), (True, True, 1), (False, True, 3)])
def test_pieces(monkeypatch, ta, tb, bias, beta, batch):
    """K in pieces with a ragged last one: bias once, the old result once, alpha in every piece."""
    M, N, K = 333, 516, 1004 if (not ta and tb) else 1000
    monkeypatch.setattr(G, "_plane_chain", lambda *s: 256)
    one = (lambda *s: torch.randn(batch, *s)) if batch > 1 else torch.randn
    a, b, bv = one(*((K, M) if ta else (M, K))), one(*((N, K) if tb else (K, N))), 30 * torch.randn(N)
    out = 30 * one(M, N)
    want = -0.5 * ((a.transpose(-1, -2) if ta else a).double() @ (b.transpose(-1, -2) if tb else b).double())
    want = want + (bv.double() if bias else 0) + (out.double() if beta else 0)
    got = G.gemm(a.cuda(), b.cuda(), trans_a=ta, trans_b=tb, alpha=-0.5, bias=bv.cuda() if bias else None,
                 out=out.cuda(), beta=beta)
    L.assert_status_ok()
    # every accumulator truncates 6 x 16 sums and every piece is rounded once: below 2^-20 together
    assert float((got.double().cpu() - want).norm() / want.norm()) < 2.0 ** -20


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,factor", [(1024, 1024, 1024, 1.0), (1024, 1024, 4096, 1.0), (3000, 4096, 1024, 2.0),
                                          (2048, 2048, 2048, 3.0), (4096, 4096, 4096, 4.5)])
def test_error_relative_to_the_fma_kernel(M, N, K, factor):
    """One accumulator truncates K / 16 sums where an FMA chain rounds K: measured ratios on normal inputs 1.7 at K = 1024, 2.6 at
    2048, 3.8 at 4096, and below 0.5 where few tiles cut K into slices."""
    torch.manual_seed(K)
    a, b = torch.randn(M, K, device="cuda"), torch.randn(K, N, device="cuda")
    want = a.double() @ b.double()
    err = {}
    for mode in ("bf16x3", "simt"):
        old = G.set_fp32_gemm_mode(mode)
        try:
            err[mode] = float((G.gemm(a, b).double() - want).norm() / want.norm())
        finally:
            G.set_fp32_gemm_mode(old)
    assert err["bf16x3"] <= factor * err["simt"], err


@pytest.mark.parametrize("M,N,K,batch,part", [(4096, 1024, 3001, 1, 384), (4096, 1024, 3583, 1, 384), (4096, 2048, 4095, 1, 512),
                                              (2048, 512, 1001, 1, 192), (1024, 1024, 1025, 1, 256), (512, 512, 513, 1, 192),
                                              (1024, 512, 333, 1, 0), (4096, 256, 391, 1, 128), (4096, 1023, 3001, 1, 0)])
def test_ragged_rule(M, N, K, batch, part):
    assert G._ragged_part(M, N, K, batch) == part


@pytest.mark.gpu
@pytest.mark.parametrize("draw", [torch.randn, torch.rand])
@pytest.mark.parametrize("M,N,K,ta,tb", [(1031, 516, 513, True, False), (130, 1000, 1537, False, False), (2050, 128, 1025, True, True),
                                         (516, 260, 4097, True, False), (1030, 1028, 2305, True, False), (2048, 1024, 257, True, False),
                                         (512, 3000, 386, True, True)])
def test_ragged_contractions_are_no_less_exact_than_fma(draw, M, N, K, ta, tb):
    assert G._ragged_part(M, N, K, 1) > 0
    a, b = draw(*((K, M) if ta else (M, K)), device="cuda"), draw(*((N, K) if tb else (K, N)), device="cuda")
    want = (a.t() if ta else a).double() @ (b.t() if tb else b).double()
    err = {}
    for mode in ("bf16x3", "simt"):
        old = G.set_fp32_gemm_mode(mode)
        try:
            err[mode] = float((G.gemm(a, b, trans_a=ta, trans_b=tb).double() - want).norm() / want.norm())
        finally:
            G.set_fp32_gemm_mode(old)
    L.assert_status_ok()
    assert err["bf16x3"] <= err["simt"], err


@pytest.mark.gpu
@pytest.mark.parametrize("room", ["slices", "two slices", "pieces", "none"])
@pytest.mark.parametrize("ta,tb,batch", [(True, False, 1), (False, False, 3), (True, True, 1)])
def test_ragged_scratch(monkeypatch, room, ta, tb, batch):
    """Slices in one launch, two slices a launch, pieces without slices, and the FMA kernel where memory is short: bias and the
    old result once, alpha in every slice."""
    M, N, K = 333, 516, 1001
    if room == "two slices":
        monkeypatch.setattr(G, "_WS_BYTES", 2 * 4 * M * N * batch + 64)
    if room == "pieces":
        monkeypatch.setattr(G, "_WS_BYTES", 4 * M * N * batch - 4)
    if room == "none":
        def short(*_):
            raise torch.OutOfMemoryError("short")
        monkeypatch.setattr(G, "_x3_workspace", short)
    one = (lambda *s: torch.randn(batch, *s)) if batch > 1 else torch.randn
    a, b, bv = one(*((K, M) if ta else (M, K))), one(*((N, K) if tb else (K, N))), 30 * torch.randn(N)
    out = 30 * one(M, N)
    want = -0.5 * ((a.transpose(-1, -2) if ta else a).double() @ (b.transpose(-1, -2) if tb else b).double())
    want = want + bv.double() + out.double()
    got = G.gemm(a.cuda(), b.cuda(), trans_a=ta, trans_b=tb, alpha=-0.5, bias=bv.cuda(), out=out.cuda(), beta=True)
    L.assert_status_ok()
    # as in test_pieces: every accumulator truncates 6 x 12 sums, every slice is rounded once; an FMA chain of 1001 is below too
    assert float((got.double().cpu() - want).norm() / want.norm()) < 2.0 ** -20


def _both_ways(a, b, **kw):
    got = {}
    for mode in ("bf16x3", "simt"):
        old = G.set_fp32_gemm_mode(mode)
        try:
            out = kw["out"].clone() if "out" in kw else None
            got[mode] = G.gemm(a, b, **{**kw, "out": out})
        finally:
            G.set_fp32_gemm_mode(old)
    L.assert_status_ok()
    return got["bf16x3"], got["simt"]


def _same(x, y):
    return bool(((x == y) | (x.isnan() & y.isnan())).all())


_ODD_OPERANDS = {
    "overflow": lambda t: t.mul_(3e37), "one large": lambda t: t[7, 5].fill_(1e35), "tiny": lambda t: t.mul_(1e-36),
    "one tiny": lambda t: t[7, 5].fill_(2e-33), "a tiny row": lambda t: t[:, 3].mul_(1e-34), "one infinity": lambda t: t[7, 5].fill_(float("inf")),
    "one nan": lambda t: t[7, 5].fill_(float("nan")), "one subnormal": lambda t: t[7, 5].fill_(1e-40), "products that vanish": lambda t: t.mul_(1e-17),
}


@pytest.mark.gpu
@pytest.mark.parametrize("what", sorted(_ODD_OPERANDS))
@pytest.mark.parametrize("M,N,K,ta,tb", [(516, 260, 1001, True, False), (384, 1024, 2049, False, False), (1031, 516, 513, True, True)])
def test_ragged_operands_outside_the_planes_range(what, M, N, K, ta, tb):
    """What would overflow between the planes, or whose parts would be subnormal: the bits of the FMA kernel."""
    assert G._ragged_part(M, N, K, 1) > 0
    torch.manual_seed(K)
    a, b = torch.randn(*((K, M) if ta else (M, K)), device="cuda"), torch.randn(*((N, K) if tb else (K, N)), device="cuda")
    bias, out = torch.randn(N, device="cuda"), torch.randn(M, N, device="cuda")
    change = _ODD_OPERANDS[what]
    if what in ("overflow", "tiny", "products that vanish"):
        change(a)
    change(b)
    for kw in (dict(), dict(bias=bias, alpha=0.5), dict(out=out, beta=True)):
        x, y = _both_ways(a, b, trans_a=ta, trans_b=tb, **kw)
        assert _same(x, y)
    assert what != "overflow" or bool(y.isinf().any())


@pytest.mark.gpu
@pytest.mark.parametrize("room", ["slices", "two slices", "pieces"])
def test_ragged_infinities_with_little_scratch(monkeypatch, room):
    M, N, K = 333, 516, 1001
    if room != "slices":
        monkeypatch.setattr(G, "_WS_BYTES", 2 * 4 * M * N + 64 if room == "two slices" else 4 * M * N - 4)
    a, b, out = torch.rand(K, M, device="cuda") + 0.5, torch.rand(K, N, device="cuda") + 0.5, torch.randn(M, N, device="cuda")
    a[K - 3, 9], b[K - 3, 11], a[5, 20] = 1e30, -1e30, 1e30
    x, y = _both_ways(a, b, trans_a=True, out=out, beta=True, bias=torch.ones(N, device="cuda"))
    assert x[9, 11] == y[9, 11] == -float("inf") and torch.equal(x.isinf(), y.isinf()) and not x.isnan().any()
    # FMA sums of 1001 products and of the pieces
    ok = y.isfinite()
    assert float((x[ok].double() - y[ok].double()).norm() / y[ok].double().norm()) < 2.0 ** -20


@pytest.mark.gpu
def test_ragged_ordinary_operands_are_products_of_planes():
    """Zeros, and magnitudes from 2^-50 to 2^48, do not send a product to the FMA kernel."""
    torch.manual_seed(3)
    a, b = torch.randn(1001, 516, device="cuda"), torch.randn(1001, 260, device="cuda")
    a[:, ::3], b[5] = 0, 0
    a[3, 1], b[9, 9] = 2.0 ** 48, 2.0 ** -50
    x, y = _both_ways(a, b, trans_a=True)
    assert not torch.equal(x, y)
    want = a.double().t() @ b.double()
    assert float((x.double() - want).norm()) <= float((y.double() - want).norm())
