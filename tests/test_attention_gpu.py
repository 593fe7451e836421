"""Flash attention kernels against materialised fp32 attention (forward, LSE, backward).
Pattern: benchmark/flashattn/main.go:102-123 (kernel vs CPU reference) and
benchmark/flashbwd/main.go:40-95 (gradient check) of the reference."""
import math

import pytest
import torch

from gonn_b200.ops import attention as A
from gonn_b200.ops.attention import attention_ref, flash_attention, flash_bwd, flash_fwd

pytestmark = pytest.mark.gpu

CASES = [(1, 128, 1, 128, False), (1, 128, 1, 64, True), (2, 256, 2, 128, True), (2, 512, 3, 64, True),
         (1, 200, 2, 128, True), (1, 333, 1, 64, False), (2, 1024, 4, 128, True),
         # the benchmark shapes' sequence lengths
         (1, 2048, 2, 128, True), (1, 4096, 2, 128, True), (1, 2048, 2, 64, False),
         # head sizes between the two compiled ones: zero-filled by the loads, clipped by the stores
         (2, 256, 2, 32, True), (1, 333, 3, 96, False), (1, 200, 2, 8, True), (2, 128, 1, 40, False),
         (1, 384, 2, 72, True), (1, 256, 2, 112, True)]


@pytest.mark.parametrize("B,S,H,D,causal", CASES)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_forward_backward(B, S, H, D, causal, dtype, status_ok):
    q, k, v = (torch.randn(B, S, H, D, device="cuda", dtype=dtype) for _ in range(3))
    scale = 1 / math.sqrt(D)
    out, lse = flash_fwd(q, k, v, causal, scale)
    qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
    ref = attention_ref(qf, kf, vf, causal, scale)
    assert (out.float() - ref).abs().max().item() < 0.02
    s = torch.einsum("bqhd,bkhd->bhqk", qf, kf) * scale
    if causal:
        s = s + torch.triu(torch.ones(S, S, device="cuda"), 1) * -1e30
    assert (lse - torch.logsumexp(s, -1)).abs().max().item() < 1e-3
    do = torch.randn_like(out)
    dq, dk, dv, _ = flash_bwd(q, k, v, out, do, lse, causal, scale)
    ref.backward(do.float())
    for got, want in ((dq, qf.grad), (dk, kf.grad), (dv, vf.grad)):
        assert (got.float() - want).abs().max().item() < 0.01 * want.abs().max().item() + 0.03


def test_strided_qkv_views(status_ok):
    B, S, H, D = 2, 256, 4, 64
    qkv = torch.randn(B, S, 3, H, D, device="cuda", dtype=torch.bfloat16)
    q, k, v = qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2]
    out = flash_attention(q, k, v, causal=True)
    ref = attention_ref(q.float(), k.float(), v.float(), True)
    assert (out.float() - ref).abs().max().item() < 0.02


def test_cross_attention_lengths(status_ok):
    q = torch.randn(2, 130, 2, 64, device="cuda", dtype=torch.bfloat16)
    k = torch.randn(2, 300, 2, 64, device="cuda", dtype=torch.bfloat16)
    v = torch.randn(2, 300, 2, 64, device="cuda", dtype=torch.bfloat16)
    q.requires_grad_(True)
    out = flash_attention(q, k, v)
    ref = attention_ref(q.float(), k.float(), v.float(), False)
    assert (out.float() - ref).abs().max().item() < 0.02
    out.sum().backward()
    assert torch.isfinite(q.grad).all()


def test_deterministic(status_ok):
    q, k, v = (torch.randn(2, 512, 4, 128, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    o1, l1 = flash_fwd(q, k, v, True, 0.1)
    do = torch.randn_like(o1)
    g1 = flash_bwd(q, k, v, o1, do, l1, True, 0.1)[:3]
    o2, l2 = flash_fwd(q, k, v, True, 0.1)
    g2 = flash_bwd(q, k, v, o2, do, l2, True, 0.1)[:3]
    assert torch.equal(o1, o2)
    for a, b in zip(g1, g2):
        assert torch.equal(a, b)


@pytest.mark.parametrize("B,Sq,Sk,H,D,causal", [(2, 512, 512, 3, 64, True), (1, 200, 200, 2, 128, True),
                                                (2, 130, 300, 2, 64, False), (1, 1024, 1024, 2, 64, True),
                                                (1, 333, 333, 1, 96, False), (2, 192, 192, 2, 64, True)])
def test_backward_with_and_without_the_dS_workspace(B, Sq, Sk, H, D, causal, status_ok):
    """The two ways to get dQ (one product with the spilled dS^T; a second pass that recomputes the
    scores) give the same dK / dV bit for bit and the same dQ up to the summation order, and both
    match fp32 attention."""
    q = torch.randn(B, Sq, H, D, device="cuda", dtype=torch.bfloat16)
    k, v = (torch.randn(B, Sk, H, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    scale = 1 / math.sqrt(D)
    out, lse = flash_fwd(q, k, v, causal, scale)
    do = torch.randn_like(out)
    old = A.DS_SPILL_LIMIT_BYTES
    try:
        A.set_ds_spill_limit(1 << 30)
        g_spill = flash_bwd(q, k, v, out, do, lse, causal, scale)[:3]
        A.set_ds_spill_limit(0)
        g_two = flash_bwd(q, k, v, out, do, lse, causal, scale)[:3]
    finally:
        A.set_ds_spill_limit(old)
    assert torch.equal(g_spill[1], g_two[1]) and torch.equal(g_spill[2], g_two[2])
    qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
    attention_ref(qf, kf, vf, causal, scale).backward(do.float())
    for got in (g_spill[0], g_two[0]):
        assert (got.float() - qf.grad).abs().max().item() < 0.01 * qf.grad.abs().max().item() + 0.03
    assert (g_spill[0].float() - g_two[0].float()).abs().max().item() < 0.02 * qf.grad.abs().max().item() + 0.01


@pytest.mark.parametrize("scale", [1e-33, 3e-38, 0.3, 4.0])
@pytest.mark.parametrize("Sq,Sk,D,causal", [(1, 1, 64, False), (65, 129, 64, False), (191, 191, 128, True), (257, 63, 128, False)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_backward_folds_the_row_statistics(scale, Sq, Sk, D, causal, dtype, status_ok):
    """The dK / dV kernel adds -LSE / scale to the scores: also where that quotient would overflow, at edges of its
    64-query steps and 128-key tiles, and where large scores make the statistics large beside their differences."""
    torch.manual_seed(Sq)
    q = torch.randn(2, Sq, 2, D, device="cuda", dtype=dtype)
    k, v = (torch.randn(2, Sk, 2, D, device="cuda", dtype=dtype) for _ in range(2))
    out, lse = flash_fwd(q, k, v, causal, scale)
    do = torch.randn_like(out)
    grads = flash_bwd(q, k, v, out, do, lse, causal, scale)[:3]
    qd, kd, vd = (t.double().requires_grad_(True) for t in (q, k, v))
    attention_ref(qd, kd, vd, causal, scale).backward(do.double())
    # roundings to the inputs' type of at most one unit each (2^-8 or 2^-11): P, the output inside Delta, dS and the result; the
    # statistics take the scores, up to 4 * 4 sqrt(D) * 4 here, to fp32: 2^-24 of that in the exponent
    unit = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    for got, want in zip(grads, (qd.grad, kd.grad, vd.grad)):
        assert torch.isfinite(got).all()
        floor = 1e-2 * unit * want.numel() ** 0.5          # gradients that vanish (scale 0, one key): rounding of P * (dP - Delta)
        assert (got.double() - want).norm() <= 4 * unit * want.norm() + floor


@pytest.mark.parametrize("B,H,Sq,Sk,D,causal", [(8, 74, 130, 130, 64, True), (8, 74, 129, 191, 64, False), (37, 32, 65, 65, 32, True),
                                                (8, 74, 256, 64, 40, False), (4, 74, 450, 450, 64, True)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_forward_of_many_tiles(B, H, Sq, Sk, D, causal, dtype, status_ok):
    """1 184 query tiles and more of heads up to 64 run with one score buffer and four CTAs per SM: edges of the 64-key steps, rows
    whose last steps are masked, a single step, running maxima that grow (scores of a few tens)."""
    torch.manual_seed(Sq)
    q = torch.randn(B, Sq, H, D, device="cuda", dtype=dtype) * 3
    k, v = (torch.randn(B, Sk, H, D, device="cuda", dtype=dtype) for _ in range(2))
    k = k * torch.linspace(0.2, 3, Sk, device="cuda")[None, :, None, None].to(dtype)
    out, lse = flash_fwd(q, k, v, causal, 0.5)
    qd, kd, vd = (t.float().transpose(1, 2) for t in (q, k, v))
    s = qd @ kd.transpose(-1, -2) * 0.5
    if causal:
        s = s.masked_fill(torch.ones(Sq, Sk, dtype=torch.bool, device="cuda").triu(1), -float("inf"))
    assert (lse - torch.logsumexp(s, -1)).abs().max().item() < 1e-3
    ref = (s.softmax(-1) @ vd).transpose(1, 2)
    # P and the result are rounded to the inputs' type: half a unit of 2^-8 or 2^-11 each, relative to sum |P V| <= max |V|
    unit = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert (out.float() - ref).abs().max().item() <= 2 * unit * vd.abs().max().item()


@pytest.mark.parametrize("bad", [float("inf"), -float("inf"), float("nan")])
@pytest.mark.parametrize("D,causal", [(64, True), (64, False), (128, True), (32, False)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_what_an_infinity_reaches_in_the_backward(bad, D, causal, dtype, status_ok):
    """One infinity or NaN in dO: its column of dV, its query's dQ and the keys that this query sees in dK.  One in V makes the output
    and Delta of many queries infinite, but dV depends on neither.  Everything else keeps its bits."""
    torch.manual_seed(D)
    q, k, v = (torch.randn(1, 200, 2, D, device="cuda", dtype=dtype) for _ in range(3))
    scale = D ** -0.5
    out, lse = flash_fwd(q, k, v, causal, scale)
    do = torch.randn_like(out)
    do[0, 70, 1, 5] = 0
    dq, dk, dv = flash_bwd(q, k, v, out, do, lse, causal, scale)[:3]
    g = do.clone()
    g[0, 70, 1, 5] = bad
    gq, gk, gv = flash_bwd(q, k, v, out, g, lse, causal, scale)[:3]
    seen = 71 if causal else 200
    other = [d for d in range(D) if d != 5]
    assert torch.equal(gv[..., other], dv[..., other]) and not torch.isfinite(gv[0, :seen, 1, 5]).any()
    rows = [r for r in range(200) if r != 70]
    assert torch.equal(gq[0, rows, 1], dq[0, rows, 1]) and not torch.isfinite(gq[0, 70, 1]).any()
    assert not torch.isfinite(gk[0, :seen, 1]).any()
    for a, b in ((gq, dq), (gk, dk), (gv, dv)):
        assert torch.equal(a[:, :, 0], b[:, :, 0])
    w = v.clone()
    w[0, 30, 1, 3] = bad
    o2, lse2 = flash_fwd(q, k, w, causal, scale)
    assert torch.equal(lse, lse2) and not torch.isfinite(o2[0, 30:, 1, 3]).any()
    assert torch.equal(flash_bwd(q, k, w, o2, do, lse2, causal, scale)[2], dv)
