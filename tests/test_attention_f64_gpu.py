"""The fp64 tensor-core attention kernels (csrc/attn_f64.cu) against the materialised oracle in float64."""
import pytest
import torch

from gonn_b200 import lib as L
from gonn_b200.ops import attention as A

pytestmark = pytest.mark.gpu

# row blocks of 16 / 32 / 64, tiles of 16 / 32, head sizes around 8 / 16 / 32 / 64 columns (odd ones take
# the 8-byte copies), unequal lengths
SHAPES = [(1, 1, 1, 1, 1), (2, 3, 17, 17, 16), (1, 2, 65, 33, 24), (2, 2, 64, 130, 40), (1, 3, 100, 100, 7), (1, 2, 129, 129, 64),
          (2, 1, 31, 15, 33)]


@pytest.fixture(params=[0, 1, 2, 4])
def split(request):
    L.call("gb_attn_f64_tune", L.I(request.param))
    yield request.param
    L.call("gb_attn_f64_tune", L.I(0))


@pytest.fixture(params=[True, False])
def spill(request, monkeypatch):
    """dQ from the dS that the dK / dV kernel left in memory, or recomputed."""
    monkeypatch.setattr(A, "DS_MIN_SCORES", 0 if request.param else 1 << 62)
    return request.param


def _check(B, H, Tq, Tk, D, causal, masks, p_drop, strided=False):
    torch.manual_seed(Tq * 7 + Tk * 3 + D)
    mk = lambda n: torch.randn(B, n, H, D, dtype=torch.float64)
    q, k, v, dy = mk(Tq), mk(Tk), mk(Tk), mk(Tq)
    mask = kpm = None
    if masks:
        mask = torch.randn(Tq, Tk).masked_fill(torch.rand(Tq, Tk) < 0.2, float("-inf"))
        mask[:, 0] = 0.5                                        # no row without a finite score, causal ones neither
        kpm = torch.rand(B, Tk) < 0.2
    scale = 0.37
    qc, kc, vc = (t.cuda().requires_grad_() for t in (q, k, v))
    if strided:                                                 # (B, H, S, D) storage with a padded row: odd strides
        qc, kc, vc = (torch.cat([t.detach().permute(0, 2, 1, 3)] * 2, -1).cuda()[..., 1:D + 1].permute(0, 2, 1, 3)
                      for t in (q, k, v))
        q, k, v = (t.detach().cpu() for t in (qc, kc, vc))
        qc, kc, vc = (t.requires_grad_() for t in (qc, kc, vc))
    out = A.general_attention(qc, kc, vc, causal, scale, None if mask is None else mask.cuda(),
                              None if kpm is None else kpm.cuda(), p_drop, seed=1234)
    out.backward(dy.cuda())
    L.assert_status_ok()
    keep = None
    if p_drop:
        keep = torch.empty(B, H, Tq, Tk, dtype=torch.uint8, device="cuda")
        L.call("gb_attn_keep_mask", L.ptr(keep), L.I(B), L.I(H), L.I(Tq), L.I(Tk), L.D(p_drop), L.L(1234), L.stream_ptr())
        keep = keep.cpu().bool()
    qr, kr, vr = (t.clone().requires_grad_() for t in (q, k, v))
    want = A.masked_attention_ref(qr, kr, vr, causal, scale, mask, kpm, keep, p_drop)
    want.backward(dy)
    for n, a, b in (("out", out, want), ("dq", qc.grad, qr.grad), ("dk", kc.grad, kr.grad), ("dv", vc.grad, vr.grad)):
        # sums of at most 130 products and exponentials of arguments below 64: a few hundred units of 2^-53
        err = float((a.detach().cpu() - b.detach()).norm() / b.detach().norm().clamp_min(1e-300))
        assert err < 5e-14 or float(b.detach().norm()) < 1e-12 and float(a.detach().norm()) < 1e-12, f"{n}: {err:.3g}"


@pytest.mark.parametrize("B,H,Tq,Tk,D", SHAPES)
@pytest.mark.parametrize("causal", [False, True])
def test_plain(split, spill, B, H, Tq, Tk, D, causal):
    _check(B, H, Tq, Tk, D, causal, False, 0.0)


@pytest.mark.parametrize("p_drop", [0.0, 0.3])
@pytest.mark.parametrize("causal", [False, True])
def test_masks_and_dropout(split, spill, causal, p_drop):
    # (a mask beside the causal flag: no tile is skipped, and dS above the diagonal counts)
    _check(2, 2, 70, 50, 24, causal, True, p_drop)
    _check(1, 2, 130, 130, 40, causal, True, p_drop)
    _check(2, 2, 45, 45, 64, causal, False, p_drop)


def test_unaligned_strides(split, spill):
    _check(1, 2, 40, 40, 15, True, False, 0.0, strided=True)


def test_rows_without_finite_scores_and_nan():
    q, k, v = (torch.randn(1, 40, 1, 16, dtype=torch.float64, device="cuda") for _ in range(3))
    mask = torch.zeros(40, 40)
    mask[3] = float("-inf")
    out = A.general_attention(q, k, v, False, 1.0, mask.cuda())
    assert out[:, 3].isnan().all() and out[:, :3].isfinite().all() and out[:, 4:].isfinite().all()
    q2 = q.clone()
    q2[0, 5, 0, 0] = float("nan")
    out = A.general_attention(q2, k, v, False, 1.0)
    assert out[:, 5].isnan().all() and out[:, :5].isfinite().all() and out[:, 6:].isfinite().all()


def test_the_handed_over_ds_lives_for_one_call(monkeypatch):
    """The fp64 backward leaves no workspace behind, and without memory for it gives the same gradients."""
    monkeypatch.setattr(A, "DS_MIN_SCORES", 0)
    q, k, v = (torch.randn(2, 300, 2, 32, dtype=torch.float64, device="cuda", requires_grad=True) for _ in range(3))
    dy = torch.randn(2, 300, 2, 32, dtype=torch.float64, device="cuda")
    need = 8 * 4 * 320 * 320
    out = A.flash_attention(q, k, v, causal=True)

    def gradients():
        return torch.autograd.grad(out, (q, k, v), dy, retain_graph=True)

    del_me = gradients()
    del del_me
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    with_ds = gradients()
    assert torch.cuda.max_memory_allocated() - before >= need                     # it was used
    kept = sum(g.numel() * 8 for g in with_ds)
    assert torch.cuda.memory_allocated() - before <= kept + 4096                  # and given back
    empty = torch.empty

    def no_room(*size, **kw):
        if kw.get("dtype") is torch.uint8:
            raise torch.OutOfMemoryError("no room")
        return empty(*size, **kw)

    monkeypatch.setattr(torch, "empty", no_room)
    without = gradients()
    monkeypatch.setattr(torch, "empty", empty)
    L.assert_status_ok()
    for a, b in zip(with_ds, without):
        assert float((a - b).norm() / b.norm()) < 5e-14                           # (as in _check)
