"""The channels-last and the short-contraction convolution kernels (csrc/conv_cl.cu, csrc/conv.cu) against float64."""
import pytest
import torch

from gonn_b200 import lib as L, nn

pytestmark = pytest.mark.gpu

# (images, C_in, C_out, (H, W), kernel, stride, padding, dilation): channel counts around the 8-wide pieces, the
# 64-wide k-blocks and the 128-wide tiles, k-blocks that span taps, ragged positions, one position
CL = [(3, 64, 128, (15, 15), 3, 1, 0, 1), (2, 8, 16, (9, 7), 3, 1, 1, 1), (5, 24, 136, (11, 6), 3, 2, 1, 1),
      (2, 72, 40, (8, 8), 2, 1, 0, 2), (1, 128, 64, (5, 5), 5, 1, 2, 1), (7, 16, 8, (1, 1), 1, 1, 0, 1), (4, 200, 264, (6, 7), 1, 1, 0, 1)]
# C * T <= 32: plane sizes that are multiples of 8, 4, 2 and odd (width of the runs), channel counts off 16
SMALL = [(3, 3, 64, (32, 32), 3, 1, 0, 1), (2, 3, 32, (10, 10), 3, 1, 1, 1), (5, 1, 128, (9, 10), 5, 1, 2, 1),
         (3, 2, 20, (7, 7), 3, 2, 1, 1), (40, 3, 64, (3, 3), 3, 1, 0, 1), (2, 4, 32, (9, 5), 2, 1, 0, 1), (2, 32, 64, (5, 7), 1, 1, 0, 1)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("case", CL + SMALL)
def test_forward_and_gradients(case, dtype):
    N, Ci, Co, hw, k, s, p, d = case
    torch.manual_seed(Ci * 31 + Co)
    net = nn.Conv2d(Ci, Co, k, s, p, d, dtype=dtype, device="cuda")
    x = torch.randn(N, Ci, *hw, device="cuda").to(dtype).requires_grad_()
    y = net(x)
    dy = torch.randn_like(y)
    y.backward(dy)
    L.assert_status_ok()
    xr, wr, br = (t.detach().double().cpu().requires_grad_() for t in (x, net.weight, net.bias))
    want = torch.nn.functional.conv2d(xr, wr, br, s, p, d)
    want.backward(dy.double().cpu())
    # products of 16-bit values are exact in fp32; what remains is the rounding of the result (half a unit of
    # 2^-8 or 2^-11) and fp32 sums, far below it
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for n, a, b in (("y", y, want), ("dx", x.grad, xr.grad), ("dw", net.weight.grad, wr.grad), ("db", net.bias.grad, br.grad)):
        err = float((a.detach().double().cpu() - b.detach()).norm() / b.detach().norm())
        assert err < tol, f"{n}: {err:.3g}"


def test_padding_and_tiles_ignore_non_finite_neighbours():
    """Rows past the channel count or the positions never reach a result: an infinity in one image stays there."""
    net = nn.Conv2d(16, 24, 3, 1, 1, dtype=torch.bfloat16, device="cuda")
    x = torch.randn(3, 16, 6, 6, device="cuda").bfloat16()
    x[1, 0, 0, 0] = float("inf")
    y = net(x)
    assert y[0].isfinite().all() and y[2].isfinite().all() and not y[1, :, :2, :2].isfinite().all()
    assert y[1, :, 2:, 2:].isfinite().all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("Co", [32, 64, 128, 372])
@pytest.mark.parametrize("case", ["conv1d_32", "conv2d_4x8"])
def test_windows_of_32_taps(dtype, Co, case):
    """One input channel and 32 taps: the longest windows of the short-contraction kernels (49 KB of shared memory)."""
    torch.manual_seed(Co)
    kw = dict(dtype=dtype, device="cuda")
    net = nn.Conv1d(1, Co, 32, **kw) if case == "conv1d_32" else nn.Conv2d(1, Co, (4, 8), **kw)
    x = torch.randn(*((3, 1, 75) if case == "conv1d_32" else (3, 1, 9, 13)), device="cuda").to(dtype).requires_grad_()
    y = net(x)
    dy = torch.randn_like(y)
    y.backward(dy)
    L.assert_status_ok()
    xr, wr, br = (t.detach().double().cpu().requires_grad_() for t in (x, net.weight, net.bias))
    conv = torch.nn.functional.conv1d if case == "conv1d_32" else torch.nn.functional.conv2d
    want = conv(xr, wr.view(Co, *((1, 32) if case == "conv1d_32" else (1, 4, 8))), br)
    want.backward(dy.double().cpu())
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11      # one rounding of exact products' fp32 sums
    for n, a, b in (("y", y, want), ("dx", x.grad, xr.grad), ("dw", net.weight.grad, wr.grad), ("db", net.bias.grad, br.grad)):
        err = float((a.detach().double().cpu() - b.detach()).norm() / b.detach().norm())
        assert err < tol, f"{n}: {err:.3g}"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_without_memory_for_the_channels_last_copies(monkeypatch, dtype):
    """The kernels that need no scratch take a convolution for which it cannot be had."""
    from gonn_b200.nn import conv
    net = nn.Conv2d(24, 40, 3, 1, 1, dtype=dtype, device="cuda")
    x = torch.randn(5, 24, 11, 9, device="cuda").to(dtype).requires_grad_()
    y = net(x)
    dy = torch.randn_like(y)
    want = [y] + list(torch.autograd.grad(y, [x, *net.parameters()], dy))
    seen = []
    L.set_call_hook(lambda name, fn, args: (seen.append(name), fn(*args))[1])
    monkeypatch.setattr(conv, "_scratch", lambda *a: None)
    try:
        y = net(x)
        got = [y] + list(torch.autograd.grad(y, [x, *net.parameters()], dy))
    finally:
        L.set_call_hook(None)
    L.assert_status_ok()
    assert "gb_conv_igemm" in seen and not any(n.startswith("gb_conv_cl") for n in seen)
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11      # one rounding of the result on either side
    for a, b in zip(got, want):
        a, b = a.detach().double(), b.detach().double()
        assert float((a - b).norm() / b.norm()) < 2 * tol


def test_scratch_is_none_when_memory_runs_out(monkeypatch):
    from gonn_b200.nn import conv

    def no_room(*a, **kw):
        raise torch.OutOfMemoryError("no room")

    assert conv._scratch(8, torch.bfloat16, "cuda").numel() == 8
    monkeypatch.setattr(torch, "empty", no_room)
    assert conv._scratch(8, torch.bfloat16, "cuda") is None
