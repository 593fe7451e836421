"""The persistent LSTM kernels (csrc/lstm_seq.cu) against the step-by-step oracle in float64."""
import copy

import pytest
import torch

from gonn_b200 import lib as L, nn
from gonn_b200.nn import rnn as R

pytestmark = pytest.mark.gpu

# hidden sizes around the slices of 4 / 8 / 16 units and the exchange tile of 8 sequences, batches
# that leave a sub-tile ragged or need several per CTA, the widest layer that fits
SIZES = [(1, 1, 8, 4), (3, 5, 7, 20), (8, 3, 16, 64), (9, 4, 12, 68), (17, 7, 40, 132), (32, 5, 64, 512),
         (70, 3, 24, 512), (5, 2, 16, 880)]


def _close(a, b, tol, what):
    a, b = a.detach().double().cpu(), b.detach()
    err = float((a - b).norm() / b.norm().clamp_min(1e-30))
    assert err < tol, f"{what}: relative error {err:.3g}"


@pytest.mark.parametrize("B,T,I,H", SIZES)
@pytest.mark.parametrize("state", [False, True])
def test_lstm_sequence_matches_float64(B, T, I, H, state):
    torch.manual_seed(B * 1000 + H)
    ref = nn.LSTM(I, H, bidirectional=state, dtype=torch.float64)
    net = copy.deepcopy(ref).float().cuda()
    x = torch.randn(B, T, I, dtype=torch.float64)
    D = 2 if state else 1
    st = tuple(torch.randn(D, B, H, dtype=torch.float64) for _ in range(2)) if state else None
    dy = torch.randn(B, T, D * H, dtype=torch.float64)
    dh, dc = torch.randn(D, B, H, dtype=torch.float64), torch.randn(D, B, H, dtype=torch.float64)
    xg = x.float().cuda().requires_grad_()
    assert R._sequence_kernel_takes(net.cells[0], xg, None)
    got, want = [], []
    for net_, x_, conv, acc in ((net, xg, lambda t: t.float().cuda(), got),
                                (ref, x.clone().requires_grad_(), lambda t: t, want)):
        s_ = tuple(conv(t).requires_grad_() for t in st) if state else None
        y, (h, c) = net_.ForwardWithState(x_, s_)
        ((y * conv(dy)).sum() + (h * conv(dh)).sum() + (c * conv(dc)).sum()).backward()
        acc += [("y", y), ("h", h), ("c", c), ("dx", x_.grad)] + [(n, p.grad) for n, p in net_.named_parameters()]
        if state:
            acc += [("dh0", s_[0].grad), ("dc0", s_[1].grad)]
    L.assert_status_ok()
    for (n, a), (_, b) in zip(got, want):
        # fp32 sums of up to 4H terms and the fast-math exponential / tanh of the gate arithmetic
        # (a few 1e-6 per step), carried through T steps
        _close(a, b, 3e-5, n)


@pytest.mark.parametrize("B,T,H,scattered", [(8, 9, 132, True), (300, 3, 256, True), (512, 2, 512, True), (513, 3, 512, False), (9, 5, 876, True)])
def test_backward_either_way_round_matches_float64(B, T, H, scattered):
    """The scattered exchange with several sub-tiles and slices that the units do not fill, up to the most words it takes, and the
    gathered one behind that."""
    words = L.lib().gb_lstm_seq_bwd_words(L.I(B), L.I(H))
    assert (words > 74) == scattered and 8 * words <= 128 << 20
    torch.manual_seed(H)
    net = nn.LSTM(8, H, device="cuda")
    x = torch.randn(B, T, 8, device="cuda", requires_grad=True)
    dy = torch.randn(B, T, H, device="cuda")
    y, (_, c) = net.ForwardWithState(x)
    ((y * dy).sum() + c.sum()).backward()
    L.assert_status_ok()
    ref = copy.deepcopy(net).double().cpu()
    ref.zero_grad()
    xr = x.detach().double().cpu().requires_grad_()
    yr, (_, cr) = ref.ForwardWithState(xr)
    ((yr * dy.double().cpu()).sum() + cr.sum()).backward()
    for n, a, b in [("y", y, yr), ("dx", x.grad, xr.grad)] + [(n, p.grad, q.grad) for (n, p), q in zip(net.named_parameters(), ref.parameters())]:
        _close(a, b, 3e-5, n)          # as in test_lstm_sequence_matches_float64


def test_step_path_where_the_kernel_does_not_apply():
    net = nn.LSTM(8, 16, device="cuda")
    x = torch.randn(2, 3, 8, device="cuda")
    y = net(x)
    seen = []
    handle = net.cells[0].register_forward_hook(lambda m, a, o: seen.append(1))
    y2 = net(x)
    handle.remove()
    assert len(seen) == 3                                     # every step is observed
    assert (y - y2).abs().max() < 1e-5
    assert not R._sequence_kernel_takes(nn.LSTM(8, 6, device="cuda").cells[0], x, None)      # 6 % 4 != 0
    assert not R._sequence_kernel_takes(net.cells[0].to(torch.bfloat16), x.bfloat16(), None)


@pytest.mark.parametrize("B,H", [(20, 896), (150, 880)])
def test_layers_at_the_limit_of_shared_memory_train(B, H):
    """Layers whose backward would need a whole block's shared memory beside its static flag take the steps."""
    torch.manual_seed(H)
    net = nn.LSTM(16, H, device="cuda")
    x = torch.randn(B, 2, 16, device="cuda", requires_grad=True)
    y = net(x)
    y.sum().backward()
    ref = copy.deepcopy(net).double().cpu()
    xr = x.detach().double().cpu().requires_grad_()
    yr = ref(xr)
    yr.sum().backward()
    L.assert_status_ok()
    _close(y, yr, 3e-5, "y")
    _close(x.grad, xr.grad, 3e-5, "dx")


@pytest.mark.parametrize("edit", [lambda t: t.relu_(), lambda t: t.mul_(2.0), lambda t: t[:, 0].zero_()])
@pytest.mark.parametrize("layers,bidirectional,state", [(1, False, False), (1, False, True), (2, True, False)])
def test_the_output_may_be_changed_in_place(edit, layers, bidirectional, state):
    """The backward keeps nothing that the caller of a layer gets: in-place work on the output differentiates."""
    torch.manual_seed(5)
    ref = nn.LSTM(12, 20, layers, bidirectional=bidirectional, dtype=torch.float64)
    net = copy.deepcopy(ref).float().cuda()
    x = torch.randn(3, 5, 12, dtype=torch.float64)
    D = (2 if bidirectional else 1) * layers
    st = tuple(torch.randn(D, 3, 20, dtype=torch.float64) for _ in range(2)) if state else None
    grads = []
    for m, conv in ((net, lambda t: t.float().cuda()), (ref, lambda t: t.clone())):
        xi = conv(x).requires_grad_()
        y, (h, c) = m.ForwardWithState(xi, None if st is None else tuple(conv(t) for t in st))
        edit(y)
        edit(h)
        edit(c)
        (y.sum() + (h * h).sum() + c.sum()).backward()
        grads.append([y, h, c, xi.grad] + [p.grad for p in m.parameters()])
    L.assert_status_ok()
    for a, b in zip(*grads):
        _close(a, b, 3e-5, "in-place")


@pytest.mark.parametrize("state", [False, True])
@pytest.mark.parametrize("T", [1, 6, 7, 8, 50])
def test_evaluation_in_pieces(monkeypatch, T, state):
    """Without a tape a sequence may run in pieces (here of 7 steps): the outputs and the last states of a whole one."""
    B, I, H = 5, 24, 64
    net = nn.LSTM(I, H, 2, bidirectional=True, device="cuda")
    x = torch.randn(B, T, I, device="cuda")
    st = tuple(torch.randn(4, B, H, device="cuda") for _ in range(2)) if state else None
    want, (h, c) = net.ForwardWithState(x, st)                       # with a tape
    monkeypatch.setattr(R._rnn_ops, "PROJECTION_BYTES", 7 * 16 * B * H + 1)
    with torch.no_grad():
        got, (h2, c2) = net.ForwardWithState(x, st)
    L.assert_status_ok()
    for n, a, b in (("y", got, want), ("h", h2, h), ("c", c2, c)):
        # the same kernel; the projections of fewer rows may be summed in another order
        assert a.shape == b.shape and not a.requires_grad
        _close(a, b.double().cpu(), 2e-6, n)


def test_evaluation_keeps_neither_gates_nor_cell_states(monkeypatch):
    B, T, I, H = 64, 512, 16, 128
    net = nn.LSTM(I, H, device="cuda")
    x = torch.randn(B, T, I, device="cuda")
    piece = 8 << 20
    monkeypatch.setattr(R._rnn_ops, "PROJECTION_BYTES", piece)
    with torch.no_grad():
        net(x)
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        y = net(x)
    # the output and two pieces of the projections (one of them the ragged last); the states are small
    assert torch.cuda.max_memory_allocated() - before < y.numel() * 4 + 2 * piece + (4 << 20)


@pytest.mark.parametrize("value", [float("inf"), -float("inf"), 3.4e38, -3.4e38])
def test_an_infinite_input_saturates_the_gates(value):
    """The projections of the whole input are large enough for the plane products: an infinity must arrive as one."""
    net = nn.LSTM(512, 512, device="cuda")
    x = torch.randn(32, 64, 512, device="cuda")
    x[3, 2, 5] = value
    with torch.no_grad():
        y = net(x)
    assert y.isfinite().all()


def test_tangents_and_transforms_are_not_dropped_without_a_tape():
    """Forward-mode tangents and vmap reach the autograd function, which refuses them, also where no gradient is recorded."""
    net = nn.LSTM(12, 20, device="cuda")
    x = torch.randn(3, 5, 12, device="cuda")
    fw = torch.autograd.forward_ad
    with torch.no_grad(), fw.dual_level():
        with pytest.raises(Exception):
            net(fw.make_dual(x, torch.ones_like(x)))
    with torch.no_grad(), pytest.raises(Exception):
        torch.func.vmap(net)(torch.randn(2, 3, 5, 12, device="cuda"))
    with torch.no_grad():
        assert net(x).isfinite().all()


@pytest.mark.parametrize("B,T,H", [(9, 5, 692), (70, 4, 720), (200, 3, 744)])
def test_forward_with_one_buffer_of_partial_sums(B, T, H):
    """Widths at which 16 units leave room for one: alone, several sub-tiles to a group, the widest."""
    test_lstm_sequence_matches_float64(B, T, 8, H, True)


def _no_words(monkeypatch, asked):
    """Memory for the words of the scattered exchange (more than any other whole-number buffer here) is short."""
    real = torch.empty

    def empty(*size, **kw):
        if kw.get("dtype") is torch.int64 and size[0] > 1 << 16:
            asked.append(size[0])
            raise torch.OutOfMemoryError("short")
        return real(*size, **kw)
    monkeypatch.setattr(torch, "empty", empty)


@pytest.mark.parametrize("B,H", [(16, 256), (200, 132)])
def test_backward_where_memory_for_the_exchange_is_short(monkeypatch, B, H):
    assert L.lib().gb_lstm_seq_bwd_words(L.I(B), L.I(H)) > 1 << 16 > 2 * B * H
    asked = []
    _no_words(monkeypatch, asked)
    test_lstm_sequence_matches_float64(B, 5, 8, H, True)
    assert asked


def test_one_step_takes_no_words(monkeypatch):
    asked = []
    _no_words(monkeypatch, asked)
    test_lstm_sequence_matches_float64(70, 1, 8, 256, True)
    assert not asked


@pytest.mark.parametrize("B,H", [(70, 256), (9, 132)])
def test_two_steps_take_no_words(monkeypatch, B, H):
    asked = []
    real = torch.empty

    def empty(*size, **kw):
        if kw.get("dtype") is torch.int64 and size[0] > max(2 * B * H, 74):      # (the forward's words are 2 B H)
            asked.append(size[0])
        return real(*size, **kw)
    monkeypatch.setattr(torch, "empty", empty)
    test_lstm_sequence_matches_float64(B, 2, 8, H, True)
    assert not asked
    test_lstm_sequence_matches_float64(B, 3, 8, H, True)
    assert asked


def test_backward_with_the_most_words_it_takes():
    test_backward_either_way_round_matches_float64(512, 3, 512, True)
