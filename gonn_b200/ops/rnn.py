"""Fused gate arithmetic of the LSTM / GRU cells (kernels in ``csrc/rnn.cu``).

``lstm_gates(gates, c) -> (h', c')`` with gate order i, f, g, o and
``gru_gates(xg, hg, h) -> h'`` with gates r, z, n (nn/rnn.go:159-286 of the reference).
CUDA tensors of fp32 / fp16 / bf16 run one kernel per direction; other tensors take the
torch expression with the same formulas (the oracle of the tests).

``lstm_sequence`` runs a whole fp32 LSTM layer: the input projections of all steps as one GEMM, the
recurrence as one persistent kernel per direction (``csrc/lstm_seq.cu``), and the weight and input
gradients as one GEMM each over all steps.  Measured forward + backward at B = 32, T = 64,
I = H = 512: 0.96 ms, 22.6 ms step by step.  The products of all steps are large enough for the bf16 planes (``ops/gemm.py``),
where those of one step were FMA sums; the layer's error against 64 bits, which the fast-math gates set, is the same
within 2 % up to 64 x 64 steps (output 5.5e-6, dx 3.9e-6 against 4.0e-6, dW_ih 3.9e-6, dW_hh 6.2e-6) and
up to 6 % larger where a gradient sums 8192 rows (32 x 256 steps: dx 4.2e-6 against 4.0e-6).
"""
from __future__ import annotations

import torch

from .. import lib as _l

_KERNEL_DTYPES = (torch.float32, torch.float16, torch.bfloat16)


def _on_kernels(t: torch.Tensor) -> bool:
    return t.is_cuda and t.dtype in _KERNEL_DTYPES


def lstm_gates_ref(gates, c):
    H = c.shape[-1]
    i, f = torch.sigmoid(gates[:, :H]), torch.sigmoid(gates[:, H:2 * H])
    g, o = torch.tanh(gates[:, 2 * H:3 * H]), torch.sigmoid(gates[:, 3 * H:])
    c_new = f * c + i * g
    return o * torch.tanh(c_new), c_new


def gru_gates_ref(xg, hg, h):
    H = h.shape[-1]
    r = torch.sigmoid(xg[:, :H] + hg[:, :H])
    z = torch.sigmoid(xg[:, H:2 * H] + hg[:, H:2 * H])
    n = torch.tanh(xg[:, 2 * H:] + r * hg[:, 2 * H:])
    return (1 - z) * n + z * h


class _LSTMGates(torch.autograd.Function):
    @staticmethod
    def forward(ctx, gates, c):
        B, H = c.shape
        gates, c = gates.contiguous(), c.contiguous()
        h_new, c_new = torch.empty_like(c), torch.empty_like(c)
        act = torch.empty_like(gates)
        _l.call("gb_lstm_gates_fwd", _l.I(_l.dtype_code(c.dtype)), _l.ptr(gates), _l.ptr(c), _l.ptr(h_new),
                _l.ptr(c_new), _l.ptr(act), _l.L(B), _l.I(H), _l.stream_ptr())
        ctx.save_for_backward(act, c, c_new)
        return h_new, c_new

    @staticmethod
    def backward(ctx, dh, dc):
        act, c, c_new = ctx.saved_tensors
        B, H = c.shape
        dh = dh.contiguous() if dh is not None else None
        dc = dc.contiguous() if dc is not None else None
        dgates, dc_prev = torch.empty_like(act), torch.empty_like(c)
        _l.call("gb_lstm_gates_bwd", _l.I(_l.dtype_code(c.dtype)), _l.ptr(act), _l.ptr(c), _l.ptr(c_new),
                _l.ptr(dh), _l.ptr(dc), _l.ptr(dgates), _l.ptr(dc_prev), _l.L(B), _l.I(H), _l.stream_ptr())
        return dgates, dc_prev


class _GRUGates(torch.autograd.Function):
    @staticmethod
    def forward(ctx, xg, hg, h):
        B, H = h.shape
        xg, hg, h = xg.contiguous(), hg.contiguous(), h.contiguous()
        h_new = torch.empty_like(h)
        act = torch.empty((B, 4 * H), dtype=h.dtype, device=h.device)
        _l.call("gb_gru_gates_fwd", _l.I(_l.dtype_code(h.dtype)), _l.ptr(xg), _l.ptr(hg), _l.ptr(h),
                _l.ptr(h_new), _l.ptr(act), _l.L(B), _l.I(H), _l.stream_ptr())
        ctx.save_for_backward(act, h)
        return h_new

    @staticmethod
    def backward(ctx, dh):
        act, h = ctx.saved_tensors
        B, H = h.shape
        dh = dh.contiguous()
        dxg = torch.empty((B, 3 * H), dtype=h.dtype, device=h.device)
        dhg = torch.empty_like(dxg)
        dh_prev = torch.empty_like(h)
        _l.call("gb_gru_gates_bwd", _l.I(_l.dtype_code(h.dtype)), _l.ptr(act), _l.ptr(h), _l.ptr(dh),
                _l.ptr(dxg), _l.ptr(dhg), _l.ptr(dh_prev), _l.L(B), _l.I(H), _l.stream_ptr())
        return dxg, dhg, dh_prev


def _aligned(t):
    """Contiguous and 16-byte aligned (the persistent kernels read rows in 16-byte pieces)."""
    if t is None:
        return None
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


# Without a tape the projections of the whole input (four times the output) live for a moment only: longer sequences go in
# pieces of at most this many bytes, each from the state that the one before it left.
PROJECTION_BYTES = 256 << 20
LEAST_WORDS = 74       # 64-bit words: a flag per CTA of the backward that gathers (the one that scatters takes up to 128 MiB)


def _lstm_forward(x, w_ih, b_ih, w_hh, h0, c0, tape: bool):
    """(out (B, T, H), c, hprev, gates, x2): with ``tape`` c and hprev are (B, T, H), gates (B * T, 4H) and x2 the input's rows, what the
    backward reads; without it c is the last cell state (B, H) and nothing else is kept."""
    from .gemm import gemm
    B, T, I = x.shape
    H = w_hh.shape[1]
    steps = T if tape or 16 * B * T * H <= PROJECTION_BYTES else max(1, PROJECTION_BYTES // (16 * B * H))
    # the product first: the rest of the host's work hides behind it
    x2 = (x if steps == T else x[:, :steps]).reshape(B * steps, I)
    xg = gemm(x2, w_ih, trans_b=True)
    dev, s = x.device, _l.stream_ptr()
    whh, h0, c0 = _aligned(w_hh.detach()), _aligned(h0), _aligned(c0)
    bias = b_ih.detach().contiguous() if b_ih is not None else None
    out = torch.empty((B, T, H), dtype=x.dtype, device=dev)
    xch = torch.empty(2 * B * H, dtype=torch.int64, device=dev)
    hprev = torch.empty((B, T, H), dtype=x.dtype, device=dev) if tape else None
    c = torch.empty((B, T, H) if tape else (B, H), dtype=x.dtype, device=dev)
    for t in range(0, T, steps):
        n = min(steps, T - t)
        if t > 0:
            xg = gemm(x[:, t:t + n].reshape(B * n, I), w_ih, trans_b=True, out=xg if n == steps else None)
        _l.call("gb_lstm_seq_fwd", _l.ptr(xg), _l.ptr(bias), _l.ptr(whh), _l.ptr(h0), _l.ptr(c0), _l.P(out.data_ptr() + 4 * t * H),
                _l.L(T * H), _l.ptr(hprev), _l.ptr(c), _l.ptr(xch), _l.I(B), _l.I(n), _l.I(H), s)
        if t + n < T:
            h0, c0 = _aligned(out[:, t + n - 1]), c
    return out, c, hprev, xg, x2


class _LSTMSequence(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w_ih, b_ih, w_hh, h0, c0):
        # the backward reads h_{t-1} from a buffer of its own: the output belongs to the caller, who may change it in place
        c0 = _aligned(c0)
        out, cseq, hprev, act, x2 = _lstm_forward(x, w_ih, b_ih, w_hh, h0, c0, True)
        ctx.save_for_backward(x2, w_ih, w_hh, c0, hprev, cseq, act)
        ctx.b_ih, ctx.xshape = b_ih, x.shape
        ctx.set_materialize_grads(False)
        return out, cseq[:, -1].clone()

    @staticmethod
    def backward(ctx, dout, dcn):
        from .gemm import gemm
        from .linear import emit_vector_grad, emit_weight_grad
        x2, w_ih, w_hh, c0, hprev, cseq, act = ctx.saved_tensors
        B, T, H = cseq.shape
        dev = cseq.device
        dout = dout.contiguous() if dout is not None else None
        dcn = dcn.contiguous() if dcn is not None else None
        whh = _aligned(w_hh.detach())
        dgates = torch.empty_like(act)                     # (B * T, 4H)
        dc0 = torch.empty((B, H), dtype=cseq.dtype, device=dev) if ctx.needs_input_grad[5] else None
        # (sequences of up to two steps gather: one step of B = H = 512 takes 160 us with the words allocated and cleared, 131 without)
        words = _l.lib().gb_lstm_seq_bwd_words(_l.I(B), _l.I(H)) if T > 2 else LEAST_WORDS
        try:
            scratch = torch.empty(words, dtype=torch.int64, device=dev)
        except torch.OutOfMemoryError:
            words = LEAST_WORDS
            scratch = torch.empty(words, dtype=torch.int64, device=dev)
        _l.call("gb_lstm_seq_bwd", _l.ptr(whh), _l.ptr(c0), _l.ptr(cseq), _l.ptr(act), _l.ptr(dout), _l.ptr(dcn),
                _l.ptr(dgates), _l.ptr(dc0), _l.ptr(scratch), _l.L(words), _l.I(B), _l.I(T), _l.I(H), _l.stream_ptr())
        dx = dwih = db = dwhh = dh0 = None
        # every read of a weight comes before its gradient is declared ready (ops/linear.py)
        if ctx.needs_input_grad[0]:
            dx = gemm(dgates, w_ih).view(ctx.xshape)
        if ctx.needs_input_grad[4]:
            dh0 = gemm(dgates.view(B, T, 4 * H)[:, 0], w_hh)
        if ctx.needs_input_grad[1]:
            dwih = emit_weight_grad(w_ih, dgates, x2, True, False)
        if ctx.b_ih is not None and ctx.needs_input_grad[2]:
            db = emit_vector_grad(ctx.b_ih, dgates)
        if ctx.needs_input_grad[3]:
            dwhh = emit_weight_grad(w_hh, dgates, hprev.view(B * T, H), True, False)
        return dx, dwih, db, dwhh, dh0, dc0


def lstm_sequence_fits(B: int, H: int) -> bool:
    """Whether a layer of ``H`` units over ``B`` sequences fits the persistent kernels."""
    return bool(_l.lib().gb_lstm_seq_fits(_l.I(B), _l.I(H)))


def _transformed() -> bool:
    """Forward-mode tangents, a function transform, tracing or compilation: these must see the autograd function."""
    return bool(torch.autograd.forward_ad._current_level >= 0 or torch._C._functorch.peek_interpreter_stack() is not None
                or torch.jit.is_tracing() or torch.compiler.is_compiling())


def lstm_sequence(x, w_ih, b_ih, w_hh, h0=None, c0=None):
    """(h_1 .. h_T (B, T, H), c_T (B, H)) of an fp32 LSTM layer over (B, T, I) on CUDA."""
    if (torch.is_grad_enabled() and (x.requires_grad or w_ih.requires_grad or w_hh.requires_grad
                                     or any(t is not None and t.requires_grad for t in (b_ih, h0, c0)))
            or _transformed()):
        return _LSTMSequence.apply(x, w_ih, b_ih, w_hh, h0, c0)
    return _lstm_forward(x, w_ih, b_ih, w_hh, h0, c0, False)[:2]


def lstm_gates(gates: torch.Tensor, c: torch.Tensor):
    """(h', c') from the (B, 4H) gate pre-activations and the cell state."""
    if _on_kernels(c) and gates.dtype == c.dtype:
        return _LSTMGates.apply(gates, c)
    return lstm_gates_ref(gates, c)


def gru_gates(xg: torch.Tensor, hg: torch.Tensor, h: torch.Tensor):
    """h' from the (B, 3H) input / hidden pre-activations and the previous state."""
    if _on_kernels(h) and xg.dtype == h.dtype and hg.dtype == h.dtype:
        return _GRUGates.apply(xg, hg, h)
    return gru_gates_ref(xg, hg, h)
