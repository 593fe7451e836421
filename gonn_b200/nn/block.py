"""Transformer blocks without a tape in one native call (``csrc/block.cu``).

``evaluate`` serves ``TransformerEncoderLayer.forward`` and ``GPTBlock.forward`` under ``torch.no_grad``, ``evaluate_stack`` the
models that chain them: the same kernels in the same order as the operators, launched from one call.  They return None, and the
caller runs block by block or operator by operator, whenever something could observe or change a single block or operator: hooks, a
subclass or a replaced forward, a parametrization, an active tracer, forward-mode tangents, a transform, tracing or
compilation, or a type, layout or size outside the fused path of the operators.  At one prompt of 77
tokens through the 12-layer 768-wide model, host time: 3.5 ms operator by operator, 0.75 ms block by block, 0.55 ms in one call.
"""
from __future__ import annotations

import ctypes
import math

import torch

from .. import lib as _l
from .activation import Activation
from .attention import MultiHeadAttention
from .linear import Linear
from .module import ModuleList
from .norm import LayerNorm, RMSNorm

_ACT = {"relu": 1, "gelu": 2, "geluexact": 3}
_DTYPES = {torch.bfloat16: 0, torch.float16: 1}
_fwd_ad = torch.autograd.forward_ad
_tm = torch.nn.modules.module
_ABSENT = object()
_WORDS = 26                 # argument words of a block
_GROUP = 4                  # blocks that a native call asks for at most at a time
_More = ctypes.CFUNCTYPE(None)


def plain(m, cls) -> bool:
    """``m`` is exactly a ``cls`` whose call is its class's forward: no hook, no replaced forward."""
    if type(m) is not cls:
        return False
    d = m.__dict__
    return not (d["_forward_hooks"] or d["_forward_pre_hooks"] or d["_backward_hooks"] or d["_backward_pre_hooks"]
                or "forward" in d)


def _observed() -> bool:
    return bool(_l._call_hook is not None or _tm._global_forward_hooks or _tm._global_forward_pre_hooks
                or _tm._global_backward_hooks or _tm._global_backward_pre_hooks or _fwd_ad._current_level >= 0
                or torch._C._functorch.peek_interpreter_stack() is not None or torch._C._len_torch_dispatch_stack()
                or torch._C._len_torch_function_stack() or torch.jit.is_tracing() or torch.compiler.is_compiling())


def _addresses(m, cls, dtype, device, shapes, out):
    """Appends the addresses of the parameters ``shapes`` (name, shape; 0 for a missing bias) of a plain ``cls`` to ``out`` if
    the kernels can read them as they stand (else returns False).  ``device``: its index."""
    if type(m) is not cls:
        return False
    d = m.__dict__
    if d["_forward_hooks"] or d["_forward_pre_hooks"] or d["_backward_hooks"] or d["_backward_pre_hooks"] or "forward" in d:
        return False
    ps = d["_parameters"]
    for name, shape in shapes:
        p = ps.get(name, _ABSENT)
        if p is None and name == "bias" and cls is Linear:
            out.append(0)
            continue
        if p is _ABSENT or p is None or p.dtype is not dtype or p.get_device() != device or p.shape != shape or not p.is_contiguous():
            return False
        at = p.data_ptr()
        if at & 15:
            return False
        out.append(at)
    return True


def _input_ok(x) -> bool:
    return not (torch.is_grad_enabled() or type(x) is not torch.Tensor or not x.is_cuda or x.dim() != 3 or x.dtype not in _DTYPES
                or x.numel() == 0 or _observed() or not x.is_contiguous() or x.data_ptr() & 15
                or x.get_device() != torch.cuda.current_device())


def _block_words(B, S, E, dt, dev, parts):
    """(F, H, code, rms, pre_norm, causal, weights, eps1, eps2, scale) of a block of plain layers whose parameters the kernels can
    read as they stand, or None.  ``weights``: addresses of norm1, norm2, the fused QKV projection, outproj, ff1, ff2."""
    attn, norm1, norm2, ff1, ff2, act, pre_norm, causal = parts
    if not plain(attn, MultiHeadAttention):
        return None
    if isinstance(act, str):
        kind = act
    elif plain(act, Activation):
        kind = act.kind
    else:
        return None
    code = _ACT.get(kind)
    ad = attn.__dict__
    H = ad["num_heads"]
    D = E // H
    if (code is None or not E == ad["embed_dim"] == ad["kdim"] == ad["vdim"] or E % 8 or D % 8 or not 8 <= D <= 128
            or type(ff1) is not Linear):
        return None
    F = ff1.out_features
    if F % 8 or F == 0 or B * S * max(3 * E, F) >= 2 ** 31:
        return None
    rms = type(norm1) is RMSNorm
    norm_cls, norm_shapes = (RMSNorm, (("weight", (E,)),)) if rms else (LayerNorm, (("weight", (E,)), ("bias", (E,))))
    square, am = (("weight", (E, E)), ("bias", (E,))), ad["_modules"]
    q, k, v, o = am["qproj"], am["kproj"], am["vproj"], am["outproj"]
    n1, n2, qkv, rest = [], [], [], []
    if not (_addresses(norm1, norm_cls, dt, dev, norm_shapes, n1) and _addresses(norm2, norm_cls, dt, dev, norm_shapes, n2)
            and _addresses(q, Linear, dt, dev, square, qkv) and _addresses(k, Linear, dt, dev, square, qkv)
            and _addresses(v, Linear, dt, dev, square, qkv) and _addresses(o, Linear, dt, dev, square, rest)
            and _addresses(ff1, Linear, dt, dev, (("weight", (F, E)), ("bias", (F,))), rest)
            and _addresses(ff2, Linear, dt, dev, (("weight", (E, F)), ("bias", (E,))), rest)):
        return None
    for m in (q, k, v, o, ff1, ff2):
        if m.activation not in (None, "none"):
            return None
    # the three projections are one product when they lie back to back
    wq, bq, wk, bk, wv, bv = qkv
    if wk != wq + 2 * E * E or wv != wk + 2 * E * E:
        return None
    if bq:
        if bk != bq + 2 * E or bv != bk + 2 * E:
            return None
    elif bk or bv:
        return None
    if rms:
        n1.append(0)
        n2.append(0)
    return F, H, code, rms, bool(pre_norm), bool(causal), (*n1, *n2, wq, bq, *rest), norm1.eps, norm2.eps, 1.0 / math.sqrt(D)


class _Run:
    """How far a native call over a chain of blocks has come."""
    __slots__ = ("group", "done", "y", "spare", "sized", "ws", "keep", "error")

    def __init__(self, group):
        self.group, self.done, self.keep = group, 0, []
        self.y = self.spare = self.sized = self.ws = self.error = None


def evaluate_stack(x, blocks):
    """The output of a chain of blocks for ``x`` (B, S, E) and how many of them it stands for: one native call, up to the first
    block that it cannot take (see the module docstring).  ``blocks``: the parts of each (attn, norm1, norm2, ff1, ff2, act,
    pre_norm, causal); ``act``: an Activation module, or the name of a fusable activation.

    It starts with the first one and asks for the others by and by, so that the first kernel waits for the checks of one block only
    (about 20 us of the host) and the GPU works while the others are checked: one, three, then four at a time, since going to and
    fro costs the host 5 to 10 us.  One call on an idle GPU, us, all checked first | so: 12 layers, 1 x 77 858 | 711; 24 layers, 4 x 512
    2 440 | 2 083; 24 layers of 2 048, 1 x 1024 3 880 | 3 560; 4 layers, 4 x 512 621 | 577; calls back to back the same.  A few
    blocks that the host alone bounds go at once (4 layers, 1 x 77 384 | 369, but back to back 307 | 321)."""
    if not blocks or not _input_ok(x):
        return x, 0
    B, S, E = x.shape
    dt, dev, code_dt = x.dtype, x.get_device(), _DTYPES[x.dtype]
    counts, words, scalars = (ctypes.c_int * 3)(), (_l.L * (_WORDS * _GROUP))(), (_l.F * (3 * _GROUP))()
    run = _Run(len(blocks) if len(blocks) <= _GROUP and B * S < 512 else 1)

    def more():
        try:
            n = 0
            while n < run.group and run.done < len(blocks):
                w = _block_words(B, S, E, dt, dev, blocks[run.done])
                if w is None:
                    run.group = 0
                    break
                F, H, code, rms, pre_norm, causal, weights, eps1, eps2, scale = w
                if run.sized != (H, F):
                    run.sized = H, F
                    need = int(_l.lib().gb_block_ws(B, S, E, H, F))
                    if run.ws is None or run.ws.numel() < need:
                        run.keep.append(run.ws)        # (blocks of this group may use it)
                        run.ws = torch.empty(need, dtype=torch.uint8, device=x.device)
                frm, to = (x if run.y is None else run.y), (torch.empty_like(x) if run.spare is None else run.spare)
                words[_WORDS * n:_WORDS * (n + 1)] = (code_dt, B, S, E, H, F, rms, pre_norm, causal, code, frm.data_ptr(), to.data_ptr(), *weights,
                                                      run.ws.data_ptr(), run.ws.numel())
                scalars[3 * n:3 * (n + 1)] = eps1, eps2, scale
                run.spare, run.y = run.y, to           # by turns
                run.done += 1
                n += 1
            run.group = 0 if run.group == 0 else 3 if run.done == 1 else _GROUP
            counts[2] = run.group > 0 and run.done < len(blocks)
            counts[0] = n
        except BaseException as e:                     # (nothing passes through the native call)
            run.error = e

    more()
    if run.done == 0 and run.error is None:
        return x, 0
    _l.call("gb_stack_fwd", _More(more), counts, words, scalars, _l.I(_WORDS), _l.I(_GROUP), _l.stream_ptr())
    _l.kernel_count += 7 * counts[1]
    if run.error is not None or counts[1] != run.done:
        raise run.error or RuntimeError("the checks of a transformer block were interrupted")
    return (x if run.y is None else run.y), run.done


def evaluate(x, *parts):
    """The output of a single block, or None."""
    if not _input_ok(x):
        return None
    B, S, E = x.shape
    w = _block_words(B, S, E, x.dtype, x.get_device(), parts)
    if w is None:
        return None
    F, H, code, rms, pre_norm, causal, weights, eps1, eps2, scale = w
    need = int(_l.lib().gb_block_ws(B, S, E, H, F))
    ws = torch.empty(need, dtype=torch.uint8, device=x.device)
    y = torch.empty_like(x)
    words = (_l.L * _WORDS)(_DTYPES[x.dtype], B, S, E, H, F, rms, pre_norm, causal, code, x.data_ptr(), y.data_ptr(), *weights,
                            ws.data_ptr(), need)
    _l.call("gb_block_fwd", words, _l.I(_WORDS), _l.F(eps1), _l.F(eps2), _l.F(scale), _l.stream_ptr())
    return y


def chain(x, layers, cls, forward):
    """``layers`` (a ModuleList) applied one after another: without a tape in one native call, if all of them are plain ``cls``
    layers whose class's forward is still ``forward``, as far as it can take them, and layer by layer from there."""
    done = 0
    if not torch.is_grad_enabled() and type(layers) is ModuleList and cls.forward is forward:
        blocks = [l._parts() if plain(l, cls) else None for l in layers]
        if None not in blocks:
            x, done = evaluate_stack(x, blocks)
    for i, l in enumerate(layers):
        if i >= done:
            x = l(x)
    return x
