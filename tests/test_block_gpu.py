"""A transformer block in one native call (nn/block.py) against the same block operator by operator."""
import copy

import pytest
import torch

from gonn_b200 import lib as L, nn
from gonn_b200.models.lm import GPTBlock
from gonn_b200.nn import block

pytestmark = pytest.mark.gpu


def _encoder(act, pre_norm, causal, dtype):
    return nn.TransformerEncoderLayer(128, 4, 264, pre_norm=pre_norm, activation=act, causal=causal, dtype=dtype, device="cuda")


def _calls(fn):
    n = L.launch_count
    with torch.no_grad():
        y = fn()
    return y, L.launch_count - n


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("pre_norm,causal", [(True, True), (True, False), (False, False)])
@pytest.mark.parametrize("act", [nn.ReLU, nn.GELU, nn.GELUExact])
@pytest.mark.parametrize("B,S", [(1, 1), (3, 77), (2, 130)])
def test_same_bits_as_the_operators(dtype, pre_norm, causal, act, B, S):
    torch.manual_seed(S)
    m = _encoder(act(), pre_norm, causal, dtype)
    for p in m.parameters():
        p.data += 0.1 * torch.randn_like(p)
    x = torch.randn(B, S, 128, device="cuda").to(dtype)
    y, n = _calls(lambda: m(x))
    assert n == 1
    h = m.norm2.register_forward_hook(lambda *a: None)
    want, n = _calls(lambda: m(x))                  # a hook: operator by operator
    h.remove()
    assert n > 1
    # the same kernels in the same order, the pre-activation aside
    assert torch.equal(y, want)
    L.assert_status_ok()


def test_gpt_block_and_missing_biases():
    m = GPTBlock(128, 2, 256, dtype=torch.bfloat16, device="cuda")
    x = torch.randn(2, 50, 128, device="cuda").bfloat16()
    y, n = _calls(lambda: m(x))
    assert n == 1
    assert torch.equal(y, m(x).detach())            # with gradients: operator by operator
    for q in (m.attn.outproj, m.ff1, m.ff2):
        q.bias = None
    y2, n = _calls(lambda: m(x))
    assert n == 1 and torch.equal(y2, m(x).detach())


def test_what_runs_operator_by_operator():
    x = torch.randn(2, 40, 128, device="cuda").bfloat16()
    base = _encoder(nn.GELU(), True, True, torch.bfloat16)

    def counts(change, x=x):
        m = copy.deepcopy(base)
        m.attn._pack_qkv()
        undo = change(m)
        y, n = _calls(lambda: m(x))
        if undo is not None:
            undo.remove()
        return n

    assert counts(lambda m: None) == 1
    assert counts(lambda m: m.attn.register_forward_hook(lambda *a: None)) > 1
    assert counts(lambda m: m.drop1.register_forward_pre_hook(lambda *a: None)) > 1
    assert counts(lambda m: setattr(m.ff1, "forward", m.ff1.forward)) > 1
    assert counts(lambda m: m.norm1.float() and None) > 1                     # fp32 norm weights
    assert counts(lambda m: torch.nn.utils.parametrizations.weight_norm(m.ff2) and None) > 1
    assert counts(lambda m: None, x.transpose(0, 1).contiguous().transpose(0, 1)) > 1
    assert counts(lambda m: torch.nn.modules.module.register_module_forward_hook(lambda *a: None)) > 1

    class Sub(type(base)):
        pass
    sub = Sub(128, 4, 264, pre_norm=True, dtype=torch.bfloat16, device="cuda")
    assert _calls(lambda: sub(x))[1] > 1
    # training mode with dropout draws its masks; evaluation mode does not
    d = nn.TransformerEncoderLayer(128, 4, 264, pre_norm=True, dropout=0.5, dtype=torch.bfloat16, device="cuda")
    assert _calls(lambda: d(x))[1] > 1
    d.eval()
    assert _calls(lambda: d(x))[1] == 1
    assert block.evaluate(x, base.attn, base.norm1, base.norm2, base.ff1, base.ff2, base.act, True, True) is None   # tape on


@pytest.mark.parametrize("layers", [1, 2, 5])
def test_a_chain_of_blocks_is_one_call(layers):
    """The models' chains: the same bits as block by block, an input that stays as it is, and block by block as soon as one of
    them is observed, replaced or cannot be taken."""
    from gonn_b200.models.lm import GPT
    torch.manual_seed(layers)
    enc = nn.TransformerEncoder(layers, 128, 4, 264, pre_norm=True, activation=nn.GELU(), dtype=torch.bfloat16, device="cuda")
    gpt = GPT(64, 128, layers, 4, 256, 64, dtype=torch.bfloat16, device="cuda").layers
    for stack, run in ((enc.layers, enc), (gpt, lambda x: block.chain(x, gpt, GPTBlock, GPTBlock.forward))):
        for p in stack.parameters():
            p.data += 0.05 * torch.randn_like(p)
        x = torch.randn(2, 33, 128, device="cuda").bfloat16()
        keep = x.clone()
        y, n = _calls(lambda: run(x))
        assert n == 1 and torch.equal(x, keep)
        want = x
        with torch.no_grad():
            for l in stack:
                want = l(want)
        assert torch.equal(y, want)
        last = stack[layers - 1]
        h = last.register_forward_hook(lambda *a: None)
        y2, n = _calls(lambda: run(x))
        h.remove()
        assert n == layers and torch.equal(y2, want)              # each by itself still one call
        last.forward = last.forward
        assert _calls(lambda: run(x))[1] == layers
        del last.__dict__["forward"]
        last.norm2.float()
        assert _calls(lambda: run(x))[1] > layers
        last.norm2.to(torch.bfloat16)
        assert _calls(lambda: run(x))[1] == 1
    seen = []
    original = nn.TransformerEncoderLayer.forward
    try:
        nn.TransformerEncoderLayer.forward = lambda self, x: seen.append(1) or original(self, x)
        _calls(lambda: enc(x))
    finally:
        nn.TransformerEncoderLayer.forward = original
    assert len(seen) == layers


def test_a_chain_up_to_a_block_that_it_cannot_take(monkeypatch):
    """One native call up to that block, whose output goes on from there; nothing is computed or looked at twice."""
    torch.manual_seed(0)
    enc = nn.TransformerEncoder(9, 128, 4, 264, pre_norm=True, activation=nn.GELU(), dtype=torch.bfloat16, device="cuda")
    x = torch.randn(2, 33, 128, device="cuda").bfloat16()
    looked = []
    real = block._block_words
    monkeypatch.setattr(block, "_block_words", lambda *a: looked.append(1) or real(*a))
    for at in (0, 1, 2, 5, 8):
        layer = enc.layers[at]
        layer.norm2.float()
        want = [x]
        with torch.no_grad():
            for l in enc.layers:
                want.append(l(want[-1]))
        alone = _calls(lambda: layer(want[at]))[1]
        looked.clear()
        y, n = _calls(lambda: enc(x))
        # the chain (if it has a first block), the block operator by operator, the others each by itself
        assert n == (at > 0) + alone + (8 - at) and len(looked) == 10 and torch.equal(y, want[-1])
        layer.norm2.to(torch.bfloat16)
    L.assert_status_ok()


def test_a_chain_of_unlike_blocks():
    """Feed-forward layers and heads that differ: the workspace grows on the way."""
    torch.manual_seed(1)
    stack = nn.ModuleList([nn.TransformerEncoderLayer(128, h, f, pre_norm=i % 2 == 0, causal=i % 3 == 0, activation=nn.ReLU(), dtype=torch.bfloat16,
                                                      device="cuda") for i, (h, f) in enumerate([(4, 64), (8, 512), (2, 128), (4, 1024), (4, 1024), (1, 8)])])
    x = torch.randn(3, 70, 128, device="cuda").bfloat16()
    cls = nn.TransformerEncoderLayer
    y, n = _calls(lambda: block.chain(x, stack, cls, cls.forward))
    want = x
    with torch.no_grad():
        for l in stack:
            want = l(want)
    assert n == 1 and torch.equal(y, want)


def test_an_error_among_the_checks_reaches_the_caller(monkeypatch):
    enc = nn.TransformerEncoder(4, 128, 4, 264, pre_norm=True, activation=nn.GELU(), dtype=torch.bfloat16, device="cuda")
    x = torch.randn(1, 5, 128, device="cuda").bfloat16()
    with torch.no_grad():
        want = enc(x)
        q = enc.layers[2].attn._modules.pop("qproj")
        with pytest.raises(KeyError):
            enc(x)
        enc.layers[2].attn._modules["qproj"] = q
        assert torch.equal(enc(x), want)
