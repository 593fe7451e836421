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
