"""The work this framework is measured on: training steps, evaluation and single operators.

Every case goes through the entry points that a user's program calls and is described by plain
values.  Twelve kinds of work are covered; ``listed()`` has one case of each, at the size that the
repository's benchmarks and configurations use, and ``draw()`` gives other sizes of the same kinds,
ragged ones among them.

    kind              what it stands for
    mlp_train         the quick-start classifier: a small fp32 model stepped eagerly by ``optim.SGD``
    lm_eval           logits of a few sequences from the 12-layer language model (no tape, short calls)
    lm_train          one captured data-parallel training step of that language model
    gpt_eval          logits of whole documents from the 1.3 B decoder (prefill)
    cnn_train         one captured training step of the convolutional classifier
    attention         bf16 / fp16 attention, forward and backward: causal self-attention over long
                      sequences, or cross-attention between ragged lengths
    attention_f64     double-precision attention, forward and backward (the reference's own precision)
    matmul_f64        a double-precision matrix product
    linear_f32        an ``nn.Linear`` in the layers' default type (fp32): forward and all gradients
    lstm_train        an fp32 LSTM over a batch of sequences: forward and backpropagation through time
    int8_linear       a dynamically quantised ``Linear`` on bf16 activations
"""
from __future__ import annotations

import math

import torch

LM = dict(vocab=32000, d_model=768, n_heads=12, d_ff=3072, max_seq=1024)
GPT_1B = dict(vocab=50304, d_model=2048, n_heads=16, d_ff=8192, max_seq=2048)
_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # the smallest calls: every launch and every microsecond of host work counts
        dict(name="mlp_train_64", kind="mlp_train", batch=64, hidden1=256, hidden2=128),
        # scoring one short prompt with the language model: latency, few rows per product
        dict(name="lm_eval_1x77", kind="lm_eval", layers=12, batch=1, seq=77),
        # the repository's flagship benchmark
        dict(name="lm_train_16x1024", kind="lm_train", layers=12, batch=16, seq=1024),
        # head size 128, RMSNorm and the widest products
        dict(name="gpt_eval_4x2048", kind="gpt_eval", layers=24, batch=4, seq=2048),
        # the image benchmark
        dict(name="cnn_train_256", kind="cnn_train", batch=256),
        # the attention benchmark: long causal sequences
        dict(name="attention_8x4096_d128", kind="attention", batch=8, heads=16, queries=4096, keys=4096, dim=128,
             causal=True, dtype="bf16"),
        # cross-attention of an encoder-decoder: unequal lengths that are no multiple of a tile
        dict(name="attention_cross_1000x1531", kind="attention", batch=6, heads=12, queries=1000, keys=1531, dim=64,
             causal=False, dtype="fp16"),
        # the reference's attention benchmark shape, in its precision
        dict(name="attention_f64_16x2048", kind="attention_f64", batch=1, heads=16, seq=2048, dim=64, causal=True),
        # the reference's matrix benchmark, in its precision
        dict(name="matmul_f64_2048", kind="matmul_f64", m=2048, n=2048, k=2048),
        # a feed-forward layer in the default type, with a row count that no tile divides
        dict(name="linear_f32_3000x1024", kind="linear_f32", rows=3000, inputs=1024, outputs=4096),
        dict(name="lstm_train_32x64", kind="lstm_train", layers=1, batch=32, steps=64, inputs=512, hidden=512),
        dict(name="int8_linear_8192", kind="int8_linear", rows=8192, inputs=4096, outputs=4096, per_channel=True),
    ]


def _log(rng, lo, hi):
    """A whole number from lo to hi, spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("mlp_train", "lm_eval", "lm_train", "gpt_eval", "cnn_train", "attention", "attention_f64",
                       "matmul_f64", "linear_f32", "lstm_train", "int8_linear"))
    if kind == "mlp_train":
        return dict(kind=kind, batch=_log(rng, 16, 512), hidden1=_log(rng, 64, 1024), hidden2=_log(rng, 32, 512))
    if kind == "lm_eval":
        return dict(kind=kind, layers=rng.randint(2, 12), batch=rng.randint(1, 4), seq=_log(rng, 16, 1024))
    if kind == "lm_train":
        return dict(kind=kind, layers=rng.randint(2, 12), batch=rng.randint(1, 16), seq=_log(rng, 96, 1024))
    if kind == "gpt_eval":
        return dict(kind=kind, layers=rng.randint(2, 24), batch=rng.randint(1, 4), seq=_log(rng, 128, 2048))
    if kind == "cnn_train":
        return dict(kind=kind, batch=rng.randint(16, 256))
    if kind == "attention":
        causal = rng.random() < 0.5
        q = _log(rng, 100, 4096)
        return dict(kind=kind, batch=rng.randint(1, 8), heads=rng.randint(4, 16), queries=q,
                    keys=q if causal else _log(rng, 100, 4096), dim=rng.choice((32, 64, 80, 96, 128)), causal=causal,
                    dtype=rng.choice(("bf16", "fp16")))
    if kind == "attention_f64":
        return dict(kind=kind, batch=rng.randint(1, 2), heads=rng.randint(2, 8), seq=_log(rng, 64, 2048),
                    dim=rng.choice((16, 32, 64)), causal=rng.random() < 0.5)
    if kind == "matmul_f64":
        return dict(kind=kind, m=_log(rng, 64, 2048), n=_log(rng, 64, 2048), k=_log(rng, 64, 2048))
    if kind == "linear_f32":
        return dict(kind=kind, rows=_log(rng, 64, 4096), inputs=8 * _log(rng, 16, 256), outputs=8 * _log(rng, 16, 512))
    if kind == "lstm_train":
        return dict(kind=kind, layers=rng.randint(1, 2), batch=rng.randint(4, 64), steps=rng.randint(8, 64),
                    inputs=8 * _log(rng, 8, 64), hidden=8 * _log(rng, 8, 64))
    return dict(kind=kind, rows=_log(rng, 64, 8192), inputs=16 * _log(rng, 16, 256), outputs=8 * _log(rng, 32, 512),
                per_channel=rng.random() < 0.5)


# ---------------------------------------------------------------------------------------
# preparation: what a program holds before the call
# ---------------------------------------------------------------------------------------
def prepare(case, seed):
    torch.manual_seed(seed)
    return _PREPARE[case["kind"]](case)


def _randn(*shape, dtype=torch.float32):
    return torch.randn(*shape, dtype=dtype, device="cuda")


def _prepare_mlp(c):
    from gonn_b200 import optim
    from gonn_b200.models.mlp import MLP
    model = MLP((784, c["hidden1"], c["hidden2"], 10), device="cuda")
    return dict(run=_run_mlp, model=model, opt=optim.SGD(model.parameters(), lr=0.01, momentum=0.9),
                x=torch.rand(c["batch"], 1, 28, 28, device="cuda"), y=torch.randint(0, 10, (c["batch"],), device="cuda"))


def _run_mlp(s):
    from gonn_b200 import nn
    s["opt"].zero_grad()
    loss = nn.CrossEntropyLoss(s["model"](s["x"]), s["y"])
    loss.backward()
    s["opt"].step()
    params = list(s["model"].parameters())
    return dict(loss=loss, params=params, grads=[p.grad for p in params])


def _language_model(c):
    from gonn_b200.models import GPT, TransformerLM
    cls, conf = (GPT, GPT_1B) if c["kind"] == "gpt_eval" else (TransformerLM, LM)
    model = cls(n_layers=c["layers"], dtype=torch.bfloat16, device="cuda", **conf)
    return model, torch.randint(0, conf["vocab"], (c["batch"], c["seq"]), device="cuda")


def _prepare_eval(c):
    model, ids = _language_model(c)
    model.eval()
    return dict(run=_run_eval, model=model, ids=ids)


def _run_eval(s):
    with torch.no_grad():
        return s["model"](s["ids"])


def _captured_step(model, x, y):
    """The step as the training benchmark runs it: the data-parallel engine with its fused AdamW,
    captured once and replayed."""
    from gonn_b200.distributed.ddp import DistributedDataParallel
    from gonn_b200.utils.graph import GraphedStep
    ddp = DistributedDataParallel(model, optimizer=dict(kind="adamw", lr=3e-4, weight_decay=0.1))

    def step(a, b):
        loss = model.loss(a, b)
        loss.backward()
        ddp.step()
        return loss

    return dict(run=_run_captured, model=model, ddp=ddp, step=GraphedStep(step, ddp, (x, y), warmup=1), x=x, y=y)


def _prepare_lm_train(c):
    model, ids = _language_model(c)
    return _captured_step(model, ids, torch.roll(ids, -1, 1))


def _prepare_cnn(c):
    from gonn_b200.models.cnn import SmallCNN
    model = SmallCNN(dtype=torch.bfloat16, device="cuda")
    return _captured_step(model, _randn(c["batch"], 3, 32, 32).bfloat16(),
                          torch.randint(0, 10, (c["batch"],), device="cuda"))


def _run_captured(s):
    loss = s["step"](s["x"], s["y"])
    return dict(loss=loss, params=s["ddp"].flat_params, grads=s["ddp"].flat_grads, buffers=list(s["model"].buffers()))


def _prepare_attention(c):
    dt = _DTYPES.get(c.get("dtype"), torch.float64)
    b, h, d = c["batch"], c["heads"], c["dim"]
    nq, nk = (c["seq"], c["seq"]) if "seq" in c else (c["queries"], c["keys"])
    q, k, v = (_randn(b, n, h, d, dtype=dt).requires_grad_() for n in (nq, nk, nk))
    return dict(run=_run_attention, q=q, k=k, v=v, dout=_randn(b, nq, h, d, dtype=dt), causal=c["causal"])


def _run_attention(s):
    from gonn_b200.ops.attention import flash_attention
    for t in (s["q"], s["k"], s["v"]):
        t.grad = None
    out = flash_attention(s["q"], s["k"], s["v"], causal=s["causal"])
    out.backward(s["dout"])
    return dict(out=out, dq=s["q"].grad, dk=s["k"].grad, dv=s["v"].grad)


def _prepare_matmul(c):
    return dict(run=_run_matmul, a=_randn(c["m"], c["k"], dtype=torch.float64), b=_randn(c["k"], c["n"], dtype=torch.float64))


def _run_matmul(s):
    from gonn_b200 import tensor as T
    return T.MatMul(s["a"], s["b"])


def _prepare_linear(c):
    from gonn_b200 import nn
    return dict(run=_run_linear, layer=nn.Linear(c["inputs"], c["outputs"], device="cuda"),
                x=_randn(c["rows"], c["inputs"]).requires_grad_(), dy=_randn(c["rows"], c["outputs"]))


def _run_linear(s):
    layer, x = s["layer"], s["x"]
    x.grad = layer.weight.grad = layer.bias.grad = None
    y = layer(x)
    y.backward(s["dy"])
    return dict(y=y, dx=x.grad, dw=layer.weight.grad, db=layer.bias.grad)


def _prepare_lstm(c):
    from gonn_b200 import nn
    return dict(run=_run_lstm, layer=nn.LSTM(c["inputs"], c["hidden"], c["layers"], device="cuda"),
                x=_randn(c["batch"], c["steps"], c["inputs"]).requires_grad_(),
                dy=_randn(c["batch"], c["steps"], c["hidden"]))


def _run_lstm(s):
    layer, x = s["layer"], s["x"]
    x.grad = None
    for p in layer.parameters():
        p.grad = None
    out, (h, cell) = layer.ForwardWithState(x)
    out.backward(s["dy"])
    return dict(out=out, h=h, c=cell, dx=x.grad, grads=[p.grad for p in layer.parameters()])


def _prepare_int8(c):
    from gonn_b200 import nn, quant
    lin = nn.Linear(c["inputs"], c["outputs"], device="cuda", dtype=torch.bfloat16)
    layer = quant.DynamicLinear(lin, per_channel_weights=c["per_channel"])
    return dict(run=_run_int8, layer=layer, x=_randn(c["rows"], c["inputs"]).bfloat16())


def _run_int8(s):
    return s["layer"](s["x"])


_PREPARE = dict(mlp_train=_prepare_mlp, lm_eval=_prepare_eval, lm_train=_prepare_lm_train, gpt_eval=_prepare_eval,
                cnn_train=_prepare_cnn, attention=_prepare_attention, attention_f64=_prepare_attention,
                matmul_f64=_prepare_matmul, linear_f32=_prepare_linear, lstm_train=_prepare_lstm, int8_linear=_prepare_int8)


def run(state):
    return state["run"](state)


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
def _transformer_work(c, conf, train):
    """(bytes, flops) of the language models; a training step does three times the products of a
    forward pass, reads and writes the AdamW state (fp32 master and moments, 16-bit gradients) once."""
    tokens, d = c["batch"] * c["seq"], conf["d_model"]
    weights = c["layers"] * (4 * d * d + 2 * d * conf["d_ff"]) + d * conf["vocab"]
    attention = c["layers"] * 2.0 * c["batch"] * c["seq"] ** 2 * d             # causal: half of the pairs
    flops = 2.0 * tokens * weights + attention
    tables = (conf["vocab"] + conf["max_seq"]) * d
    if train:
        return (weights + tables) * (2 + 2 + 2 + 24) + 16.0 * tokens, 6.0 * tokens * weights + 3.5 * attention
    return 2.0 * weights + 2.0 * tokens * (conf["vocab"] + d), flops


def work(case):
    c, kind = case, case["kind"]
    if kind == "mlp_train":
        w = 784 * c["hidden1"] + c["hidden1"] * c["hidden2"] + 10 * c["hidden2"]
        nbytes, flops = 4.0 * (c["batch"] * 784 + 6 * w), 6.0 * c["batch"] * w
    elif kind in ("lm_eval", "gpt_eval"):
        nbytes, flops = _transformer_work(c, GPT_1B if kind == "gpt_eval" else LM, False)
    elif kind == "lm_train":
        nbytes, flops = _transformer_work(c, LM, True)
    elif kind == "cnn_train":
        b = c["batch"]
        # input, the first convolution's activations (30 x 30 x 64) in both directions, the pooled
        # ones and the second convolution's (13 x 13 x 128) in both directions, 16-bit
        nbytes = 2.0 * b * (3072 + 4 * 57600 + 4 * 14400 + 4 * 21632)
        flops = b * (4.0 * 900 * 27 * 64 + 6.0 * 169 * 576 * 128)
    elif kind in ("attention", "attention_f64"):
        nq, nk = (c["seq"], c["seq"]) if "seq" in c else (c["queries"], c["keys"])
        bh, d, size = c["batch"] * c["heads"], c["dim"], 8 if kind == "attention_f64" else 2
        nbytes = size * bh * d * (4.0 * nq + 4.0 * nk)
        flops = 14.0 * bh * nq * nk * d * (0.5 if c["causal"] else 1.0)
    elif kind == "matmul_f64":
        nbytes = 8.0 * (c["m"] * c["k"] + c["k"] * c["n"] + c["m"] * c["n"])
        flops = 2.0 * c["m"] * c["n"] * c["k"]
    elif kind == "linear_f32":
        r, i, o = c["rows"], c["inputs"], c["outputs"]
        nbytes, flops = 4.0 * (2 * r * i + 2 * r * o + 2 * i * o), 6.0 * r * i * o
    elif kind == "lstm_train":
        rows, h = c["batch"] * c["steps"], c["hidden"]
        nbytes = flops = 0.0
        for layer in range(c["layers"]):
            i = c["inputs"] if layer == 0 else h
            nbytes += 4.0 * (2 * rows * (i + h) + 2 * 4 * h * (i + h))
            flops += 6.0 * rows * 4 * h * (i + h)
    else:
        r, i, o = c["rows"], c["inputs"], c["outputs"]
        nbytes, flops = 2.0 * r * i + i * o + 2.0 * r * o, 2.0 * r * i * o
    return dict(bytes=nbytes, flops=flops)


# Four times the largest error seen against the same path evaluated in 64 bits (the single operators
# and the fp32 layers) or in fp32 / with other kernels of the same precision (the 16-bit models).
_TOLERANCE = {
    "mlp_train": dict(rel=5e-6),
    "lm_eval": dict(rel=3e-2),
    "lm_train": dict(rel=3e-2),
    "gpt_eval": dict(rel=2.5e-2),
    "cnn_train": dict(rel=4e-2),
    "attention_bf16": dict(rel=1e-2),
    "attention_fp16": dict(rel=1.4e-3),
    "attention_f64": dict(rel=1e-14),
    "matmul_f64": dict(rel=6e-15),
    "linear_f32": dict(rel=1.2e-5),
    "lstm_train": dict(rel=2.5e-5),
    "int8_linear": dict(rel=1.2e-2),
}


def tolerance(case):
    kind = case["kind"]
    return dict(_TOLERANCE[kind + "_" + case["dtype"] if kind == "attention" else kind])
