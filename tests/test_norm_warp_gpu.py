"""The warp-per-row norm forward (csrc/norm.cu): every vector count per lane, ragged rows, weights it cannot load whole."""
import pytest
import torch

from gonn_b200 import lib as L
from gonn_b200.ops import norm as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,wdtype", [(torch.bfloat16, torch.bfloat16), (torch.float16, torch.float32), (torch.float32, torch.float32)])
@pytest.mark.parametrize("nvec", [1, 31, 33, 64, 65, 97, 129, 192, 193, 256, 257])
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("shift", [0, 1])
def test_forward(dtype, wdtype, nvec, rms, shift):
    D, rows = nvec * (4 if dtype == torch.float32 else 8), 7
    torch.manual_seed(nvec)
    x = (torch.randn(rows, D) * 3 + 50 * (not rms)).to(dtype)             # a mean far above the spread
    w, b = (torch.randn(D + 1)[shift:shift + D].to(wdtype) for _ in range(2))
    wc, bc = (torch.empty(D + 1, dtype=wdtype, device="cuda")[shift:shift + D].copy_(t) for t in (w, b))
    got = (N.rms_norm(x.cuda(), wc, 1e-6) if rms else N.layer_norm(x.cuda(), wc, bc, 1e-5)).double().cpu()
    L.assert_status_ok()
    want = N.norm_ref(x.double(), w.double(), None if rms else b.double(), 1e-6 if rms else 1e-5, rms)
    # one rounding of the result; the fp32 sums of the shifted row stay far below it (fp32: 2^-24 per term, D terms, and the
    # cancellation of the offset, 50 / 3 of it)
    tol = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 1e-5}[dtype]
    assert float((got - want).norm() / want.norm()) < tol


@pytest.mark.parametrize("dtype,wdtype", [(torch.bfloat16, torch.bfloat16), (torch.float16, torch.float32), (torch.float32, torch.float32)])
@pytest.mark.parametrize("nvec,rows", [(3, 9473), (70, 9480), (129, 4737), (256, 9500)])
@pytest.mark.parametrize("rms", [False, True])
def test_staged_weights_over_many_rows(dtype, wdtype, nvec, rows, rms):
    """Weights that are not 16-byte aligned stand in shared memory while a warp takes row after row: the bits of aligned ones."""
    D = nvec * (4 if dtype == torch.float32 else 8)
    x = (torch.randn(rows, D, device="cuda") * 3 + 5).to(dtype)
    w, b = (torch.randn(D, device="cuda").to(wdtype) for _ in range(2))
    wu, bu = (torch.empty(D + 1, dtype=wdtype, device="cuda")[1:].copy_(t) for t in (w, b))
    f = (lambda p, q: N.rms_norm(x, p, 1e-6)) if rms else (lambda p, q: N.layer_norm(x, p, q, 1e-5))
    assert wu.data_ptr() % 16 and torch.equal(f(wu, bu), f(w, b))
    L.assert_status_ok()
