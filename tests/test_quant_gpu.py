"""int8 tcgen05 GEMM with the dequantising epilogue, device-side observers and fake quantisation
against the host restatement of the reference's integer loop."""
import pytest
import torch

from gonn_b200 import lib as _l
from gonn_b200 import quant as Q
from gonn_b200.nn import Linear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_channel", [False, True])
@pytest.mark.parametrize("shape", [(64, 128, 96), (300, 200, 130), (1024, 768, 3072),
                                   (2300, 400, 2312), (2300, 400, 2311), (2049, 16, 2304)])   # two-CTA tiles: ragged edges, unaligned rows, one k-block
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_dynamic_linear_matches_integer_reference(per_channel, shape, dtype, status_ok):
    M, K, N = shape
    torch.manual_seed(0)
    lin = Linear(K, N, dtype=torch.float32)
    x = torch.randn(M, K) * 2
    dl = Q.DynamicLinear(lin, per_channel)
    xd = x.to("cuda", dtype)
    y = dl(xd)
    # host reference with the q-parameters of the (dtype-rounded) input
    xr = xd.double().cpu()
    sx, zx = Q.affine_qparams(float(xr.min()), float(xr.max()))
    ref = dl.core.forward_host(xr, sx, zx)
    tol = 2e-2 if dtype == torch.bfloat16 else 2e-4
    assert ((y.double().cpu() - ref).abs() / (1 + ref.abs())).max().item() < tol
    f = lin(x.double().float())
    assert (y.float().cpu() - f).abs().max().item() < 0.06 * f.abs().max().item()


def test_static_linear_and_observer(status_ok):
    torch.manual_seed(1)
    lin = Linear(256, 64)
    sl = Q.StaticLinear(lin, True)
    x = torch.randn(128, 256)
    sl.Calibrate(x)
    y = sl(x.cuda())
    ref = sl.core.forward_host(x.double(), sl.InScale, sl.InZeroPoint)
    assert (y.double().cpu() - ref).abs().max().item() < 1e-3
    qp4, zp = Q._observe_device(x.cuda())
    s, z = Q.affine_qparams(float(x.min()), float(x.max()))
    assert abs(qp4[2].item() - s) < 1e-7 and int(zp.item()) == z


def test_fake_quant_kernel_matches_host(status_ok):
    fq = Q.FakeQuant()
    x = torch.randn(10000) * 2
    fq.train()
    yh = fq(x.double().requires_grad_(True))
    fq.eval()
    xd = x.cuda().requires_grad_(True)
    yd = fq(xd)
    xh = x.double().requires_grad_(True)
    yh = fq(xh)
    assert (yd.double().cpu() - yh).abs().max().item() < 1e-5
    g = torch.randn(10000)
    yd.backward(g.cuda())
    yh.backward(g.double())
    assert (xd.grad.double().cpu() - xh.grad).abs().max().item() < 1e-6


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(1, 1), (3, 5), (7, 16), (64, 256), (513, 1531), (2000, 1024)])
@pytest.mark.parametrize("offset", [0, 1])     # 1: rows that are not 16-byte aligned
def test_dynamic_quantisation_bytes(dtype, shape, offset, status_ok):
    """One call that observes and quantises leaves the bytes of the two calls, zeros in the padding, and follows the rule of
    the reference (halves away from zero) wherever x / scale is exact: steps of a half and a range of 255 make the scale 1."""
    M, K = shape
    pitch = (K + 15) // 16 * 16
    torch.manual_seed(M)
    flat = torch.randint(-256, 255, (M * K + offset,)).double() / 2
    if M * K >= 2:
        flat[offset], flat[-1] = -128.0, 127.0
    x = flat.to("cuda", dtype)[offset:].view(M, K)
    scratch = torch.empty(_l.lib().gb_q_scratch_floats(), device="cuda")
    qp, zp = torch.empty(4, device="cuda"), torch.empty(1, dtype=torch.int32, device="cuda")
    q = torch.full((M, pitch), 77, dtype=torch.int8, device="cuda")
    _l.call("gb_q_dynamic", _l.I(_l.dtype_code(dtype)), _l.ptr(x), _l.ptr(q), _l.L(M), _l.L(K), _l.L(pitch), _l.ptr(scratch),
            _l.ptr(qp), _l.ptr(zp), _l.stream_ptr())
    qp2, zp2 = Q._observe_device(x)
    q2 = torch.zeros((M, pitch), dtype=torch.int8, device="cuda")
    _l.call("gb_q_quantize", _l.I(_l.dtype_code(dtype)), _l.ptr(x), _l.ptr(q2), _l.L(M), _l.L(K), _l.L(pitch), _l.ptr(qp2[2:]),
            _l.ptr(zp2), _l.I(0), _l.stream_ptr())
    assert torch.equal(q, q2) and torch.equal(qp, qp2) and torch.equal(zp, zp2)
    if M * K >= 2:
        assert qp[2].item() == 1.0 and zp.item() == 0
        assert torch.equal(q[:, :K].cpu(), Q.quantize_value(flat[offset:].view(M, K), 1.0, 0).to(torch.int8))
