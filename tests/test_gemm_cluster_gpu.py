"""The cluster kernel for products with few tiles (csrc/gemm.cu): K cut over 1 .. 8 CTAs, the whole epilogue."""
import pytest
import torch

from gonn_b200 import lib as L
from gonn_b200.ops.gemm import _dact_ref, gemm

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[0, 1, 2, 4, 8])
def splits(request):
    L.call("gb_gemm_cluster_tune", L.I(request.param))
    yield request.param
    L.call("gb_gemm_cluster_tune", L.I(0))


def _close(got, want, dtype, what):
    # fp32 sums, one rounding of the result to 8 or 11 bits
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    err = float((got.double().cpu() - want).norm() / want.norm())
    assert err < tol, f"{what}: {err:.3g}"


# around the 128 x 64 x 64 tile, one row, a K of one k-block that leaves seven CTAs of a cluster empty, ragged N
@pytest.mark.parametrize("M,N,K", [(1, 64, 64), (77, 768, 768), (128, 72, 40), (129, 200, 520), (300, 130, 1000), (77, 99, 264)])
@pytest.mark.parametrize("ta,tb", [(False, True), (False, False), (True, False), (True, True)])
def test_forms(splits, M, N, K, ta, tb):
    torch.manual_seed(M + N + K)
    dt = torch.float16 if M % 2 else torch.bfloat16
    a, b = torch.randn((K, M) if ta else (M, K)).to(dt), torch.randn((N, K) if tb else (K, N)).to(dt)
    want = (a.t() if ta else a).double() @ (b.t() if tb else b).double()
    got = gemm(a.cuda(), b.cuda(), trans_a=ta, trans_b=tb)
    _close(got, want, dt, "plain")
    f32 = torch.randn(M, N, device="cuda")
    base = f32.double().cpu()
    gemm(a.cuda(), b.cuda(), trans_a=ta, trans_b=tb, out=f32, beta=True, alpha=0.5)
    err = float((f32.double().cpu() - base - 0.5 * want).norm() / want.norm())
    assert err < 1e-6, err                       # exact products, fp32 sums of at most 1000 terms
    L.assert_status_ok()
    assert torch.equal(gemm(a.cuda(), b.cuda(), trans_a=ta, trans_b=tb), got)


# (a derivative factor goes with a plain product)
@pytest.mark.parametrize("act,aux_mode", [(a, x) for a in (None, "relu", "gelu", "geluexact") for x in (None, "add", "store_pre")]
                         + [(None, x) for x in ("mul_dgelu", "mul_drelu", "mul_dgeluexact")])
@pytest.mark.parametrize("N", [192, 200, 77])
def test_epilogue(splits, act, aux_mode, N):
    torch.manual_seed(N)
    dt, M, K = torch.bfloat16, 150, 320
    a, b, bias = torch.randn(M, K).to(dt), (torch.randn(N, K) * 0.1).to(dt), torch.randn(N).to(dt)
    aux = torch.randn(M, N).to(dt) if aux_mode else None
    auxc = None if aux is None else aux.cuda()
    got = gemm(a.cuda(), b.cuda(), trans_b=True, bias=bias.cuda(), act=act, aux=auxc, aux_mode=aux_mode)
    pre = a.double() @ b.double().t() + bias.double()
    f = torch.nn.functional
    want = {None: pre, "relu": torch.relu(pre), "gelu": f.gelu(pre, approximate="tanh"), "geluexact": f.gelu(pre)}[act]
    if aux_mode == "add":
        want = want + aux.double()
    elif aux_mode == "store_pre":
        _close(auxc, pre, dt, "pre")
    elif aux_mode:
        want = want * _dact_ref(aux.double(), {"mul_dgelu": 3, "mul_drelu": 4, "mul_dgeluexact": 5}[aux_mode])
    _close(got, want, dt, "out")


def test_batches(splits):
    a, b = torch.randn(3, 60, 96).bfloat16(), torch.randn(96, 72).bfloat16()
    _close(gemm(a.cuda(), b.cuda()), a.double() @ b.double(), torch.bfloat16, "batched")
