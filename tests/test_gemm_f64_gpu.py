"""The fp64 tensor-core product (csrc/gemm_exact.cu): tile edges, both storage forms, K cut over a cluster."""
import pytest
import torch

from gonn_b200 import lib as L
from gonn_b200.ops.gemm import gemm

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[0, 1, 2, 8])
def splits(request):
    L.call("gb_gemm_f64_tune", L.I(request.param))
    yield request.param
    L.call("gb_gemm_f64_tune", L.I(0))


# around the 64 x 64 x 16 tile, odd pitches (8-byte copies), a K that leaves the last parts of a cluster empty
@pytest.mark.parametrize("M,N,K", [(64, 64, 16), (65, 127, 17), (128, 64, 257), (100, 190, 33), (193, 66, 1000), (64, 64, 2048)])
@pytest.mark.parametrize("ta", [False, True])
@pytest.mark.parametrize("tb", [False, True])
def test_matches_float64(splits, M, N, K, ta, tb):
    torch.manual_seed(M + N + K)
    a = torch.randn((K, M) if ta else (M, K), dtype=torch.float64)
    b = torch.randn((N, K) if tb else (K, N), dtype=torch.float64)
    want = (a.t() if ta else a) @ (b.t() if tb else b)
    got = gemm(a.cuda(), b.cuda(), trans_a=ta, trans_b=tb)
    # K rounded products and sums on both sides: sqrt(K) units of 2^-53 each, with room for the order
    tol = 8 * 2.0 ** -53 * K ** 0.5
    assert float((got.cpu() - want).norm() / want.norm()) < tol
    out = torch.randn(M, N + 3, dtype=torch.float64, device="cuda")[:, 1:N + 1]      # odd pitch, 8-byte aligned
    base = out.clone()
    gemm(a.cuda(), b.cuda(), trans_a=ta, trans_b=tb, out=out, beta=True, alpha=-0.5)
    want2 = base.cpu() - 0.5 * want
    assert float((out.cpu() - want2).norm() / want2.norm()) < tol
    assert torch.equal(gemm(a.cuda(), b.cuda(), trans_a=ta, trans_b=tb), got)        # bit-reproducible


def test_batched_and_broadcast(splits):
    a = torch.randn(3, 70, 90, dtype=torch.float64, device="cuda")
    b = torch.randn(90, 66, dtype=torch.float64, device="cuda")
    got = gemm(a, b)
    want = a.cpu() @ b.cpu()
    assert float((got.cpu() - want).norm() / want.norm()) < 1e-14
