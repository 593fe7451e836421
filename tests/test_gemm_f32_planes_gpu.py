"""fp32 products as bf16 planes (csrc/gemm_exact.cu): one launch for the six plane products, K slices, the fused bias."""
import pytest
import torch

from gonn_b200 import lib as L
from gonn_b200.ops.gemm import gemm

pytestmark = pytest.mark.gpu


# one tile row, K that 64 does not divide (K % 8 == 0 where an operand is stored along K), split and cluster sizes, two-CTA tiles
@pytest.mark.parametrize("M,N,K,ta,tb", [(128, 256, 4100, False, True), (333, 512, 1000, False, False), (136, 132, 8200, True, False),
                                         (1100, 768, 520, True, True), (3000, 1028, 264, False, True)])
@pytest.mark.parametrize("bias,beta", [(False, False), (True, False), (True, True), (False, True)])
def test_against_float64(M, N, K, ta, tb, bias, beta):
    torch.manual_seed(K)
    a, b = torch.randn((K, M) if ta else (M, K)), torch.randn((N, K) if tb else (K, N))
    bv = torch.randn(N) * K ** 0.5 if bias else None
    want = (a.t() if ta else a).double() @ (b.t() if tb else b).double()
    out = torch.randn(M, N).cuda() if beta else None
    if bias:
        want = want + bv.double()
    if beta:
        want = want + out.double().cpu()
    got = gemm(a.cuda(), b.cuda(), trans_a=ta, trans_b=tb, bias=None if bv is None else bv.cuda(), out=out, beta=beta)
    L.assert_status_ok()
    # planes drop less than 2^-24 of each product; the accumulator truncates once per 16 products: K / 16 units of 2^-24
    # of a partial sum at worst, half that on average over the chain
    assert float((got.double().cpu() - want).norm() / want.norm()) < (K / 32 + 4) * 2.0 ** -24


def test_batches_share_an_operand_and_infinities_stay_in_their_row():
    a, b = torch.randn(3, 256, 512), torch.randn(512, 512)
    a[1, 5, 7] = float("inf")
    got = gemm(a.cuda(), b.cuda()).cpu()
    want = a.double() @ b.double()
    fin = torch.ones(3, 256, dtype=torch.bool)
    fin[1, 5] = False
    assert not got[~fin].isfinite().any()      # (the planes of b have both signs)
    assert float((got[fin].double() - want[fin]).norm() / want[fin].norm()) < 20 * 2.0 ** -24


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("M,N,K", [(1, 1, 3), (64, 10, 128), (65, 67, 40), (30, 130, 17), (1500, 1200, 33)])
def test_bias_of_the_simt_kernel(dtype, M, N, K):
    a, b, bias = torch.randn(M, K, dtype=dtype), torch.randn(N, K, dtype=dtype), torch.randn(N, dtype=dtype)
    out = torch.randn(M, N, dtype=dtype)
    got = gemm(a.cuda(), b.cuda(), trans_b=True, bias=bias.cuda(), out=out.cuda(), beta=True)
    want = a.double() @ b.double().t() + bias.double() + out.double()
    # rounding of K products and sums
    assert float((got.double().cpu() - want).norm() / want.norm()) < 4 * (K + 2) ** 0.5 * torch.finfo(dtype).eps


@pytest.mark.parametrize("ta,tb", [(False, True), (False, False), (True, False), (True, True)])
def test_infinities_nan_and_the_largest_values_as_in_fp32(ta, tb):
    """Every entry is finite, an infinity of one sign or NaN exactly where an fp32 product has it."""
    torch.manual_seed(3)
    M, N, K = 264, 520, 2048
    a, b = torch.randn(M, K), torch.randn(K, N)
    inf, big = float("inf"), torch.finfo(torch.float32).max
    a[3, 5] = inf                       # meets ordinary values of both signs
    a[4, 6] = -inf
    b[5, 7] = 0.0                       # inf * 0
    a[9, 10], b[10, 11] = inf, -inf     # both sides at one k
    a[12, 20], a[12, 21] = inf, inf     # two of them: NaN where their partners' signs differ
    a[15, 1] = float("nan")
    b[100, 200] = float("nan")
    b[101, 300] = inf
    a[30, 40], a[31, 41], a[32, 42] = big, -big, -3.4e38          # masks of the type's lowest value
    b[40] *= 1e-3
    b[41] *= 1e-3
    b[42] *= 1e-3
    a[50, 60], b[60, 70] = 3.395e38, 1.0      # between bf16's largest value and the rounding to infinity
    put = lambda t, tr: (t.t().contiguous().cuda().t() if tr else t.cuda())
    got = gemm(put(a, ta).t() if ta else a.cuda(), put(b, tb).t() if tb else b.cuda(), trans_a=ta, trans_b=tb).cpu()
    want = a @ b
    L.assert_status_ok()
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got == inf, want == inf) and torch.equal(got == -inf, want == -inf)
    fin = want.isfinite()
    exact = a.double() @ b.double()
    assert not fin.all() and fin[30].sum() > 0 and fin[32].sum() > 0
    for rows in (slice(30, 33), slice(50, 51), slice(60, M)):
        f = fin[rows]
        err = float((got[rows][f].double() - exact[rows][f]).norm() / exact[rows][f].norm())
        assert err < (K / 32 + 4) * 2.0 ** -24, err


def test_split_values_add_up():
    """A product with the identity returns the operand: finite values of all sizes, the largest ones among them."""
    n = 1024
    # (below 2^-100 the lo part would be subnormal, which is flushed to zero)
    x = torch.randn(n, n).abs().clamp_min(1e-5) * torch.logspace(-24, 38, n)[:, None]
    x[:, 0], x[:, 1], x[:, 2] = torch.finfo(torch.float32).max, -3.4e38, 3.3961775e38
    x = x.clamp(-torch.finfo(torch.float32).max, torch.finfo(torch.float32).max)
    got = gemm(x.cuda(), torch.eye(n).cuda()).cpu()
    # three roundings to 8 bits leave nothing of a 24-bit value; the accumulator, aligned to the hi part, which may lie in the
    # binade above, cuts each of the two sums by less than 2^-23 of it
    assert got.isfinite().all()
    assert float(((got.double() - x.double()) / x.double()).abs().max()) <= 2.0 ** -22
