"""Which 16-bit products take the cluster kernel (host code of csrc/gemm.cu; no GPU needed)."""
import pytest

from gonn_b200 import lib as L

pytestmark = pytest.mark.skipif(not L.available(), reason="the native library is not built")


# the sizes measured beside the rule: parts where the cluster kernel is ahead, 0 where one CTA per tile is, or not behind
@pytest.mark.parametrize("M,N,K,parts", [
    (77, 768, 3072, 8), (77, 768, 768, 8), (1, 768, 768, 8), (64, 576, 512, 8), (128, 128, 1024, 8), (64, 64, 256, 0),
    (256, 256, 256, 0), (512, 512, 512, 0), (64, 784, 256, 0), (128, 512, 640, 0), (128, 512, 768, 8),
    (128, 1280, 768, 0), (128, 1280, 1024, 4), (512, 320, 1024, 4), (128, 1280, 4096, 8), (64, 1280, 512, 4),
    (32, 2304, 512, 4), (16, 2304, 768, 4), (77, 2304, 768, 0), (77, 2304, 1024, 4), (256, 1024, 768, 0), (256, 1024, 1024, 4),
    (64, 2624, 768, 0), (64, 2624, 1024, 4), (128, 2048, 8192, 4), (300, 768, 3072, 4), (2048, 64, 2048, 4),
    (700, 768, 3072, 2), (77, 3072, 768, 0), (128, 8192, 2048, 0), (300, 2304, 768, 0), (1000, 1000, 1000, 0)])
def test_parts(M, N, K, parts):
    assert L.lib().gb_gemm_cluster_parts(L.I(M), L.I(N), L.I(K), L.I(1)) == parts
