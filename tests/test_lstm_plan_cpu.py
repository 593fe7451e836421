"""Which LSTM layers the persistent kernels accept (host code of csrc/lstm_seq.cu; no GPU needed)."""
import pytest

from gonn_b200 import lib as L

pytestmark = pytest.mark.skipif(not L.available(), reason="the native library is not built")

BLOCK = 227 * 1024        # shared memory of a block of sm_100a, static and dynamic together


def test_accepted_layers_leave_room_for_static_shared_memory():
    l = L.lib()
    widest = 0
    for H in range(4, 1100, 4):
        for B in range(1, 602, 8):                 # a plan depends on the batch through its tiles of 8 sequences
            if not l.gb_lstm_seq_fits(L.I(B), L.I(H)):
                continue
            for bwd in (0, 1):
                dyn = int(l.gb_lstm_seq_smem(L.I(B), L.I(H), L.I(bwd)))
                # both kernels hold a 4-byte static flag beside it
                assert 0 < dyn <= BLOCK - 4, (B, H, bwd, dyn)
                widest = max(widest, dyn)
    assert widest > BLOCK - 2048                   # the boundary is in the range above


@pytest.mark.parametrize("B,H", [(20, 896), (50, 892), (85, 888), (115, 884), (150, 880), (180, 876), (210, 872), (245, 868)])
def test_layers_that_would_need_the_whole_block_are_refused(B, H):
    assert not L.lib().gb_lstm_seq_fits(L.I(B), L.I(H))


def test_fewer_sms_fit_fewer_layers():
    """Every CTA of the cooperative launch needs an SM of its own: on a part of a GPU the steps take over."""
    l = L.lib()
    fits = lambda sms, B, H: bool(l.gb_lstm_seq_fits_on(L.I(sms), L.I(B), L.I(H)))
    assert fits(148, 32, 512) and fits(32, 32, 512) and not fits(31, 32, 512)     # 32 slices of 16 units
    assert fits(148, 5, 880) and not fits(100, 5, 880)                            # 110 slices of 8 units
    assert fits(1, 1, 16) and not fits(1, 300, 16)                                # one CTA, 32 tiles of 8 sequences at most
    for H in (64, 512, 800):
        assert [fits(s, 64, H) for s in range(1, 149)] == sorted(fits(s, 64, H) for s in range(1, 149))


@pytest.mark.parametrize("H", [4 * h for h in range(160, 187)])
def test_sixteen_units_a_cta_as_long_as_their_weights_fit(H):
    """Forward: 16 units and the exchange tile are 72 rows of H + 4 floats, and a buffer of partial sums beside them takes 16 KB.  Up to
    H = 744 that fits, and so 16 units it is where many sequences would otherwise wait for one another in a single group."""
    need = 4 * 72 * (H + 4) + (16 << 10)
    assert need <= BLOCK - 16
    got = int(L.lib().gb_lstm_seq_smem(L.I(256), L.I(H), L.I(0)))
    assert got in (need, need + (16 << 10))
    assert got == need + (16 << 10) or need + (16 << 10) > BLOCK - 16          # two buffers wherever there is room
