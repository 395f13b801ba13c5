"""Rules of the launchers about grids and the choice of a kernel (the products' are in ``test_gemm_plan``); no GPU needed."""

import pytest

from torchure_b200 import ops

_C = ops.ext()
pytestmark = pytest.mark.skipif(_C is None, reason="the CUDA extension is not built")


@pytest.mark.parametrize("Hq,Hkv", [(2, 1), (16, 4), (16, 8), (32, 8), (6, 3)])
@pytest.mark.parametrize("acc", [True, False])
def test_qknorm_backward_leaves_room_for_communication(Hq, Hkv, acc):
    """All CTAs of the persistent QK-norm backward are resident at once where communication CTAs, which take half of an SM's
    register file, are on some SMs: such an SM has room for one.  Without them the grid fills the chip."""
    for sms, shared in ((148, 0), (148, 16), (148, 148), (132, 16), (148, 500)):
        cols, chunks, per_sm = _C.qknorm_rope_bwd_grid(8192, Hq, Hkv, acc, sms, shared)
        room = sms * per_sm - min(shared, sms) * (per_sm - 1)
        assert room - chunks < cols * chunks <= room and 2 <= per_sm <= 3
    assert _C.qknorm_rope_bwd_grid(9, Hq, Hkv, acc, 148, 16)[0] == 2          # eight rows per CTA
    assert _C.qknorm_rope_bwd_grid(8192, 512, 64, acc, 8, 8)[0] == 1


def test_attention_backward_counts_the_sms_it_has():
    """Which kernel takes an attention backward, and how many CTAs share a key block, on all SMs of a B200 (the measured
    choices) and on those that are left beside reserved ones: clusters that share a key block run at once."""
    taken = [(2, 4096, 16, 8), (1, 16384, 16, 8), (1, 2048, 16, 8), (8, 512, 16, 8), (8, 256, 16, 8), (8, 640, 16, 8)]
    left = [(1, 1024, 16, 8), (1, 4096, 8, 2), (8, 384, 16, 8), (2, 512, 16, 8)]
    pairs = lambda c, sms: _C.attn_bwd_on_pairs(c[0], c[1], c[1], c[2], c[3], True, sms)
    assert all(pairs(c, 148) for c in taken) and not any(pairs(c, 148) for c in left)
    assert not pairs((8, 256, 16, 8), 100)              # 64 pairs no longer fit at once
    assert pairs((1, 1024, 16, 8), 100)                 # nor do 64 clusters of two
    for sms in (148, 132, 100, 64):
        for tiles in range(1, 160):
            parts = _C.attn_bwd_parts(tiles, 40, sms)
            assert parts in (1, 2, 4) and (parts == 1 or tiles * parts <= sms)
    assert [_C.attn_bwd_parts(t, 40, 148) for t in (32, 33, 74, 75)] == [4, 2, 2, 1]
