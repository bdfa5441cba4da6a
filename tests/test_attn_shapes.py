"""Which shapes the attention kernels are given: their index arithmetic takes k's and v's sizes from q, so any other shape has to be
turned away before the launch."""
import pytest


@pytest.mark.parametrize("q,k,v,causal,covered", [
    ((4, 8, 2, 32), (4, 8, 2, 32), (4, 8, 2, 32), True, True),
    ((4, 8, 2, 32), (4, 20, 2, 32), (4, 20, 2, 32), True, True),
    ((4, 8, 2, 32), (1, 8, 2, 32), (1, 8, 2, 32), True, False),        # k's batch: read, and dK written, beyond its end
    ((1, 8, 2, 32), (4, 8, 2, 32), (4, 8, 2, 32), True, False),
    ((4, 8, 2, 32), (4, 8, 2, 16), (4, 8, 2, 16), True, False),        # its head size
    ((4, 8, 2, 32), (4, 8, 1, 32), (4, 8, 1, 32), True, False),        # shared key heads
    ((4, 8, 2, 32), (4, 8, 2, 32), (4, 9, 2, 32), True, False),
    ((4, 8, 2, 32), (4, 8, 2, 32), (4, 8, 2, 16), True, False),
    ((4, 8, 2, 24), (4, 8, 2, 24), (4, 8, 2, 24), True, False),
    ((4, 8, 2, 32), (4, 7, 2, 32), (4, 7, 2, 32), True, False),        # a row without keys
    ((4, 8, 2, 32), (4, 7, 2, 32), (4, 7, 2, 32), False, True),
    ((8, 2, 32), (8, 2, 32), (8, 2, 32), True, False),
])
def test_32_bit_heads(q, k, v, causal, covered):
    from rumus_b200.ops.attention import f32_covers
    assert f32_covers(q, k, v, causal) is covered
