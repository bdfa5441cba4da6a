"""Which shapes the attention kernels are given: their index arithmetic takes k's and v's sizes from q, so any other shape has to be
turned away before the launch."""
import pytest
import torch


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
    ((65535, 2, 2, 16), (65535, 2, 2, 16), (65535, 2, 2, 16), True, True),
    ((65536, 2, 2, 16), (65536, 2, 2, 16), (65536, 2, 2, 16), True, False),
    ((1, 2, 65536, 16), (1, 2, 65536, 16), (1, 2, 65536, 16), True, False),
])
def test_32_bit_heads(q, k, v, causal, covered):
    from rumus_b200.ops.attention import f32_covers
    assert f32_covers(q, k, v, causal) is covered


@pytest.mark.parametrize("heads,kv_heads,hd,dtype", [
    (4, 2, 32, torch.float32),          # key heads h >= kv_heads lie beyond the rows
    (4, 4, 24, torch.float32),
    (2, 2, 64, torch.bfloat16),         # forward only
])
def test_packed_heads_that_no_kernel_takes(heads, kv_heads, hd, dtype):
    from rumus_b200.ops import functional as F
    with pytest.raises(ValueError):
        F.flash_attention_packed(torch.zeros(2, 8, (heads + 2 * kv_heads) * hd, dtype=dtype), heads, kv_heads, True)


def test_32_bit_forward_turns_other_shapes_away():
    from rumus_b200.ops.attention import attention_f32
    q, k = torch.zeros(4, 8, 2, 32), torch.zeros(1, 8, 2, 32)
    with pytest.raises(ValueError):
        attention_f32(q, k, k, True)


@pytest.mark.parametrize("q,k,v,types", [
    ((2, 8, 4, 64), (1, 8, 4, 64), (1, 8, 4, 64), "bbb"),              # k's batch
    ((2, 8, 4, 64), (2, 8, 4, 128), (2, 8, 4, 128), "bbb"),            # its head size
    ((2, 8, 4, 64), (2, 9, 4, 64), (2, 8, 4, 64), "bbb"),
    ((2, 8, 4, 64), (2, 8, 3, 64), (2, 8, 3, 64), "bbb"),              # heads that cannot be shared evenly
    ((2, 8, 4, 64), (2, 8, 0, 64), (2, 8, 0, 64), "bbb"),
    ((2, 8, 4, 64), (2, 8, 4, 64), (2, 8, 4, 64), "bhb"),
])
def test_16_bit_forward_turns_other_shapes_away(q, k, v, types):
    from rumus_b200.ops.attention import fa_forward
    dt = {"b": torch.bfloat16, "h": torch.float16}
    with pytest.raises(ValueError):
        fa_forward(*(torch.zeros(s, dtype=dt[t]) for s, t in zip((q, k, v), types)), True, 0.1)


@pytest.mark.parametrize("Sq,Sk,D,causal,rows", [
    (1024, 1024, 128, True, 1024), (1024, 1024, 32, False, 1024), (1024, 1024, 64, False, 768), (256, 256, 128, False, 192),
    (16, 512, 64, True, 384), (16, 512, 16, False, 384), (64, 256, 128, True, 192),
])
def test_32_bit_rows_go_to_the_quicker_kernels(Sq, Sk, D, causal, rows):
    from rumus_b200.ops.attention import f32_max_rows
    assert f32_max_rows(Sq, Sk, D, causal) == rows
