"""FlashAttention forward at the edges of its tiles and arguments, against the same operation in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one key tile, an odd and an even number of them (the two warpgroups take them in turn), ragged ends, fewer query than key rows and the
# other way round (rows that see no key give zeros), shared key heads, scales that are negative or zero
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Sq,Sk,H,Hkv,causal,scale", [(1, 1, 2, 2, True, 0.1), (128, 128, 2, 1, True, 0.1), (129, 129, 2, 2, True, 0.1),
                                                       (100, 300, 2, 2, True, 0.1), (300, 130, 2, 2, True, 0.1), (260, 384, 4, 2, False, 0.1),
                                                       (300, 300, 2, 2, True, -0.1), (130, 257, 2, 2, True, 0.0), (520, 513, 1, 1, False, -0.1)])
def test_flash_forward_edges(D, Sq, Sk, H, Hkv, causal, scale):
    from rumus_b200.ops import native
    from rumus_b200.ops.attention import fa_forward
    torch.manual_seed(Sq + Sk)
    q, k, v = (torch.randn(2, S, h, D, device="cuda").bfloat16() for S, h in ((Sq, H), (Sk, Hkv), (Sk, Hkv)))
    o, lse, _ = fa_forward(q, k, v, causal, scale)
    kd, vd = (t.double().repeat_interleave(H // Hkv, 2) for t in (k, v))
    s = torch.einsum("bihd,bjhd->bhij", q.double(), kd) * scale
    if causal:
        s = s.masked_fill(~torch.ones(Sq, Sk, dtype=torch.bool, device="cuda").tril(Sk - Sq), float("-inf"))
    ref = torch.einsum("bhij,bjhd->bihd", s.softmax(-1).nan_to_num(0.0), vd)
    # weights and results are rounded to 8 bits: 2^-9 of each on average, the weights' part smaller by averaging
    assert ((o.double() - ref).norm() / ref.norm()).item() < 2 ** -8
    want = torch.logsumexp(s, -1)
    seen = torch.isfinite(want)
    assert torch.equal(torch.isfinite(lse), seen) and (lse.double() - want)[seen].abs().max() < 1e-4
    assert native.read_status() == 0


# rows that see no key of a tile (Sk - Sq no multiple of 128), and scores that range beyond what 16 bits hold of exp2
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("Sq,Sk,causal,scale", [(100, 300, True, -0.1), (130, 257, True, -0.1), (300, 130, True, -0.1), (1, 129, True, -0.1),
                                                 (200, 384, False, -2.0), (260, 384, True, -2.0), (260, 384, True, 2.0), (100, 300, True, 2.0)])
def test_flash_forward_negative_scales(D, dtype, Sq, Sk, causal, scale):
    from rumus_b200.ops import native
    from rumus_b200.ops.attention import fa_forward
    torch.manual_seed(Sq + Sk)
    q, k, v = (torch.randn(2, S, 2, D, device="cuda").to(dtype) for S in (Sq, Sk, Sk))
    o, lse, _ = fa_forward(q, k, v, causal, scale)
    s = torch.einsum("bihd,bjhd->bhij", q.double(), k.double()) * scale
    if causal:
        s = s.masked_fill(~torch.ones(Sq, Sk, dtype=torch.bool, device="cuda").tril(Sk - Sq), float("-inf"))
    ref = torch.einsum("bhij,bjhd->bihd", s.softmax(-1).nan_to_num(0.0), v.double())
    # weights and results rounded to 8 (11) bits; the scores' own rounding, 2^-24 of up to 2 * 128 each way, is below that
    assert torch.isfinite(o).all() and ((o.double() - ref).norm() / ref.norm()).item() < 2 ** -8
    want = torch.logsumexp(s, -1)
    seen = torch.isfinite(want)
    assert torch.equal(torch.isfinite(lse), seen) and not torch.isnan(lse).any()
    assert (lse.double() - want)[seen].abs().max() < 1e-4 * max(1.0, want[seen].abs().max().item() / 10)
    assert native.read_status() == 0
