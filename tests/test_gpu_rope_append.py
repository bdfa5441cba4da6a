"""Rotation and cache append in one pass against the two rotations and the append that it replaces."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


# both layouts, block sizes that are no power of two, head sizes below, between and beyond a warp's pieces, shared key heads, rows of a wider buffer,
# tokens whose place is not theirs to write, and both sides of the count from which a token has one CTA
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("head_major", [False, True])
@pytest.mark.parametrize("T,H,Hkv,hd,bs,pad", [(1, 4, 4, 128, 16, 0), (5, 8, 2, 16, 16, 0), (147, 4, 1, 48, 12, 16), (148, 2, 2, 128, 16, 0),
                                               (300, 3, 3, 64, 5, 8), (33, 2, 1, 1024, 8, 0)])
def test_rope_append(dtype, head_major, T, H, Hkv, hd, bs, pad):
    from rumus_b200.serve import llama
    from rumus_b200.serve.cache import PagedKVCache
    torch.manual_seed(T + hd)
    cfg = SimpleNamespace(num_blocks=T // bs + 3, block_size=bs, kv_head_major=head_major, dtype=dtype, model=SimpleNamespace(num_layers=2))
    ours, theirs = (PagedKVCache(cfg, Hkv, hd, "cuda") for _ in range(2))
    for c in (ours, theirs):
        for t in c.k + c.v:
            t.fill_(7.0)
    width = (H + 2 * Hkv) * hd
    qkv = torch.randn(T, width + pad, device="cuda").to(dtype)[:, :width]
    pos = torch.randint(0, 5000, (T,), device="cuda")
    slots = torch.randperm(cfg.num_blocks * bs, device="cuda")[:T]
    slots[::7] = -1
    rest = qkv.clone()
    q, k, v = rest[:, :H * hd], rest[:, H * hd:(H + Hkv) * hd], rest[:, (H + Hkv) * hd:]
    llama._rope(q, pos, H, hd, 10000.0)
    llama._rope(k, pos, Hkv, hd, 10000.0)
    theirs.append(1, k, v, slots)
    ours.rope_append(1, qkv, H, pos, slots, 10000.0)
    # the same angles and the same two products a number; whether they are contracted is the compiler's choice: 2^-24 of each before the rounding
    eps = 2 ** -8 if dtype is torch.bfloat16 else 2 ** -11
    assert torch.equal(qkv[:, (H + Hkv) * hd:], v)
    assert ((qkv.double() - rest.double()).abs() <= 2 * eps * rest.double().abs() + 2 ** -20).all()
    for a, b in zip(ours.v, theirs.v):
        assert torch.equal(a, b)
    assert torch.equal(ours.k[0], theirs.k[0]) and ((ours.k[1].double() - theirs.k[1].double()).abs() <= 2 * eps * theirs.k[1].double().abs() + 2 ** -20).all()
    # what is stored is what stands in the rows
    blk, off = slots.clamp(min=0) // bs, slots.clamp(min=0) % bs
    stored = (ours.k[1][blk, :, off] if head_major else ours.k[1][blk, off])[slots >= 0]
    assert torch.equal(stored, qkv[:, H * hd:(H + Hkv) * hd].reshape(T, Hkv, hd)[slots >= 0])
