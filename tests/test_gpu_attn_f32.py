"""32-bit attention kernels (``csrc/kernels/attn_f32.cu``) against the same operation in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(q, k, v, causal, scale):
    s = torch.einsum("bihd,bjhd->bhij", q, k) * scale
    if causal:
        see = torch.ones(q.shape[1], k.shape[1], dtype=torch.bool, device=q.device).tril(k.shape[1] - q.shape[1])
        s = s.masked_fill(~see, float("-inf"))
    return torch.einsum("bhij,bjhd->bihd", s.softmax(-1), v)


# tile and block edges: 32 keys a tile, 128 / (D / 16) rows a block; one row; more keys than rows
@pytest.mark.parametrize("D", [16, 32, 64, 128])
@pytest.mark.parametrize("B,H,Sq,Sk,causal", [(2, 3, 64, 64, True), (1, 2, 1, 1, True), (1, 2, 33, 33, False), (2, 1, 17, 80, True),
                                               (1, 2, 130, 97, False), (1, 1, 257, 257, True)])
def test_attention_f32(D, B, H, Sq, Sk, causal):
    from rumus_b200.ops import functional as F
    from rumus_b200.ops.attention import f32_covered
    torch.manual_seed(D + Sq)
    q, k, v = (torch.randn(B, S, H, D, device="cuda", requires_grad=True) for S in (Sq, Sk, Sk))
    g = torch.randn(B, Sq, H, D, device="cuda")
    assert f32_covered(q, k, v, causal)
    o = F.flash_attention(q, k, v, causal)
    got = (o,) + torch.autograd.grad(o, (q, k, v), g)
    qd, kd, vd = (t.detach().double().requires_grad_() for t in (q, k, v))
    od = _ref(qd, kd, vd, causal, D ** -0.5)
    want = (od,) + torch.autograd.grad(od, (qd, kd, vd), g.double())
    for a, b in zip(got, want):
        # sums of up to 257 products of 32-bit numbers, 2^-24 each, times what cancels in dP - delta (up to some tens); with one key the
        # gradients of q and k are nothing but that cancellation
        assert (a.double() - b).norm() < 1e-5 * b.norm() + 1e-5 * (Sk == 1) * g.norm()


def test_attention_f32_packed_is_the_same_and_the_rest_is_composed():
    from rumus_b200.ops import functional as F
    from rumus_b200.ops.attention import f32_covered
    torch.manual_seed(0)
    B, S, H, D = 2, 40, 4, 32
    qkv = torch.randn(B, S, 3 * H * D, device="cuda", requires_grad=True)
    g = torch.randn(B, S, H, D, device="cuda")
    packed = F.flash_attention_packed(qkv, H, H, True)
    split = F.flash_attention(*(t.view(B, S, H, D) for t in qkv.split(H * D, -1)), True)
    assert torch.equal(packed, split)
    assert torch.equal(torch.autograd.grad(packed, qkv, g)[0], torch.autograd.grad(split, qkv, g)[0])
    q, k, v = (torch.randn(1, S, H, 24, device="cuda") for _ in range(3))
    assert not f32_covered(q, k, v, True)
    ref = _ref(q.double(), k.double(), v.double(), True, 24 ** -0.5)
    assert ((F.flash_attention(q, k, v, True).double() - ref).norm() / ref.norm()).item() < 1e-5


@pytest.mark.parametrize("layout", ["four bytes on", "batch second"])
def test_packed_rows_of_other_layouts(layout):
    from rumus_b200.ops import functional as F
    torch.manual_seed(1)
    B, S, H, D = 2, 33, 2, 32
    rows = torch.randn(B, S, 3 * H * D, device="cuda")
    if layout == "batch second":
        qkv = rows.transpose(0, 1).contiguous().transpose(0, 1)
    else:
        qkv = torch.empty(rows.numel() + 1, device="cuda")[1:].view_as(rows).copy_(rows)
    g = torch.randn(B, S, H, D, device="cuda")
    got, want = [], []
    for t, out in ((qkv, got), (rows, want)):
        t.requires_grad_()
        o = F.flash_attention_packed(t, H, H, True)
        out += [o, torch.autograd.grad(o, t, g)[0]]
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("D", [16, 128])
def test_numbers_that_are_none(D, causal):
    """NaN and infinite scores reach the result where a softmax in 64 bits has them, also as the first keys of a row."""
    from rumus_b200.ops.attention import attention_f32
    torch.manual_seed(D)
    q, k, v = (torch.randn(2, 40, 2, D, device="cuda") for _ in range(3))
    k[0, :4, 0] = float("nan")              # one group of keys, the first
    k[0, 9, 1, 0] = float("inf")            # scores of +inf and -inf
    k[1, 33, 0, 1] = float("nan")
    v[1, 2, 1, 3] = float("inf")
    o = attention_f32(q, k, v, causal)
    ref = _ref(q.double(), k.double(), v.double(), causal, D ** -0.5)
    some = torch.isfinite(ref)
    assert torch.equal(torch.isnan(o[0, :, 0]), torch.isnan(ref[0, :, 0])) and torch.isnan(o[0, :, 0]).all()
    assert torch.equal(torch.isfinite(o)[0], some[0]) and torch.equal(torch.isfinite(o)[1, :, 0], some[1, :, 0])
    seen = torch.arange(40, device="cuda") >= 2 if causal else torch.ones(40, dtype=torch.bool, device="cuda")
    assert torch.isinf(o[1, seen, 1, 3]).all()
    assert ((o - ref)[some & torch.isfinite(o)].norm() / ref[some].norm()).item() < 1e-5
