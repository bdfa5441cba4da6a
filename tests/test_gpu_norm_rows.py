"""Norms of rows at the edges of what a CTA keeps in registers, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("D", [1288, 2048, 4096, 8192, 8200])
def test_rms_norm_wide_rows(dtype, D):
    from rumus_b200.ops import functional as F
    torch.manual_seed(D)
    x, w = torch.randn(5, D, device="cuda").to(dtype), torch.randn(D, device="cuda").to(dtype)
    r = torch.randn(5, D, device="cuda").to(dtype)
    h = (x.float() + r.float()).to(dtype)
    y, hh = F.rms_norm(x, w, 1e-6, residual=r)
    assert torch.equal(h, hh)
    for got, v in ((F.rms_norm(x, w, 1e-6), x), (y, h)):
        ref = v.double() * torch.rsqrt(v.double().pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
        # one rounding of the result, and of the sum and root in 32 bits
        assert ((got.double() - ref).norm() / ref.norm()).item() < {torch.bfloat16: 2 ** -8, torch.float16: 2 ** -11}.get(dtype, 1e-6)


# rows of one vector a thread: a CTA each up to 2048 (1024 in 32 bits), a warp each beyond
@pytest.mark.parametrize("dtype,D", [(torch.bfloat16, 1288), (torch.float16, 2048), (torch.float32, 1024)])
@pytest.mark.parametrize("rows", [1, 1024, 1025, 2048, 2049, 3001])
def test_rms_norm_many_rows(dtype, D, rows):
    from rumus_b200.ops import functional as F
    torch.manual_seed(rows)
    x, w = torch.randn(rows, D, device="cuda").to(dtype), torch.randn(D, device="cuda").to(dtype)
    y = F.rms_norm(x, w, 1e-6)
    ref = x.double() * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    assert ((y.double() - ref).norm() / ref.norm()).item() < {torch.bfloat16: 2 ** -8, torch.float16: 2 ** -11}.get(dtype, 1e-6)
