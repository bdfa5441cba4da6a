"""SwiGLU at the edges of its two kernels: rows narrower than a CTA, pieces that end inside one, widths and bases off 16 bytes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,F,layout", [(1, 8, "plain"), (33, 8, "plain"), (4097, 8, "plain"), (1366, 24, "plain"), (17, 2056, "plain"),
                                            (3000, 12, "plain"), (3, 7, "plain"), (5000, 7, "plain"), (2100, 16, "pitch"), (600, 64, "offset"),
                                            (0, 64, "plain")])
def test_swiglu(dtype, rows, F, layout):
    from rumus_b200.ops import functional as Fn
    torch.manual_seed(rows + F)
    gu = torch.randn(rows, 2 * F, device="cuda").to(dtype)
    x = gu
    if layout == "pitch":
        x = torch.empty(rows, 2 * F + 16, device="cuda", dtype=dtype)[:, :2 * F].copy_(gu)
    elif layout == "offset":
        x = torch.empty(gu.numel() + 1, device="cuda", dtype=dtype)[1:].view_as(gu).copy_(gu)
    y = Fn.swiglu(x)
    g, u = gu.double().chunk(2, -1)
    ref = g * torch.sigmoid(g) * u
    assert y.shape == ref.shape and y.dtype == dtype
    # one rounding of the result; the sigmoid and the products in 32 bits (a few 2^-22)
    eps = {torch.bfloat16: 2 ** -8, torch.float16: 2 ** -11}.get(dtype, 2 ** -20)
    tiny = {torch.float16: 2 ** -24}.get(dtype, 0)      # halves below 2^-14 are multiples of it
    assert ((y.double() - ref).abs() <= eps * 1.01 * ref.abs() + tiny).all()
