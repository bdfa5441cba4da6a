"""Column sums at the edges of what is in flight: rows of a slab, what is left of it, more slabs than one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows", [0, 1, 7, 8, 9, 15, 16, 17, 23, 24, 31, 63, 64, 65, 129, 1555, 33001])
@pytest.mark.parametrize("N,pitch", [(64, 64), (1032, 1040), (12, 13)])
def test_colsum(dtype, rows, N, pitch):
    from rumus_b200.ops import native
    torch.manual_seed(rows + N)
    x = torch.randn(rows, pitch, device="cuda").to(dtype)[:, :N]
    out = torch.full((N + 1,), 7.0, dtype=dtype, device="cuda")
    for got in (native.colsum(x), native.colsum(x, out=out[:N])):
        ref = x.double().sum(0)
        # every addition in 32 bits errs by at most 2^-24 of its sum, which is at most the sum of the sizes, and the longest chain of additions
        # is a slab's rows, an eighth of the slabs and the eight parts of those; then one rounding of the result
        slabs = max(1, min(512, (rows + 63) // 64))
        chain = (rows + slabs - 1) // slabs + (slabs + 7) // 8 + 8
        eps = {torch.bfloat16: 2 ** -8, torch.float16: 2 ** -11}.get(dtype, 2 ** -24)
        assert ((got.double() - ref).abs() <= eps * ref.abs() + chain * 2 ** -24 * x.double().abs().sum(0)).all()
    assert out[N] == 7
