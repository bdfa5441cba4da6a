"""16-bit pools, eight channels a thread (``csrc/kernels/vision.cu``), against PyTorch in 64 bits: values, argmax and gradients."""
import pytest
import torch
import torch.nn.functional as TF

pytestmark = pytest.mark.gpu
EPS = {torch.bfloat16: 2 ** -8, torch.float16: 2 ** -11}


def _input(dtype, shape, layout):
    x = torch.randn(shape, device="cuda").to(dtype)
    return (x.contiguous(memory_format=torch.channels_last) if layout == "last" else x).requires_grad_()


# windows with loads unrolled (2, 3) and of any size, strides beyond and below the window, rows that no window covers, windows over the edge;
# 12 channels: the kernel of one channel a thread
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("C,layout", [(8, "last"), (24, "first"), (12, "last")])
@pytest.mark.parametrize("k,stride,pad", [(3, 2, 1), (2, 2, 0), (3, 1, 1), (5, 3, 2), (2, 3, 0), (7, 7, 0), (4, 3, 1), (1, 2, 0)])
def test_max_pool(dtype, C, layout, k, stride, pad):
    from rumus_b200.ops import vision as V
    torch.manual_seed(k + C)
    x = _input(dtype, (2, C, 13, 16), layout)
    y = V.max_pool2d(x, k, stride, pad)
    g = torch.randn_like(y)
    dx, = torch.autograd.grad(y, x, g)
    xd = x.detach().double().requires_grad_()
    yd = TF.max_pool2d(xd, k, stride, pad)
    dd, = torch.autograd.grad(yd, xd, g.double())
    assert torch.equal(y.double(), yd)
    # sums of up to k * k 16-bit gradients in 32 bits, rounded once; of equal maxima the first has the gradient on both sides
    assert ((dx.double() - dd).abs() <= EPS[dtype] * dd.abs() + 2 ** -20 * k * k).all()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("k", [2, 3, 4])
def test_max_pool_of_extremes(dtype, k):
    """Infinities, the type's lowest value, and NaN (which a comparison never replaces and never takes over) as one channel a thread has them."""
    from rumus_b200.ops import vision as V
    torch.manual_seed(k)
    x = torch.randn(2, 8, 12, 12, device="cuda").to(dtype)
    pick = torch.randint(0, 8, x.shape, device="cuda")
    for code, v in enumerate((float("inf"), float("-inf"), torch.finfo(dtype).min, float("nan"))):
        x[pick == code] = v
    x[0, 0] = float("-inf")
    x = x.contiguous(memory_format=torch.channels_last)
    wide, ref = V.max_pool2d(x, k, k), V.max_pool2d(x[:, :7].contiguous(memory_format=torch.channels_last), k, k)
    assert torch.equal(wide[:, :7].isnan(), ref.isnan()) and torch.equal(wide[:, :7].nan_to_num(7.0), ref.nan_to_num(7.0))


# one bin, bins that overlap, more bins than pixels, windows longer than what is in flight
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("C,layout", [(8, "last"), (24, "first"), (12, "last")])
@pytest.mark.parametrize("H,W,out", [(7, 7, (1, 1)), (7, 7, (3, 2)), (13, 9, (5, 4)), (3, 5, (6, 7)), (40, 33, (1, 2)), (1, 1, (1, 1)), (17, 1, (1, 1))])
def test_adaptive_avg_pool(dtype, C, layout, H, W, out):
    from rumus_b200.ops import vision as V
    torch.manual_seed(H + C)
    x = _input(dtype, (2, C, H, W), layout)
    y = V.adaptive_avg_pool2d(x, out)
    g = torch.randn_like(y)
    dx, = torch.autograd.grad(y, x, g)
    xd = x.detach().double().requires_grad_()
    yd = TF.adaptive_avg_pool2d(xd, out)
    dd, = torch.autograd.grad(yd, xd, g.double())
    # one rounding of the result; sums of up to H * W numbers in 32 bits
    for a, b in ((y, yd), (dx, dd)):
        assert ((a.double() - b).abs() <= EPS[dtype] * b.abs() + 2 ** -22 * H * W).all()
