"""A 1x1 convolution that hands its input on as the skip connection: values and gradients are those of the two operations."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# pixels below and above the row tiles of the GEMM kernels, channels at and beyond their column tiles
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,Cin,Cout,H", [(1, 8, 8, 3), (2, 64, 64, 17), (4, 256, 64, 24), (2, 72, 200, 31)])
def test_conv_skip_is_conv_and_skip(dtype, B, Cin, Cout, H):
    from rumus_b200.ops import vision as V
    torch.manual_seed(H)
    x = torch.randn(B, Cin, H, H, device="cuda").to(dtype).contiguous(memory_format=torch.channels_last).requires_grad_()
    w = (torch.randn(Cout, Cin, 1, 1, device="cuda") * 0.1).to(dtype).requires_grad_()
    gy, gs = torch.randn(B, Cout, H, H, device="cuda").to(dtype), torch.randn(B, Cin, H, H, device="cuda").to(dtype)
    y0 = V.conv2d(x, w)
    want = (y0,) + torch.autograd.grad((y0, x * 1), (x, w), (gy, gs))
    y1, skip = V.conv2d_skip(x, w)
    got = (y1,) + torch.autograd.grad((y1, skip), (x, w), (gy, gs))
    assert torch.equal(skip, x)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def test_a_block_whose_convolution_is_listened_to():
    from rumus_b200.models.resnet import Bottleneck
    torch.manual_seed(0)
    block = Bottleneck(64, 16, device="cuda", dtype=torch.float16)
    x = torch.randn(2, 64, 9, 9, device="cuda").half().contiguous(memory_format=torch.channels_last).requires_grad_()
    grads, seen = [], []
    for _ in range(2):
        y = block(x)
        grads.append(torch.autograd.grad(y, [x, *block.parameters()], torch.ones_like(y)))
        block.conv1.register_forward_hook(lambda m, a, out: seen.append(out.shape))
    assert seen == [(2, 16, 9, 9)]
    for a, b in zip(*grads):
        assert torch.equal(a, b)
