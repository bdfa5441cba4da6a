"""The register-fed INT4 kernel (``csrc/kernels/int4_rows.cu``) against the 64-bit product with the dequantised weight."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(M, K, N, dtype, scale_dtype, seed, group=128):
    from rumus_b200.nn.quant import QuantizedTensor
    torch.manual_seed(seed)
    q = QuantizedTensor.from_f32(torch.randn(K, N) * 0.05 + 0.01, group, scale_dtype).to("cuda")
    return (torch.randn(M, K, device="cuda") + 0.2).to(dtype), q


def _rel(y, ref):
    return ((y.double() - ref).norm() / ref.norm()).item()


# edges: one row to a full launch, every row bucket; K that is no multiple of a group, one step, more steps than warps;
# N below, at and beyond a tile; slices of a cluster that differ in length
@pytest.mark.parametrize("M", [1, 8, 9, 17, 25, 33, 47, 48])
@pytest.mark.parametrize("K,N,split", [(1000, 264, 0), (128, 4, 0), (4096, 132, 0), (2944, 516, 5), (11008, 384, 8), (11008, 128, 1)])
def test_int4_rows(M, K, N, split):
    from rumus_b200.ops import quant_cuda as Q
    x, q = _case(M, K, N, torch.bfloat16, torch.float16, M + K)
    ref = x.double() @ q.dequantize(torch.float32).double()
    y = Q.int4_matmul_rows(x, q, split=split)
    # the result is rounded once to the 8 bits of bfloat16, which moves each value by at most 2^-8 of it (half of the 2^-7
    # between neighbours at 1); the fp32 sums' own error is below 1e-5.  Above eight rows the weights are rounded too: scale,
    # offset and weight by at most 2^-8 each, independently from weight to weight
    assert _rel(y, ref) < (2 ** -8 if M <= 8 else 2 ** -7)
    assert torch.equal(y, Q.int4_matmul_rows(x, q, split=split))


@pytest.mark.parametrize("dtype,scale_dtype", [(torch.float16, torch.float16), (torch.float16, torch.float32), (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("M,group", [(3, 128), (16, 256), (40, 128)])
def test_int4_rows_types_bias_residual(dtype, scale_dtype, M, group):
    from rumus_b200.ops import quant_cuda as Q
    x, q = _case(M, 1160, 300, dtype, scale_dtype, M, group)
    bias, res = torch.randn(300, device="cuda").to(dtype), torch.randn(M, 300, device="cuda").to(dtype)
    ref = x.double() @ q.dequantize(torch.float32).double() + bias.double() + res.double()
    y = Q.int4_matmul(x, q, bias, residual=res)
    assert _rel(y, ref) < (2 ** -8 if dtype is torch.bfloat16 else 2 ** -11) * (1 if M <= 8 else 2)
    out = torch.empty_like(y)
    assert Q.int4_matmul(x, q, bias, out=out, residual=res) is out and torch.equal(out, y)
    # above the kernel's rows: the same sum by the dense product
    big = torch.cat([x] * (80 // M + 1))
    y2 = Q.int4_matmul(big, q, bias, residual=torch.cat([res] * (80 // M + 1)))
    assert _rel(y2[:M], ref) < 1e-2


def test_int4_rows_not_covered_shapes_take_the_other_kernels():
    from rumus_b200.ops import quant_cuda as Q
    for group, N, K in ((64, 264, 1024), (128, 266, 1024), (128, 264, 1004)):
        x, q = _case(5, K, N, torch.bfloat16, torch.float16, 0, group)
        assert Q.int4_matmul_rows(x, q) is None
        assert _rel(Q.int4_matmul(x, q), x.double() @ q.dequantize(torch.float32).double()) < 1e-2


def test_int4_rows_infinite_activations():
    """An infinity reaches the sums with the weight's sign, as in a product with the dequantised weight."""
    from rumus_b200.ops import quant_cuda as Q
    x, q = _case(5, 512, 64, torch.bfloat16, torch.float16, 3)
    x[1, 70], x[3, 300], x[4, 2] = float("inf"), float("-inf"), float("nan")
    ref = (x.double() @ q.dequantize(torch.float32).double()).bfloat16()
    y = Q.int4_matmul_rows(x, q)
    assert torch.equal(torch.isnan(y), torch.isnan(ref)) and torch.equal(y[torch.isinf(ref)], ref[torch.isinf(ref)])
    assert _rel(y[[0, 2]], ref[[0, 2]].double()) < 2 ** -8


@pytest.mark.parametrize("M,dense", [(8, False), (9, True), (48, True)])
def test_int4_dense_weights_on_request(M, dense, monkeypatch):
    """RB_W4A16=0: more than eight rows are multiplied with the weights of a dense copy, rounded once."""
    from rumus_b200.ops import native, quant_cuda as Q
    monkeypatch.setenv("RB_W4A16", "0")
    x, q = _case(M, 1024, 264, torch.bfloat16, torch.float32, M)
    res = torch.randn(M, 264, device="cuda").bfloat16()
    want = native.gemm(x, Q.int4_dequant(q, x.dtype))
    assert torch.equal(Q.int4_matmul(x, q), want) is dense
    assert _rel(Q.int4_matmul(x, q, residual=res), want.double() + res.double()) < 2 ** -7
