"""The FP8 Linear on a few rows, which the split GEMM quantises itself, against the row quantiser and the GEMM one after the other:
the same bits.  One row per group of eight, two, four and eight (the warps a row's maximum is shared by), nine (the general way);
K and N at the edges of k-steps and tiles, more values than the launch takes on (16384), strided rows."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9])
@pytest.mark.parametrize("K,N", [(16, 8), (144, 136), (3072, 18432), (15360, 72), (2064, 1000), (16384, 64), (2048, 64)])
@pytest.mark.parametrize("dtype,static", [(torch.bfloat16, False), (torch.float16, False), (torch.bfloat16, True)])
def test_linear_of_a_few_rows_is_quantiser_then_gemm(M, K, N, dtype, static):
    from ksanadit_b200 import _lib, ops
    from ksanadit_b200.linear import B200Fp8Linear
    g = torch.Generator(device="cuda").manual_seed(M * K + N)
    dense = torch.nn.Linear(K, N, device="cuda")
    lin = B200Fp8Linear.from_float(dense, dtype=dtype)
    if static:
        lin.scale_input = torch.nn.Parameter(torch.tensor(0.03, device="cuda"), requires_grad=False)
    x = torch.randn(M, 2 * K, device="cuda", generator=g, dtype=dtype)[:, :K]
    x[0, K // 2] = 300.0
    if M > 1:
        x[1] = 0.0
    xq, sx = lin.quantize_input(x)
    ref = ops.fp8_gemm(xq, sx, lin.weight.data, lin.weight_scale_vector(), lin.bias, out_dtype=dtype)
    out = lin(x)
    again = [lin(x) for _ in range(2)][-1]  # through the call in C++
    _lib.assert_device_ok()
    assert torch.equal(out, ref) and torch.equal(again, ref)
