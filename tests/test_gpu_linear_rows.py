"""The FP8 Linear on a few rows, which the split GEMM quantises itself, against the row quantiser and the GEMM one after the other:
the same bits.  One row per group of eight, two, four and eight (the warps a row's maximum is shared by), nine (the general way);
K and N at the edges of k-steps and tiles, as many values as the launch takes on (10240, 6144 over a large weight) and more,
strided rows."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 8, 9])
@pytest.mark.parametrize("K,N", [(16, 8), (144, 136), (3072, 18432), (15360, 72), (2064, 1000), (16384, 64), (2048, 64)])
@pytest.mark.parametrize("dtype,static", [(torch.bfloat16, False), (torch.float16, False), (torch.bfloat16, True), (torch.float16, True)])
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
    assert lin._call.host and lin._call.host.run(lin, x, _lib.EPI_NONE) is not None
    _lib.assert_device_ok()
    assert torch.equal(out, ref) and torch.equal(again, ref)


@pytest.mark.parametrize("writer", ["rowwise kernel", "set_weight"])
@pytest.mark.parametrize("M,K,N", [(1, 3072, 18432), (1, 1536, 1536), (3, 3072, 3072)])
def test_weight_written_by_the_kernel_ahead_of_the_call(writer, M, K, N):
    """The one-launch form is the call's first kernel and may start while the kernel ahead, here the one that writes the weight,
    drains (the row quantiser releases its successor before it has written anything): it has to read the new weight."""
    from ksanadit_b200 import _lib, ops
    from ksanadit_b200.linear import B200Fp8Linear
    g = torch.Generator(device="cuda").manual_seed(N)
    lin = B200Fp8Linear.from_float(torch.nn.Linear(K, N, bias=False, device="cuda"))
    x = torch.randn(M, K, device="cuda", generator=g, dtype=torch.bfloat16)
    dense = [torch.randn(N, K, device="cuda", generator=g, dtype=torch.bfloat16) * 0.02 * (i + 1) for i in range(3)]
    scales = lin.weight_scale_vector()

    def write(w):
        if writer == "set_weight":
            lin.set_weight(w, inplace_update=True)
        else:
            ops.quant_fp8_rowwise(w, out=(lin.weight.data, scales))

    refs = []
    for w in dense:
        write(w)
        torch.cuda.synchronize()
        refs.append(lin(x))
        torch.cuda.synchronize()
    n = ops.STATS.kernels
    lin(x)
    assert ops.STATS.kernels - n == 1
    outs = []
    for i in range(60):
        write(dense[i % 3])
        outs.append(lin(x))
    _lib.assert_device_ok()
    assert all(torch.equal(o, refs[i % 3]) for i, o in enumerate(outs))
    assert not torch.equal(refs[0], refs[1])


@pytest.mark.parametrize("M,K,shift", [(1, 1536, 0), (4, 1536, 0), (3, 3072, 0), (4, 1536, 1536), (2, 1536, -1536), (8, 1024, 8), (9, 1536, 0)])
@pytest.mark.parametrize("static", [False, True])
def test_output_over_the_input(M, K, shift, static):
    """The C interface takes an `out` that overlaps x (``shift``: by how many elements it lies behind it): two launches, since a CTA of
    the one-launch form may store while another still quantises.  Next to x, not over it, one launch."""
    import ctypes

    from ksanadit_b200 import _lib, native
    from ksanadit_b200.linear import B200Fp8Linear
    lin = B200Fp8Linear.from_float(torch.nn.Linear(K, K, device="cuda"))
    desc = native.Watch().linear_of(lin, torch.bfloat16)
    lib = _lib.load()
    scale = torch.full((1,), 0.03, device="cuda")
    ws = native.workspace(lib.ksb_linear_workspace(M, K), torch.device("cuda"))

    def run(buf, x0, o0):
        return lib.ksb_linear_forward(ctypes.addressof(desc), buf[x0:].data_ptr(), _lib.BF16, M, K, static, scale.data_ptr() if static else None,
                                      buf[o0:].data_ptr(), _lib.EPI_NONE, None, 0, None, 0, ws.data_ptr(), native.stream())

    n = M * K
    data = torch.randn(n, device="cuda", dtype=torch.bfloat16)
    far = torch.cat([data, torch.zeros_like(data)])
    assert run(far, 0, n) == (1 if M <= 8 else 2)
    ref = far[n:].clone()
    for _ in range(20):
        buf = torch.zeros(3 * n, device="cuda", dtype=torch.bfloat16)
        buf[n:2 * n] = data
        assert run(buf, n, n + shift) == 2
        assert torch.equal(buf[n + shift:2 * n + shift], ref)
    _lib.assert_device_ok()


# kernels queued: one up to eight rows of 10240 values, of 6144 over a weight above 48 MiB; two beyond
@pytest.mark.parametrize("M,K,N,kernels", [(1, 16, 8, 1), (8, 144, 136, 1), (9, 144, 136, 2), (8, 1280, 200, 1), (8, 1296, 200, 2), (1, 10240, 64, 1),
                                           (1, 10256, 64, 2), (2, 3072, 18432, 1), (3, 3072, 18432, 2)])
@pytest.mark.parametrize("epilogue", ["none", "gelu", "gate", "gate rows"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_epilogues_of_both_forms(M, K, N, kernels, epilogue, dtype):
    from ksanadit_b200 import _lib, ops
    from ksanadit_b200.linear import B200Fp8Linear
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    lin = B200Fp8Linear.from_float(torch.nn.Linear(K, N, device="cuda"), dtype=dtype)
    x = torch.randn(M, K, device="cuda", generator=g, dtype=dtype)
    kw = dict(epilogue={"none": _lib.EPI_NONE, "gelu": _lib.EPI_GELU_TANH}.get(epilogue, _lib.EPI_GATE_RESIDUAL))
    if epilogue.startswith("gate"):
        kw["resid"] = torch.randn(M, N, device="cuda", generator=g, dtype=dtype)
        kw["gate"] = torch.randn(M if epilogue == "gate rows" else 1, N, device="cuda", generator=g, dtype=dtype)
    xq, sx = ops.quant_fp8_rowwise(x)
    ref = ops.fp8_gemm(xq, sx, lin.weight.data, lin.weight_scale_vector(), lin.bias, out_dtype=dtype, **kw)
    for _ in range(3):
        n = ops.STATS.kernels
        assert torch.equal(lin(x, **kw), ref)
        assert ops.STATS.kernels - n == kernels
    _lib.assert_device_ok()


@pytest.mark.parametrize("M", [1, 2, 4, 8])
@pytest.mark.parametrize("dtype,static", [(torch.bfloat16, False), (torch.float16, False), (torch.bfloat16, True), (torch.float16, True)])
def test_rows_without_a_finite_maximum(M, dtype, static):
    """Infinities, NaN, the type's largest and smallest values, zeros of either sign: the row quantisers' bytes and scales."""
    from ksanadit_b200 import _lib, ops
    from ksanadit_b200.linear import B200Fp8Linear
    info = torch.finfo(dtype)
    lin = B200Fp8Linear.from_float(torch.nn.Linear(1024, 136, device="cuda"), dtype=dtype)
    if static:
        lin.scale_input = torch.nn.Parameter(torch.tensor(0.03, device="cuda"), requires_grad=False)
    plain = torch.randn(1024, device="cuda", dtype=dtype)
    special = [float("inf"), float("-inf"), float("nan"), info.max, info.min, info.smallest_normal, info.smallest_normal / 4, -0.0]
    for fill in (False, True):  # one such value in a row, or nothing else
        rows = []
        for i, v in enumerate(special):
            row = torch.full_like(plain, v) if fill else plain.clone()
            row[129 * i % 1024] = v
            rows.append(row)
        for i in range(0, len(rows), M):
            x = torch.stack(rows[i:i + M])
            xq, sx = lin.quantize_input(x)
            ref = ops.fp8_gemm(xq, sx, lin.weight.data, lin.weight_scale_vector(), lin.bias, out_dtype=dtype)
            n = ops.STATS.kernels
            out = lin(x)
            assert ops.STATS.kernels - n == 1
            assert torch.equal(out.isnan(), ref.isnan()) and torch.equal(out.nan_to_num(), ref.nan_to_num()), (fill, special[i:i + M])
    _lib.assert_device_ok()
