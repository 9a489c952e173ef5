"""Whole-operator calls (attention, Wan and Qwen-Image blocks as one call of the library) against the same operator kernel by
kernel, at the sizes where the folded statistics, the shared launches and the job lists can go wrong; and the inputs and
parameter changes that have to reach the right one of the two."""

import pytest
import torch

from conftest import cosine

pytestmark = pytest.mark.gpu


def _rel(a, b):
    a, b = a.double().flatten(), b.double().flatten()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


def _qkv(B, Lq, Lk, H, dtype, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + Lq + Lk)
    q = torch.randn(B, Lq, H, 128, device="cuda", generator=g, dtype=dtype)
    # K and V as views into one fused buffer
    kv = torch.randn(B, Lk, 2, H, 128, device="cuda", generator=g, dtype=dtype)
    kv[:, :, 0] += 0.5 * torch.randn(H, 128, device="cuda", generator=g, dtype=dtype)
    return q, kv[:, :, 0], kv[:, :, 1]


def _by_kernels(q, k, v):
    from ksanadit_b200 import ops
    outs = []
    for b in range(q.shape[0]):
        km = ops.sage_kmean(k[b])
        q8, qs = ops.sage_quant_int8(q[b], ops.Q_BLOCK, premul=ops.q_premul(128))
        k8, ks = ops.sage_quant_int8(k[b], ops.K_BLOCK, mean=km)
        vt, vs = ops.sage_quant_v(v[b])
        outs.append(ops.sage_attn_core(q8, qs, k8, ks, vt, vs, q.shape[1], k.shape[1], q.dtype))
    return torch.stack(outs)


# 1 token; tile edges; the statistics' sums left to the quantisers (<= 64 tiles) or finished first; more samples than a launch
# takes (four); more CTAs' worth of heads than SMs
@pytest.mark.parametrize("B,Lq,Lk,H", [(1, 1, 1, 1), (1, 129, 127, 3), (2, 64, 8192, 2), (2, 200, 8193, 1), (5, 130, 65, 3), (1, 300, 257, 40)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_attention_call_matches_kernels(B, Lq, Lk, H, dtype):
    from ksanadit_b200 import _lib, ops
    q, k, v = _qkv(B, Lq, Lk, H, dtype)
    out = torch.full((B, Lq, H, 128), float("nan"), device="cuda", dtype=dtype)
    ops.sage_attention_batched(q, k, v, out)
    ref = _by_kernels(q, k, v)
    _lib.assert_device_ok()
    # the K mean's fp32 sums may be added in another order; one rounding of K to INT8 (1/127 of its block's maximum) more or less
    assert _rel(out, ref) < 1e-2


@pytest.mark.parametrize("offset", [0, 1, 4])
def test_attention_v_scale_table_at_any_address(offset):
    """The output stage reads the V scales 16 bytes at a time where their address allows it."""
    from ksanadit_b200 import ops
    q, k, v = (t[0] for t in _qkv(1, 129, 200, 2, torch.bfloat16))
    q8, qs = ops.sage_quant_int8(q, ops.Q_BLOCK, premul=ops.q_premul(128))
    k8, ks = ops.sage_quant_int8(k, ops.K_BLOCK, mean=ops.sage_kmean(k))
    vt, vs = ops.sage_quant_v(v)
    shifted = torch.zeros(vs.numel() + offset, device="cuda")[offset:].view_as(vs).copy_(vs)
    ref = ops.sage_attn_core(q8, qs, k8, ks, vt, vs, 129, 200)
    assert torch.equal(ops.sage_attn_core(q8, qs, k8, ks, vt, shifted, 129, 200), ref)


def test_attention_of_one_sample_with_any_batch_stride():
    """The stride between samples says nothing where there is one (a row of a packed buffer of odd length)."""
    from ksanadit_b200 import ops
    q, k, v = _qkv(1, 130, 70, 2, torch.bfloat16)

    def packed(t):
        buf = torch.empty(2, t.numel() + 4, dtype=t.dtype, device="cuda")
        row = buf[:, :t.numel()].view(2, *t.shape[1:])[:1]
        assert row.stride(0) % 8 != 0
        return row.copy_(t)

    ref, out = torch.empty_like(q), packed(q)
    ops.sage_attention_batched(q, k.contiguous(), v.contiguous(), ref)
    ops.sage_attention_batched(packed(q), packed(k), packed(v), out)
    assert torch.equal(out, ref)


def test_attention_inputs_the_single_call_does_not_take():
    """Operands of different half types and an empty batch go the general way."""
    from ksanadit_b200 import ops
    from ksanadit_b200.attention import KsanaAttentionOp
    from ksanadit_b200.config import KsanaAttentionBackend, KsanaAttentionConfig
    op = KsanaAttentionOp(2, 128, attention_config=KsanaAttentionConfig(backend=KsanaAttentionBackend.SAGE_ATTN))
    q, k, v = _qkv(2, 130, 70, 2, torch.bfloat16)
    ref = op(q, k, v)
    mixed = op(q, k.to(torch.float16), v)
    assert mixed.dtype == torch.bfloat16 and _rel(mixed, ref) < 2e-2
    assert _rel(ops.sage_attention(q[0], k[0].to(torch.float16), v[0]), ref[0]) < 2e-2
    assert op(q[:0], k[:0], v[:0]).shape == (0, 130, 2, 128)


def _wan(dim, ffn, heads, dtype, seed=3):
    from ksanadit_b200.wan_block import B200WanBlock
    return B200WanBlock(dim, ffn, heads, device="cuda", dtype=dtype).random_init(seed)


def _general(blk, *args, **kw):
    """The block kernel by kernel."""
    from ksanadit_b200 import native
    blk._native = lambda: native.Descriptor()
    try:
        return blk(*args, **kw)
    finally:
        del blk._native


# one token and one text token; ragged; three samples (two per launch); modulation per token; more rows than the limit of the
# in-kernel 1 / rms sums (8192); float32 modulation
@pytest.mark.parametrize("dim,ffn,B,grid,text,per_token,dtype,e_dtype", [
    (256, 512, 1, (1, 1, 1), 1, False, torch.bfloat16, torch.bfloat16),
    (512, 1040, 1, (1, 13, 10), 77, True, torch.float16, torch.float16),
    (256, 768, 3, (3, 7, 9), 33, False, torch.bfloat16, torch.float32),
    (256, 768, 2, (2, 9, 10), 65, True, torch.bfloat16, torch.bfloat16),
    (256, 512, 1, (7, 30, 40), 130, False, torch.bfloat16, torch.bfloat16),
])
def test_wan_block_call_matches_kernels(dim, ffn, B, grid, text, per_token, dtype, e_dtype):
    from ksanadit_b200 import _lib
    L = grid[0] * grid[1] * grid[2]
    blk = _wan(dim, ffn, dim // 128, dtype)
    g = torch.Generator(device="cuda").manual_seed(L)
    x = torch.randn(B, L, dim, device="cuda", generator=g, dtype=dtype)
    e = (torch.randn(B, L if per_token else 1, 6, dim, device="cuda", generator=g) * 0.1).to(e_dtype)
    c = torch.randn(B, text, dim, device="cuda", generator=g, dtype=dtype)
    with torch.no_grad():
        out = blk(x, e, grid_sizes=[grid] * B, context=c)
        assert blk._call.address is not None
        ref = _general(blk, x, e, grid_sizes=[grid] * B, context=c)
    _lib.assert_device_ok()
    assert cosine(out, ref) >= 0.999 and _rel(out, ref) < 2e-2


def test_wan_block_call_matches_kernels_where_the_quantisers_take_many_waves():
    test_wan_block_call_matches_kernels(512, 512, 1, (1, 130, 129), 33, False, torch.bfloat16, torch.bfloat16)


def test_wan_block_call_follows_its_parameters():
    """A parameter replaced, re-typed or re-laid out, and plain attributes, after the first call."""
    dim, grid = 256, (1, 6, 7)
    blk = _wan(dim, 512, 2, torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(0)
    x = torch.randn(1, 42, dim, device="cuda", generator=g, dtype=torch.bfloat16)
    e = torch.randn(1, 1, 6, dim, device="cuda", generator=g, dtype=torch.bfloat16) * 0.1
    c = torch.randn(1, 9, dim, device="cuda", generator=g, dtype=torch.bfloat16)

    def both():
        with torch.no_grad():
            return blk(x, e, grid_sizes=[grid], context=c), _general(blk, x, e, grid_sizes=[grid], context=c)

    first, ref = both()
    assert _rel(first, ref) < 2e-2
    blk.eps = 50.0
    out, ref = both()
    assert _rel(out, ref) < 0.1 * _rel(out, first)  # a stale eps gives `first` again
    blk.eps = 1e-6
    # the same place in memory holding the bits of another type: what a re-typed bias may find itself in
    bias = blk.ffn[2].bias
    bias.data = (torch.randn(dim, device="cuda", generator=g) * 4).to(torch.float16).view(torch.bfloat16)
    both()
    bias.data = bias.data.view(torch.float16)
    out, ref = both()
    assert _rel(out, ref) < 2e-2
    blk.cross_attn_norm = False
    out, ref = both()
    assert _rel(out, ref) < 2e-2


def _qwen(dim, heads, ffn, edit=False):
    from ksanadit_b200.qwen_block import B200QwenBlock
    return B200QwenBlock(dim, heads, ffn, zero_cond_t=edit).random_init(5)


@pytest.mark.parametrize("h,w,text,edit", [(1, 1, 1, False), (9, 15, 77, False), (11, 12, 130, True), (8, 16, 128, True), (70, 65, 20, False)])
def test_qwen_block_call_matches_kernels(h, w, text, edit):
    from ksanadit_b200 import _lib
    blk = _qwen(256, 2, 768, edit)
    g = torch.Generator(device="cuda").manual_seed(h * w)
    img = torch.randn(1, h * w, 256, device="cuda", generator=g, dtype=torch.bfloat16)
    txt = torch.randn(1, text, 256, device="cuda", generator=g, dtype=torch.bfloat16)
    temb = torch.randn(2 if edit else 1, 256, device="cuda", generator=g, dtype=torch.bfloat16)
    kw = dict(img_grid=(1, h, w))
    if edit:
        kw["modulate_index"] = torch.randint(0, 2, (1, h * w), device="cuda", generator=g)
    with torch.no_grad():
        out = blk(img, txt, temb, **kw)
        assert blk._call.address is not None
        ref = _general(blk, img, txt, temb, **kw)
    _lib.assert_device_ok()
    for a, b in zip(out, ref):
        assert cosine(a, b) >= 0.999 and _rel(a, b) < 2e-2


@pytest.mark.parametrize("layout", ["strided", "expanded"])
def test_modulate_index_of_any_layout(layout):
    blk = _qwen(256, 2, 768, True)
    g = torch.Generator(device="cuda").manual_seed(1)
    img = torch.randn(1, 40, 256, device="cuda", generator=g, dtype=torch.bfloat16)
    txt = torch.randn(1, 8, 256, device="cuda", generator=g, dtype=torch.bfloat16)
    temb = torch.randn(2, 256, device="cuda", generator=g, dtype=torch.bfloat16)
    if layout == "strided":
        index = torch.randint(0, 2, (1, 80), device="cuda", generator=g)[:, ::2]
    else:
        index = torch.ones(1, 1, device="cuda", dtype=torch.int64).expand(1, 40)
    with torch.no_grad():
        out, ref = (blk(img, txt, temb, img_grid=(1, 5, 8), modulate_index=i) for i in (index, index.clone(memory_format=torch.contiguous_format)))
    assert all(torch.equal(a, b) for a, b in zip(out, ref))


def test_modulate_index_out_of_range_is_reported():
    from ksanadit_b200 import _lib
    blk = _qwen(256, 2, 768, True)
    img = torch.ones(1, 40, 256, device="cuda", dtype=torch.bfloat16)
    txt = torch.ones(1, 8, 256, device="cuda", dtype=torch.bfloat16)
    temb = torch.ones(2, 256, device="cuda", dtype=torch.bfloat16)
    index = torch.zeros(1, 40, device="cuda", dtype=torch.int64)
    index[0, 3], index[0, 39] = 2, -1
    temb[1] = -1
    with torch.no_grad():
        out = blk(img, txt, temb, img_grid=(1, 5, 8), modulate_index=index)
    torch.cuda.synchronize()
    with pytest.raises(_lib.KsanaB200Error, match="modulate_index"):
        _lib.assert_device_ok()
    _lib.assert_device_ok()  # reading the status cleared it
    with torch.no_grad():  # the rows it names were modulated by row 0
        ref = blk(img, txt, temb, img_grid=(1, 5, 8), modulate_index=torch.zeros_like(index))
        other = blk(img, txt, temb, img_grid=(1, 5, 8), modulate_index=torch.ones_like(index))
    assert all(torch.equal(a, b) for a, b in zip(out, ref)) and not torch.equal(other[1], ref[1])


def test_bad_index_and_a_wait_that_runs_out_are_both_reported():
    """A bad index neither makes other kernels' waits give up nor hides one that ran out."""
    from ksanadit_b200 import _lib
    blk = _qwen(256, 2, 768, True)
    x = torch.ones(1, 40, 256, device="cuda", dtype=torch.bfloat16)
    with torch.no_grad():
        blk(x, x[:, :8], x[0, :2], img_grid=(1, 5, 8), modulate_index=torch.full((1, 40), 2, device="cuda"))
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.check(_lib.load().ksb_selftest_bounded_wait(2_000_000, flag.data_ptr(), torch.cuda.current_stream().cuda_stream), "selftest")
    with pytest.raises(_lib.KsanaB200Error, match="kernel=15 site=1"):
        _lib.assert_device_ok()
    with pytest.raises(_lib.KsanaB200Error, match="modulate_index"):
        _lib.assert_device_ok()
    _lib.assert_device_ok()


def test_linear_without_rows():
    from ksanadit_b200.linear import B200Fp8Linear
    lin = B200Fp8Linear.from_float(torch.nn.Linear(64, 48, device="cuda"))
    assert lin(torch.empty(0, 64, device="cuda", dtype=torch.bfloat16)).shape == (0, 48)
    assert lin(torch.empty(1, 0, 64, device="cuda", dtype=torch.bfloat16)).shape == (1, 0, 48)
