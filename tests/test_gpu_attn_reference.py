"""Attention where a row's reference point moves late, often, or never: scores that rise along the keys, one late spike, equal scores,
short KV whose two halves take turns, odd numbers of blocks, tile lists.  The one-block kernel against the two-block kernel: the same
bits."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _keys(kind, Lk, H, q):
    g = torch.Generator(device="cuda").manual_seed(Lk)
    k = torch.randn(Lk, H, 128, device="cuda", generator=g, dtype=torch.bfloat16)
    if kind == "rising":
        k *= torch.linspace(0.05, 4.0, Lk, device="cuda").to(k.dtype)[:, None, None]
    elif kind == "spike":  # one key close to the first queries, behind the first tiles
        k[Lk - 2] = 2 * q[0]
    elif kind == "equal":
        k.zero_()
    return k


@pytest.mark.parametrize("kind", ["plain", "rising", "spike", "equal"])
@pytest.mark.parametrize("Lq,Lk,H", [(129, 128, 3), (300, 200, 2), (257, 512, 5), (640, 513, 3), (1500, 1000, 12), (200, 2600, 2)])
def test_kernels_agree_wherever_reference_points_move(kind, Lq, Lk, H):
    from ksanadit_b200 import _lib, ops
    q = torch.randn(Lq, H, 128, device="cuda", generator=torch.Generator(device="cuda").manual_seed(7), dtype=torch.bfloat16) * 2
    k = _keys(kind, Lk, H, q)
    v = torch.randn(Lk, H, 128, device="cuda", generator=torch.Generator(device="cuda").manual_seed(8), dtype=torch.bfloat16)
    q8, qs = ops.sage_quant_int8(q, ops.Q_BLOCK, premul=ops.q_premul(128))
    k8, ks = ops.sage_quant_int8(k, ops.K_BLOCK)
    vt, vs = ops.sage_quant_v(v)
    lib = _lib.load()
    outs = []
    for mode in (1, 0):
        before = lib.ksb_attn_dual_mode(mode)
        try:
            outs.append(ops.sage_attn_core(q8, qs, k8, ks, vt, vs, Lq, Lk, torch.bfloat16))
        finally:
            lib.ksb_attn_dual_mode(before)
    _lib.assert_device_ok()
    assert torch.equal(outs[0], outs[1])
    assert outs[0].isfinite().all()


@pytest.mark.parametrize("kind", ["plain", "rising"])
@pytest.mark.parametrize("Lk", [96 * 128 - 1, 96 * 128, 96 * 128 + 1])
def test_kernels_agree_about_the_longest_kv_that_takes_turns(kind, Lk):
    test_kernels_agree_wherever_reference_points_move(kind, 300, Lk, 2)


# one Q block per head; 24 KV tiles, then more of them in launches of up to and above 540 tiles of pairs on each of 148 SMs
@pytest.mark.parametrize("Lq,Lk,H", [(100, 512, 3), (100, 513, 3), (77, 3000, 160), (20400, 3072, 40), (20200, 3200, 40), (20400, 3200, 40)])
def test_kernels_agree_about_the_launches_that_take_turns(Lq, Lk, H):
    test_kernels_agree_wherever_reference_points_move("rising", Lq, Lk, H)


def _operands_of_scores(scales, Lk, seed=0):
    """INT8 / FP8 operands of one Q block per head, with ``scales`` per unit of the INT8 product.  In one row of each warp every KV tile's
    largest score lies above the one before by the least whole number of units that exceeds the slack, on top of a large score
    that all keys share; nothing else in a tile comes near it.  The other rows have one large score, in the first tile."""
    g = torch.Generator().manual_seed(seed)
    H, nq, nk = len(scales), 1, Lk // 128
    q8 = torch.randint(-127, 128, (H, 128, 128), generator=g, dtype=torch.int8)
    k8 = torch.randint(-127, 128, (H, 1, 128), generator=g, dtype=torch.int8).repeat(1, Lk, 1)
    rises = torch.zeros(128, dtype=torch.bool)
    rises[torch.tensor([3, 32 + 14, 64 + 31, 96])] = True
    q8[:, :, :3] = 0
    q8[:, rises, 0], q8[:, rises, 1], q8[:, ~rises, 2] = 1, 100, 127
    k8[:, :, 2] = -127
    k8[:, 0, 2] = 0
    for h, sc in enumerate(scales):
        least = int(3.5 / sc) + 1
        top = 0
        for t in range(nk):
            at = top - int(12 / sc) - torch.randint(0, 50, (128,), generator=g)
            at[int(torch.randint(0, 128, (1,), generator=g))] = top
            fine = torch.remainder(at + 50, 100) - 50
            k8[h, 128 * t:128 * (t + 1), 0] = fine.to(torch.int8)
            k8[h, 128 * t:128 * (t + 1), 1] = torch.div(at - fine, 100, rounding_mode="floor").to(torch.int8)
            top += least
    qs = torch.tensor(scales, dtype=torch.float32).view(H, nq)
    ks = torch.ones(H, 2 * nk)
    vt = torch.randn(H, 128, Lk, generator=g).to(torch.float8_e4m3fn)
    return [t.cuda() for t in (q8, qs, k8, ks, vt, torch.rand(H, 128, generator=g) + 0.5)]


def _both_kernels(run):
    from ksanadit_b200 import _lib
    lib = _lib.load()
    outs = []
    for mode in (1, 0):
        before = lib.ksb_attn_dual_mode(mode)
        try:
            outs.append(run())
        finally:
            lib.ksb_attn_dual_mode(before)
    _lib.assert_device_ok()
    return outs


@pytest.mark.parametrize("Lk,seed", [(256, 0), (256, 1), (256, 2), (1024, 0)])
def test_kernels_agree_where_scores_just_exceed_the_slack(Lk, seed):
    """Scales up to 2 per unit of the INT8 product: the exponentials' argument is then rounded by up to a unit, and a value just above
    the slack may give an exponential below 2^(5 + 3.5)."""
    from ksanadit_b200 import ops
    scales = [float(s) for s in torch.logspace(-2, 0.3, 97)]
    args = _operands_of_scores(scales, Lk, seed)
    two, one = _both_kernels(lambda: ops.sage_attn_core(*args, 128, Lk, torch.bfloat16))
    assert two.isfinite().all()
    wrong = (two != one).flatten(2).any(2)  # [row, head]
    assert not wrong.any(), [(scales[h], int(wrong[:, h].sum())) for h in range(len(scales)) if wrong[:, h].any()]


@pytest.mark.parametrize("kind", ["plain", "rising", "spike", "equal", "large"])
@pytest.mark.parametrize("Lq,Lk,H", [(129, 300, 3), (640, 1100, 2), (1500, 1500, 5)])
def test_tile_lists_agree_wherever_reference_points_move(monkeypatch, kind, Lq, Lk, H):
    """Lists with dropped 64-token halves, first tiles other than tile 0 and an empty list: the one-block kernel against the pairs'."""
    import numpy as np

    from ksanadit_b200 import _lib, ops, radial_mask
    g = torch.Generator(device="cuda").manual_seed(7)
    q = torch.randn(Lq, H, 128, device="cuda", generator=g, dtype=torch.bfloat16) * (40 if kind == "large" else 2)
    k = _keys("rising" if kind == "large" else kind, Lk, H, q) * (10 if kind == "large" else 1)
    v = torch.randn(Lk, H, 128, device="cuda", generator=g, dtype=torch.bfloat16)
    q8, qs = ops.sage_quant_int8(q, ops.Q_BLOCK, premul=ops.q_premul(128))
    k8, ks = ops.sage_quant_int8(k, ops.K_BLOCK)
    vt, vs = ops.sage_quant_v(v)
    nq, nk = (Lq + 127) // 128, (Lk + 127) // 128
    mask = np.random.RandomState(Lk).random_sample((nq, 2 * nk)) < 0.5
    mask[0, 2 * nk - 1] = True
    mask[1 if nq < 3 else 2] = False
    lists = [torch.from_numpy(a).cuda() for a in radial_mask.compact_tile_lists(mask)]
    outs = []
    for overhead in (0.0, 1e9):
        monkeypatch.setattr(ops, "PAIR_LIST_MAX_OVERHEAD", overhead)
        monkeypatch.setattr(ops, "_PAIR_LISTS", {})
        assert (ops._pair_lists(*lists, False) is None) == (overhead == 0.0)
        outs.append(ops.sage_attn_core(q8, qs, k8, ks, vt, vs, Lq, Lk, torch.bfloat16, tile_offsets=lists[0], tile_entries=lists[1]))
    _lib.assert_device_ok()
    assert torch.equal(outs[0], outs[1]) and outs[0].isfinite().all()


@pytest.mark.parametrize("B,Lq,Lk,H", [(1, 128 * 26 + 7, 257, 12), (3, 128 * 13 + 1, 128, 24), (1, 128 * 25, 16 * 128, 12), (1, 128 * 25, 16 * 128 + 1, 12)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_output_in_bulk_equals_output_row_by_row(B, Lq, Lk, H, dtype):
    """More pairs than SMs over up to 16 KV tiles: stores through a tensor map, into heads that lie apart, with a ragged end, samples of a batch,
    one KV tile per pair (the next P is written where the output lies); what is beside the output stays."""
    from ksanadit_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(Lq + Lk)
    q, k, v = (torch.randn(B, n, H, 128, device="cuda", generator=g, dtype=dtype) for n in (Lq, Lk, Lk))

    def run():
        buf = torch.full((B, Lq + 3, H, 136), 7.0, device="cuda", dtype=dtype)
        ops.sage_attention_batched(q, k, v, buf[:, :Lq, :, :128])
        return buf
    two, one = _both_kernels(run)
    assert torch.equal(two, one)
    assert two.isfinite().all() and bool((two[:, Lq:] == 7).all()) and bool((two[..., 128:] == 7).all())


@pytest.mark.parametrize("axis", ["sample", "token", "head"])
def test_output_strides_that_no_tensor_map_takes(axis):
    """An output laid out backwards (a C caller's; torch has no such strides), in a launch whose output otherwise leaves in bulk: stored
    row by row, and the call that succeeds leaves the text of the last error as it was."""
    import ctypes

    from ksanadit_b200 import _lib, native, ops
    B, L, H, Lk = 2, 1000, 24, 77
    g = torch.Generator(device="cuda").manual_seed(2)
    q, k, v = (torch.randn(B, n, H, 128, device="cuda", generator=g, dtype=torch.bfloat16) for n in (L, Lk, Lk))
    ref, buf = torch.empty_like(q), torch.full_like(q, 7.0)
    ops.sage_attention_batched(q, k, v, ref)
    lib = _lib.load()
    assert lib.ksb_quant_fp8_rowwise(None, 0, 4, 24, 24, None, None, None) == -1
    text = lib.ksb_last_error()
    dim = ("sample", "token", "head").index(axis)
    strides = list(buf.stride()[:3])
    last = buf.data_ptr() + 2 * strides[dim] * (buf.shape[dim] - 1)
    strides[dim] = -strides[dim]
    layout = (ctypes.c_int64 * 12)(*q.stride()[:3], *k.stride()[:3], *v.stride()[:3], *strides)
    ws = native.workspace(lib.ksb_sage_attention_workspace(B, L, Lk, H), q.device)
    rc = lib.ksb_sage_attention(q.data_ptr(), k.data_ptr(), v.data_ptr(), _lib.BF16, B, L, Lk, H, layout, ops.q_premul(128), None, last, ws.data_ptr(), native.stream())
    _lib.assert_device_ok()
    assert rc > 0 and lib.ksb_last_error() == text
    assert torch.equal(buf.flip(dim), ref)
