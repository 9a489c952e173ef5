"""Attention where a row's reference point moves late, often, or never: scores that rise along the keys, one late spike, equal scores,
short KV whose two halves take turns, odd numbers of blocks.  The one-block kernel, which looks for maxima only where its sums ask for
it, against the two-block kernel, which always looks: the same bits."""

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
