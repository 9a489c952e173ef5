"""Row quantisers at the edges of their size classes (warps per row, 16-element chunks per thread), and their modulation forms
against one another: bytes and scales are determined bit for bit."""

import pytest
import torch

from oracle import dit_ops as D
from oracle import quantizers as Qz

pytestmark = pytest.mark.gpu

EDGES = [16, 1536, 1552, 2048, 2064, 4096, 4112, 6144, 6160, 8192, 8208, 12288, 12304, 16384]


@pytest.mark.parametrize("K", EDGES)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_plain_and_static(K, dtype):
    from ksanadit_b200 import _lib, ops
    x = D.make_activations(9, K, seed=K, dtype=dtype)
    x[1] = 0
    # small rows; in fp16 the multiplier 1 / scale overflows below a maximum of 7e-3, where the kernel saturates and torch's cast does not
    x[2] *= 1e-6 if dtype == torch.bfloat16 else 1e-3
    if dtype == torch.float16:
        x[2, 0] = 0.01
    x[3, 5], x[4, -1], x[5, 0] = float("inf"), float("nan"), -0.0
    q, s = ops.quant_fp8_rowwise(x.cuda())
    rows = [r for r in range(9) if r not in (3, 4)]
    q_ref, s_ref = Qz.act_quant_fp8_rowwise(x[rows])
    assert torch.equal(s.cpu()[rows], s_ref) and torch.equal(q.cpu()[rows].view(torch.uint8), q_ref.view(torch.uint8))
    assert torch.isinf(s[3]) and torch.isfinite(s[4])  # a NaN is not the maximum
    nan = q.cpu().float().isnan()
    assert nan[3].sum() == 1 and nan[4].sum() == 1 and nan[3, 5] and nan[4, -1]
    scale = torch.tensor([0.037], device="cuda")
    q, s = ops.quant_fp8_static(x.cuda(), scale)
    inv = (1 / scale.cpu()).to(dtype)
    ref = (x[rows] * inv).float().clamp(-448, 448).to(torch.float8_e4m3fn)
    assert torch.equal(q.cpu()[rows].view(torch.uint8), ref.view(torch.uint8)) and bool((s.cpu() == scale.cpu()).all())
    _lib.assert_device_ok()


@pytest.mark.parametrize("K", EDGES)
@pytest.mark.parametrize("rounded", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_adaln_forms_agree(K, rounded, dtype):
    from ksanadit_b200 import _lib, ops
    M = 37
    g = torch.Generator().manual_seed(K)
    x = D.make_activations(M, K, seed=K, dtype=dtype)
    shift, scale = ((torch.randn(1, K, generator=g) * 0.3).to(dtype) for _ in range(2))
    one = ops.adaln_quant_fp8(x.cuda(), shift.cuda(), scale.cuda(), want_h=True, round_product=rounded)
    rows = ops.adaln_quant_fp8(x.cuda(), shift.expand(M, K).cuda(), scale.expand(M, K).cuda(), want_h=True, round_product=rounded)
    for a, b in zip(one, rows):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
    q2, s2 = Qz.act_quant_fp8_rowwise(one[2].cpu())
    assert torch.equal(one[0].cpu().view(torch.uint8), q2.view(torch.uint8)) and torch.equal(one[1].cpu(), s2)
    # the modulation itself, from LayerNorm in 64 bits: a last-place difference of the norm (2^-8 of it, bf16) moves the result by
    # one more rounding at most
    xd = x.double()
    ln = ((xd - xd.mean(1, keepdim=True)) / (xd.var(1, unbiased=False, keepdim=True) + 1e-6).sqrt()).to(dtype)
    ref = (ln * (1 + scale) + shift) if rounded else torch.addcmul(shift, ln, 1 + scale)
    ulp = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    bound = 4 * ulp * (ln.float() * (1 + scale.float())).abs().clamp_min(1e-3) + 2 * ulp * (ref.float().abs() + shift.float().abs())
    assert bool(((one[2].cpu().float() - ref.float()).abs() <= bound).all())
    _lib.assert_device_ok()


@pytest.mark.parametrize("K", [1536, 8192, 8208, 12304, 16384])
@pytest.mark.parametrize("bias", [False, True])
def test_affine_norm(K, bias):
    """Against LayerNorm in 64 bits: the result's rounding, and fp32 sums over K elements (the mean of 16384 values up to 80)."""
    from ksanadit_b200 import _lib, ops
    g = torch.Generator().manual_seed(K)
    x = D.make_activations(21, K, seed=K)
    w, b = torch.randn(K, generator=g), torch.randn(K, generator=g)
    q, s, h = ops.layernorm_quant_fp8(x.cuda(), w.cuda(), b.cuda() if bias else None, want_h=True)
    q2, s2 = Qz.act_quant_fp8_rowwise(h.cpu())
    assert torch.equal(q.cpu().view(torch.uint8), q2.view(torch.uint8)) and torch.equal(s.cpu(), s2)
    ref = torch.nn.functional.layer_norm(x.double(), (K,), w.double(), b.double() if bias else None, 1e-6)
    assert bool(((h.cpu().double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4 * w.abs()).all())
    _lib.assert_device_ok()


@pytest.mark.parametrize("M,K", [(40001, 64), (20003, 2064), (7001, 4112)])
def test_rows_of_many_waves(M, K):
    """From eight turns per resident CTA on, a launch without a norm has more CTAs: the rows are those of two shorter ones."""
    from ksanadit_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K, device="cuda", generator=g, dtype=torch.bfloat16)
    scale = torch.tensor([0.02], device="cuda")
    for quant in (ops.quant_fp8_rowwise, lambda t: ops.quant_fp8_static(t, scale)):
        parts = [quant(t) for t in x.split(5000)]
        q, s = quant(x)
        assert torch.equal(q.view(torch.uint8), torch.cat([p[0].view(torch.uint8) for p in parts])) and torch.equal(s, torch.cat([p[1] for p in parts]))
