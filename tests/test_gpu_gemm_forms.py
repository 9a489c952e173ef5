"""GPU parity of the GEMM forms behind the size rule: the split-K form (few rows, few tiles, a K range shared by the CTAs of
a cluster) and the 128-column tiles of the persistent form, at the sizes where they can go wrong."""

import pytest
import torch

from conftest import cosine, max_abs_rel
from oracle import dit_ops as D
from oracle import quantizers as Qz

pytestmark = pytest.mark.gpu

# one 16-bit ulp of the largest output (2^-8 of it) plus the fp32 accumulation order
TOL, COS = 1e-2, 0.9999


@pytest.mark.parametrize("M,N,K", [
    (1, 8, 16),        # smallest problem: one row, one 16-byte unit of columns, an eighth of a k-step
    (1, 18432, 256),   # more CTAs than SMs, two per SM
    (7, 200, 3072),    # A box of 8 rows, columns cut inside a tile, K split over a cluster
    (33, 72, 2064),    # A box of 40 rows, K ends inside a k-step, uneven shares
    (77, 1536, 4096),  # a text prompt
    (129, 136, 8960),  # second row tile with one row, K split eight ways
    (257, 9216, 1536), # 128-column tiles of the persistent form, one row past a pair
])
@pytest.mark.parametrize("epilogue", ["none", "gelu", "gate"])
def test_small_gemm_matches_oracle(M, N, K, epilogue):
    from ksanadit_b200 import _lib, ops
    g = torch.Generator().manual_seed(M + N + K)
    dtype = torch.float16 if M % 2 else torch.bfloat16
    x = D.make_activations(M, K, seed=M + K, dtype=dtype)
    wq, sw = Qz.weight_quant_fp8_channelwise((torch.randn(N, K, generator=g) * 0.02).to(dtype))
    b = (torch.randn(N, generator=g) * 0.02).to(dtype)
    xq, sx = Qz.act_quant_fp8_rowwise(x)
    ref = Qz.fp8_linear_emulated(x, wq, sw, b, xq=xq, s_x=sx)
    kw = {}
    if epilogue == "gelu":
        ref = D.gelu_tanh(ref)
        kw = dict(epilogue=_lib.EPI_GELU_TANH)
    elif epilogue == "gate":
        resid, gate = torch.randn(M, N, generator=g).to(dtype), torch.randn(1, N, generator=g).to(dtype)
        ref = D.gate_residual(resid, ref, gate)
        kw = dict(epilogue=_lib.EPI_GATE_RESIDUAL, resid=resid.cuda(), gate=gate.cuda())
    # columns of a wider buffer: what lies beside them stays untouched
    buf = torch.full((M, N + 16), 7.0, dtype=dtype, device="cuda")
    ops.fp8_gemm(xq.cuda(), sx.cuda(), wq.cuda(), sw.cuda(), b.cuda(), out=buf[:, :N], **kw)
    _lib.assert_device_ok()
    assert max_abs_rel(buf[:, :N].cpu().float(), ref.float()) <= TOL
    assert cosine(buf[:, :N].cpu(), ref) >= COS
    assert bool((buf[:, N:] == 7).all())


@pytest.mark.parametrize("M", [5, 40])  # read ahead of the accumulator and behind it
def test_unaligned_column_parameters(M):
    """Scales and bias that do not start on 16 bytes (slices of a fused projection's vectors)."""
    from ksanadit_b200 import ops
    N, K = 64, 256
    g = torch.Generator(device="cuda").manual_seed(0)
    xq, wq = ((torch.randn(n, K, device="cuda", generator=g) * 50).clamp(-448, 448).to(torch.float8_e4m3fn) for n in (M, N))
    sx, sw = torch.rand(M, device="cuda", generator=g), torch.rand(N + 1, device="cuda", generator=g) * 1e-3
    bias = torch.randn(N + 1, device="cuda", generator=g).to(torch.bfloat16)
    assert torch.equal(ops.fp8_gemm(xq, sx, wq, sw[1:], bias[1:]), ops.fp8_gemm(xq, sx, wq, sw[1:].clone(), bias[1:].clone()))


# workers go from tiles inside the problem to ragged ones (rows and columns): an epilogue warp
# without a part in a tile must leave the part of its last tile alone until that is stored
@pytest.mark.parametrize("M,N,K", [(2384, 4680, 1536), (2640, 2392, 3072), (19536, 1480, 256)])
def test_gated_gemm_past_the_edge_equals_a_padded_problem(M, N, K):
    from ksanadit_b200 import _lib, ops
    Mp, Np = (M + 255) // 256 * 256, (N + 255) // 256 * 256
    g = torch.Generator(device="cuda").manual_seed(M)
    xq, wq = ((torch.randn(n, K, device="cuda", generator=g) * 50).clamp(-448, 448).to(torch.float8_e4m3fn) for n in (Mp, Np))
    sx, sw = torch.rand(Mp, device="cuda", generator=g), torch.rand(Np, device="cuda", generator=g) * 1e-3
    bias, gate = (torch.randn(1, Np, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    resid = torch.randn(Mp, Np, device="cuda", generator=g).to(torch.bfloat16)
    kw = dict(epilogue=_lib.EPI_GATE_RESIDUAL)
    ref = ops.fp8_gemm(xq, sx, wq, sw, bias[0], resid=resid, gate=gate, **kw)[:M, :N]
    cut = (xq[:M], sx[:M], wq[:N], sw[:N], bias[0, :N])
    for _ in range(5):  # in place, as a block's residual stream is
        x = resid[:M, :N].contiguous()
        assert torch.equal(ops.fp8_gemm(*cut, resid=x, gate=gate[:, :N], out=x, **kw), ref)
    _lib.assert_device_ok()


@pytest.mark.parametrize("M", [1, 300])  # the split form and whole tiles
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gelu_over_the_whole_range(M, dtype):
    """Every value of the type (the bias of an empty product) against 64 bits: infinities and NaN stay where they are."""
    from ksanadit_b200 import _lib, ops
    g = torch.Generator().manual_seed(0)
    x = torch.arange(65536, dtype=torch.int32).to(torch.uint16).view(dtype)[torch.randperm(65536, generator=g)].cuda()
    zero = torch.zeros(M, 16, device="cuda").to(torch.float8_e4m3fn)
    one = torch.ones(65536, device="cuda")
    out = ops.fp8_gemm(zero, one[:M], torch.zeros(65536, 16, device="cuda").to(torch.float8_e4m3fn), one, x, out_dtype=dtype, epilogue=_lib.EPI_GELU_TANH)
    assert torch.equal(out.view(torch.uint16), out[:1].view(torch.uint16).expand(M, -1))
    v = x.double()
    ref = v / (1 + torch.exp(-2 * (2 / torch.pi) ** 0.5 * (v + 0.044715 * v ** 3)))
    got = out[0].double()
    assert torch.equal(got.isnan(), ref.isnan())
    ref = torch.where(ref.abs() > torch.finfo(dtype).max, v.sign() * torch.inf, ref)
    finite = ref.isfinite()
    assert torch.equal(got[~finite & ~ref.isnan()], ref[~finite & ~ref.isnan()])
    # half a unit in the last place, and the exponential's 2 + |exponent| units of 2^-24; below the fast quotient's 2^-126 a zero
    ulp = torch.finfo(dtype).eps / 2
    tiny = 2.0 ** -24 if dtype == torch.float16 else 2.0 ** -120
    err = (got - ref).abs()[finite]
    assert bool((err <= ulp * 1.01 * ref.abs()[finite] + tiny).all())


# On 74 pairs: tiles of 192 columns, 56 in one wave; 128 columns; 224 columns, 280 in four waves, the last half piece cut, the whole last
# part past the edge with a ragged row tile; 192 columns, the last tile 88 wide (a piece whole, one cut, one past the edge).  Sums per 64
# columns and launches of two problems: test_row_sums_stay_inside_their_table, test_two_problems_in_tiles_of_192_and_224_columns.
@pytest.mark.parametrize("M,N,K,form", [(1560, 1536, 1536, 192), (1281, 1480, 272, 128), (1560, 8960, 256, 224), (1101, 3120, 400, 224), (1101, 3080, 1040, 224),
                                        (2640, 2392, 3072, 192)])
@pytest.mark.parametrize("epilogue", ["none", "gelu", "gate"])
def test_tiles_of_192_and_224_columns_equal_ctas_on_their_own(M, N, K, form, epilogue):
    from ksanadit_b200 import _lib, ops
    assert _form([(M, N)], K) == form
    g = torch.Generator(device="cuda").manual_seed(M + N)
    dtype = torch.float16 if K % 3 else torch.bfloat16
    xq, wq = ((torch.randn(n, K, device="cuda", generator=g) * 50).clamp(-448, 448).to(torch.float8_e4m3fn) for n in (M, N))
    sx, sw = torch.rand(M, device="cuda", generator=g) * 1e-2, torch.rand(N, device="cuda", generator=g) * 1e-3
    bias = torch.randn(N, device="cuda", generator=g).to(dtype)
    kw = {}
    if epilogue == "gelu":
        kw = dict(epilogue=_lib.EPI_GELU_TANH)
    elif epilogue == "gate":
        kw = dict(epilogue=_lib.EPI_GATE_RESIDUAL, resid=torch.randn(M, N, device="cuda", generator=g).to(dtype), gate=torch.randn(1, N, device="cuda", generator=g).to(dtype))
    outs = []
    for pairs in (1, 0):
        before = _lib.load().ksb_gemm_pair_mode(pairs)
        try:
            buf = torch.full((M, N + 16), 7.0, dtype=dtype, device="cuda")
            ops.fp8_gemm(xq, sx, wq, sw, bias, out=buf[:, :N], **kw)
        finally:
            _lib.load().ksb_gemm_pair_mode(before)
        outs.append(buf)
    _lib.assert_device_ok()
    assert torch.equal(outs[0], outs[1])
    assert bool((outs[0][:, N:] == 7).all()) and bool(outs[0].isfinite().all())


def _form(problems, K, sums=0):
    """The form a launch of these (M, N) takes: columns per tile of a CTA pair, 0 = split K."""
    import ctypes

    from ksanadit_b200 import _lib
    rows, cols = ((ctypes.c_int64 * len(problems))(*v) for v in zip(*problems))
    return _lib.load().ksb_gemm_form(len(problems), rows, cols, K, sums)


def _after_steps(monkeypatch, call, name, steps, pairs):
    """Workspace and output of a block call that runs ``steps`` alone in GEMM mode ``pairs``, on a workspace full of one byte."""
    from ksanadit_b200 import _lib, native
    lib, made = _lib.load(), []
    forward = getattr(lib, name)

    def workspace(n, device):
        made.append(torch.full((n,), 0xA5, dtype=torch.uint8, device=device))
        return made[-1]

    with monkeypatch.context() as m:
        m.setattr(native, "workspace", workspace)
        m.setattr(lib, name, lambda block, args, first, last, ws, stream: sum(forward(block, args, s, s, ws, stream) for s in steps))
        before = lib.ksb_gemm_pair_mode(pairs)
        try:
            with torch.no_grad():
                out = call()
        finally:
            lib.ksb_gemm_pair_mode(before)
    _lib.assert_device_ok()
    return made, out


# tiles of 192 columns where neither 2 * dim nor dim is a multiple of 192
@pytest.mark.parametrize("dim,L,text,step", [(5120, 200, 200, "WAN_QKV"), (2048, 1300, 33, "WAN_QKV"), (5120, 400, 16, "WAN_CROSS_Q"), (2048, 1200, 16, "WAN_CROSS_Q")])
def test_row_sums_stay_inside_their_table(monkeypatch, dim, L, text, step):
    """The sums of squares of a Wan block's projections end where Q and K do, in the middle of a tile: every byte of the workspace
    is what CTAs on their own, whose tiles end there, leave."""
    from ksanadit_b200 import native
    from ksanadit_b200.wan_block import B200WanBlock
    problems = [(L, 3 * dim), (text, dim), (text, dim)] if step == "WAN_QKV" else [(L, dim)]
    assert _form(problems, dim, 64) == 192 and dim % 192 != 0
    blk = B200WanBlock(dim, 256, dim // 128, device="cuda", dtype=torch.bfloat16).random_init(3)
    g = torch.Generator(device="cuda").manual_seed(L)
    x, c = (torch.randn(1, n, dim, device="cuda", generator=g, dtype=torch.bfloat16) for n in (L, text))
    e = torch.randn(1, 1, 6, dim, device="cuda", generator=g, dtype=torch.bfloat16) * 0.1
    run = lambda: blk(x, e, grid_sizes=[(1, L // 20, 20)], context=c)  # noqa: E731
    spaces = [_after_steps(monkeypatch, run, "ksb_wan_block_forward", (native.WAN_PRE, getattr(native, step)), pairs)[0] for pairs in (1, 0)]
    assert len(spaces[0]) == len(spaces[1]) >= 1
    for a, b in zip(*spaces):
        assert torch.equal(a, b)
    written = torch.cat([a.view(torch.uint8) for a in spaces[0]]) != 0xA5
    assert int(written.sum()) > L * dim  # the projection's output and the sums among it


# dim 2560 is no multiple of 192 or 224: the gated output projections end inside a tile
@pytest.mark.parametrize("Lt,Li,step,form", [(77, 1000, "QWEN_QKV", 192), (77, 1000, "QWEN_OUT", 192), (256, 1100, "QWEN_QKV", 224), (256, 1100, "QWEN_OUT", 224)])
def test_two_problems_in_tiles_of_192_and_224_columns(monkeypatch, Lt, Li, step, form):
    """Both streams' projections of a Qwen-Image block in one launch: workspace and output as CTAs on their own leave them."""
    from ksanadit_b200 import native
    from ksanadit_b200.qwen_block import B200QwenBlock
    dim = 2560
    cols = 3 * dim if step == "QWEN_QKV" else dim
    assert _form([(Lt, cols), (Li, cols)], dim) == form
    blk = B200QwenBlock(dim, dim // 128, 256).random_init(5)
    g = torch.Generator(device="cuda").manual_seed(Li)
    img, txt = (torch.randn(1, n, dim, device="cuda", generator=g, dtype=torch.bfloat16) for n in (Li, Lt))
    temb = torch.randn(1, dim, device="cuda", generator=g, dtype=torch.bfloat16)
    mods = torch.randn(1, 12 * dim, device="cuda", generator=g, dtype=torch.bfloat16) * 0.1
    run = lambda: blk(img, txt, temb, img_grid=(1, Li // 20, 20), mods=mods)  # noqa: E731
    (space, out), (space1, out1) = (_after_steps(monkeypatch, run, "ksb_qwen_block_forward", (native.QWEN_PRE, getattr(native, step)), pairs) for pairs in (1, 0))
    assert len(space) == len(space1) >= 1 and all(torch.equal(a, b) for a, b in zip(space, space1))
    if step == "QWEN_OUT":
        assert all(torch.equal(a, b) and a.isfinite().all() for a, b in zip(out, out1))
    else:
        assert int((torch.cat(space) != 0xA5).sum()) > (Lt + Li) * 3 * dim
