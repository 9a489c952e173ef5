"""CPU tests of what the whole-operator calls hand to the library: the tensors' layouts, and which calls do not reach it.

A stand-in for the library records its arguments; CPU tensors pass for tensors of one GPU, meta tensors for those of another."""

import ctypes

import pytest
import torch


class FakeLibrary:
    """Answers the whole-operator entry points and keeps what it saw of each call."""

    def __init__(self):
        self.calls = []
        self.rc = 1

    def ksb_attn_dual_mode(self, mode):
        return 0

    def ksb_last_error(self):
        return b"refused"

    def __getattr__(self, name):
        if name.endswith(("_workspace", "_bytes")):
            return lambda *a: 256
        if not name.startswith("ksb_"):
            raise AttributeError(name)

        def entry(*a):
            self.calls.append((name, self.seen(name, a)))
            return self.rc
        return entry

    @staticmethod
    def seen(name, a):
        from ksanadit_b200 import native
        if name == "ksb_qwen_block_forward":
            c = native.QwenCall.from_address(a[1])
            return dict(index=list((ctypes.c_int64 * c.img_tokens).from_address(c.mod_index)) if c.mod_index else None)
        if name == "ksb_linear_forward":
            return dict(static=bool(a[5]))
        if name == "ksb_wan_block_forward":
            return dict(compute_context=native.WanCall.from_address(a[1]).compute_context)
        return {}


@pytest.fixture
def fake(monkeypatch):
    from ksanadit_b200 import _lib, native
    lib = FakeLibrary()
    monkeypatch.setattr(_lib, "load", lambda: lib)
    monkeypatch.setattr(native, "stream", lambda: 0)
    monkeypatch.setattr(torch.Tensor, "is_cuda", property(lambda t: True), raising=False)
    return lib


def _qwen(edit=False):
    from ksanadit_b200.qwen_block import B200QwenBlock
    return B200QwenBlock(256, 2, 512, device="cpu", zero_cond_t=edit).random_init(0)


def _qwen_args(tokens=6, text=3, rows=1, dim=256):
    bf = torch.bfloat16
    return (torch.zeros(1, tokens, dim, dtype=bf), torch.zeros(1, text, dim, dtype=bf), torch.zeros(rows, dim, dtype=bf)), \
        dict(img_grid=(1, 2, tokens // 2), mods=torch.zeros(rows, 12 * dim, dtype=bf))


@pytest.mark.parametrize("index", [
    torch.tensor([[1, 0, 1, 0, 0, 0, 1, 0, 1, 1, 0, 1]])[:, ::2],         # stride 2
    torch.tensor([1, 0, 0, 0, 0, 0])[:1].expand(1, 6),                      # one value for all
    torch.tensor([[1, 1, 0, 0, 1, 0]], dtype=torch.int32),                  # another type
])
def test_modulate_index_is_read_by_its_strides(fake, index):
    args, kw = _qwen_args(rows=2)
    _qwen(edit=True)(*args, modulate_index=index, **kw)
    assert fake.calls[-1] == ("ksb_qwen_block_forward", dict(index=index.reshape(-1).tolist()))


def _wan(**kw):
    from ksanadit_b200.wan_block import B200WanBlock
    return B200WanBlock(256, 512, 2, device="cpu", **kw).random_init(0)


def _wan_args(batch=1, tokens=6, text=3, e_shape=(1, 6, 256), dim=256, text_dim=256, e_dtype=torch.bfloat16):
    bf = torch.bfloat16
    return dict(x=torch.zeros(batch, tokens, dim, dtype=bf), e=torch.zeros(batch, *e_shape, dtype=e_dtype),
                context=torch.zeros(batch, text, text_dim, dtype=bf), grid_sizes=[(1, 2, 3)] * batch)


def _wan_route(fake, blk, args):
    """The way a call takes: the whole-block call, or kernel by kernel (with the shapes of its six modulation tensors)."""
    general = []
    blk._block_one = lambda x, e6, *a: (general.append({tuple(t.shape) for t in e6}), x)[1]
    try:
        blk(**args)
    except (RuntimeError, NotImplementedError):
        general.append("refused")
    return [name for name, _ in fake.calls], general


@pytest.mark.parametrize("args", [dict(), dict(batch=2), dict(e_dtype=torch.float32), dict(e_shape=(6, 6, 256))])
def test_wan_block_call_takes(fake, args):
    assert _wan_route(fake, _wan(), _wan_args(**args)) == (["ksb_wan_block_forward"], [])


@pytest.mark.parametrize("args", [
    dict(dim=128), dict(dim=512), dict(text_dim=128), dict(text_dim=4096),  # other widths than the block's
    dict(e_shape=(1, 6, 1)), dict(e_shape=(1, 1, 256)), dict(e_shape=(2, 6, 256)),  # broadcast, or no modulation of these tokens
    dict(tokens=0), dict(text=0),
])
def test_wan_block_call_leaves_other_shapes_to_the_general_way(fake, args):
    called, general = _wan_route(fake, _wan(), _wan_args(**args))
    assert called == [] and general


def test_wan_block_general_way_broadcasts_the_modulation(fake):
    assert _wan_route(fake, _wan(), _wan_args(e_shape=(1, 1, 256)))[1] == [{(1, 256)}]
    assert _wan_route(fake, _wan(), _wan_args(e_shape=(6, 6, 1)))[1] == [{(6, 256)}]


@pytest.mark.parametrize("name", ["context", "e"])
def test_wan_block_call_refuses_tensors_of_another_device(fake, name):
    args = _wan_args()
    args[name] = args[name].to("meta")
    called, general = _wan_route(fake, _wan(), args)
    assert called == [] and general


def _qwen_route(fake, args, kw, blk=None):
    """Whether a call reaches the whole-block call; the general way ends at the stand-in, which refuses every kernel."""
    try:
        (blk or _qwen())(*args, **kw)
    except (RuntimeError, NotImplementedError, AssertionError, ValueError):
        pass
    return "ksb_qwen_block_forward" in [name for name, _ in fake.calls]


def test_qwen_block_call_takes(fake):
    assert _qwen_route(fake, *_qwen_args())


@pytest.mark.parametrize("change", ["image width", "text width", "both widths", "no text", "text elsewhere", "rows elsewhere"])
def test_qwen_block_call_leaves_other_tensors_to_the_general_way(fake, change):
    (img, txt, temb), kw = _qwen_args(text=0 if change == "no text" else 3)
    narrow = lambda t: t[..., :128]  # noqa: E731
    if change in ("image width", "both widths"):
        img, kw["mods"] = narrow(img), kw["mods"][:, :12 * 128]
    if change in ("text width", "both widths"):
        txt = narrow(txt)
    if change == "text elsewhere":
        txt = txt.to("meta")
    if change == "rows elsewhere":
        kw["mods"] = kw["mods"].to("meta")
    assert not _qwen_route(fake, (img, txt, temb), kw)


def test_qwen_block_call_leaves_rotary_embeddings_of_another_device(fake):
    args, kw = _qwen_args()
    kw.pop("img_grid")
    emb = torch.zeros(6, 64, dtype=torch.complex64), torch.zeros(3, 64, dtype=torch.complex64)
    assert _qwen_route(fake, args, dict(kw, image_rotary_emb=emb))
    fake.calls.clear()
    assert not _qwen_route(fake, args, dict(kw, image_rotary_emb=(emb[0].to("meta"), emb[1])))


@pytest.mark.parametrize("grid,whole", [((1, 1, 1024), True), ((1, 1, 1025), False), ((1, 1030, 1), False), ((1025, 1, 1), False)])
def test_qwen_grids_beyond_the_packed_positions_go_the_general_way(fake, grid, whole):
    """The folded rotation packs ten bits per axis; the general way rotates by its own kernel, without that limit."""
    args, kw = _qwen_args(tokens=2)
    assert _qwen_route(fake, args, dict(kw, img_grid=grid)) == whole


def test_qwen_rotary_embeddings_have_one_position(fake):
    args, kw = _qwen_args(tokens=1100)
    kw.pop("img_grid")
    emb = torch.zeros(1100, 64, dtype=torch.complex64), torch.zeros(3, 64, dtype=torch.complex64)
    assert _qwen_route(fake, args, dict(kw, image_rotary_emb=emb))


def _linear(k=64, n=48, **kw):
    from ksanadit_b200.linear import B200Fp8Linear
    return B200Fp8Linear.from_float(torch.nn.Linear(k, n), **kw)


def _linear_route(fake, lin, x, **kw):
    try:
        lin(x, **kw)
    except (RuntimeError, NotImplementedError, AssertionError):
        pass
    return "ksb_linear_forward" in [name for name, _ in fake.calls]


def _rows(*shape):
    return torch.zeros(*shape, dtype=torch.bfloat16)


def test_linear_call_takes(fake):
    from ksanadit_b200 import _lib
    assert _linear_route(fake, _linear(), _rows(4, 64))
    fake.calls.clear()
    assert _linear_route(fake, _linear(), _rows(2, 2, 64), epilogue=_lib.EPI_GATE_RESIDUAL, resid=_rows(2, 2, 48), gate=_rows(1, 48))


@pytest.mark.parametrize("resid,gate", [
    (_rows(4, 48).to("meta"), _rows(1, 48)), (_rows(4, 48), _rows(1, 48).to("meta")), (_rows(3, 48), _rows(1, 48)), (_rows(4, 96)[:, ::2], _rows(1, 48)),
])
def test_linear_call_refuses_a_residual_it_cannot_read(fake, resid, gate):
    """Of another device, with too few rows, or with columns apart."""
    from ksanadit_b200 import _lib
    with pytest.raises(_lib.KsanaB200Error):
        _linear()(_rows(4, 64), epilogue=_lib.EPI_GATE_RESIDUAL, resid=resid, gate=gate)
    assert not fake.calls


def test_linear_call_refuses_parameters_of_another_device(fake):
    lin = _linear()
    lin.scale_input = torch.nn.Parameter(torch.ones((), device="meta"), requires_grad=False)
    assert not _linear_route(fake, lin, _rows(4, 64))
    for name in ("weight", "bias"):
        lin = _linear()
        setattr(lin, name, torch.nn.Parameter(getattr(lin, name).to("meta"), requires_grad=False))
        assert not _linear_route(fake, lin, _rows(4, 64))


@pytest.mark.parametrize("change", ["weight rows", "weight columns", "bias", "scales"])
def test_linear_call_leaves_parameters_that_do_not_fit_to_the_general_way(fake, change):
    lin = _linear()
    if change.startswith("weight"):
        shape = (40, 64) if change == "weight rows" else (48, 32)
        lin.weight = torch.nn.Parameter(torch.zeros(shape).to(torch.float8_e4m3fn), requires_grad=False)
    if change == "bias":
        lin.bias = torch.nn.Parameter(torch.zeros(40, dtype=torch.bfloat16), requires_grad=False)
    if change == "scales":
        lin._w_scale_vec = torch.ones(40)
    assert not _linear_route(fake, lin, _rows(4, 64))


# ---------------------------------------------------------------------------------------------- parameters of the blocks


def _replace(module, name, value):
    setattr(module, name, torch.nn.Parameter(value, requires_grad=False))


WAN_CHANGES = {
    "modulation rows": lambda b: _replace(b, "modulation", torch.zeros(1, 5, 256, dtype=torch.bfloat16)),
    "norm elsewhere": lambda b: _replace(b.self_attn.norm_q, "weight", torch.ones(256, device="meta")),
    "projection width": lambda b: setattr(b.self_attn, "o", _linear(256, 128)),
    "projection depth": lambda b: setattr(b.cross_attn, "q", _linear(128, 256)),
    "hidden width": lambda b: b.ffn.__setitem__(2, _linear(384, 256)),
    "modulation elsewhere": lambda b: _replace(b, "modulation", b.modulation.to("meta")),
}


@pytest.mark.parametrize("change", WAN_CHANGES)
def test_wan_block_call_leaves_parameters_that_do_not_fit(fake, change):
    blk = _wan()
    WAN_CHANGES[change](blk)
    called, general = _wan_route(fake, blk, _wan_args())
    assert called == [] and general


QWEN_CHANGES = {
    "norm width": lambda b: _replace(b.attn.norm_k, "weight", torch.ones(64)),
    "norm elsewhere": lambda b: _replace(b.attn.norm_added_k, "weight", torch.ones(128, device="meta")),
    "projection width": lambda b: setattr(b.attn, "to_add_out", _linear(256, 128)),
    "projection depth": lambda b: setattr(b.attn, "to_qkv", _linear(128, 768)),
    "hidden width": lambda b: setattr(b.img_mlp.net[0], "proj", _linear(256, 384)),
    "streams of other hidden widths": lambda b: (setattr(b.txt_mlp.net[0], "proj", _linear(256, 384)), b.txt_mlp.net.__setitem__(2, _linear(384, 256))),
}


@pytest.mark.parametrize("change", QWEN_CHANGES)
def test_qwen_block_call_leaves_parameters_that_do_not_fit(fake, change):
    blk = _qwen()
    QWEN_CHANGES[change](blk)
    assert not _qwen_route(fake, *_qwen_args(), blk)


@pytest.mark.parametrize("which", [0, 1, 2])
def test_tile_lists_of_another_device_are_refused(fake, monkeypatch, which):
    """A list on the host, which is no GPU tensor, must not reach the library."""
    from ksanadit_b200 import _lib, native
    lists = [torch.tensor([0, 1], dtype=torch.int32), torch.tensor([3], dtype=torch.int32), torch.tensor([0], dtype=torch.int32)]
    assert native.tile_lists(*lists, 1)[0] is not None
    host = lists[which]
    monkeypatch.setattr(torch.Tensor, "is_cuda", property(lambda t: t is not host), raising=False)
    with pytest.raises(_lib.KsanaB200Error):
        native.tile_lists(*lists, 1)


def test_context_cache_keeps_nothing_of_a_refused_call(fake):
    from ksanadit_b200 import _lib
    blk, args = _wan(cache_context=True), _wan_args()
    fake.rc = -1
    with pytest.raises(_lib.KsanaB200Error):
        blk(**args)
    fake.rc = 1
    for _ in range(2):
        blk(**args)
    assert [seen["compute_context"] for _, seen in fake.calls] == [1, 1, 0]  # refused; filled; reused


def test_context_cache_serves_both_ways_of_a_block(fake):
    """The whole-block call keeps one buffer, the kernels one by one keep four tensors; a block may change between them."""
    from ksanadit_b200 import native
    fake.rc = 0
    blk, args = _wan(cache_context=True), _wan_args()

    def general():
        blk._native = lambda: native.Descriptor()
        blk(**args)
        del blk._native

    computed = []
    for run in (lambda: blk(**args), general) * 2:
        n = len(fake.calls)
        run()
        # the context's V quantiser, or the whole call told to compute the context (self-attention's V is one quantiser more)
        computed.append(sum(seen.get("compute_context", 0) + (name == "ksb_sage_quant_v_fp8") for name, seen in fake.calls[n:]))
    assert computed == [1, 2, 0, 1]
    blk.random_init(1)
    assert blk._ctx_cache is None  # both forms go with the weights


# ---------------------------------------------------------------------------------------------- modules a user changes


class _Wrapped(torch.nn.Module):
    """A module around a Linear, as adapters put there."""

    def __init__(self, inner):
        super().__init__()
        self.inner = inner
        self.calls = 0

    def forward(self, x):
        self.calls += 1
        return self.inner(x)


def test_wan_block_calls_a_wrapped_context_projection(fake):
    fake.rc = 0
    blk = _wan()
    blk(**_wan_args())
    blk.cross_attn.k, blk.cross_attn.v = _Wrapped(blk.cross_attn.k), _Wrapped(blk.cross_attn.v)
    blk(**_wan_args())
    assert blk.cross_attn.k.calls == blk.cross_attn.v.calls == 1


@pytest.mark.parametrize("register", ["register_forward_hook", "register_forward_pre_hook"])
def test_wan_block_runs_hooks_of_the_context_projections(fake, register):
    fake.rc = 0
    blk, seen = _wan(), []
    blk(**_wan_args())
    handle = getattr(blk.cross_attn.v, register)(lambda *a: seen.append(1))
    blk(**_wan_args())
    assert seen == [1]
    handle.remove()
    n = len(fake.calls)
    blk(**_wan_args())
    assert seen == [1] and [name for name, _ in fake.calls[n:]] == ["ksb_wan_block_forward"]


def test_wan_block_keeps_to_a_projection_with_a_forward_of_its_own(fake):
    from ksanadit_b200.linear import B200Fp8Linear
    fake.rc = 0
    calls = []

    class Own(B200Fp8Linear):
        def forward(self, x, **kw):
            calls.append(1)
            return super().forward(x, **kw)

    blk = _wan()
    blk.cross_attn.k.__class__ = Own
    blk(**_wan_args())
    assert calls == [1]
    blk = _wan()
    plain = blk.cross_attn.k.forward
    blk.cross_attn.k.forward = lambda x: (calls.append(2), plain(x))[1]
    blk(**_wan_args())
    assert calls == [1, 2]


class _Same(torch.nn.Module):
    def forward(self, w):
        return w


def test_linear_with_a_parametrised_weight_goes_the_general_way(fake):
    fake.rc = 0
    lin = _linear()
    torch.nn.utils.parametrize.register_parametrization(lin, "weight", _Same(), unsafe=True)
    assert lin(_rows(4, 64)).shape == (4, 48)
    assert [name for name, _ in fake.calls] == ["ksb_quant_fp8_rowwise", "ksb_fp8_gemm"]


def test_linear_reads_parameters_kept_as_plain_tensors(fake):
    """A weight or bias that is no Parameter any more, and an activation scale set as a plain tensor."""
    fake.rc = 0
    for name in ("weight", "bias"):
        lin = _linear()
        lin(_rows(4, 64))
        value = getattr(lin, name).data
        delattr(lin, name)
        setattr(lin, name, value)
        fake.calls.clear()
        lin(_rows(4, 64))
        assert [n for n, _ in fake.calls] == ["ksb_quant_fp8_rowwise", "ksb_fp8_gemm"], name
    lin = _linear()
    lin.scale_input = torch.full((), 0.5)
    fake.calls.clear()
    lin(_rows(4, 64))
    assert fake.calls == [("ksb_linear_forward", dict(static=True))]


def test_wan_block_honours_a_context_projections_activation_scale(fake):
    for make in (lambda t: t, lambda t: torch.nn.Parameter(t, requires_grad=False)):
        fake.rc = 0
        blk = _wan()
        blk(**_wan_args())
        blk.cross_attn.v.scale_input = make(torch.full((), 0.5))
        fake.calls.clear()
        blk(**_wan_args())
        assert "ksb_wan_block_forward" not in [name for name, _ in fake.calls]


def test_modules_saved_before_there_were_descriptors(fake):
    """A module pickled whole by an earlier version comes back without the attribute that holds its descriptor."""
    lin, wan, qwen = _linear(), _wan(), _qwen()
    for m in [lin, wan, qwen] + [c for b in (wan, qwen) for c in b.modules()]:
        m.__dict__.pop("_call", None)
    assert _linear_route(fake, lin, _rows(4, 64))
    assert _wan_route(fake, wan, _wan_args())[0][-1] == "ksb_wan_block_forward"
    assert _qwen_route(fake, *_qwen_args(), qwen)
