"""What this package is used for, as measurable cases: the calls a denoise step is made of, from one modulation row to a
full block at 75 600 tokens.

Five kinds of calls, each through the entry point a model uses:

* ``linear``     the FP8 Linear (``B200Fp8Linear.from_float`` / ``b200_fp8_ops``), per-token or static activation scales
* ``attention``  ``KsanaAttentionOp`` with the Sage backend, self- or cross-attention
* ``radial``     ``KsanaAttentionOp`` with the radial block-sparse backend past its dense steps and blocks
* ``wan``        ``B200WanDenoiseStep``: fused Wan blocks, one sample or a cond / uncond batch
* ``qwen``       ``B200QwenDenoiseStep``: fused Qwen-Image dual-stream blocks, optionally with per-token modulation
                 (``zero_cond_t``, the image-editing models)

Activations are N(0, 1) with one channel in a hundred scaled by 20, weights N(0, 0.02), K and the Q / K projections carry
a per-channel offset of N(0, 0.5) (what K smoothing removes), adaLN modulation is N(0, 0.1).
"""

import math

import torch

from ksanadit_b200.attention import KsanaAttentionOp
from ksanadit_b200.config import KsanaAttentionBackend, KsanaAttentionConfig, KsanaRadialSageAttentionConfig
from ksanadit_b200.linear import B200Fp8Linear, b200_fp8_ops, quantize_weight_per_channel
from ksanadit_b200.qwen_block import B200QwenBlock, B200QwenDenoiseStep
from ksanadit_b200.wan_block import B200WanDenoiseStep

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
HEAD = 128
# block widths: (dim, heads, FFN)
WAN_SMALL, WAN_LARGE = (1536, 12, 8960), (5120, 40, 13824)
QWEN = (3072, 24, 12288)
WIDTHS = (1536, 3072, 4608, 5120, 8960, 9216, 12288, 13824, 15360)
MAX_TOKENS = 75600


# ---------------------------------------------------------------------------------------------- cases


def _linear(m, k, n, dtype="bf16", bias=True, static=False):
    return dict(kind="linear", m=m, k=k, n=n, dtype=dtype, bias=bias, static=static)


def _attention(batch, lq, lk, heads, dtype="bf16"):
    return dict(kind="attention", batch=batch, lq=lq, lk=lk, heads=heads, dtype=dtype)


def _radial(frames, lat_h, lat_w, heads, block=128, decay=0.02, extra=0):
    return dict(kind="radial", frames=frames, lat_h=lat_h, lat_w=lat_w, heads=heads, block=block, decay=decay, extra=extra)


def _wan(model, layers, frames, h, w, text=512, batch=1, dtype="bf16"):
    dim, heads, ffn = model
    return dict(kind="wan", layers=layers, dim=dim, heads=heads, ffn=ffn, frames=frames, h=h, w=w, text=text, batch=batch, dtype=dtype)


def _qwen(layers, h, w, text, edit=False):
    dim, heads, ffn = QWEN
    return dict(kind="qwen", layers=layers, dim=dim, heads=heads, ffn=ffn, h=h, w=w, text=text, edit=edit)


def listed():
    return [
        # one row: the modulation Linear of a Qwen-Image stream, once per block and step; streams its weight
        dict(_linear(1, 3072, 18432), name="linear_modulation_row"),
        # the text K / V projection of the small Wan model in fp16, the smallest Linear of a step
        dict(_linear(512, 1536, 1536, dtype="fp16"), name="linear_text_projection"),
        # FFN up-projection of the large Wan model at 480p x 81 frames
        dict(_linear(32760, 5120, 13824), name="linear_ffn_480p"),
        # self-attention of the small Wan model on one 480p frame
        dict(_attention(1, 1560, 1560, 12), name="attention_one_frame"),
        # cross-attention of a 480p x 81-frame video to 512 text tokens, large Wan model
        dict(_attention(1, 32760, 512, 40), name="attention_cross_480p"),
        # joint text + image attention of a 1328 x 1328 Qwen-Image picture: a ragged length, in fp16
        dict(_attention(1, 7145, 7145, 24, dtype="fp16"), name="attention_joint_ragged"),
        # radial block-sparse self-attention, 21 latent frames of 64 x 96, with the backend's default decay
        dict(_radial(21, 64, 96, 40), name="radial_81_frames"),
        # two blocks of the small Wan model on one 480p frame (1560 tokens): launches and latency
        dict(_wan(WAN_SMALL, 2, 1, 30, 52), name="wan_small_one_frame"),
        # a block of the small Wan model at 480p x 81 frames, cond and uncond sample in one batch
        dict(_wan(WAN_SMALL, 1, 21, 30, 52, batch=2), name="wan_small_480p_cfg"),
        # a block of the large Wan model at 720p x 81 frames: the largest call
        dict(_wan(WAN_LARGE, 1, 21, 45, 80), name="wan_large_720p"),
        # two dual-stream blocks on a 512 x 512 picture being edited, a short ragged prompt
        dict(_qwen(2, 32, 32, 77, edit=True), name="qwen_edit_512"),
        # two dual-stream blocks on a 1328 x 1328 picture
        dict(_qwen(2, 83, 83, 256), name="qwen_1328"),
    ]


def _log_uniform(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _width(rng):
    return rng.choice(WIDTHS) if rng.random() < 0.75 else 16 * _log_uniform(rng, 4, 864)


def draw(rng):
    kind = rng.choice(("linear", "linear", "linear", "attention", "attention", "attention", "radial", "wan", "wan", "wan", "qwen", "qwen"))
    dtype = rng.choice(("bf16", "bf16", "fp16"))
    if kind == "linear":
        return _linear(_log_uniform(rng, 1, MAX_TOKENS), _width(rng), _width(rng), dtype, rng.random() < 0.8, rng.random() < 0.2)
    if kind == "attention":
        lq = _log_uniform(rng, 64, 40000)
        lk = lq if rng.random() < 0.5 else _log_uniform(rng, 32, 1024)
        return _attention(rng.choice((1, 1, 2)), lq, lk, rng.choice((3, 5, 12, 24, 40)), dtype)
    if kind == "radial":
        return _radial(rng.randint(2, 21), 16 * rng.randint(1, 5), 16 * rng.randint(1, 6), rng.choice((12, 40)), rng.choice((64, 128)),
                       rng.choice((0.02, 0.2)), rng.choice((0, 0, rng.randint(1, 300))))
    if kind == "wan":
        batch = rng.choice((1, 1, 2))
        tokens = _log_uniform(rng, 200, MAX_TOKENS // batch)
        frames = rng.choice([f for f in (1, 3, 5, 9, 13, 21) if f * 64 <= tokens])
        h = max(1, int(math.sqrt(tokens / frames * rng.uniform(0.5, 1.0))))
        w = max(1, tokens // (frames * h))
        return _wan(rng.choice((WAN_SMALL, WAN_LARGE)), 1, frames, h, w, rng.choice((512, 512, rng.randint(16, 512))), batch, dtype)
    return _qwen(rng.randint(1, 2), rng.randint(16, 96), rng.randint(16, 96), _log_uniform(rng, 8, 512), rng.random() < 0.3)


# ---------------------------------------------------------------------------------------------- inputs


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _activations(g, *shape, dtype=torch.bfloat16):
    x = torch.randn(*shape, device="cuda", generator=g, dtype=dtype)
    width = shape[-1]
    loud = torch.randperm(width, device="cuda", generator=g)[: max(1, width // 100)]
    x[..., loud] *= 20
    return x


def _prepare_linear(c, g):
    dtype = DTYPES[c["dtype"]]
    x = _activations(g, 1, c["m"], c["k"], dtype=dtype)
    dense = torch.nn.Linear(c["k"], c["n"], bias=c["bias"], device="meta")
    dense.weight = torch.nn.Parameter(torch.randn(c["n"], c["k"], device="cuda", generator=g) * 0.02, requires_grad=False)
    if c["bias"]:
        dense.bias = torch.nn.Parameter(torch.randn(c["n"], device="cuda", generator=g) * 0.02, requires_grad=False)
    if not c["static"]:
        return dict(call=B200Fp8Linear.from_float(dense, dtype=dtype), args=(x,), kwargs={})
    # a scaled-FP8 checkpoint with one scale per tensor, the activations' included
    lin = b200_fp8_ops(scale_input=True)(c["k"], c["n"], bias=c["bias"], device="cuda", dtype=dtype)
    scale = dense.weight.abs().max() / 448
    sd = {"weight": (dense.weight / scale).to(torch.float8_e4m3fn), "scale_weight": scale,
          "scale_input": torch.tensor(100.0 / 448, device="cuda")}
    if c["bias"]:
        sd["bias"] = dense.bias.to(dtype)
    lin.load_state_dict(sd)
    return dict(call=lin, args=(x,), kwargs={})


def _qkv(c, g, batch, lq, lk, heads, dtype):
    q = torch.randn(batch, lq, heads, HEAD, device="cuda", generator=g, dtype=dtype)
    k = torch.randn(batch, lk, heads, HEAD, device="cuda", generator=g, dtype=dtype)
    k += 0.5 * torch.randn(1, 1, heads, HEAD, device="cuda", generator=g, dtype=dtype)
    v = torch.randn(batch, lk, heads, HEAD, device="cuda", generator=g, dtype=dtype)
    return q, k, v


def _prepare_attention(c, g):
    op = KsanaAttentionOp(c["heads"], HEAD, attention_config=KsanaAttentionConfig(backend=KsanaAttentionBackend.SAGE_ATTN))
    qkv = _qkv(c, g, c["batch"], c["lq"], c["lk"], c["heads"], DTYPES[c["dtype"]])
    return dict(call=op, args=qkv, kwargs=dict(k_lens=torch.tensor([c["lk"]] * c["batch"])))


def _radial_tokens(c):
    video = c["frames"] * (c["lat_h"] // 2) * (c["lat_w"] // 2)
    return video, video + c["extra"]


def _prepare_radial(c, g):
    video, tokens = _radial_tokens(c)
    cfg = KsanaRadialSageAttentionConfig(dense_blocks_num=1, dense_attn_steps=1, decay_factor=c["decay"], block_size=c["block"])
    op = KsanaAttentionOp(c["heads"], HEAD, attention_config=cfg)
    kwargs = dict(k_lens=torch.tensor([video]), latent_shape=[1, 16, c["frames"], c["lat_h"], c["lat_w"]], step_iter=5, block_id=3)
    return dict(call=op, args=_qkv(c, g, 1, tokens, tokens, c["heads"], torch.bfloat16), kwargs=kwargs)


def _prepare_wan(c, g):
    dtype = DTYPES[c["dtype"]]
    tokens = c["frames"] * c["h"] * c["w"]
    step = B200WanDenoiseStep(c["layers"], c["dim"], c["ffn"], c["heads"], device="cuda", dtype=dtype, seed=g.initial_seed() % (1 << 20))
    x = _activations(g, c["batch"], tokens, c["dim"], dtype=dtype)
    e = (torch.randn(c["batch"], 1, 6, c["dim"], device="cuda", generator=g) * 0.1).to(dtype)
    context = torch.randn(c["batch"], c["text"], c["dim"], device="cuda", generator=g, dtype=dtype)
    grid = torch.tensor([[c["frames"], c["h"], c["w"]]] * c["batch"])
    return dict(call=step, args=(x, e, grid, context), kwargs={})


def _prepare_qwen(c, g):
    seed = g.initial_seed() % (1 << 20)
    blocks = [B200QwenBlock(c["dim"], c["heads"], c["ffn"], zero_cond_t=c["edit"]).random_init(seed + i) for i in range(c["layers"])]
    tokens = c["h"] * c["w"]
    img = _activations(g, 1, tokens, c["dim"])
    txt = _activations(g, 1, c["text"], c["dim"])
    temb = torch.randn(2 if c["edit"] else 1, c["dim"], device="cuda", generator=g, dtype=torch.bfloat16)
    kwargs = dict(img_grid=(1, c["h"], c["w"]))
    if c["edit"]:  # the second half of the image tokens belongs to the reference picture
        kwargs["modulate_index"] = (torch.arange(tokens, device="cuda") >= tokens // 2).long()[None]
    return dict(call=B200QwenDenoiseStep(blocks), args=(img, txt, temb), kwargs=kwargs)


def prepare(case, seed):
    make = {"linear": _prepare_linear, "attention": _prepare_attention, "radial": _prepare_radial, "wan": _prepare_wan, "qwen": _prepare_qwen}
    return make[case["kind"]](case, _generator(seed))


def run(state):
    with torch.no_grad():
        return state["call"](*state["args"], **state["kwargs"])


# ---------------------------------------------------------------------------------------------- floors


def _kept_share(c):
    """Share of the score tiles that the radial mask of the case keeps."""
    from ksanadit_b200 import radial_mask
    video, tokens = _radial_tokens(c)
    return float(radial_mask.build_radial_tile_mask(tokens, video, c["frames"], c["block"], c["decay"]).mean()) if tokens >= c["block"] else 1.0


def work(case):
    c = case
    if c["kind"] == "linear":
        m, k, n = c["m"], c["k"], c["n"]
        return dict(bytes=2 * m * k + n * k + 2 * m * n + 4 * n, flops=2 * m * n * k)
    if c["kind"] == "attention":
        return dict(bytes=4 * c["batch"] * c["heads"] * HEAD * (c["lq"] + c["lk"]), flops=4 * c["batch"] * c["heads"] * c["lq"] * c["lk"] * HEAD)
    if c["kind"] == "radial":
        tokens = _radial_tokens(c)[1]
        return dict(bytes=8 * c["heads"] * HEAD * tokens, flops=4 * c["heads"] * tokens * tokens * HEAD * _kept_share(c))
    d, f = c["dim"], c["ffn"]
    if c["kind"] == "wan":
        tokens, text, b = c["frames"] * c["h"] * c["w"], c["text"], c["batch"]
        weights = 8 * d * d + 2 * d * f
        flops = 2 * tokens * (6 * d * d + 2 * d * f) + 4 * text * d * d + 4 * tokens * (tokens + text) * d
        return dict(bytes=c["layers"] * weights + b * (4 * tokens * d + 2 * text * d), flops=c["layers"] * b * flops)
    tokens, text = c["h"] * c["w"], c["text"]
    stream = 4 * d * d + 2 * d * f  # weights of one stream besides its modulation
    rows = 2 if c["edit"] else 1
    flops = 2 * (tokens + text) * stream + 2 * rows * 12 * d * d + 4 * (tokens + text) ** 2 * d
    return dict(bytes=c["layers"] * (2 * stream + 12 * d * d) + 4 * (tokens + text) * d, flops=c["layers"] * flops)


def tolerance(case):
    # A Linear's quantised operands are determined bit for bit; what is left is the fp32 summation order and the rounding
    # of the 16-bit result.  Attention rounds its probabilities to e4m3 (steps of 2^-3 of a value) against a running
    # reference point, and a block quantises its activations to e4m3 again behind every normalisation, where one 16-bit
    # rounding more or less moves a value by a whole step.
    return {"rel": 5e-3} if case["kind"] == "linear" else {"rel": 2e-2}
