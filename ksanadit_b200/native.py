"""Host side of the whole-operator calls of the C ABI (ksb_linear_forward, ksb_sage_attention, ksb_*_block_forward).

A call hands the library one descriptor of the module's parameters, one of the call's tensors and one workspace, and the
library queues all kernels.  The descriptor of a module is built once and checked on every call against the parameters it
was built from: a parameter that was replaced, or whose storage was, makes it be rebuilt.
"""

from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import os
import sysconfig
import warnings
from ctypes import c_float, c_int, c_int64, c_void_p

import torch

from . import _lib


class Linear(ctypes.Structure):
    _fields_ = [("w", c_void_p), ("w_scale", c_void_p), ("bias", c_void_p), ("N", c_int64), ("K", c_int64)]


class TileLists(ctypes.Structure):
    _fields_ = [("offsets", c_void_p), ("entries", c_void_p), ("order", c_void_p), ("pairs", c_int)]


class WanBlock(ctypes.Structure):
    _fields_ = [("dim", c_int64), ("heads", c_int64), ("eps", c_float)] + \
        [(n, Linear) for n in ("qkv", "o", "cross_q", "cross_k", "cross_v", "cross_o", "ffn_up", "ffn_down")] + \
        [(n, c_void_p) for n in ("norm_q", "norm_k", "cross_norm_q", "cross_norm_k", "norm3_w", "norm3_b", "modulation")]


class WanCall(ctypes.Structure):
    _fields_ = [(n, c_void_p) for n in ("x", "e", "context", "out", "context_operands")] + \
        [(n, c_int64) for n in ("batch", "tokens", "text", "e_rows")] + [("rope_table", c_void_p), ("lists", c_void_p)] + \
        [(n, c_int) for n in ("dtype", "e_dtype", "compute_context", "rope_len", "rope_nf", "rope_nh", "grid_f", "grid_h", "grid_w")] + \
        [("premul", c_float)]


class QwenBlock(ctypes.Structure):
    _fields_ = [("dim", c_int64), ("heads", c_int64), ("eps", c_float)] + \
        [(n, Linear) for n in ("img_qkv", "txt_qkv", "img_out", "txt_out", "img_up", "txt_up", "img_down", "txt_down")] + \
        [(n, c_void_p) for n in ("img_norm_q", "img_norm_k", "txt_norm_q", "txt_norm_k")]


class QwenCall(ctypes.Structure):
    _fields_ = [(n, c_void_p) for n in ("img", "txt", "mods", "mod_index", "out")] + [(n, c_int64) for n in ("mod_rows", "img_tokens", "text_tokens")] + \
        [(n, c_void_p) for n in ("img_rope", "txt_rope")] + \
        [(n, c_int) for n in ("img_rope_len", "txt_rope_len", "rope_nf", "rope_nh", "img_f", "img_h", "img_w", "img_diag", "txt_grid", "dtype")] + \
        [("premul", c_float)]


# the enums of the header
(WAN_PRE, WAN_QKV, WAN_SELF_PREP, WAN_SELF_ATTN, WAN_SELF_POST, WAN_O, WAN_CROSS_PRE, WAN_CROSS_Q, WAN_CROSS_PREP, WAN_CROSS_ATTN,
 WAN_CROSS_POST, WAN_CROSS_O, WAN_FFN_PRE, WAN_FFN_UP, WAN_FFN_MID, WAN_FFN_DOWN) = range(16)
(QWEN_PRE, QWEN_QKV, QWEN_PREP, QWEN_ATTN, QWEN_POST, QWEN_OUT, QWEN_MLP_PRE, QWEN_MLP_UP, QWEN_MLP_MID, QWEN_MLP_DOWN) = range(10)

MAX_GRID_AXIS = 1024  # positions per axis that the quantisers' folded rotation can decode (ten bits each)
DTYPES = {torch.bfloat16: _lib.BF16, torch.float16: _lib.FP16, torch.float32: 2}

_raw_stream = torch._C._cuda_getCurrentRawStream if hasattr(torch._C, "_cuda_getCurrentRawStream") else None


def stream() -> int:
    """The current stream's handle, without building a Stream object."""
    if _raw_stream is None:
        return torch.cuda.current_stream().cuda_stream
    return _raw_stream(torch.cuda.current_device())


def queued(rc: int, what: str) -> int:
    """Kernels queued by a whole-operator call; raises on a rejected one."""
    if rc < 0:
        _lib.check(rc, what)
    return rc


def workspace(nbytes: int, device) -> torch.Tensor:
    return torch.empty(nbytes, dtype=torch.uint8, device=device)


def _layout(t):
    return t.data_ptr(), t.dtype, t.shape, t.stride()


class Watch:
    """What a descriptor was built from: modules by identity, tensors by the place, type and layout they have now.
    ``current`` is false once a name holds another module or a tensor differs in any of these (the allocator may hand a
    replaced tensor's address to its successor, so the address alone would not do)."""

    def __init__(self):
        self.entries = []

    def tensor(self, namespace, name):
        t = namespace.get(name)
        self.entries.append((namespace, name, t, None if t is None else _layout(t)))
        return t

    def module(self, parent, name):
        m = parent._modules.get(name)
        self.entries.append((parent._modules, name, m, None))
        return m

    def linear(self, parent, name, dtype):
        """Descriptor of a B200Fp8Linear child, or None when the fused path cannot read it as it is (a bias of another
        type; another module, or one that multiplies in its own way)."""
        from .linear import B200Fp8Linear
        lin = self.module(parent, name)
        stock = lin is not None and B200Fp8Linear.is_stock(lin, "forward_quantized", "forward_quantized_rowstats", "weight_scale_vector")
        return self.linear_of(lin, dtype) if stock else None

    def linear_of(self, lin, dtype):
        """Descriptor of a B200Fp8Linear, or None: see ``linear``; also where a weight or a bias is computed, or kept as a plain
        tensor, and not one of the module's parameters."""
        if lin._parameters.get("weight") is None or "bias" not in lin._parameters:
            return None
        vec = lin.weight_scale_vector()
        w, b = self.tensor(lin._parameters, "weight"), self.tensor(lin._parameters, "bias")
        self.tensor(lin.__dict__, "_w_scale_vec")
        shape = (lin.out_features, lin.in_features)
        if w.dtype != torch.float8_e4m3fn or w.shape != shape or not w.is_contiguous() or not w.is_cuda:
            return None
        if vec.shape != shape[:1] or vec.device != w.device:
            return None
        if b is not None and (b.dtype != dtype or b.shape != shape[:1] or not b.is_contiguous() or b.device != w.device):
            return None
        return Linear(w.data_ptr(), vec.data_ptr(), None if b is None else b.data_ptr(), w.shape[0], w.shape[1])

    def one_device(self) -> bool:
        """Whether all tensors are on the same device."""
        return len({obj.device for _, _, obj, layout in self.entries if layout is not None}) == 1

    def current(self) -> bool:
        for namespace, name, obj, layout in self.entries:
            now = namespace.get(name)
            if now is not obj or (layout is not None and _layout(now) != layout):
                return False
        return True


def have_shapes(linears, shapes) -> bool:
    """Whether each Linear's descriptor is there and of the (rows, columns) the block's widths ask for."""
    return all(lin is not None and (lin.N, lin.K) == shape for lin, shape in zip(linears, shapes, strict=True))


class Descriptor:
    """A module's descriptor with what it was built from.  Copies and pickles of the module start without one."""

    __slots__ = ("watch", "desc", "config", "address", "sizes", "host")

    def __init__(self, watch=None, desc=None, config=None):
        self.watch, self.desc, self.config = watch, desc, config
        self.address = None if desc is None else ctypes.addressof(desc)
        self.sizes = {}  # workspace bytes per call shape
        self.host = None  # the call in C++ (linear_call); False: tried, and there is none

    def __reduce__(self):
        return Descriptor, ()

    def valid_for(self, config) -> bool:
        """``config``: the plain values (types, sizes, eps) that went into the descriptor besides the tensors."""
        return self.watch is not None and self.config == config and self.watch.current()


_host = None  # False: tried, and it is not there


def host_path() -> str:
    """Where the extension for this torch and this Python lies: built for another one it is not looked for."""
    tag = f"torch{torch.__version__}-{sysconfig.get_config_var('SOABI')}"
    return os.path.join(os.path.dirname(os.path.abspath(__file__)), "lib", f"ksana_b200_host.{tag}.so")


def host_module():
    """The extension with the single calls' C++ side, or None where it is not built or does not load (said once): every call then
    goes the general way, through the same kernels."""
    global _host
    if _host is None:
        name, path = "ksana_b200_host", host_path()
        try:
            loader = importlib.machinery.ExtensionFileLoader(name, path)
            module = importlib.util.module_from_spec(importlib.util.spec_from_file_location(name, path, loader=loader))
            loader.exec_module(module)
            _host = module
        except ImportError as e:
            _host = False
            warnings.warn(f"single calls go through Python, about 10 us slower: {e}; `python -m ksanadit_b200.build` builds the extension")
    return _host or None


def linear_call(lin, call, dtype, device, quantize):
    """The C++ call of a Linear with descriptor ``call``; False where it has none, is not on a GPU, or was built from what a LinearCall
    cannot watch (a parameter of a tensor subclass, say): its calls go the general way."""
    if call.address is None or device.type != "cuda" or host_module() is None:
        return False
    from . import ops
    lib = _lib.load()
    place = lambda fn: ctypes.cast(fn, c_void_p).value  # noqa: E731
    try:
        return host_module().LinearCall(call.watch.entries, lin._parameters, call.address, dtype, device.index, quantize, vars(ops), queued,
                                        place(lib.ksb_linear_forward), place(lib.ksb_linear_workspace))
    except TypeError:
        return False


def tile_lists(offsets, entries, order, n_blocks):
    """(descriptor, tensors to keep alive) of a block-sparse call's lists, merged per pair of Q blocks where that pays."""
    from . import ops
    if offsets is None:
        return None, None
    ops._cuda(offsets, entries, order)
    if offsets.numel() != n_blocks + 1 or offsets.dtype != torch.int32 or entries.dtype != torch.int32:
        raise _lib.KsanaB200Error(f"tile_offsets must hold ceil(Lq/128)+1 = {n_blocks + 1} int32 values, got {offsets.numel()}")
    if order is not None and (order.numel() != n_blocks or order.dtype != torch.int32):
        raise _lib.KsanaB200Error(f"tile_order must hold ceil(Lq/128) = {n_blocks} int32 values, got {order.numel()}")
    pairs = 0
    if _lib.load().ksb_attn_dual_mode(-1) == 1:
        merged = ops._pair_lists(offsets, entries, order is not None)
        if merged is not None:
            offsets, entries, order = merged
            pairs = 1
    keep = (offsets, entries, order)
    return TileLists(offsets.data_ptr(), entries.data_ptr(), None if order is None else order.data_ptr(), pairs), keep
