"""The Linear's single call in C++: it hands back what is not a plain call, follows the module's parameters, and does not keep a
module alive."""

import ctypes
import gc
import weakref

import pytest
import torch


def _linear(device, k=64, n=48, **kw):
    from ksanadit_b200.linear import B200Fp8Linear
    return B200Fp8Linear.from_float(torch.nn.Linear(k, n, device=device), **kw)


def _call(lin, dtype=torch.bfloat16):
    """The C++ call of a module on the CPU; it takes tensors of GPU 0 only."""
    from ksanadit_b200 import native, ops
    from ksanadit_b200.linear import _QUANTIZE_INPUT
    watch = native.Watch()
    watch.linear_of(lin, dtype)
    desc = native.Linear(None, None, None, lin.out_features, lin.in_features)
    call = native.Descriptor(watch, desc, None)
    call.host = native.host_module().LinearCall(watch.entries, lin._parameters, ctypes.addressof(desc), dtype, 0, _QUANTIZE_INPUT, vars(ops),
                                                native.queued, 0, 0)
    lin._call = call
    return call.host


def test_tensors_elsewhere_are_handed_back():
    lin = _linear("cpu")
    host = _call(lin)
    for x in (torch.zeros(2, 64, dtype=torch.bfloat16), torch.zeros(2, 64, dtype=torch.bfloat16, device="meta"), None, 3):
        assert host.run(lin, x, 0) is None


def test_module_with_a_call_is_collected():
    lin = _linear("cpu")
    _call(lin)
    gone = weakref.ref(lin)
    del lin
    gc.collect()
    assert gone() is None


def test_arguments_are_checked():
    from ksanadit_b200 import native
    lin = _linear("cpu")
    host = _call(lin)
    with pytest.raises(TypeError):
        host.run(lin)
    with pytest.raises(TypeError):
        native.host_module().LinearCall([], {}, 0, "bf16", 0, None, {}, None, 0, 0)


class _Sub(torch.Tensor):
    pass


class _SubParameter(torch.nn.Parameter):
    pass


def _subclassed(lin, name):
    """The module with one parameter of a tensor subclass."""
    if name == "scale_weight":
        lin.scale_weight = torch.nn.Parameter(lin.scale_weight.data.as_subclass(_Sub), requires_grad=False)
        lin._w_scale_vec = None  # made anew, and of the subclass
    else:
        setattr(lin, name, _SubParameter(getattr(lin, name).data, requires_grad=False))
    return lin


@pytest.mark.parametrize("name", ["weight", "bias", "scale_weight"])
def test_module_with_a_tensor_subclass_has_no_call(name):
    from ksanadit_b200 import native
    from ksanadit_b200.linear import _QUANTIZE_INPUT

    def call_of(lin):
        watch = native.Watch()
        watch.linear_of(lin, torch.bfloat16)
        call = native.Descriptor(watch, native.Linear(None, None, None, lin.out_features, lin.in_features), None)
        return native.linear_call(lin, call, torch.bfloat16, torch.device("cuda", 0), _QUANTIZE_INPUT)

    assert call_of(_linear("cpu"))
    assert call_of(_subclassed(_linear("cpu"), name)) is False


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["weight", "bias", "scale_weight"])
def test_module_with_a_tensor_subclass_goes_the_general_way(name):
    from ksanadit_b200 import _lib
    lin = _linear("cuda", 256, 128)
    x = torch.randn(3, 256, device="cuda", dtype=torch.bfloat16)
    ref = lin(x)
    _subclassed(lin, name)
    for _ in range(4):
        assert torch.equal(lin(x), ref)
    assert lin._call.host is False
    _lib.assert_device_ok()


@pytest.mark.gpu
def test_plain_calls_are_taken_and_others_go_the_general_way():
    from ksanadit_b200 import _lib, ops
    from ksanadit_b200.linear import B200Fp8Linear
    lin = _linear("cuda", 256, 128)
    x = torch.randn(2, 3, 256, device="cuda", dtype=torch.bfloat16)
    ref = lin(x)
    lin(x)  # the second call makes the one in C++
    host = lin._call.host

    def taken(m, v, epilogue=0):
        m(v, epilogue)
        return m._call.host.run(m, v, epilogue) is not None

    assert taken(lin, x) and taken(lin, x[0]) and taken(lin, x[:, :1]) and taken(lin, x[:1]) and taken(lin, x.flatten(0, 1)[::2])
    assert torch.equal(lin(x), ref) and torch.equal(lin(x[:, 1]), ref[:, 1])
    wide = torch.randn(2, 4, 512, device="cuda", dtype=torch.bfloat16)
    for v in (x.half(), x.cpu(), x[..., :128], wide[:, :3, ::2], wide[:, :3, :256], x[None], x[:0], x.as_subclass(_Sub), x.float()):
        assert host.run(lin, v, 0) is None
    assert torch.equal(lin(wide[:, :3, :256]), lin(wide[:, :3, :256].contiguous()))
    assert host.run(lin, x, 2) is None and host.run(lin, x, None) is None
    with torch.overrides.BaseTorchFunctionMode():
        assert host.run(lin, x, 0) is None
    q, s = ops.quant_fp8_rowwise(x.flatten(0, 1))
    gelu = ops.fp8_gemm(q, s, lin.weight.data, lin.weight_scale_vector(), lin.bias, out_dtype=x.dtype, epilogue=_lib.EPI_GELU_TANH)
    assert torch.equal(lin(x, epilogue=_lib.EPI_GELU_TANH), gelu.view(2, 3, 128))
    ops.STATS.timing = True
    try:
        assert host.run(lin, x, 0) is None
    finally:
        ops.STATS.timing = False
    other = _linear("cuda", 256, 128)
    assert host.run(other, x, 0) is None  # another module's descriptor
    lin.quantize_input = lambda t: ops.quant_fp8_rowwise(t * 2)
    assert host.run(lin, x, 0) is None and not torch.equal(lin(x), ref)
    del lin.quantize_input
    n = ops.STATS.kernels
    assert taken(lin, x) and ops.STATS.kernels > n
    lin.weight = torch.nn.Parameter(lin.weight.data.clone(), requires_grad=False)
    assert host.run(lin, x, 0) is None and torch.equal(lin(x), ref) and torch.equal(lin(x), ref) and taken(lin, x)
    lin.bias.data = lin.bias.data + 1
    assert host.run(lin, x, 0) is None and not torch.equal(lin(x), ref)

    class Doubled(B200Fp8Linear):
        def quantize_input(self, t):
            return super().quantize_input(t * 2)

    lin(x)
    lin.__class__ = Doubled
    assert lin._call.host.run(lin, x, 0) is None
    _lib.assert_device_ok()


def _no_extension(monkeypatch, path):
    from ksanadit_b200 import native
    monkeypatch.setattr(native, "_host", None)
    monkeypatch.setattr(native, "host_path", lambda: str(path))


@pytest.mark.parametrize("content", [None, b"not a library"])
def test_extension_that_does_not_load_is_said_once(monkeypatch, tmp_path, content):
    import warnings

    from ksanadit_b200 import native
    from ksanadit_b200.linear import _QUANTIZE_INPUT
    lin = _linear("cpu")
    _call(lin)
    path = tmp_path / "ksana_b200_host.so"
    if content is not None:
        path.write_bytes(content)
    _no_extension(monkeypatch, path)
    with warnings.catch_warnings(record=True) as said:
        warnings.simplefilter("always")
        for _ in range(3):
            assert native.linear_call(lin, lin._call, torch.bfloat16, torch.device("cuda", 0), _QUANTIZE_INPUT) is False
    assert len(said) == 1 and "ksanadit_b200.build" in str(said[0].message)


@pytest.mark.gpu
def test_linear_without_the_extension(monkeypatch, tmp_path):
    lin = _linear("cuda", 256, 128)
    x = torch.randn(3, 256, device="cuda", dtype=torch.bfloat16)
    ref = lin(x)
    _no_extension(monkeypatch, tmp_path / "absent.so")
    with pytest.warns(UserWarning, match="single calls"):
        assert torch.equal(lin(x), ref)
    assert all(torch.equal(lin(x), ref) for _ in range(3))


@pytest.mark.parametrize("compiler", ["/absent/c++", "false"])
def test_library_is_built_without_a_host_compiler(monkeypatch, capsys, compiler):
    """The extension's build fails softly and leaves what is there; and one for another torch lies under another name."""
    import os

    from ksanadit_b200 import build, native
    path = native.host_path()
    assert torch.__version__ in path
    before = os.path.getmtime(path)
    monkeypatch.setenv("CXX", compiler)
    assert build.build_host(force=True) is False
    assert "was not built" in capsys.readouterr().err
    assert os.path.getmtime(path) == before
    assert build.build() == build.LIB


@pytest.mark.gpu
def test_what_another_thread_replaces_outlives_the_launch():
    """A call lets go of the interpreter while it queues kernels; the activation scale and the counters it uses stay alive until it is
    done.  The launch is a stand-in that replaces both, as another thread may."""
    from ksanadit_b200 import _lib, native, ops
    from ksanadit_b200.linear import _QUANTIZE_INPUT
    lin = _linear("cuda", 256, 128)
    lin.scale_input = torch.nn.Parameter(torch.full((), 0.5, device="cuda"), requires_grad=False)
    watch = native.Watch()
    desc = watch.linear_of(lin, torch.bfloat16)
    space = {"STATS": ops.LaunchStats()}
    scale, stats, seen = weakref.ref(lin.scale_input), weakref.ref(space["STATS"]), []

    def launch(*a):
        lin.scale_input = None
        space["STATS"] = ops.LaunchStats()
        gc.collect()
        seen.append((scale() is not None, stats() is not None, a[6] == scale().data_ptr() if scale() is not None else None))
        return 1

    restype, argtypes = _lib.SIGNATURES["ksb_linear_forward"]
    launch_c = ctypes.CFUNCTYPE(restype, *argtypes)(launch)
    host = native.host_module().LinearCall(watch.entries, lin._parameters, ctypes.addressof(desc), torch.bfloat16, 0, _QUANTIZE_INPUT, space,
                                           native.queued, ctypes.cast(launch_c, ctypes.c_void_p).value,
                                           ctypes.cast(_lib.load().ksb_linear_workspace, ctypes.c_void_p).value)
    assert host.run(lin, torch.zeros(3, 256, device="cuda", dtype=torch.bfloat16), 0) is not None
    assert seen == [(True, True, True)]
    assert scale() is None and stats() is None
