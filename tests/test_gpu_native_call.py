"""The C++ call path of the layers and of the decoder's element-wise neighbours answers, and refuses, what the Python
path does."""
import ctypes

import pytest
import torch

from qfactory import QLinear, ops

pytestmark = pytest.mark.gpu


def _layer(m=4, n=256, k=512, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    codes = torch.randint(0, 16, (k, n), generator=g, dtype=torch.int32, device="cuda")
    s = (torch.rand(k // 128, n, generator=g, device="cuda") * 0.018 + 0.002).half()
    z = torch.randint(0, 16, (k // 128, n), generator=g, dtype=torch.int32, device="cuda")
    return QLinear.init(m, k, n, 4, codes, 128, s, z), torch.randn(m, k, generator=g, device="cuda").half()


@pytest.mark.parametrize("eps", ["1e-5", None, 10 ** 400])
def test_an_eps_that_is_no_number_is_refused(eps):
    x, w = torch.randn(2, 256, device="cuda").half(), torch.ones(256, device="cuda").half()
    with pytest.raises(ctypes.ArgumentError):
        ops.rmsnorm(x, w, eps)
    with pytest.raises(ctypes.ArgumentError):
        ops.add_rmsnorm(x.clone(), x, w, eps)
    assert torch.equal(ops.rmsnorm(x, w, 1), ops.rmsnorm(x, w, 1.0))


def test_the_sum_with_no_residual_is_refused():
    x, w = torch.randn(2, 256, device="cuda").half(), torch.ones(256, device="cuda").half()
    before = x.clone()
    for none in (None, x[:1], x.float()):
        with pytest.raises((AttributeError, AssertionError)):
            ops.add_rmsnorm(x, none, w)
    assert torch.equal(x, before)


def test_head_counts_that_are_no_numbers_are_refused():
    qkv = torch.zeros(1, 1, 3, 128, dtype=torch.float16, device="cuda")
    cos = sin = torch.zeros(8, 64, dtype=torch.float16, device="cuda")
    cache = torch.zeros(1, 1, 8, 128, dtype=torch.float16, device="cuda")
    pos = torch.zeros(1, dtype=torch.int64, device="cuda")
    with pytest.raises((AssertionError, TypeError)):
        ops.decode_attention_rope(qkv, cos, sin, pos, cache, cache.clone(), "1", 1)
    with pytest.raises((AssertionError, TypeError)):
        ops.decode_attention_rope(qkv, cos, sin, pos, cache, cache.clone(), 1, 2 ** 70)


def _counting(target, calls):
    def wrapped(self, *a, **kw):
        calls.append(self)
        return target(self, *a, **kw)
    return wrapped


@pytest.mark.parametrize("where", ["forward", "_call_impl", "__call__ of nn.Module", "_call_impl of nn.Module"])
def test_what_replaces_a_part_of_the_call_is_seen(where, monkeypatch):
    layer, x = _layer()
    want = layer(x)
    calls = []
    name, cls = where.split(" ")[0], torch.nn.Module if "nn.Module" in where else type(layer)
    monkeypatch.setattr(cls, name, _counting(getattr(cls, name), calls))
    assert torch.equal(layer(x), want) and torch.equal(layer(x, torch.empty_like(want)), want)
    assert len(calls) == 2
    monkeypatch.undo()
    assert torch.equal(layer(x), want) and len(calls) == 2


def test_a_tracer_gets_the_call_it_asks_for(monkeypatch):
    layer, x = _layer()
    layer(x)
    monkeypatch.setattr(type(layer), "_slow_forward", lambda self, t: t + 1)   # what nn.Module calls under a tracer
    traced = torch.jit.trace(lambda t: layer(t), x, check_trace=False)
    assert torch.equal(traced(x), x + 1)


def test_a_replaced_forward_of_one_layer_and_hooks():
    layer, x = _layer()
    want = layer(x)
    layer.forward = lambda t: "own"
    assert layer(x) == "own"
    del layer.forward
    module = torch.nn.modules.module
    seen = []
    hooks = [(lambda: layer.register_forward_pre_hook(lambda m, a: seen.append("pre")), "pre"),
             (lambda: layer.register_forward_hook(lambda m, a, y: seen.append("post")), "post"),
             (lambda: layer.register_full_backward_pre_hook(lambda m, go: None), None),
             (lambda: layer.register_full_backward_hook(lambda m, gi, go: None), None),
             (lambda: module.register_module_forward_pre_hook(lambda m, a: seen.append("all pre")), "all pre"),
             (lambda: module.register_module_forward_hook(lambda m, a, y: seen.append("all post")), "all post"),
             (lambda: module.register_module_full_backward_pre_hook(lambda m, go: None), None),
             (lambda: module.register_module_full_backward_hook(lambda m, gi, go: None), None)]
    for register, name in hooks:
        handle = register()
        assert torch.equal(layer(x), want) and seen == ([name] if name else [])
        handle.remove()
        seen.clear()
        assert torch.equal(layer(x), want) and not seen
    handle = layer.register_forward_hook(lambda m, a, y: y + 1)
    assert torch.equal(layer(x), want + 1)
    handle.remove()
    assert torch.equal(layer(x), want)


def test_modes_see_the_operations():
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    layer, x = _layer()
    w = torch.ones(512, dtype=torch.float16, device="cuda")
    runs = [lambda: layer(x), lambda: layer.forward(x), lambda: ops.silu_mul(x), lambda: ops.rmsnorm(x, w)]
    want = [f() for f in runs]
    seen = []

    class Dispatch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    class Function(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    for f, y in zip(runs, want):
        for mode in (Dispatch(), Function()):
            seen.clear()
            with mode:
                got = f()
            assert torch.equal(got, y) and any("empty" in s for s in seen), seen
        with torch.device("cpu"):   # a default device, which names none of ours
            assert f().is_cuda


def test_outputs_ranks_strides_and_streams():
    layer, x = _layer(m=6)
    want = layer(x)
    out = torch.empty_like(want)
    assert layer(x, out) is out and torch.equal(out, want)
    out = torch.empty_like(want)
    assert layer(x, out=out) is out and torch.equal(out, want)
    flat = torch.empty(want.numel(), dtype=torch.float16, device="cuda")
    assert layer(x, out=flat) is flat and torch.equal(flat.view_as(want), want)
    for lead in ((), (1,), (2, 3), (3, 1, 2), (1, 6)):
        xr = x[0] if lead == () else x.reshape(*lead, 512) if torch.Size(lead).numel() == 6 else x[:1]
        y = layer(xr)
        assert y.shape == (*xr.shape[:-1], 256) and torch.equal(y.reshape(-1, 256), layer(xr.reshape(-1, 512)))
    wide = torch.randn(6, 1024, device="cuda").half()
    wide[:, ::2] = x
    assert torch.equal(layer(wide[:, ::2]), want) and torch.equal(layer(x.t().contiguous().t()), want)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        y = layer(x)
    side.synchronize()
    assert torch.equal(y, want)
    assert layer(x[:0]).shape == (0, 256) and layer(x[:0].view(2, 0, 512)).shape == (2, 0, 256)
    for bad in (x.float(), x[:, :256], x.cpu()):
        with pytest.raises((AssertionError, RuntimeError)):
            layer(bad)
    out = torch.empty_like(want)
    for bad in (out[:5], out.float(), torch.empty(256, 6, dtype=torch.float16, device="cuda").t()):
        with pytest.raises(AssertionError):
            layer(x, bad)
    assert torch.equal(layer(x), want)


@pytest.mark.parametrize("m", [1, 6])
def test_the_fused_activation_gives_the_shape_of_the_rows(m):
    layer, _ = _layer(m=m)
    gu = torch.randn(m, 1024, device="cuda").half()
    want = layer.forward_silu_mul(gu)
    assert want.shape == (m, 256) and torch.equal(want, layer(ops.silu_mul(gu)))
    for shape in ((m, 256), (m * 256,), (1, m, 256), (m * 2, 128)):
        out = torch.empty(shape, dtype=torch.float16, device="cuda")
        y = layer.forward_silu_mul(gu, out)
        assert y.shape == (m, 256) and y.data_ptr() == out.data_ptr() and torch.equal(y, want)
    y = layer.forward_silu_mul(gu.view(m, 1, 1024), torch.empty_like(want))
    assert y.shape == (m, 1, 256) and torch.equal(y.view(m, 256), want)


def test_flags_and_workspace_changed_after_the_first_call():
    from qfactory import _native

    layer, x = _layer(m=24, k=4096)
    want = layer(x)
    assert _native.last_launch()["kernel"] == 2
    layer.flags = _native.FLAG_FORCE_SIMT
    layer(x)
    assert _native.last_launch()["kernel"] == 3
    layer.flags = 0
    layer._ws = torch.zeros_like(layer._ws)
    assert torch.equal(layer(x), want)
    held = layer._ws
    assert layer._native_call.hold == (layer.w, layer.s, layer.z, held) and layer._native_call.ws_ptr == held.data_ptr()
    layer._ws_bytes = 0
    with pytest.raises(_native.NativeError):   # a split without room for its partial sums
        layer(x)
    layer._ws_bytes = held.numel()
    assert torch.equal(layer(x), want)
