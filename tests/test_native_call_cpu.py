"""The native call path's behaviour that needs no GPU: what torch throws inside it arrives as a Python exception."""
import os
import subprocess
import sys

import pytest

from qfactory import _native

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.skipif(not os.path.exists(_native.TORCH_MODULE_PATH), reason="native module not built")

# A functional tensor says it is a CUDA tensor and has no storage (and without a GPU there is no current device): torch
# throws in the middle of the entry.
THROWS = """
import sys, torch
from torch._subclasses.fake_tensor import FakeTensorMode
sys.path.insert(0, %r)
from qfactory import ops
with FakeTensorMode():
    t = torch._to_functional_tensor(torch.empty(4, 256, dtype=torch.float16, device="cuda"))
    w = torch._to_functional_tensor(torch.empty(256, dtype=torch.float16, device="cuda"))
class F(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        return call(x)
def silu(x): return ops.silu_mul(x)
def norm(x): return ops.rmsnorm(x, w)
def add_norm(x): return ops.add_rmsnorm(x, x, w)
for call in (silu, norm, add_norm):
    for way in (call, F.apply):
        try:
            way(t)
        except RuntimeError as e:
            print("raised", call.__name__, type(e).__name__)
        sum([list(range(100)) for _ in range(100)], [])   # the interpreter's frames are whole
print("alive")
"""


def test_what_torch_throws_is_a_python_exception():
    r = subprocess.run([sys.executable, "-c", THROWS % os.path.join(ROOT, "qfactory-ae_b200")], capture_output=True, text=True)
    lines = r.stdout.split("\n")
    assert r.returncode == 0 and "alive" in lines, (r.returncode, r.stdout[-500:], r.stderr[-800:])
    assert sum(line.startswith("raised") for line in lines) == 6, r.stdout


def _layers():
    from qfactory import QLinear

    _native.torch_module()   # (its `__call__` is in the classes from here on)
    return [QLinear.empty(1, 256, 128, 4, 128, False, device="cpu"), QLinear.empty(1, 256, 128, 4, -1, True, device="cpu")]


def test_a_wrapped_module_call_sees_the_layers():
    import torch

    for layer in _layers():
        net = torch.nn.Sequential(layer, torch.nn.ReLU())

        class Tracer(torch.fx.Tracer):
            def is_leaf_module(self, m, name):
                return m is layer or super().is_leaf_module(m, name)

        graph = Tracer().trace(net)
        assert [n.op for n in graph.nodes] == ["placeholder", "call_module", "call_module", "output"]


def test_calls_go_where_python_would_send_them():
    import torch

    seen = []

    class Mixin(torch.nn.Module):
        def __call__(self, *a, **kw):
            seen.append("mixin")
            return super().__call__(*a, **kw)

    for layer in _layers():
        cls = type(layer)

        class Sub(cls, Mixin):
            def __call__(self, *a, **kw):
                seen.append("sub")
                return super().__call__(*a, **kw)

            def forward(self, x, out=None):
                return ("forward", x, out)

        sub = Sub.__new__(Sub)
        sub.__dict__.update(layer.__dict__)
        seen.clear()
        assert sub(1, out=2) == ("forward", 1, 2) and seen == ["sub", "mixin"]
        assert sub(1, 3) == ("forward", 1, 3) and sub(x=4) == ("forward", 4, None)
        with pytest.raises(TypeError):
            sub()
        with pytest.raises(_native.NativeError):   # no CPU path
            layer(torch.zeros(1, 256, dtype=torch.float16))
        with pytest.raises(TypeError):
            cls.__call__(object(), 1)
