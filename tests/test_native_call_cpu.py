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
