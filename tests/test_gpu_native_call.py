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


def test_head_counts_that_are_no_numbers_are_refused():
    qkv = torch.zeros(1, 1, 3, 128, dtype=torch.float16, device="cuda")
    cos = sin = torch.zeros(8, 64, dtype=torch.float16, device="cuda")
    cache = torch.zeros(1, 1, 8, 128, dtype=torch.float16, device="cuda")
    pos = torch.zeros(1, dtype=torch.int64, device="cuda")
    with pytest.raises((AssertionError, TypeError)):
        ops.decode_attention_rope(qkv, cos, sin, pos, cache, cache.clone(), "1", 1)
    with pytest.raises((AssertionError, TypeError)):
        ops.decode_attention_rope(qkv, cos, sin, pos, cache, cache.clone(), 1, 2 ** 70)
