"""K an odd multiple of 64 beyond one pass of the CUDA-core kernel: the tcgen05 kernels with a half-filled last stage."""
import ctypes

import pytest
import torch

from qfactory import QLinear, _native

pytestmark = pytest.mark.gpu


def _case(m, n, k, bits, group, sym, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    codes = torch.randint(0, 1 << bits, (k, n), generator=g, dtype=torch.int32, device="cuda")
    x = torch.randn(m, k, generator=g, device="cuda").mul_(2.0 ** -bits if group == -1 else 1.0).half()
    if group == -1:
        return QLinear.init(m, k, n, bits, codes), codes.half(), x
    s = (torch.rand(k // group, n, generator=g, device="cuda") * 0.018 + 0.002).half()
    z = None if sym else torch.randint(0, 1 << bits, (k // group, n), generator=g, dtype=torch.int32, device="cuda")
    layer = QLinear.init(m, k, n, bits, codes, group, s, z)
    zz = torch.full_like(codes[: k // group], 1 << (bits - 1)) if z is None else (z + 1).clamp(max=(1 << bits) - 1)
    return layer, s.repeat_interleave(group, 0) * (codes - zz.repeat_interleave(group, 0)).half(), x


def _check(y, x, w):
    ref = x.double() @ w.double()
    # one rounding to fp16, and k / 16 additions to an fp32 running sum no larger than the largest result
    bound = 2.0 ** -10 * ref.abs() + x.shape[1] / 16 * 2.0 ** -23 * ref.abs().max()
    assert bool(((y.double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("m,n,k,bits,group,sym", [
    (9, 200, 192, 4, 64, False), (16, 128, 64, 8, 64, True), (16, 200, 64, 4, -1, True), (32, 128, 64, 2, -1, True), (17, 1000, 1088, 2, -1, True), (32, 256, 704, 4, -1, True),
    (37, 3000, 2752, 4, 64, False), (64, 384, 4160, 8, 64, False), (65, 300, 1344, 2, 64, True), (128, 19200, 320, 4, 64, False),
    (200, 8192, 11072, 4, 64, False), (300, 9472, 2752, 8, -1, True), (600, 640, 2112, 4, 64, True)])
def test_half_filled_last_stage(m, n, k, bits, group, sym):
    layer, w, x = _case(m, n, k, bits, group, sym, m + n + k)
    # whatever an earlier launch left in shared memory must not show in the half of a stage that is not filled
    other, _, xo = _case(m, 256, 1024, bits, -1, True, 1)
    other(torch.full_like(xo, float("inf")))
    y = layer(x)
    torch.cuda.synchronize()
    assert _native.last_launch()["kernel"] == 2
    st = ctypes.c_uint(0)
    assert _native.lib().qfb_read_status(layer._ws.data_ptr(), None, ctypes.byref(st)) == 0 and st.value == 0
    _check(y, x, w)
    layer._ws_bytes = 4096   # without room for partial sums the splits are dropped, the call is not refused
    _check(layer(x), x, w)
