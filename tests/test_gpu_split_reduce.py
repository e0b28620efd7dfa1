"""The sum of K splits of the tiles with per-stage accumulators (up to 32 rows): four rows of a column per lane, stored as
8 bytes where the output allows it."""
import pytest
import torch

from qfactory import QLinear, _native

pytestmark = pytest.mark.gpu

# rows a multiple of 8, of 4, of 2, odd; one row in the last tile; batches around a run of 4 and of 16 columns
CASES = [(17, 1000, 11008, 4, "fragment"), (32, 4096, 4096, 8, "fragment"), (31, 260, 2048, 2, "fragment"),
         (24, 130, 11008, 3, "fragment"), (20, 129, 1024, 4, "fragment"), (2, 1000, 11008, 4, "tile"), (5, 131, 2048, 8, "tile"),
         (16, 4096, 11008, 4, "tile"), (15, 257, 4096, 2, "tile"), (32, 300, 28672, 3, "tile")]


@pytest.mark.parametrize("odd_place", [False, True])
@pytest.mark.parametrize("m,n,k,bits,layout", CASES)
def test_against_double_precision(m, n, k, bits, layout, odd_place):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    codes = torch.randint(0, 1 << bits, (k, n), generator=g, dtype=torch.int32, device="cuda")
    s = (torch.rand(k // 128, n, generator=g, device="cuda") * 0.018 + 0.002).half()
    z = torch.randint(0, 1 << bits, (k // 128, n), generator=g, dtype=torch.int32, device="cuda")
    layer = QLinear.init(m, k, n, bits, codes, 128, s, z, layout=layout)
    x = torch.randn(m, k, generator=g, device="cuda").half()
    flat = torch.full((m * n + 9,), 7.0, dtype=torch.float16, device="cuda")
    at = 1 if odd_place else 8
    y = flat[at:at + m * n].view(m, n)
    assert layer(x, y) is y
    info = _native.last_launch()
    assert info["kernel"] == 2 and info["grid_y"] > 1 and info["smem"] == (16 if m <= 16 else 32), info
    assert bool((flat[:at] == 7.0).all()) and bool((flat[at + m * n:] == 7.0).all())
    zz = (z + 1).clamp(max=(1 << bits) - 1)
    ref = x.double() @ (s.double().repeat_interleave(128, 0) * (codes - zz.repeat_interleave(128, 0)))
    # one rounding to fp16; the codes are exact, and k / 16 + k / 128 additions run in fp32
    bound = 2.0 ** -10 * ref.abs() + k / 14 * 2.0 ** -23 * ref.abs().max()
    assert bool(((y.double() - ref).abs() <= bound).all())
    again = torch.empty_like(y)
    layer(x, again)
    assert torch.equal(again, y)   # the splits are summed in their order, the counters reset
