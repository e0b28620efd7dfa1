"""With two CTAs per SM the row tiles beyond a whole number per SM are cut along K where their parts find an SM each."""
import pytest
import torch

from qfactory import QLinear, _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [64, 100])
@pytest.mark.parametrize("rest_of,parts", [((1, 2), 2), ((1, 3), 3), ((1, 4), 4), ((2, 3), 1)])
def test_the_rest_is_cut_where_its_parts_find_an_sm_each(m, rest_of, parts):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rest = sms * rest_of[0] // rest_of[1]
    n, k = (sms + rest) * 128, 4096
    g = torch.Generator(device="cuda").manual_seed(rest + m)
    codes = torch.randint(0, 16, (k, n), generator=g, dtype=torch.int32, device="cuda")
    s = (torch.rand(k // 128, n, generator=g, device="cuda") * 0.018 + 0.002).half()
    layer = QLinear.init(m, k, n, 4, codes, 128, s, None)
    x = torch.randn(m, k, generator=g, device="cuda").half()
    y = layer(x)
    info = _native.last_launch()
    assert (info["grid_x"], info["grid_y"]) == (sms + rest * parts, parts) if parts > 1 else info["grid_x"] == sms + rest, info
    for c0 in range(0, n, 8192):   # the kernel's weights are the fp16 products s * (q - 8)
        c1 = min(n, c0 + 8192)
        ref = x.double() @ (s[:, c0:c1].repeat_interleave(128, 0) * (codes[:, c0:c1] - 8).half()).double()
        bound = 2.0 ** -10 * ref.abs() + k / 16 * 2.0 ** -23 * ref.abs().max()
        assert bool(((y[:, c0:c1].double() - ref).abs() <= bound).all())
