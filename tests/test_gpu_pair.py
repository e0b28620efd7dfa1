"""The CTA-pair kernel of wide batches: whole and cut units, odd numbers of row tiles, batches that do not fill their
tiles, rows whose output stores cannot be vectorised, every bit width and layout, against a double-precision product."""
import ctypes

import pytest
import torch

from qfactory import QLinear, _native

pytestmark = pytest.mark.gpu

CASES = [
    # m, n, k, bits, group, sym, layout, cut
    (129, 8292, 6144, 4, 128, False, "fragment", True),    # 65 row tiles, n no multiple of 8: scalar stores
    (256, 8192, 8192, 4, 64, False, "tile", True),
    (257, 8200, 6144, 4, 128, True, "fragment", False),    # the last row tile holds 8 rows
    (600, 8200, 6144, 8, 256, False, "fragment", True),
    (1024, 9472, 1280, 3, 128, True, "fragment", False),   # 148 units: two whole ones per pair
    (1000, 9472, 1280, 2, -1, True, "tile", False),
    (300, 18944, 2560, 2, 128, False, "fragment", False),
    (512, 16384, 4096, 8, 128, False, "tile", False),
    (160, 1024, 45056, 4, 128, False, "fragment", True),   # 4 units over 74 pairs: many pieces a unit
    (2048, 28672, 1024, 4, 128, False, "fragment", False),
]


def _is_pair_launch(m, n, k, cut):
    """The launch as it is planned for CTA pairs.  (The single-CTA kernel has a CTA for every row tile and batch tile, or
    for every part of one, and batch tiles of 64, 128 or 256 columns.)"""
    slots = torch.cuda.get_device_properties(0).multi_processor_count // 2
    mtiles = -(-m // 256)
    nb = -(-(-(-m // mtiles)) // 32) * 32
    units = (-(-n // 128) + 1) // 2 * mtiles
    pairs = min(slots, units * -(-k // 128) // 16) if cut else min(slots, units)
    info = _native.last_launch()
    assert info == {"kernel": 2, "grid_x": 2 * pairs, "grid_y": 2 if cut else 1, "block": 768, "smem": nb}, info


@pytest.mark.parametrize("m,n,k,bits,group,sym,layout,cut", CASES)
def test_against_double_precision(m, n, k, bits, group, sym, layout, cut):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    codes = torch.randint(0, 1 << bits, (k, n), generator=g, dtype=torch.int32, device="cuda")
    x = torch.randn(m, k, generator=g, device="cuda").mul_(2.0 ** -bits if group == -1 else 1.0).half()
    if group == -1:
        layer = QLinear.init(m, k, n, bits, codes, layout=layout)
        w = codes.half()
    else:
        s = (torch.rand(k // group, n, generator=g, device="cuda") * 0.018 + 0.002).half()
        z = None if sym else torch.randint(0, 1 << bits, (k // group, n), generator=g, dtype=torch.int32, device="cuda")
        layer = QLinear.init(m, k, n, bits, codes, group, s, z, layout=layout)
        zz = torch.full_like(codes[: k // group], 1 << (bits - 1)) if z is None else (z + 1).clamp(max=(1 << bits) - 1)
        # the kernel's weights are the fp16 products s * (q - effective zero)
        w = s.repeat_interleave(group, 0) * (codes - zz.repeat_interleave(group, 0)).half()
    y = layer(x)
    torch.cuda.synchronize()
    _is_pair_launch(m, n, k, cut)
    st = ctypes.c_uint(0)
    assert _native.lib().qfb_read_status(layer._ws.data_ptr(), None, ctypes.byref(st)) == 0 and st.value == 0
    for c0 in range(0, n, 4096):
        ref = x.double() @ w[:, c0:c0 + 4096].double()
        err = (y[:, c0:c0 + 4096].double() - ref).abs()
        # one rounding to fp16, and k / 16 additions to an fp32 running sum no larger than the largest result
        bound = 2.0 ** -10 * ref.abs() + k / 16 * 2.0 ** -23 * ref.abs().max()
        assert bool((err <= bound).all()), float((err / bound).max())
    assert torch.equal(layer(x), y)   # the sums of cut units are in a fixed order, the counters reset


def test_without_room_for_partial_sums_units_run_whole():
    m, n, k = 200, 8192, 8192
    g = torch.Generator(device="cuda").manual_seed(5)
    codes = torch.randint(0, 16, (k, n), generator=g, dtype=torch.int32, device="cuda")
    s = (torch.rand(k // 128, n, generator=g, device="cuda") * 0.018 + 0.002).half()
    layer = QLinear.init(m, k, n, 4, codes, 128, s, None)
    x = torch.randn(m, k, generator=g, device="cuda").half()
    y = layer(x)
    _is_pair_launch(m, n, k, True)
    layer._ws_bytes = 1 << 20
    y2 = layer(x)
    _is_pair_launch(m, n, k, False)
    # fp32 sums in another order, both rounded to fp16
    bound = 2.0 ** -9 * y.float().abs() + k / 16 * 2.0 ** -22 * y.float().abs().max()
    assert bool(((y.float() - y2.float()).abs() <= bound).all())


def test_split_tiles_of_33_to_64_rows_without_a_workspace():
    m, n, k = 40, 1000, 4096
    g = torch.Generator(device="cuda").manual_seed(6)
    codes = torch.randint(0, 16, (k, n), generator=g, dtype=torch.int32, device="cuda")
    s = (torch.rand(k // 128, n, generator=g, device="cuda") * 0.018 + 0.002).half()
    layer = QLinear.init(m, k, n, 4, codes, 128, s, None)
    x = torch.randn(m, k, generator=g, device="cuda").half()
    y = layer(x)
    assert _native.last_launch()["grid_y"] > 1
    layer._ws_bytes = 4096   # (such calls ran whole, and without a workspace, before their K was split)
    y2 = layer(x)
    assert _native.last_launch()["grid_y"] == 1
    bound = 2.0 ** -9 * y.float().abs() + k / 16 * 2.0 ** -22 * y.float().abs().max()
    assert bool(((y.float() - y2.float()).abs() <= bound).all())


@pytest.mark.parametrize("m,n,k,layout,cut", [(200, 8192, 8192, "fragment", True), (300, 18944, 2560, "tile", False)])
def test_a_wait_that_runs_out_abandons_the_launch_in_both_ctas(m, n, k, layout, cut):
    """The test flag of test_gpu_bounded_waits.py: 16 bytes that never come on the first weight barrier of every CTA, waits
    of about 100 us.  Nothing is stored, the status word is raised, and the layer then runs as before: its counters are
    untouched and tensor memory is free in both CTAs of every pair."""
    g = torch.Generator(device="cuda").manual_seed(7)
    codes = torch.randint(0, 16, (k, n), generator=g, dtype=torch.int32, device="cuda")
    s = (torch.rand(k // 128, n, generator=g, device="cuda") * 0.018 + 0.002).half()
    layer = QLinear.init(m, k, n, 4, codes, 128, s, None, layout=layout)
    x = torch.randn(m, k, generator=g, device="cuda").half()
    st = ctypes.c_uint(0)
    status = lambda: (_native.lib().qfb_read_status(layer._ws.data_ptr(), None, ctypes.byref(st)), st.value)  # noqa: E731
    want = layer(x)
    _is_pair_launch(m, n, k, cut)
    assert status() == (0, 0)
    out = torch.full_like(want, 7.0)
    layer.flags = _native.FLAG_TEST_STALLED_WAIT
    layer(x, out)
    torch.cuda.synchronize()
    _is_pair_launch(m, n, k, cut)
    assert status() == (8, 1) and bool((out == 7.0).all())   # QFB_ERR_DEVICE_FLAG
    layer.flags = 0
    _native.check(_native.lib().qfb_workspace_init(layer._ws.data_ptr(), layer._ws_bytes, torch.cuda.current_stream().cuda_stream))
    for _ in range(3):
        assert torch.equal(layer(x), want)
    assert status() == (0, 0)
