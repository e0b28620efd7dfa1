"""Conversion on the GPU (fp16 weight, GPTQ words or int32 codes -> packed bytes) against the torch packers on the
CPU: every byte equal, at the edges of the 128 x 128 blocks."""
import pytest
import torch

from oracle import qf_oracle as O
from qfactory import QLinear, convert_params, gptq
from qfactory.quantize import asymmetric_quant

pytestmark = pytest.mark.gpu

# (bits, group, K, N): one block, a K tail of 64, N tails (odd too), groups of 64, of several blocks and of 192
CASES = [(4, 128, 128, 128), (4, 64, 320, 200), (4, 256, 768, 1000), (2, 128, 384, 96), (2, 64, 192, 264), (8, 128, 256, 136),
         (8, 64, 192, 40), (4, 192, 384, 264), (3, 128, 384, 72), (3, 256, 512, 129), (4, 512, 1024, 131), (8, 1024, 1024, 257)]


def _same(a, b):
    for x, y in zip((a.w, a.s, a.z), (b.w, b.s, b.z)):
        assert (x is None) == (y is None)
        if x is not None:
            assert torch.equal(x.cpu(), y)


@pytest.mark.parametrize("layout", ["tile", "auto"])
@pytest.mark.parametrize("bits,group,K,N", CASES)
def test_float_weight(bits, group, K, N, layout):
    g = torch.Generator().manual_seed(K + N + bits)
    w = torch.randn(K, N, generator=g).half()
    w[:group, 1] *= 6e-7         # subnormal differences
    if K > group:
        w[group:2 * group, 2] *= 100.0
    _same(QLinear.from_float(w.cuda(), bits, group, layout=layout), QLinear.from_float(w, bits, group, layout=layout))
    # a constant group (0 / 0, whose conversion to an integer is the GPU's): against the separate quantiser's codes
    w[:group, 0] = 0.0
    q, s, z = (t.cpu() for t in asymmetric_quant(w.cuda(), group, bits))
    _same(QLinear.from_float(w.cuda(), bits, group, layout=layout), QLinear.init(1, K, N, bits, q, group, s, z, layout=layout))


@pytest.mark.parametrize("bits,group,K,N", [(4, 64, 192, 200), (8, 128, 256, 131)])
def test_float_weight_at_an_odd_place_of_a_buffer(bits, group, K, N):
    w = torch.randn(K, N, generator=torch.Generator().manual_seed(N)).half()
    flat = torch.empty(K * N + 1, dtype=torch.float16, device="cuda")
    view = flat[1:].view(K, N)
    view.copy_(w)
    assert view.is_contiguous() and view.data_ptr() % 4 == 2
    _same(QLinear.from_float(view, bits, group), QLinear.from_float(w, bits, group))


@pytest.mark.parametrize("sym", [False, True])
@pytest.mark.parametrize("bits,group,K,N", [c for c in CASES if c[0] != 3 and c[3] % 16 == 0 or c[3] == 1000])
def test_gptq_words(bits, group, K, N, sym):
    if N % (32 // bits):
        pytest.skip("the checkpoint's zeros come in whole words")
    _, q, s, z = O.make_case(1, N, K, bits, group, False, seed=K + N)
    words, zeros = gptq.pack_qweight(q, bits), gptq.pack_qzeros(z, bits)
    _same(gptq.layer_from_gptq(words.cuda(), zeros.cuda(), s.cuda(), bits, group, sym=sym),
          gptq.layer_from_gptq(words, zeros, s, bits, group, sym=sym))


def test_values_out_of_range_are_reported():
    K, N, group = 256, 200, 128
    _, q, s, z = O.make_case(1, N, K, 4, group, False, seed=5)
    args = {"K": K, "N": N, "NBITS": 4, "GS": group}
    for bad in (16, -1):
        q2, z2 = q.clone(), z.clone()
        q2[K - 1, N - 1] = bad
        z2[0, 3] = bad
        with pytest.raises(AssertionError, match="codes"):
            convert_params(args, (q2.cuda(), s.cuda(), z.cuda()))
        with pytest.raises(AssertionError, match="zero"):
            convert_params(args, (q.cuda(), s.cuda(), z2.cuda()))
        with pytest.raises(AssertionError, match="zero"):   # codes on the CPU, zero points on the GPU
            convert_params(args, (q, s, z2.cuda()))
    with pytest.raises(AssertionError, match="zero"):   # a group far below zero has a zero point no code can hold
        QLinear.from_float(torch.full((K, N), -3.0).half().cuda() + torch.rand(K, N).half().cuda(), 4, group)


def test_more_blocks_along_k_than_a_grid_has_in_its_second_dimension():
    # 65536 blocks of 128: the last of them must hold what a layer made of the last rows alone holds
    K, N, tail = 65536 * 128, 8, 1024
    g = torch.Generator(device="cuda").manual_seed(9)
    w = torch.randn(K, N, generator=g, dtype=torch.float16, device="cuda")
    q = torch.randint(0, 16, (K, N), generator=g, dtype=torch.int32, device="cuda")
    s = torch.rand(K // 128, N, generator=g, device="cuda").half()
    words = torch.randint(-2 ** 31, 2 ** 31, (K // 8, N), generator=g, dtype=torch.int64, device="cuda").to(torch.int32)
    for make in (lambda a: QLinear.from_float(w[-a:], 4, 128, layout="tile"),
                 lambda a: QLinear.init(1, a, N, 4, q[-a:], 128, s[-(a // 128):], None, layout="tile"),
                 lambda a: gptq.layer_from_gptq(words[-(a // 8):], None, s[-(a // 128):], 4, 128, sym=True)):
        whole, last = make(K), make(tail)
        if whole.packed_layout == last.packed_layout == 0:   # tile layout: the units of the one row tile follow each other
            assert torch.equal(whole.w.view(-1)[-last.w.numel():], last.w.view(-1))
        else:                                                # fragment layout: a run for each half of the tile
            assert torch.equal(whole.w.view(2, -1)[:, -(last.w.numel() // 2):], last.w.view(2, -1))
        assert torch.equal(whole.s.view(-1)[-last.s.numel():], last.s.view(-1))
