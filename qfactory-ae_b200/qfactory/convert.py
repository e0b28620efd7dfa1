"""Offline packing entry point: GPTQ-style tensors -> the B200 tile-128 layout.

Keeps the call contract of the reference's `convert_params(args, params)`
(reference: qfactory/convert.py:84-97): `args` holds K, N, NBITS and, for the grouped
path, GS; `params` is `(weight,)` for the group-less path and `(weight, scale, zero)`
otherwise, `zero=None` meaning symmetric.  Wrong arity raises ValueError, wrong
shape / dtype / value range raises AssertionError (reference: qfactory/convert.py:3-47).

What changed is the layout that comes back (see layout.py); `unpack_params` inverts it.
CUDA tensors are packed by the native `qfb_pack` kernel, CPU tensors by the torch code
in layout.py; both produce identical bytes.
"""
from __future__ import annotations

import torch

from . import layout


def _check_weight(K, N, weight, nbits):
    assert weight.shape == (K, N), f"weight must be [K={K}, N={N}]"
    assert weight.dtype == torch.int32
    if weight.is_cuda:
        return   # the range is checked by the packing kernel, which reads every code anyway (_pack_native)
    lo, hi = torch.aminmax(weight)
    assert lo >= 0 and hi < 2 ** nbits, "codes out of range"


def _check_scale(K, N, GS, scale):
    assert scale.shape == (K // GS, N)
    assert scale.dtype == torch.float16


def _check_zero(K, N, GS, zero, nbits, in_kernel):
    assert zero.shape == (K // GS, N)
    assert zero.dtype == torch.int32
    if in_kernel:
        return   # as in _check_weight: the packing kernel goes where the codes are
    lo, hi = torch.aminmax(zero)
    assert lo >= 0 and hi < 2 ** nbits, "zero-points out of range"


def _empty_packed(K, N, nbits, GS, has_zero, dev):
    Np = layout.padded_rows(N)
    w = torch.empty(Np, K * nbits // 8, dtype=torch.int8, device=dev)
    s = torch.empty(Np, K // GS, dtype=torch.float16, device=dev) if GS != -1 else None
    z = torch.empty(Np, K // GS, dtype=torch.int8, device=dev) if has_zero else None
    return w, s, z


class _NoGuard:
    def __enter__(self):
        return self

    def __exit__(self, *exc):
        return False


_NO_GUARD = _NoGuard()


def _on(dev):
    """Makes `dev` current for a launch; nothing where it is already (the usual case)."""
    return _NO_GUARD if dev.index == torch.cuda.current_device() else torch.cuda.device(dev)


def _ptr(t):
    return t.data_ptr() if t is not None else None


def raise_out_of_range(flags):
    """What the packing kernel reported (the one synchronisation of a conversion)."""
    f = int(flags)
    assert not f & 1, "codes out of range"
    assert not f & 2, "zero-points out of range"


def _pack_native(K, N, nbits, GS, weight, scale, zero, lay=layout.LAYOUT_TILE):
    from . import _native

    L = _native.lib()
    dev = weight.device
    w, s, z = _empty_packed(K, N, nbits, GS, zero is not None, dev)
    weight = weight.contiguous()
    scale_c = scale.contiguous() if scale is not None else None
    zero_c = zero.contiguous() if zero is not None else None
    with _on(dev):
        flags = torch.zeros(1, dtype=torch.int32, device=dev)
        st = L.qfb_pack_checked(weight.data_ptr(), _ptr(scale_c), _ptr(zero_c), N, K, nbits, GS, lay, w.data_ptr(), _ptr(s),
                                _ptr(z), flags.data_ptr(), torch.cuda.current_stream(dev).cuda_stream)
    _native.check(st, "qfb_pack")
    raise_out_of_range(flags)
    return w, s, z


def pack_gptq(K, N, nbits, GS, qweight, scale, qzeros, lay):
    """`(w, s, z)` of `convert_params` straight from a GPTQ checkpoint's CUDA tensors: qweight int32
    [K * nbits / 32, N], scale fp16 [K/GS, N], qzeros int32 [K/GS, >= N * nbits / 32] or None (symmetric).
    Fields of nbits bits are always in range, so nothing is checked and nothing is waited for."""
    from . import _native

    layout.check_shape(N, K, nbits, GS)
    _check_scale(K, N, GS, scale)
    dev = qweight.device
    w, s, z = _empty_packed(K, N, nbits, GS, qzeros is not None, dev)
    qweight, scale = qweight.contiguous(), scale.contiguous()
    qzeros = qzeros.contiguous() if qzeros is not None else None
    with _on(dev):
        st = _native.lib().qfb_pack_gptq(qweight.data_ptr(), scale.data_ptr(), _ptr(qzeros),
                                         qzeros.shape[1] if qzeros is not None else 0, N, K, nbits, GS, lay, w.data_ptr(),
                                         s.data_ptr(), _ptr(z), torch.cuda.current_stream(dev).cuda_stream)
    _native.check(st, "qfb_pack_gptq")
    return w, s, z


def quantize_pack(weight, n_bits, group_size, lay):
    """`asymmetric_quant` followed by `convert_params` of a CUDA fp16 weight [K, N], in one pass over it.  Returns
    (w, s, z, flags): `raise_out_of_range(flags)` waits for the kernel and raises what `convert_params` raises."""
    from . import _native

    K, N = weight.shape
    layout.check_shape(N, K, n_bits, group_size)
    dev = weight.device
    w, s, z = _empty_packed(K, N, n_bits, group_size, True, dev)
    weight = weight.contiguous()
    with _on(dev):
        flags = torch.zeros(1, dtype=torch.int32, device=dev)
        st = _native.lib().qfb_quantize_pack(weight.data_ptr(), N, K, n_bits, group_size, lay, w.data_ptr(), s.data_ptr(),
                                             z.data_ptr(), flags.data_ptr(), torch.cuda.current_stream(dev).cuda_stream)
    _native.check(st, "qfb_quantize_pack")
    return w, s, z, flags


def convert_params(args, params):
    """Pack one layer.  Returns `w` (group-less) or `(w, s, z)`:
        w  int8 [Npad, K*NBITS/8]   s  fp16 [Npad, K/GS]   z  int8 [Npad, K/GS] or None
    with Npad = N rounded up to 128.  The stored zero is min(zero+1, 2^NBITS-1), as in the
    reference packer (reference: qfactory/convert.py:76).  The optional key LAYOUT ('tile', the
    default, or 'fragment') selects the packed layout (layout.py)."""
    K, N, NBITS = args["K"], args["N"], args["NBITS"]
    lay = layout.resolve_layout(args.get("LAYOUT", "tile"), N, K, NBITS, args.get("GS", -1))
    frag = lay == layout.LAYOUT_FRAGMENT
    if "GS" not in args:
        if len(params) != 1:
            raise ValueError("gemv requires 1 parameters")
        (weight,) = params
        layout.check_shape(N, K, NBITS, -1)
        _check_weight(K, N, weight, NBITS)
        if weight.is_cuda:
            return _pack_native(K, N, NBITS, -1, weight, None, None, lay)[0]
        return layout.pack_weight_fragment(weight, NBITS) if frag else layout.pack_weight(weight, NBITS)
    if len(params) != 3:
        raise ValueError("gptq_gemv requires 3 parameters")
    weight, scale, zero = params
    GS = args["GS"]
    layout.check_shape(N, K, NBITS, GS)
    _check_weight(K, N, weight, NBITS)
    _check_scale(K, N, GS, scale)
    if zero is not None:
        _check_zero(K, N, GS, zero, NBITS, weight.is_cuda and zero.is_cuda)
    if weight.is_cuda:
        return _pack_native(K, N, NBITS, GS, weight, scale, zero, lay)
    if frag:
        return (layout.pack_weight_fragment(weight, NBITS), layout.pack_scale_fragment(scale),
                layout.pack_zero_fragment(zero, NBITS) if zero is not None else None)
    w = layout.pack_weight(weight, NBITS)
    s = layout.pack_scale(scale)
    z = layout.pack_zero(zero, NBITS) if zero is not None else None
    return w, s, z


def unpack_params(args, packed):
    """Inverse of convert_params: returns codes int32 [K,N] (group-less) or
    (codes, scales fp16 [K/GS,N], effective zeros int32 [K/GS,N] or None)."""
    K, N, NBITS = args["K"], args["N"], args["NBITS"]
    frag = layout.resolve_layout(args.get("LAYOUT", "tile"), N, K, NBITS, args.get("GS", -1)) == layout.LAYOUT_FRAGMENT
    if "GS" not in args:
        w = packed[0] if isinstance(packed, (tuple, list)) else packed
        return layout.unpack_weight_fragment(w, N, K, NBITS) if frag else layout.unpack_weight(w, N, K, NBITS)
    w, s, z = packed
    if frag:
        return (layout.unpack_weight_fragment(w, N, K, NBITS), layout.unpack_scale_fragment(s, N),
                layout.unpack_zero_fragment(z, N) if z is not None else None)
    return (
        layout.unpack_weight(w, N, K, NBITS),
        layout.unpack_scale(s, N),
        layout.unpack_zero(z, N) if z is not None else None,
    )
