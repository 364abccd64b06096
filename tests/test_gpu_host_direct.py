"""GPU: the host entry points on textures below the size where kernels read host memory themselves, and at it, give the device
entry points' bytes from the library's pinned blocks, from pageable memory, from memory pinned elsewhere and from
any mix, unaligned addresses included; a texture returned by value keeps its bytes."""

import ctypes

import numpy as np
import pytest

import quicktex_b200 as qt
import workloads as syn
from quicktex_b200 import capi
from quicktex_b200.s3tc.bc1 import BC1Decoder, BC1Encoder

pytestmark = pytest.mark.gpu


class _Own:
    def __init__(self, n):
        self.p = ctypes.c_void_p()
        capi.check(capi.lib().qt_host_alloc(n, ctypes.byref(self.p)))
        self.a = np.ctypeslib.as_array(ctypes.cast(self.p, ctypes.POINTER(ctypes.c_uint8)), (n,))

    def __del__(self):
        capi.lib().qt_host_free(self.p)


def _buffer(kind, n):
    """(array, owner) of n bytes"""
    import torch

    if kind == "own":
        o = _Own(max(n, 1 << 18))  # pinned from 256 KiB
        return o.a[:n], o
    if kind == "pinned":
        t = torch.zeros(n, dtype=torch.uint8).pin_memory()
        return t.numpy(), t
    a = np.zeros(n + 1, np.uint8)
    return (a[1:] if kind == "odd" else a[:n]), a


@pytest.mark.parametrize("w,h", [(4, 4), (61, 47), (512, 508), (512, 512), (510, 513)])
@pytest.mark.parametrize("src_kind,dst_kind", [("own", "own"), ("own", "pageable"), ("odd", "own"), ("pageable", "odd"), ("pinned", "own"), ("own", "pinned")])
def test_every_kind_of_memory(w, h, src_kind, dst_kind):
    import torch

    L, v = capi.lib(), capi._vp
    img = np.ascontiguousarray(syn.alpha_mix(w, h, workload=18, stream=w)[:h, :w]).reshape(-1)
    nb = capi.nblocks(w, h)
    d_img = torch.from_numpy(img.copy()).cuda()
    s = v(torch.cuda.current_stream().cuda_stream)
    for level, fmt in ((5, 1), (18, 3)):
        p = capi.params_for_level(level)
        size = 8 if fmt == 1 else 16
        dev = torch.zeros(nb * size, dtype=torch.uint8, device="cuda")
        enc_d, enc_h = (L.qt_bc1_encode_device, L.qt_bc1_encode_host) if fmt == 1 else (L.qt_bc3_encode_device, L.qt_bc3_encode_host)
        capi.check(enc_d(v(d_img.data_ptr()), w, h, ctypes.byref(p), v(dev.data_ptr()), s))
        exp = dev.cpu().numpy()
        src, keep_s = _buffer(src_kind, img.size)
        dst, keep_d = _buffer(dst_kind, exp.size)
        src[:] = img
        capi.check(enc_h(v(src.ctypes.data), w, h, ctypes.byref(p), v(dst.ctypes.data)))
        assert np.array_equal(dst, exp), (fmt, "encode")
        tex = torch.zeros(w * h * 4, dtype=torch.uint8, device="cuda")
        blk, keep_b = _buffer(src_kind, exp.size)
        out, keep_o = _buffer(dst_kind, w * h * 4)
        blk[:] = exp
        if fmt == 1:
            capi.check(L.qt_bc1_decode_device(v(dev.data_ptr()), w, h, 0, 1, v(tex.data_ptr()), s))
            capi.check(L.qt_bc1_decode_host(v(blk.ctypes.data), w, h, 0, 1, v(out.ctypes.data)))
        else:
            capi.check(L.qt_bc3_decode_device(v(dev.data_ptr()), w, h, 0, v(tex.data_ptr()), s))
            capi.check(L.qt_bc3_decode_host(v(blk.ctypes.data), w, h, 0, v(out.ctypes.data)))
        assert np.array_equal(out, tex.cpu().numpy()), (fmt, "decode")


@pytest.mark.parametrize("fmt,w,h", [(1, 508, 512), (3, 512, 508), (4, 254, 260), (5, 505, 509)])
def test_in_place(fmt, w, h):
    """One block of memory as both source and destination: every texel is read before the first block is written over it (and
    the other way round), as with buffers of their own."""
    L, v = capi.lib(), capi._vp
    img = np.ascontiguousarray(syn.alpha_mix(w, h, workload=18, stream=w + h)[:h, :w]).reshape(-1)
    n = capi.nblocks(w, h) * (16 if fmt in (3, 5) else 8)
    p = ctypes.byref(capi.params_for_level(18))
    enc = {1: lambda s, d: L.qt_bc1_encode_host(s, w, h, p, d), 3: lambda s, d: L.qt_bc3_encode_host(s, w, h, p, d),
           4: lambda s, d: L.qt_bc4_encode_host(s, w, h, 1, d), 5: lambda s, d: L.qt_bc5_encode_host(s, w, h, 2, 0, d)}[fmt]
    dec = {1: lambda s, d: L.qt_bc1_decode_host(s, w, h, 0, 1, d), 3: lambda s, d: L.qt_bc3_decode_host(s, w, h, 0, d),
           4: lambda s, d: L.qt_bc4_decode_host(s, w, h, 1, d), 5: lambda s, d: L.qt_bc5_decode_host(s, w, h, 2, 0, d)}[fmt]
    a, b, c = (np.zeros(max(img.size, n) + 1, np.uint8) for _ in range(3))
    a[:img.size] = img
    capi.check(enc(v(a.ctypes.data), v(b.ctypes.data)))
    capi.check(dec(v(b.ctypes.data), v(c.ctypes.data)))
    own = _Own(max(img.size, n))
    at = v(own.a.ctypes.data)
    own.a[:img.size] = img
    capi.check(enc(at, at))
    assert np.array_equal(own.a[:n], b[:n]), "encode"
    capi.check(dec(at, at))
    assert np.array_equal(own.a[:img.size], c[:img.size]), "decode"


def test_results_keep_their_bytes(oracle_lib):
    img = syn.block_mix(260, 252, workload=18, stream=9)
    outs = [BC1Encoder(5).encode(qt.RawTexture.frombytes(img.tobytes(), 260, 252)) for _ in range(3)]
    raws = [BC1Decoder().decode(t) for t in outs]
    exp = capi.bc1_encode(img, 260, 252, capi.params_for_level(5))
    assert all(t.tobytes() == exp for t in outs)
    assert all(r.tobytes() == oracle_lib.bc1_decode(exp, 260, 252, 0, False) for r in raws)
