"""GPU: BC4/BC5 encode and every decoder on textures whose rows are off the 16-byte grid, by their width or by the base
address, with and without interior blocks, against the oracle; texels around the texture stay as they were."""

import numpy as np
import pytest

import workloads as syn
from quicktex_b200 import capi

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (3, 9), (4, 4), (5, 4), (6, 13), (7, 8), (8, 8), (127, 9), (129, 12), (130, 31), (132, 16), (259, 21)]
FENCE = 64  # bytes kept on both sides


def _at(data, offset):
    """A device copy of data starting `offset` bytes past a 16-byte boundary, inside a fence of 0xA5."""
    import torch

    buf = torch.full((FENCE + offset + data.size + FENCE,), 0xA5, dtype=torch.uint8, device="cuda")
    buf[FENCE + offset: FENCE + offset + data.size] = torch.from_numpy(data.reshape(-1).copy()).cuda()
    return buf, buf.data_ptr() + FENCE + offset


@pytest.mark.parametrize("offset", [0, 4, 8, 12])
@pytest.mark.parametrize("w,h", SIZES)
def test_off_the_grid(oracle_lib, w, h, offset):
    import torch

    L, v = capi.lib(), capi._vp
    s = v(torch.cuda.current_stream().cuda_stream)
    img = np.ascontiguousarray(syn.alpha_mix(w, h, workload=16, stream=w * 64 + h))
    nb = capi.nblocks(w, h)
    keep, src = _at(img, offset)
    for size, call, exp in (
        (8, lambda d: L.qt_bc4_encode_device(v(src), w, h, 3, v(d), s), oracle_lib.bc4_encode(img, w, h, 3)),
        (16, lambda d: L.qt_bc5_encode_device(v(src), w, h, 1, 3, v(d), s), oracle_lib.bc5_encode(img, w, h, 1, 3)),
    ):
        out = torch.zeros(nb * size, dtype=torch.uint8, device="cuda")
        capi.check(call(out.data_ptr()))
        assert out.cpu().numpy().tobytes() == exp, (size, w, h, offset)
    rng = np.random.default_rng(w + h)
    b8, b16 = (rng.integers(0, 256, nb * k, dtype=np.uint8) for k in (8, 16))
    d8, d16 = (torch.from_numpy(b).cuda() for b in (b8, b16))
    p8, p16 = v(d8.data_ptr()), v(d16.data_ptr())
    for call, exp in (
        (lambda d: L.qt_bc1_decode_device(p8, w, h, 2, 1, v(d), s), oracle_lib.bc1_decode(b8, w, h, 2, True)),
        (lambda d: L.qt_bc3_decode_device(p16, w, h, 0, v(d), s), oracle_lib.bc3_decode(b16, w, h, 0)),
        (lambda d: L.qt_bc4_decode_device(p8, w, h, 1, v(d), s), oracle_lib.bc4_decode(b8, w, h, 1)),
        (lambda d: L.qt_bc5_decode_device(p16, w, h, 0, 1, v(d), s), oracle_lib.bc5_decode(b16, w, h, 0, 1)),
    ):
        buf, dst = _at(np.zeros(w * h * 4, np.uint8), offset)
        capi.check(call(dst))
        got = buf.cpu().numpy()
        assert got[FENCE + offset: -FENCE].tobytes() == exp, (w, h, offset)
        assert (got[: FENCE + offset] == 0xA5).all() and (got[-FENCE:] == 0xA5).all()
