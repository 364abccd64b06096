"""GPU: the split pass's list at its edges: the smallest texture that takes it, a last thread block that is partly filled,
textures of solid blocks only and of none, and more blocks than its grid holds in one step. The same texture encoded in
strips below the split's size, which take no split pass, gives the expected blocks (a strip is a whole number of block rows)."""

import ctypes

import numpy as np
import pytest

import workloads as syn
from quicktex_b200 import capi

pytestmark = pytest.mark.gpu


def _texture(w, h, kind):
    if kind == "mix":
        tile = np.ascontiguousarray(syn.alpha_mix(256, 256, workload=18, stream=w + h))
        return np.ascontiguousarray(np.tile(tile, ((h + 255) // 256, (w + 255) // 256, 1))[:h, :w])
    img = np.full((h, w, 4), 77, np.uint8)
    if kind == "none solid":
        img[::4, ::4, 0] = 5
    return img


@pytest.mark.parametrize("fmt", ["bc1", "bc3"])
@pytest.mark.parametrize(
    "w,h,kind", [(512, 512, "mix"), (516, 516, "mix"), (1023, 520, "mix"), (516, 516, "solid"), (516, 516, "none solid"), (8192, 6144, "mix")]
)
def test_split_matches_strips(fmt, w, h, kind):
    import torch

    L, v = capi.lib(), capi._vp
    call = L.qt_bc1_encode_device if fmt == "bc1" else L.qt_bc3_encode_device
    size = 8 if fmt == "bc1" else 16
    s = v(torch.cuda.current_stream().cuda_stream)
    p = ctypes.byref(capi.params_for_level(0))
    bw = (w + 3) // 4
    src = torch.from_numpy(_texture(w, h, kind).reshape(-1)).cuda()
    whole, strips = (torch.zeros(capi.nblocks(w, h) * size, dtype=torch.uint8, device="cuda") for _ in range(2))
    capi.check(call(v(src.data_ptr()), w, h, p, v(whole.data_ptr()), s))
    rows = 4 * (16383 // bw)
    for y in range(0, h, rows):
        capi.check(call(v(src.data_ptr() + y * w * 4), w, min(rows, h - y), p, v(strips.data_ptr() + (y // 4) * bw * size), s))
    assert torch.equal(whole, strips)
