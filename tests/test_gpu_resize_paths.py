"""GPU: the resize's kernels against Pillow where their shapes can go wrong: both sides of the one-kernel path's size, every
number of lanes per output, power-of-two and other scales, one direction only, few and many columns."""

import numpy as np
import pytest

import workloads as syn
from quicktex_b200.image_utils import resize_device, resize_no_premultiply

pytestmark = pytest.mark.gpu

CASES = [(128, 128, (64, 128)), (128, 128, (1, 1)), (128, 128, (3, 77)), (129, 128, (64, 64)), (129, 127, (2, 1)), (16384, 1, (40, 1)),
         (1, 16384, (1, 9)), (1, 20000, (1, 3)), (4096, 5, (1, 2)), (700, 300, (10, 4)), (513, 511, (256, 255)), (640, 480, (640, 1)),
         (640, 480, (1, 480)), (300, 200, (37, 200)), (2048, 64, (64, 2)), (100, 4096, (100, 2)), (64, 64, (200, 130)), (5, 7, (300, 2))]


@pytest.mark.parametrize("w,h,to", CASES)
def test_equals_pillow(w, h, to):
    import torch
    from PIL import Image

    img = np.ascontiguousarray(syn.alpha_mix(w, h, workload=17, stream=w + 7 * h))
    src = torch.from_numpy(img).cuda()
    dst = torch.full((to[1], to[0], 4), 0xA5, dtype=torch.uint8, device="cuda")
    resize_device(src.data_ptr(), w, h, dst.data_ptr(), to[0], to[1], torch.cuda.current_stream().cuda_stream)
    ref = np.asarray(resize_no_premultiply(Image.fromarray(img, "RGBA"), to))
    assert np.array_equal(dst.cpu().numpy(), ref)


@pytest.mark.parametrize("w,h,to", [(512, 512, (300, 200)), (500, 333, (400, 666)), (300, 200, (333, 600)), (700, 600, (350, 300))])
def test_in_place(w, h, to):
    """Both directions change: the result may lie over the source, at its start or further on."""
    import torch
    from PIL import Image

    img = np.ascontiguousarray(syn.alpha_mix(w, h, workload=17, stream=w + 7 * h))
    ref = np.asarray(resize_no_premultiply(Image.fromarray(img, "RGBA"), to))
    s = torch.cuda.current_stream().cuda_stream
    for at in (0, 4 * w):
        buf = torch.zeros(at + 4 * max(w * h, to[0] * to[1]), dtype=torch.uint8, device="cuda")
        buf[:img.size] = torch.from_numpy(img.reshape(-1)).cuda()
        resize_device(buf.data_ptr(), w, h, buf.data_ptr() + at, to[0], to[1], s)
        assert np.array_equal(buf.cpu().numpy()[at:at + ref.size], ref.reshape(-1)), at


@pytest.mark.parametrize("w,h,to", [(6144, 2, (1, 1)), (1, 6144, (1, 1)), (6144, 60, (1, 30)), (1999, 333, (1, 1)), (1999, 333, (7, 2)), (33, 4097, (33, 4001)),
                                    (4099, 3, (1, 3)), (1086, 109, (66, 1)), (1000, 1000, (1, 1)), (3000, 1000, (46, 15)), (4, 65536, (4, 32768))])
def test_many_taps(w, h, to):
    """Weights whose sum is taken in another order than Pillow's: 6144 to 1 puts some on the boundary between two fixed-point
    values ((j + 1/2) / 3072^2 * 2^22 is a half for 2j + 1 = 9), where the sum has to be taken again in Pillow's order."""
    test_equals_pillow(w, h, to)
