"""CPU: rules that choose a kernel, at sizes no test runs and on devices no test has."""

import ctypes

import pytest

from quicktex_b200 import capi


@pytest.mark.parametrize("w,h,to", [(64, 64, (1 << 28, 1)), (64, 64, (215_000_000, 1)), (64, 64, (430_000_000, 1)), (8, 8, ((1 << 31) - 1, 1)),
                                    (64, 64, (1, 1 << 28)), (64, 64, (1, (1 << 29) + 1)), (8, 8, (1, (1 << 31) - 1)), (8, 8, (46341, 46341))])
def test_resize_to_a_huge_result_is_not_small(w, h, to):
    """The one-launch path's shared-memory layout and grid are 32-bit: results whose products pass 2^31 take the general path."""
    assert capi.lib().qtk_resize_is_small(w, h, *to) == 0


def test_resize_small_rule():
    small = capi.lib().qtk_resize_is_small
    assert small(256, 256, 64, 64) == 1
    assert small(512, 513, 64, 64) == 0
    assert small(512, 512, 1 << 19, 1) == 0


@pytest.mark.parametrize("w,h,to", [(500, 500, (1000, 1000)), (300, 300, (1024, 1024)), (1, 1, (1000, 1000)), (512, 512, (256, 256)), (512, 512, (511, 512)),
                                    (64, 64, (64, 1024)), (1086, 109, (66, 1)), (729, 12, (2, 988))])
def test_resize_with_much_to_do_per_row_is_not_small(w, h, to):
    """Sizes at which the one-launch path took 1.3 to 14 times the general path's time."""
    assert capi.lib().qtk_resize_is_small(w, h, *to) == 0


@pytest.mark.parametrize("w,h,to", [(128, 128, (64, 64)), (256, 256, (32, 32)), (500, 500, (62, 62)), (250, 167, (3, 2)), (64, 64, (1, 1)), (512, 512, (1, 1)), (915, 77, (19, 2))])
def test_small_chains_stay_small(w, h, to):
    assert capi.lib().qtk_resize_is_small(w, h, *to) == 1


def _coop(level, interp, n, defer_min):
    p = capi.params_for_level(level, capi.FOUR_COLOR, interp)
    return capi.lib().qtk_coop_rule(ctypes.byref(p), ctypes.c_long(n), ctypes.c_long(defer_min))


@pytest.mark.parametrize("sms", [1, 10, 19, 20, 148])
@pytest.mark.parametrize("level", range(13, 20))
def test_deferred_nvidia_never_runs_cooperatively(sms, level):
    """The deferred path (1024 blocks per SM and more) has cooperative kernels for the other interpolations only, so on a device of any
    size Nvidia's textures that reach it stay with the one-block-per-lane kernels."""
    defer_min = 1024 * sms
    sizes = (defer_min, defer_min + 1, 16384, 20000, 400000, 1 << 24)
    assert [n for n in sizes if n >= defer_min and _coop(level, capi.NVIDIA, n, defer_min)] == []


def test_coop_rule_on_148_sms():
    d = 1024 * 148
    assert [_coop(18, i, d - 1, d) for i in range(4)] == [1, 1, 1, 1] and [_coop(18, i, d, d) for i in range(4)] == [1, 1, 0, 1]
    assert [_coop(17, i, 20000, d) for i in range(4)] == [1, 1, 1, 1] and [_coop(17, i, 20001, d) for i in range(4)] == [1, 1, 0, 1]
    assert [_coop(13, i, 5000, d) for i in range(4)] == [1, 1, 0, 1] and _coop(13, 0, 5001, d) == 0 and _coop(12, 0, 100, d) == 0


# sizes at which the kernel took longer on host memory than with the copies around it, and at which it was faster
STAGED = [(0, 1, 8, 24000), (0, 4, 4, 24000), (0, 3, 12, 8000), (0, 1, 33, 7000), (0, 1, 17, 2400), (0, 1, 125, 1500), (0, 4, 191, 1000), (0, 5, 33, 7000),
          (0, 3, 99, 1200), (1, 5, 500, 508), (1, 5, 12, 12000), (1, 4, 8, 32000), (1, 1, 512, 512), (0, 1, 512, 512), (0, 1, 511, 513)]
DIRECT = [(0, 1, 256, 256), (0, 1, 401, 399), (0, 1, 510, 334), (0, 3, 128, 128), (0, 5, 129, 127), (0, 1, 64, 64), (0, 1, 63, 61), (0, 1, 7, 5), (0, 4, 250, 250),
          (1, 5, 480, 528), (1, 5, 500, 200), (1, 5, 501, 500), (1, 4, 12, 8000), (1, 1, 2, 30000), (1, 1, 508, 508), (1, 3, 17, 12000)]


@pytest.mark.parametrize("encode,fmt,w,h", STAGED)
def test_host_textures_with_many_small_pieces_are_staged(encode, fmt, w, h):
    assert capi.lib().qtk_host_direct(encode, fmt, w, h) == 0


@pytest.mark.parametrize("encode,fmt,w,h", DIRECT)
def test_other_small_host_textures_are_direct(encode, fmt, w, h):
    assert capi.lib().qtk_host_direct(encode, fmt, w, h) == 1
