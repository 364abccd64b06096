"""CPU: rules that choose a kernel, at sizes no test runs and on devices no test has."""

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


@pytest.mark.parametrize("w,h,to", [(128, 128, (64, 64)), (256, 256, (32, 32)), (500, 500, (62, 62)), (250, 167, (3, 2)), (64, 64, (1, 1))])
def test_small_chains_stay_small(w, h, to):
    assert capi.lib().qtk_resize_is_small(w, h, *to) == 1
