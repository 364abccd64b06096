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
