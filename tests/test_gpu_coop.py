"""GPU: the warp-cooperative cluster fit and EndpointSearch (levels 13-19) give the oracle's blocks where their shapes
can go wrong: one block, blocks that do not fill a warp's share, orderings that do not fill a step of 32, searches that
end inside, at and after a window of candidates, and both sides of the block counts at which the mapping changes."""

import numpy as np
import pytest

import workloads as syn
from oracle import BC1Params
from quicktex_b200 import capi

pytestmark = pytest.mark.gpu

MODES = [capi.FOUR_COLOR, capi.THREE_COLOR, capi.THREE_COLOR_BLACK]
HAZARDS = syn.hazard_mix()


def _check(oracle_lib, img, level, mode, interp, **over):
    h, w = img.shape[:2]
    img = np.ascontiguousarray(img)
    got = np.frombuffer(capi.bc1_encode(img, w, h, capi.params_for_level(level, mode, interp, **over)), np.uint64)
    exp = np.frombuffer(oracle_lib.bc1_encode(img, w, h, BC1Params(level=level, color_mode=mode, interpolator=interp, **over)), np.uint64)
    bad = np.flatnonzero(got != exp)
    assert bad.size == 0, f"L{level} mode {mode} interp {interp} {w}x{h} {over}: {bad.size} of {exp.size} blocks, first {bad[0]}"


@pytest.mark.parametrize("w,h", [(4, 4), (3, 5), (36, 4), (132, 4), (61, 47)])
@pytest.mark.parametrize("level", [13, 15, 16, 18, 19])
def test_few_blocks(oracle_lib, level, w, h):
    img = syn.block_mix(w, h, workload=15, stream=level)
    for mode in MODES:
        for interp in range(4):
            _check(oracle_lib, img, level, mode, interp)


@pytest.mark.parametrize("level", range(13, 19))
@pytest.mark.parametrize("interp", range(4))
def test_rare_branches(oracle_lib, level, interp):
    """Blocks of the corpus's every class, few enough for the cooperative mapping at every level."""
    y = 4 * np.arange(0, HAZARDS.shape[0] // 4, 3)
    rows = np.concatenate([HAZARDS[k:k + 4] for k in y])[:, :256]  # 32 x 64 blocks
    for mode in MODES:
        _check(oracle_lib, rows, level, mode, interp)


@pytest.mark.parametrize("over", [dict(orderings4=1), dict(orderings4=33, orderings3=5), dict(orderings4=127), dict(search_rounds=1),
                                  dict(search_rounds=15), dict(search_rounds=17), dict(search_rounds=32), dict(search_rounds=33),
                                  dict(search_rounds=1000), dict(exhaustive=1), dict(two_cf_passes=0), dict(two_ep_passes=0)])
@pytest.mark.parametrize("interp", [0, 2])
def test_settings(oracle_lib, over, interp):
    img = syn.block_mix(76, 52, workload=15, stream=77)
    for mode in MODES:
        _check(oracle_lib, img, 18, mode, interp, **over)


@pytest.mark.parametrize("level,interp,blocks", [(13, 0, 5000), (13, 2, 3000), (15, 0, 16384), (15, 2, 9216), (17, 2, 20000)])
def test_both_sides_of_the_limits(oracle_lib, level, interp, blocks):
    for n in (blocks, blocks + 1):
        bw = 100 if n % 100 == 0 else 1
        img = syn.block_mix(4 * bw, 4 * (n // bw), workload=15, stream=n)
        _check(oracle_lib, img, level, capi.FOUR_COLOR, interp)
