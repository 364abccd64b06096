"""GPU: every kernel of a batch and every size of tile against the oracle: the 24 specialised encoders (four interpolations, the
Faster and Check2 error modes, three colour modes), BC3's four-colour ones, and levels 13-19 on both sides of the cooperative
encoder's rule."""

import numpy as np
import pytest

import workloads as syn
from oracle import BC1Params
from quicktex_b200.batch import Batch, Job, run_jobs

pytestmark = pytest.mark.gpu

FAST = [(lv, m, i) for lv in (1, 5, 8, 10) for m in (0x04, 0x03, 0x13) for i in range(4)]
SEARCH = [(lv, m, i) for lv in (13, 14, 15, 16, 17, 18) for m, i in ((0x04, 0), (0x13, 1), (0x03, 2), (0x13, 3))] + [(19, 0x04, 2), (19, 0x13, 0)]


def _expected(oracle_lib, fmt, img, w, h, lv, m, i):
    p = BC1Params(level=lv, color_mode=m, interpolator=i)
    return (oracle_lib.bc1_encode if fmt == "bc1" else oracle_lib.bc3_encode)(img, w, h, p)


@pytest.mark.parametrize("settings", [FAST, SEARCH], ids=["fast", "search"])
@pytest.mark.parametrize("tile", [1, 7, 31, 33, 64])
def test_every_kernel_and_tile(oracle_lib, settings, tile):
    w, h = 61, 38  # 160 blocks, both sides ragged
    img = np.ascontiguousarray(syn.alpha_mix(w, h, workload=19, stream=tile))
    jobs, expected = [], []
    for lv, m, i in settings:
        for fmt in ("bc1", "bc3"):
            if fmt == "bc3" and m != 0x04:
                continue
            jobs.append(Job.encode(fmt, img, w, h, level=lv, color_mode=m, interpolator=i))
            expected.append(_expected(oracle_lib, fmt, img, w, h, lv, m, i))
    b = Batch(0, use_default_tuning=False)
    try:
        b.set_rules([{"op": 0, "format": f, "level": -1, "tile_blocks": tile, "cost_per_block": 1.0} for f in (1, 3)])
        outs = run_jobs(jobs, batch=b)
        assert [k for k, (o, e) in enumerate(zip(outs, expected)) if o != e] == []
    finally:
        b.close()
