"""GPU: a batch keeps one graph of kernels whatever mixes it runs, and cuts a short run into enough tiles to fill the GPU."""

import random

import pytest

from quicktex_b200 import capi
from quicktex_b200.batch import Batch, Job, run_jobs

import numpy as np
import workloads as syn

pytestmark = pytest.mark.gpu


def _graphs(b):
    return capi.lib().qtk_batch_graphs(b.handle)


def _mixes(seed, n):
    """n sets of kernels: small textures at levels 0 (Check2), 5 (Faster), 4 (no kernel of its own) and 18, any mode and interpolation"""
    rng = random.Random(seed)
    img = syn.block_mix(16, 12, workload=3, stream=seed)
    every = [Job.encode("bc1", img, 16, 12, level=lv, color_mode=m, interpolator=i) for lv in (0, 5) for m in (0x04, 0x03, 0x13) for i in range(4)]
    every += [Job.encode("bc1", img, 16, 12, level=18), Job.encode("bc4", img, 16, 12, channel=0)]
    return every, [rng.sample(every, rng.randint(1, 5)) for _ in range(n)]


def test_mixes_do_not_add_graphs():
    every, mixes = _mixes(5, 60)
    expected = {id(j): out for j, out in zip(every, run_jobs(every))}
    b = Batch(0)
    try:
        b.reserve(64, 64)
        assert _graphs(b) == 0
        for mix in mixes:
            assert run_jobs(mix, batch=b) == [expected[id(j)] for j in mix]
        run_jobs(every, batch=b)
        whole = _graphs(b)
        for mix in _mixes(6, 60)[1]:
            run_jobs(mix, batch=b)
        assert _graphs(b) == whole <= len(every)
    finally:
        b.close()


def test_a_larger_queue_keeps_its_kernels():
    every, _ = _mixes(7, 1)
    b = Batch(0)
    try:
        first = run_jobs(every[:3], batch=b)
        n = _graphs(b)
        big = [Job.encode("bc1", np.zeros((4, 4, 4), np.uint8), 4, 4, level=0)] * 200  # more textures than the queue holds
        run_jobs(big, batch=b)
        assert _graphs(b) == n + 1
        assert run_jobs(every[:3], batch=b) == first
    finally:
        b.close()


def _tiles(b, jobs):
    run_jobs(jobs, batch=b)
    return b.last_tiles()


def test_a_short_run_is_cut_finer_whatever_ran_before():
    import torch

    warps = 16 * torch.cuda.get_device_properties(0).multi_processor_count
    img = syn.alpha_mix(260, 252, workload=3, stream=8)
    short = [Job.encode("bc1", img, 260, 252, level=5), Job.encode("bc3", img, 260, 252, level=18), Job.encode("bc4", img, 260, 252, channel=0)]
    blocks = 65 * 63
    fresh, b = Batch(0), Batch(0)
    try:
        b.reserve(100, 1 << 17)
        n = _tiles(fresh, short)
        # a block per lane or, for the cooperative encoder, at most one warp's share; no more than a tile per warp and texture
        assert n >= 2 * ((blocks + 31) // 32) + min(blocks, warps // 2)
        assert n <= 2 * warps + 3 * blocks // 256 + 3
        assert _tiles(b, short) == n
        _tiles(fresh, short * 40)
        assert _tiles(fresh, short) == n
        assert run_jobs(short, batch=fresh) == [run_jobs([j])[0] for j in short]
    finally:
        b.close()
        fresh.close()


@pytest.mark.parametrize("cost", [1e-38, 1e-3, 1.0, 3e38, float("inf")])
def test_any_cost_gives_tiles_of_every_block(cost):
    img = syn.block_mix(60, 52, workload=3, stream=9)
    jobs = [Job.encode("bc1", img, 60, 52, level=18), Job.encode("bc1", img, 60, 52, level=0), Job.encode("bc4", img, 60, 52, channel=0)]
    b = Batch(0, use_default_tuning=False)
    try:
        b.set_rules([{"op": 0, "format": 1, "level": 18, "tile_blocks": 64, "cost_per_block": cost}, {"op": 0, "format": 4, "tile_blocks": 7, "cost_per_block": 1.0}])
        assert run_jobs(jobs, batch=b) == run_jobs(jobs)
    finally:
        b.close()
