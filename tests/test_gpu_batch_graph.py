"""GPU: a batch keeps one graph of kernels whatever mixes it runs."""

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
