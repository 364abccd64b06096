"""GPU: the grid and CTA size that a batch was given hold for all of its kernels, as they stand in its graph."""

import ctypes

import numpy as np
import pytest

import workloads as syn
from quicktex_b200 import capi
from quicktex_b200.batch import Batch, Job, run_jobs

pytestmark = pytest.mark.gpu


def _jobs():
    img = np.ascontiguousarray(syn.alpha_mix(300, 260, workload=3, stream=12))
    jobs = [Job.encode("bc1", img, 300, 260, level=lv, color_mode=m, interpolator=i) for lv, m, i in ((0, 0x04, 0), (5, 0x03, 1), (10, 0x13, 3), (18, 0x13, 2))]
    return jobs + [Job.encode("bc3", img, 300, 260, level=17), Job.encode("bc4", img, 300, 260, channel=1)]


def _kernels(b, jobs):
    """The outputs, (CTAs, threads per CTA) of each kernel that the last run launched, and how many of them wait for another."""
    out = run_jobs(jobs, batch=b)
    grid, block = ((ctypes.c_uint * 26)() for _ in range(2))
    n = capi.lib().qtk_batch_kernels(b.handle, grid, block)
    return out, list(zip(grid[:n], block[:n])), capi.lib().qtk_batch_edges(b.handle)


@pytest.mark.parametrize("threads,ctas", [(128, 1), (128, 3), (64, 1), (64, 3), (32, 1), (32, 2), (32, 3)])
def test_a_limited_grid_holds_for_every_kernel(threads, ctas):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    jobs = _jobs()
    ref = run_jobs(jobs)
    b = Batch(0)
    try:
        b.set_threads(threads)
        b.set_grid(ctas)
        out, kernels, edges = _kernels(b, jobs)
    finally:
        b.close()
    assert out == ref
    assert len(kernels) == 5  # BC4; cooperative; Check2 four-colour; Faster three-colour; Check2 three-colour + black
    assert max(n * t for n, t in kernels) <= sms * ctas * threads
    assert edges == 4  # one after the other


def test_without_a_limit_each_kernel_fills_the_gpu():
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    jobs = _jobs()
    b = Batch(0)
    try:
        for threads, ctas in ((128, 0), (128, 4), (64, 8), (32, 0)):
            b.set_threads(threads)
            b.set_grid(ctas)
            out, kernels, edges = _kernels(b, jobs)
            assert edges == 0 and len(kernels) == 5 and min(n for n, _ in kernels) >= 4 * sms
            assert {t for _, t in kernels} == {threads, 128}
    finally:
        b.close()
