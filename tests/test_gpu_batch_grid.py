"""GPU: the grid and CTA size that a batch was given hold for all of its kernels, as the CUDA profiler records them."""

import json

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


def _kernels(b, jobs, tmp_path):
    import torch
    from torch.profiler import ProfilerActivity, profile

    run_jobs(jobs, batch=b)
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        out = run_jobs(jobs, batch=b)
        torch.cuda.synchronize()
    path = tmp_path / "trace.json"
    prof.export_chrome_trace(str(path))
    ev = [e for e in json.loads(path.read_text())["traceEvents"] if e.get("cat") == "kernel" and "k_batch" in e["name"]]
    return out, sorted(ev, key=lambda e: e["ts"])


@pytest.mark.parametrize("threads,ctas", [(128, 1), (128, 3), (64, 1), (64, 3), (32, 1), (32, 2), (32, 3)])
def test_a_limited_grid_holds_for_every_kernel(threads, ctas, tmp_path):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    jobs = _jobs()
    ref = run_jobs(jobs)
    b = Batch(0)
    try:
        b.set_threads(threads)
        b.set_grid(ctas)
        out, ev = _kernels(b, jobs, tmp_path)
        edges = capi.lib().qtk_batch_edges(b.handle)
    finally:
        b.close()
    assert out == ref
    assert len(ev) == 5  # BC4; cooperative; Check2 four-colour; Faster three-colour; Check2 three-colour + black
    for e in ev:
        grid, block = (np.prod(e["args"][k]) for k in ("grid", "block"))
        assert grid * block <= sms * ctas * threads, e["name"]
    assert edges == len(ev) - 1  # one after the other


def test_without_a_limit_each_kernel_fills_the_gpu(tmp_path):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    jobs = _jobs()
    b = Batch(0)
    try:
        for threads, ctas in ((128, 0), (128, 4), (64, 8), (32, 0)):
            b.set_threads(threads)
            b.set_grid(ctas)
            out, ev = _kernels(b, jobs, tmp_path)
            assert capi.lib().qtk_batch_edges(b.handle) == 0
            assert len(ev) == 5 and all(np.prod(e["args"]["grid"]) >= 4 * sms for e in ev)
            assert {int(np.prod(e["args"]["block"])) for e in ev} == {threads, 128}
    finally:
        b.close()
