"""CPU: bench.py's figures of the reference's CPU encoder, where that is not built."""

import numpy as np

import bench
import oracle


def test_a_missing_reference_does_not_lose_the_line(monkeypatch):
    monkeypatch.setattr(oracle, "reference_available", lambda: False)
    line = bench.cpu_lines(np.zeros((512, 512, 4), np.uint8))
    assert set(line) == {"cpu_baseline"} and "not built" in line["cpu_baseline"]["unavailable"]
