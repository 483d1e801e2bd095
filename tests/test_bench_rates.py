"""The rates that the bench lines divide by."""

from __future__ import annotations

import re
from pathlib import Path

BENCH = (Path(__file__).resolve().parents[1] / "bench.py").read_text()


def test_the_fp64_rate_is_the_measured_one():
    """148 SMs at 1,965 MHz: a loop of independent DFMAs measured 36.8 TFLOP/s, within 2% of 64 FMAs per SM and cycle."""
    per_cycle = int(re.search(r"^FP64_FMA_PER_SM_CYCLE = (\d+)$", BENCH, re.M).group(1))
    assert abs(148 * per_cycle * 2 * 1965e6 / 36.8e12 - 1) < 0.02
    assert "peak = fp64_core_tflops(" in BENCH and "sms * 32 *" not in BENCH
