"""The product of a short series with many directions takes no longer than the tiled product it replaces, also for few
rows, where spreading it over the SMs counts."""

from __future__ import annotations

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize(("ca", "ncoef", "rows"), [(6, 642, 500), (15, 642, 32), (15, 642, 4000), (45, 300, 500),
                                                   (45, 642, 1), (45, 642, 2000), (48, 2562, 500)])
def test_the_expansion_of_few_rows_is_spread_over_the_sms(cuda, ca, ncoef, rows):
    """exact_integral takes the tiled product of the same shape. The least of twenty launches each; a launch is a few
    microseconds, so a quarter more is within their spread, where unspread the expansion took 1.5 to 4 times as long."""
    from larmor_b200 import _core

    rng = np.random.default_rng(ca)
    projector = _core.ShProjector(rng.normal(size=(ncoef, ca)))
    rows = cuda.from_numpy(rng.normal(size=(rows, ca))).cuda()
    ms = {}
    for tiled in (False, True):
        times = []
        for _ in range(22):
            _core.kernel_timing(True)
            _core.project_sh_device(projector, rows, tiled)
            cuda.cuda.synchronize()
            times.append(_core.kernel_time("project_sh_kernel")[0])
            _core.kernel_timing(False)
        ms[tiled] = min(times[2:])
    assert ms[False] <= 1.25 * ms[True], ms
