"""A log-signal design holds its matrices on the device and nothing that no kernel reads."""

from __future__ import annotations

import gc

import numpy as np
import pytest


@pytest.mark.gpu
def test_a_design_holds_its_matrices_and_no_products(cuda):
    """X and its pseudo-inverse, in double and in float: 24 p bytes per measurement (10.6 MB here), each array rounded
    up to an allocation's granularity (2 MiB). The products of X's columns would add 12 p (p + 1) / 2 (60 MB)."""
    from larmor_b200 import _core

    n, p = 20_000, 22
    x = np.random.default_rng(1).normal(size=(n, p))
    _core.LogDesign(x[:100], np.zeros((0, p)))  # the library's own state
    gc.collect()
    cuda.cuda.synchronize()
    before = cuda.cuda.mem_get_info()[0]
    design = _core.LogDesign(x, np.zeros((0, p)))
    used = before - cuda.cuda.mem_get_info()[0]
    assert design.handle is not None
    assert used <= 24 * n * p + 8 * (2 << 20), used
