"""A DTI voxel's fit does not depend on the call it is part of: the same bits in a whole volume and in its pieces, and
the same tables accepted, whatever the number of voxels."""

from __future__ import annotations

import numpy as np
import pytest

from larmor_b200 import _lib
from larmor_b200.dwi.dti import dti_design
from larmor_b200.synthetic import unit_directions
from larmor_b200.types import GradientTable

pytestmark = pytest.mark.gpu


def _problem(torch, n, v):
    rng = np.random.default_rng(n)
    g = GradientTable(np.concatenate([[0.0], np.full(n - 1, 1000.0)]), np.vstack([np.zeros(3), unit_directions(rng, n - 1)]))
    s = np.abs(800.0 * np.exp(-1.2 * rng.uniform(0.2, 1.5, (v, n))) + rng.normal(0, 30.0, (v, n))) + 1.0
    return dti_design(g), torch.from_numpy(s.astype(np.float32)).cuda()


def _fit(torch, design, s, weighted, precision):
    from larmor_b200 import _core

    v = len(s)
    maps = torch.empty((16, v), dtype=torch.float32, device="cuda")
    npd = torch.empty(v, dtype=torch.uint8, device="cuda")
    params = torch.empty((v, 7), dtype=torch.float64, device="cuda")
    floor = torch.ones(v, dtype=torch.float64, device="cuda")
    _core.fit_dti_maps_device(design, s, floor, weighted, maps, npd, params, precision=precision)
    fitted = torch.empty((v, 7), dtype=torch.float64, device="cuda")
    broke = torch.empty(v, dtype=torch.uint8, device="cuda")
    steps = torch.empty(v, dtype=torch.int32, device="cuda")
    _core.fit_log_signal_device(design, torch.log(s.double()), weighted, 20, 1e-6, fitted, broke, steps, precision)
    return params.cpu().numpy(), maps.T.cpu().numpy(), fitted.cpu().numpy(), steps.cpu().numpy()


# Tables of a voxel's smallest share of measurements, of whole and ragged shares, and around the table size where the
# lanes' classes change; the pieces lie on both sides of every voxel count where the lanes per voxel do.
@pytest.mark.parametrize("n", [7, 8, 31, 37, 64, 95, 96, 135])
@pytest.mark.parametrize(("weighted", "precision"), [(True, _lib.LAR_FP64), (False, _lib.LAR_FP64), (True, _lib.LAR_FP32)])
def test_a_voxel_has_the_same_bits_in_any_call(cuda, n, weighted, precision):
    from larmor_b200 import _core

    design, s = _problem(cuda, n, 32_000)
    handle = _core.LogDesign(design, np.zeros((0, 7)))
    whole = _fit(cuda, handle, s, weighted, precision)
    ends = [0, 1, 18, 1_001, 5_001, 15_001, 32_000]  # pieces of 1, 17, 983, 4,000, 10,000 and 16,999 voxels
    pieces = [_fit(cuda, handle, s[a:b].contiguous(), weighted, precision) for a, b in zip(ends, ends[1:])]
    for k, all_at_once in enumerate(whole):
        np.testing.assert_array_equal(np.concatenate([p[k] for p in pieces]), all_at_once)


def test_large_tables_are_accepted_at_every_call_size(cuda):
    """1,200 measurements fit the shared memory at eight lanes per voxel, in small and in large calls."""
    from larmor_b200 import _core

    design, s = _problem(cuda, 1_200, 5_001)
    handle = _core.LogDesign(design, np.zeros((0, 7)))
    small, large = _fit(cuda, handle, s[:300].contiguous(), True, _lib.LAR_FP64), _fit(cuda, handle, s, True, _lib.LAR_FP64)
    for a, b in zip(small, large):
        np.testing.assert_array_equal(a, b[:300])


@pytest.mark.parametrize("n", [31, 64, 95, 96, 135])
@pytest.mark.parametrize("v", [50, 9_000, 25_000])
def test_the_fallback_is_the_unweighted_fit(cuda, n, v):
    """Every third voxel's diffusion-weighted signals lie e^2000 below its one b0: all their weights are exactly 0, the
    normal matrix has exactly zero pivots, and the ordinary fit stands: the bits of an unweighted call's, whatever the
    lanes of either."""
    from larmor_b200 import _core

    design, s = _problem(cuda, n, v)
    handle = _core.LogDesign(design, np.zeros((0, 7)))
    log_s = cuda.log(s.double())
    log_s[::3, 1:] -= 2000.0
    fits = []
    for weighted in (True, False):
        params = cuda.empty((v, 7), dtype=cuda.float64, device="cuda")
        broke, steps = (cuda.empty(v, dtype=kind, device="cuda") for kind in (cuda.uint8, cuda.int32))
        _core.fit_log_signal_device(handle, log_s, weighted, 20, 1e-6, params, broke, steps)
        fits.append(params.cpu().numpy())
    np.testing.assert_array_equal(fits[0][::3], fits[1][::3])
    assert (fits[0][1::3] != fits[1][1::3]).any()
