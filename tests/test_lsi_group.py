"""The LSI group kernel (a group of warps per voxel, E^T and the voxels' factors in shared memory)
at the edges of its sizes, against the oracle: constraint counts around its lanes' shares, active
sets on both sides of 32, problems it hands to the one-warp kernel, voxel counts around a CTA's
eight, near-dependent constraints (the QR variant), and signals with f = 0 or NaN."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(seed, m, n, k):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((m, n))
    g = np.vstack([np.eye(n), rng.uniform(0.0, 1.0, (max(0, k - n), n))])[:k]
    return rng, np.ascontiguousarray(a), np.ascontiguousarray(g)


def _fit(a, g, signals):
    from larmor_b200 import _core

    return _core.fit_lsi(np.ascontiguousarray(signals), _core.LsiDesign(a, g, 0.0), 1)


# Random orthant problems: cond(a) < 1e3, so both fits carry far less than 1e-9 of the largest.
@pytest.mark.parametrize("m, n, k, v", [
    (5, 2, 1, 1), (40, 10, 10, 7), (60, 31, 32, 8), (60, 32, 33, 9), (90, 47, 302, 33), (120, 63, 319, 17),
    (60, 33, 320, 16), (60, 33, 321, 16), (90, 47, 512, 9)])
def test_group_kernel_matches_the_oracle(cuda, oracle, m, n, k, v):
    rng, a, g = _problem(100 * n + k, m, n, k)
    signals = 3.0 * rng.standard_normal((v, m))
    x, conv = _fit(a, g, signals)
    rx, rconv, *_ = oracle.fit_lsi(a, g, 0.0, signals, details=True)
    np.testing.assert_array_equal(conv, rconv)
    assert np.abs(x - rx).max() <= 1e-9 * np.abs(rx).max()


def test_near_dependent_constraints(cuda, oracle):
    """Every constraint twice, the copies 1e-7 apart: factors whose pivots fail go to the QR
    variant. Which copy is active moves x by about their distance."""
    rng, a, g = _problem(7, 60, 12, 40)
    g = np.ascontiguousarray(np.vstack([g, g + 1e-7 * rng.standard_normal(g.shape)]))
    signals = 3.0 * rng.standard_normal((64, 60))
    x, conv = _fit(a, g, signals)
    rx, rconv, *_ = oracle.fit_lsi(a, g, 0.0, signals, details=True)
    np.testing.assert_array_equal(conv, rconv)
    assert np.abs(x - rx).max() <= 1e-5 * np.abs(rx).max()
    assert (x @ g.T).min() >= -1e-8 * np.abs(x).max()


def test_zero_and_nan_signals_among_others(cuda):
    rng, a, g = _problem(11, 60, 20, 50)
    signals = rng.standard_normal((19, 60))
    plain, _ = _fit(a, g, signals)
    odd = signals.copy()
    odd[3] = 0.0
    odd[8, 5] = np.nan
    x, _ = _fit(a, g, odd)
    keep = np.setdiff1d(np.arange(19), [3, 8])
    np.testing.assert_array_equal(x[keep], plain[keep])
    np.testing.assert_array_equal(x[3], np.zeros(20))
    assert np.isnan(x[8]).all()
