"""The lean ridge NNLS (a warp per voxel, at most 32 active columns) at the edges of its sizes inside the
multi-tissue fit, against the oracle: column counts around a lane's share and around the limits where
the general kernel takes over, active sets past 32, ragged voxel counts, and a NaN signal."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M = 120


def _case(seed, c_lr, c_hr, v, sparse=True):
    rng = np.random.default_rng(seed)
    k_lr, k_hr = (np.ascontiguousarray(np.abs(rng.standard_normal((M, c)))) for c in (c_lr, c_hr))
    iso = np.ascontiguousarray(np.stack([np.exp(-np.linspace(0, 1, M)), np.exp(-np.linspace(0, 4, M))], axis=1))
    x = rng.uniform(0.0, 1.0, (v, c_hr)) * (rng.uniform(size=(v, c_hr)) < (0.1 if sparse else 0.9))
    s = x @ k_hr.T / c_hr + rng.uniform(0.0, 0.3, (v, 2)) @ iso.T + 0.02 * rng.standard_normal((v, M))
    return k_lr, k_hr, iso, np.ascontiguousarray(np.maximum(s, 0.0))


def _device(k_lr, k_hr, iso, s):
    from larmor_b200 import _core

    lr = _core.DeconvKernel(k_lr, iso, iso, [(0, k_lr.shape[1])])
    hr = _core.DeconvKernel(k_hr, iso, iso, [(0, k_hr.shape[1])])
    return _core.fit_multi_tissue(s, np.ones(M), lr, _core.FodSolver.l2nnls(k_lr, 0.0, 1e-6), hr,
                                  _core.FodSolver.l2nnls(k_hr, 0.1, 1e-6), 20, 1e-7, 1e-2, 1)


def _oracle(oracle, k_lr, k_hr, iso, s):
    kern = lambda k, **more: dict(k_aniso=k, k_iso=iso, w_k_iso=iso, w_k_aniso=k, **more)  # noqa: E731
    return oracle.fit_multi_tissue(s, np.ones(M), kern(k_lr), kern(k_hr, blocks=[(0, k_hr.shape[1])]), max_rounds=20)


# The Gram matrices are well conditioned (|N| columns of 120 rows, ridge 0.1 at high resolution): the
# repository's bounds, FODs within 1e-9 of the voxel's largest amplitude and fractions 1e-9.
@pytest.mark.parametrize("c_lr, c_hr, v, sparse", [
    (1, 65, 1, True), (31, 64, 17, True), (32, 65, 33, True), (33, 96, 40, True), (47, 97, 31, True),
    (48, 110, 64, True), (49, 100, 30, True), (40, 100, 150, False), (20, 320, 9, True), (20, 321, 9, True)])
def test_lean_nnls_matches_the_oracle(cuda, oracle, c_lr, c_hr, v, sparse):
    k_lr, k_hr, iso, s = _case(1000 * c_lr + c_hr, c_lr, c_hr, v, sparse)
    fods, fractions = _device(k_lr, k_hr, iso, s)
    rf, rfr = _oracle(oracle, k_lr, k_hr, iso, s)
    largest = np.abs(rf).max(axis=1, keepdims=True) + 1e-300
    assert (np.abs(fods - rf) / largest).max() <= 1e-9
    assert np.abs(fractions - rfr).max() <= 1e-9
    if not sparse:
        assert ((fods > 0).sum(axis=1) > 32).any()  # some voxels outgrow the lean factor


# Kernels within [0, 1] whose maximum can lie in `top` rows only (row r is 1 but for one entry): the
# lane-per-voxel fractions take up to 16 such rows and solutions that are mostly zero; 17 rows, more
# columns, four isotropic tissues or dense solutions go the general way.
@pytest.mark.parametrize("top, c_lr, v, sparse, ci", [
    (1, 44, 1, True, 2), (1, 1, 33, True, 1), (2, 47, 64, True, 3), (16, 48, 31, True, 2), (17, 40, 20, True, 2),
    (1, 49, 20, True, 2), (1, 20, 40, True, 0), (1, 20, 40, True, 4), (1, 40, 70, False, 2)])
def test_fractions_of_bounded_kernels(cuda, oracle, top, c_lr, v, sparse, ci):
    from larmor_b200 import _core

    rng = np.random.default_rng(100 * top + c_lr)
    k_lr, k_hr = (rng.uniform(0.0, 1.0, (M, c)) ** 3 for c in (c_lr, 100))
    k_lr[:top] = 1.0
    for r in range(1, top):
        k_lr[r, r % c_lr] = 1.0 + 0.01 * r
        k_lr[r, (r + 1) % c_lr] = 0.5
    k_lr, k_hr = np.ascontiguousarray(k_lr), np.ascontiguousarray(k_hr)
    iso = np.ascontiguousarray(np.exp(-np.linspace(0, 1, M)[:, None] * (1.0 + 2.0 * np.arange(ci))))
    x = rng.uniform(0.0, 1.0, (v, c_lr)) * (rng.uniform(size=(v, c_lr)) < (0.15 if sparse else 0.95))
    s = np.ascontiguousarray(np.maximum(
        x @ k_lr.T / c_lr + rng.uniform(0.0, 0.2, (v, ci)) @ iso.T + 0.01 * rng.standard_normal((v, M)), 0.0))
    empty = ci == 0
    lr, hr = (_core.DeconvKernel(k, None if empty else iso, None if empty else iso, [(0, k.shape[1])])
              for k in (k_lr, k_hr))
    fods, fractions = _core.fit_multi_tissue(s, np.ones(M), lr, _core.FodSolver.l2nnls(k_lr, 0.0, 1e-6), hr,
                                             _core.FodSolver.l2nnls(k_hr, 0.1, 1e-6), 20, 1e-7, 1e-2, 1)
    rf, rfr = _oracle(oracle, k_lr, k_hr, iso, s)
    assert np.abs(fods - rf).max() <= 1e-8 * np.abs(rf).max()
    assert np.abs(fractions - rfr).max() <= 1e-8


def test_a_nan_voxel_leaves_the_others_alone(cuda):
    k_lr, k_hr, iso, s = _case(3, 44, 100, 50)
    plain, plain_fr = _device(k_lr, k_hr, iso, s)
    s[17, 5] = np.nan
    fods, fractions = _device(k_lr, k_hr, iso, s)
    keep = np.arange(50) != 17
    np.testing.assert_array_equal(fods[keep], plain[keep])
    np.testing.assert_array_equal(fractions[keep], plain_fr[keep])
