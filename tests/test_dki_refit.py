"""The fast constrained re-fit (DKI's D, V and bound D - V rows) at the edges of its tables, against
the oracle and against the general re-fit, which takes the same constraints in another order."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _table(n, seed):
    from larmor_b200.types import GradientTable

    rng = np.random.default_rng(seed)
    d = rng.standard_normal((n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    b = np.where(np.arange(n) % 2 == 0, 1000.0, 2000.0)
    b[0] = 0.0
    d[0] = 0.0
    return rng, GradientTable(b, d)


# Tables on both sides of whole 8-row tiles and of the fast kernel's largest (302).
@pytest.mark.parametrize("n, v, weighted", [
    (63, 40, True), (64, 400, False), (65, 1, True), (134, 300, True), (301, 50, True), (302, 50, False),
    (303, 50, True)])
def test_fast_and_general_refits_agree_with_the_oracle(cuda, oracle, n, v, weighted):
    from larmor_b200 import _core
    from larmor_b200.dwi.dki import dki_constraints, dki_design

    rng, gtab = _table(n, n)
    x, g = dki_design(gtab), np.ascontiguousarray(dki_constraints(gtab))
    axis = rng.standard_normal((v, 3))
    axis /= np.linalg.norm(axis, axis=1, keepdims=True)
    cos2 = (axis @ gtab.bvecs.T) ** 2
    clean = 0.5 * np.exp(-gtab.bvals * 2e-3 * cos2) + 0.5 * np.exp(-gtab.bvals * (0.6e-3 + 1.4e-3 * cos2))
    log_s = np.log(1000.0 * np.sqrt((clean + rng.normal(0, 1 / 20, clean.shape)) ** 2
                                    + rng.normal(0, 1 / 20, clean.shape) ** 2))
    want, want_broke = oracle.fit_log_signal(x, g, log_s, weighted)
    got, broke = _core.fit_log_signal(x, g, log_s, weighted, 20, 1e-6, 1)
    other, other_broke = _core.fit_log_signal(x, np.ascontiguousarray(g[::-1]), log_s, weighted, 20, 1e-6, 1)
    np.testing.assert_array_equal(broke, want_broke)
    np.testing.assert_array_equal(other_broke, want_broke)
    assert v == 1 or broke.any()
    # The reference's bound, 1e-10 on column-scaled parameters, holds at its table of 134; a QR's
    # forward error grows with the weighted design's condition, so 10 cond(W^1/2 X)^2 eps covers
    # the smallest tables (whose reweighting itself solves the normal equations).
    scale = np.linalg.norm(x, axis=0)
    cond = max(np.linalg.cond(np.exp(p @ x.T - (p @ x.T).max())[:, None] * (x / scale)) for p in want)
    tol = max(1e-10, 10 * cond**2 * np.finfo(np.float64).eps) * np.abs(want * scale).max()
    assert np.abs((got - want) * scale).max() <= tol
    assert np.abs((other - want) * scale).max() <= tol


def test_a_repeated_violator_list_is_walked_afresh(cuda):
    """Two calls in a row on one design: the first marks its entries done, the second fills the list again."""
    from larmor_b200 import _core
    from larmor_b200.dwi.dki import dki_constraints, dki_design

    rng, gtab = _table(90, 5)
    x, g = dki_design(gtab), np.ascontiguousarray(dki_constraints(gtab))
    log_s = np.log(1000.0 * np.exp(-gtab.bvals * 1e-3) * rng.uniform(0.7, 1.3, (200, 90)))
    first, broke = _core.fit_log_signal(x, g, log_s, True, 20, 1e-6, 1)
    again, _ = _core.fit_log_signal(x, g, log_s, True, 20, 1e-6, 1)
    assert broke.any()
    np.testing.assert_array_equal(first, again)
