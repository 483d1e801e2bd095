"""One step of damped Richardson-Lucy against its formula in exact arithmetic: f (1 + d (k - p) / (p + 1e-16)) with
d = f^8 / (f^8 + nu^8) (a constant signal has strength 1), k = K^T s and p = K^T K f. The kernel forms two steps with
one reciprocal; its roundings are counted here, and the ends of the range, where a product of the denominators would
vanish or overflow, have to come out as the formula gives them."""

from __future__ import annotations

from fractions import Fraction

import numpy as np
import pytest

U = 2.0**-53


def _step(torch, ks, gram, nu, init):
    """The amplitudes after one step from `init`, with K^T s = ks and K^T K = diag(gram)."""
    from larmor_b200 import _core
    from larmor_b200.sd.solvers import fit_single_tissue_on_device

    c = len(ks)
    k_t = np.zeros((c, 6))
    k_t[:, 0] = ks
    solver = _core.FodSolver.drl(k_t, np.diag(gram), nu, 1, init)
    return fit_single_tissue_on_device(torch.ones((3, 6), dtype=torch.float64, device="cuda"), solver).cpu().numpy()


# The kernels of up to 64, 320 and 640 directions, even and odd.
SIZES = [8, 37, 64, 65, 300, 321, 640]


@pytest.mark.gpu
@pytest.mark.parametrize("c", SIZES)
@pytest.mark.parametrize("nu", [0.0, 6e-4, 0.4])
@pytest.mark.parametrize("init", [1 / 300, 0.5, 700.0])
def test_a_step_is_the_formula_within_its_roundings(cuda, c, nu, init):
    """f^8 in the numerator and in the denominator 7 u each, and nu^8 no more; one u for each of the sum f^8 + nu^8,
    k - p, p + 1e-16, the products above and below, the product of the two below, its reciprocal, the products with the
    other and with what is above, 1 + step and the product with f."""
    rng = np.random.default_rng(c)
    ks, gram = 10.0 ** rng.uniform(-3, 3, c), 10.0 ** rng.uniform(-3, 3, c)
    got = _step(cuda, ks, gram, nu, init)
    np.testing.assert_array_equal(got, np.broadcast_to(got[0], got.shape))
    f, n8, tiny = Fraction(init), Fraction(nu) ** 8, Fraction(1e-16)
    for d in range(c):
        pred = Fraction(init * gram[d])
        step = f**8 / (f**8 + n8) * (Fraction(ks[d]) - pred) / (pred + tiny)
        want = max(f * (1 + step), Fraction(1e-6))
        assert abs(Fraction(got[0, d]) - want) <= Fraction(25 * U) * f * (1 + abs(step)), (d, got[0, d], float(want))


@pytest.mark.gpu
@pytest.mark.parametrize("c", SIZES)
def test_a_step_at_the_ends_of_the_range(cuda, c):
    # p = -1e-16 exactly: the ratio is (k + 1e-16) / 0, the amplitude infinite.
    init = 2.0**-7
    got = _step(cuda, np.ones(c), np.full(c, -1e-16 / init), 0.0, init)
    assert np.all(got == np.inf)
    # f^8 (p + 1e-16) past the largest number, f^8 / (f^8 + nu^8) and the ratio far inside.
    init, gram = 1e36, np.full(c, 1e-10)
    got = _step(cuda, np.full(c, 3e26), gram, 1e20, init)
    np.testing.assert_allclose(got, 3e36, rtol=40 * U)
    # and below the smallest.
    init = 1e-39
    got = _step(cuda, np.full(c, 1.0), np.full(c, 1e20), 0.0, init)
    np.testing.assert_allclose(got, init * (1 + (1.0 - 1e-19) / (1e-19 + 1e-16)), rtol=0.0, atol=1e-6 + 1e-12)
