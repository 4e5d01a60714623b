"""The differentiable step at particle counts on each side of its lanes-per-particle rule
(8,192 and 18,944), against the plain FP64 steps and between its forms.

Tolerances: the mean force within 1e-12 of the FP64 steps' (five steps of the same arithmetic,
last-bit differences of the sums only); each direction of the six-direction pass within 1e-9 of
its single pass (the bar of the six-direction test at one size)."""
import numpy as np
import pytest

from helpers import load_product, perturbed_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny", [20, 21, 30, 31])  # 7,970 | 8,822 and 18,310 | 19,589 particles
def test_values_and_directions(mf, ny):
    st = perturbed_scene(mf, ny=ny, seed=50 + ny, blank_frac=0.01)
    st["S"] *= 3.0
    ctx = load_product(mf, st)
    mean, d6 = ctx.tangent_mean_force_all(1, 4)
    ref = load_product(mf, st)
    ref.step(5)
    np.testing.assert_allclose(mean, ref.force_log()[1:].mean(axis=0), rtol=1e-12, atol=0.0)
    for k in (0, 5):
        m1, d = ctx.tangent_mean_force(1, 4, k)
        assert np.array_equal(m1, mean)
        np.testing.assert_allclose(d6[k], d, rtol=1e-9, atol=1e-9 * np.abs(d).max())
    # the workspace a larger call left behind does not reach a smaller one
    again, e6 = ctx.tangent_mean_force_all(1, 4)
    assert np.array_equal(again, mean) and np.array_equal(e6, d6)
