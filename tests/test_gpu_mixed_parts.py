"""The mixed pair kernel's forms at the sizes where the parts of its sums change, with rows that
overflow and non-finite records: sorted every step, on neighbour lists (a step that sorts) and in
a batch give the same bits; the rates are the FP64 form's within FP32 rounding.

Tolerance against FP64: 1e-4 of the field's largest value, the bar of the mixed form's own test
(~30 terms of FP32 rounding 6e-8 with cancellation between neighbours)."""
import numpy as np
import pytest

from conftest import bits_equal, rel_err
from helpers import load_product, perturbed_scene

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "S", "rho", "T", "pos_t", "vel_t", "S_t", "rho_t", "T_t", "blanked", "id")


def scene(mf, ny, kind):
    st = perturbed_scene(mf, ny=ny, seed=70 + ny, blank_frac=0.01)
    wp = np.flatnonzero((st["tool_p"] == 0.0) & (st["blanked"] == 0.0))
    rng = np.random.default_rng(ny)
    if kind == "crowded":  # ~150 neighbours each: more than a row holds
        st["pos"][wp[:150]] = st["pos"][wp[len(wp) // 2]] + rng.uniform(-0.5, 0.5, (150, 2)) * st["grid"][2]
    elif kind == "nonfinite":
        st["S"][wp[len(wp) // 3], 0] = np.nan
        st["vel"][wp[2 * len(wp) // 3], 1] = np.inf
    return st


# 2,724 and 28,156 particles (four parts), 29,736 and 45,724 (two), 47,733 (one)
@pytest.mark.parametrize("ny", [12, 37, 38, 47, 48])
@pytest.mark.parametrize("kind", ["plain", "crowded", "nonfinite"])
def test_forms_agree(mf, ny, kind):
    st = scene(mf, ny, kind)
    load = lambda **kw: load_product(mf, st, precision=mf.PRECISION_MIXED, **kw)  # noqa: E731
    a, b, c, d = load(), load(flags=mf.OPT_NEIGHBOUR_LISTS), load(), load()
    batch = mf.Batch([c, d], steps_per_launch=2)
    assert batch.fused
    a.step(1)
    b.step(1)
    f64 = load_product(mf, st)
    f64.step(1)
    if kind != "crowded":  # (a crowded list row is flagged as full)
        assert b.status()["error_flags"] == 0
    for f in FIELDS:
        assert bits_equal(a.get(f), b.get(f)), f
    assert np.array_equal(a.get("blanked"), f64.get("blanked"))
    live = f64.get("blanked") == 0.0
    for f in ("vel_t", "S_t", "rho_t"):
        x, y = a.get(f)[live], f64.get(f)[live]
        fin = np.isfinite(y)
        assert np.array_equal(fin, np.isfinite(x)), f
        assert rel_err(x[fin], y[fin]) <= 1e-4, f
    a.step(1)
    batch.step(1)
    for f in FIELDS:
        assert bits_equal(a.get(f), c.get(f)) and bits_equal(c.get(f), d.get(f)), f
    batch.close()
