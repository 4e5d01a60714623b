"""The FP64 pair kernel's neighbour lists at the sizes where its lanes per particle change, with
windows that overflow a list row, non-finite neighbours and particles outside the grid, against
the oracle.

Tolerance: 1e-12 of the field's largest value, the single-step bar for pair sums from identical
inputs (sums of ~30 terms, of ~400 in the crowded cell, each rounded to ~1e-16)."""
import numpy as np
import pytest

from conftest import rel_err
from helpers import load_oracle, load_product, perturbed_scene

pytestmark = pytest.mark.gpu

RATES = ("pos_t", "vel_t", "S_t", "rho_t", "T_t", "S_der", "v_der")


# 2,724 and 18,310 particles (four lanes), 19,589 and 36,475 (two), 38,139 and 116,726 (one)
@pytest.mark.parametrize("ny", [12, 30, 31, 42, 43, 75])
@pytest.mark.parametrize("kind", ["plain", "crowded", "nonfinite", "outside"])
def test_pair_sums(mf, orc, ny, kind):
    st = perturbed_scene(mf, ny=ny, seed=40 + ny, blank_frac=0.01)
    wp = np.flatnonzero((st["tool_p"] == 0.0) & (st["blanked"] == 0.0))
    rng = np.random.default_rng(ny)
    h = st["grid"][2]
    if kind == "crowded":  # ~400 particles inside one cell's width, more than any row holds
        n = min(400, len(wp) // 2)
        st["pos"][wp[:n]] = st["pos"][wp[len(wp) // 2]] + rng.uniform(-0.5, 0.5, (n, 2)) * h
    elif kind == "nonfinite":
        st["S"][wp[len(wp) // 3], 0] = np.nan
        st["vel"][wp[2 * len(wp) // 3], 1] = np.inf
        st["rho"][wp[len(wp) // 2]] = np.nan
    elif kind == "outside":  # counted in the border cells they are clamped to
        st["pos"][wp[:3]] = np.array(st["grid"][1]) + np.array([[9.0, 0.3], [9.0, 0.3 + h / 3], [9.0 + h, 7.0]])
    ctx = load_product(mf, st, flags=mf.OPT_KEEP_DERIVATIVES)
    ctx.stage(0)
    ctx.stage(1)
    if kind == "outside":  # the oracle's grid refuses them: only that nothing else is disturbed
        ctx.stage(2)
        near = load_product(mf, dict(st, pos=np.where(np.isin(np.arange(st["N"]), wp[:3])[:, None],
                                                      st["pos"] + 1e3, st["pos"])), flags=mf.OPT_KEEP_DERIVATIVES)
        for k in range(3):
            near.stage(k)
        keep = ~np.isin(ctx.get("id"), wp[:3])
        for f in RATES:
            assert np.isfinite(ctx.get(f)[keep]).all(), f
        assert ctx.status()["out_of_grid"] == near.status()["out_of_grid"] == 3
        return
    o = load_oracle(orc, st)
    o.L.orc_grid_update(o.s)
    o.L.orc_stage_predict(o.s)
    assert np.array_equal(ctx.get("idx"), o.get("idx"))
    o.set_field("R", ctx.get("R"))
    ctx.stage(2)
    o.L.orc_stage_interact(o.s)
    o.L.orc_stage_rates(o.s)
    live = ctx.get("blanked") == 0.0
    wpm = live & (ctx.get("tool_p") == 0.0)
    for f in RATES:
        m = wpm if f in ("S_der", "v_der") else live
        a, b = ctx.get(f)[m], o.get(f)[m]
        assert np.array_equal(np.isfinite(a), np.isfinite(b)), f
        fin = np.isfinite(b)
        assert rel_err(a[fin], b[fin]) <= 1e-12, f
