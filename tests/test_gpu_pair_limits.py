"""The FP64 pair term at the ends of what its reciprocals take."""
import numpy as np
import pytest

from conftest import rel_err
from helpers import load_oracle, load_product, perturbed_scene

pytestmark = pytest.mark.gpu


# 2,724 particles (four lanes), 19,589 (two), 38,139 (one)
@pytest.mark.parametrize("ny", [12, 31, 43])
def test_nearly_coincident_without_eta(mf, orc, ny):
    """The viscosity's denominator r^2 + eta^2 h^2 with eta = 0 and two approaching particles 1e-20
    apart: far below float's range, and no part of the sums (W = 0 below 1e-4). Tolerance: the
    single-step bar for pair sums, 1e-12 of the field's largest value."""
    st = perturbed_scene(mf, ny=ny, seed=60 + ny)
    st["corr"] = mf.Corr.from_buffer_copy(st["corr"])
    st["corr"].eta = 0.0
    wp = np.flatnonzero((st["tool_p"] == 0.0) & (st["fixed"] == 0.0))
    i, j = wp[np.argsort(np.abs(st["pos"][wp, 0]))[:2]]
    st["pos"][i] = (0.0, st["pos"][i, 1])
    st["pos"][j] = (1e-20, st["pos"][i, 1])
    for k in ("pos_t", "vel_t"):
        st[k][[i, j]] = 0.0
    st["vel"][i], st["vel"][j] = (1e-4, 0.0), (-1e-4, 0.0)
    ctx, o = load_product(mf, st), load_oracle(orc, st)
    ctx.stage(0)
    ctx.stage(1)
    o.L.orc_grid_update(o.s)
    o.L.orc_stage_predict(o.s)
    assert np.array_equal(ctx.get("idx"), o.get("idx"))
    o.set_field("R", ctx.get("R"))
    ctx.stage(2)
    o.L.orc_stage_interact(o.s)
    o.L.orc_stage_rates(o.s)
    for f in ("pos_t", "vel_t", "S_t", "rho_t", "T_t"):
        assert np.isfinite(ctx.get(f)).all(), f
        assert rel_err(ctx.get(f), o.get(f)) <= 1e-12, f
