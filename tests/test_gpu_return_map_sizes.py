"""The Johnson-Cook return map (two lanes per particle) with lists of a few warps, of part of the GPU
and of tens of thousands of particles: one finish stage against the oracle.

Tolerances: the solve itself is FP64 on both sides (1e-9 of the largest stress and temperature: its
powers differ by an ulp or two between the libraries, and the secant's slope, a difference over 1 % of
the increment, loses two digits); the strain adds the increment rounded to float (one unit of 6e-8 of
at most 0.05 over 0.5: 1e-8), and the rate is that float (1e-6).
"""
import numpy as np
import pytest

from conftest import rel_err
from helpers import load_oracle, load_product, perturbed_scene

pytestmark = pytest.mark.gpu

TOL = {"S": 1e-9, "T": 1e-9, "eps_pl": 1e-8, "eps_pl_dot": 1e-6}


@pytest.mark.parametrize("ny,more_than", [(10, 16), (40, 2048), (92, 28416)])
def test_return_map_at_list_lengths(mf, orc, ny, more_than):
    st = perturbed_scene(mf, ny=ny, seed=41, tensile=True)
    st["S"] *= 3.0
    ctx, o = load_product(mf, st), load_oracle(orc, st)
    ctx.stage(0)
    ctx.stage(1)
    o.L.orc_grid_update(o.s)
    o.L.orc_stage_predict(o.s)
    o.set_field("R", ctx.get("R"))
    ctx.stage(2)
    o.L.orc_stage_interact(o.s)
    o.L.orc_stage_rates(o.s)
    for f in ("pos_t", "vel_t", "S_t", "rho_t", "T_t"):
        o.set_field(f, ctx.get(f))
    ctx.stage(3)
    o.L.orc_stage_finish(o.s)
    assert np.count_nonzero(ctx.get("eps_pl_dot")) > more_than
    for f, tol in TOL.items():
        assert rel_err(ctx.get(f), o.get(f)) <= tol, f
    ctx.close()
