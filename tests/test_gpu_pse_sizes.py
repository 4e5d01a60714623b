"""The PSE heat kernels at the sizes where their lanes per particle change, blanked particles
(which they include) among the neighbours.

Tolerances: FP64 1e-12 of the field's largest value against the oracle (the single-step bar),
mixed 1e-4 against the FP64 form (the mixed form's own bar)."""
import numpy as np
import pytest

from conftest import rel_err
from helpers import load_oracle, load_product, perturbed_scene

pytestmark = pytest.mark.gpu


def rates(ctx):
    for k in range(3):
        ctx.stage(k)
    return ctx.get("T_t"), ctx.get("blanked") == 0.0


# FP64: 2,724 and 18,310 particles (four lanes), 19,589 and 36,475 (two), 38,139 (one)
@pytest.mark.parametrize("ny", [12, 30, 31, 42, 43])
def test_fp64(mf, orc, ny):
    st = perturbed_scene(mf, ny=ny, seed=80 + ny, blank_frac=0.05)
    a, live = rates(load_product(mf, st, thermal_solver=1))
    o = load_oracle(orc, st, thermal_solver=1)
    o.L.orc_grid_update(o.s)
    o.L.orc_stage_predict(o.s)
    o.L.orc_stage_interact(o.s)
    o.L.orc_stage_rates(o.s)
    assert rel_err(a[live], o.get("T_t")[live]) <= 1e-12


# mixed: 2,724 and 28,156 particles (four lanes), 29,736 and 45,724 (two), 47,733 (one)
@pytest.mark.parametrize("ny", [12, 37, 38, 47, 48])
def test_mixed(mf, ny):
    st = perturbed_scene(mf, ny=ny, seed=90 + ny, blank_frac=0.05)
    a, live = rates(load_product(mf, st, thermal_solver=1, precision=mf.PRECISION_MIXED))
    b, _ = rates(load_product(mf, st, thermal_solver=1))
    assert rel_err(a[live], b[live]) <= 1e-4
