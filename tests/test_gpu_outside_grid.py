"""Particles outside the locked grid, counted in the border cells they are clamped to: they and the
particles inside have the pair sums of their exact distances.

Inside: against the oracle, whose grid refuses such particles, with them blanked (which takes them out
of every other particle's sums, as their distance does here). Outside: two of them are each other's only
neighbours, so that their velocity gradient is one term, computed here; the third has none. Tolerance:
1e-12 of the field's largest value, the single-step bar of the FP64 pair sums."""
import numpy as np
import pytest

from conftest import rel_err
from helpers import load_oracle, load_product, perturbed_scene

pytestmark = pytest.mark.gpu

RATES = ("pos_t", "vel_t", "S_t", "rho_t", "T_t")


# 2,724 particles (four lanes), 19,589 (two), 38,139 (one)
@pytest.mark.parametrize("ny", [12, 31, 43])
def test_inside_and_outside(mf, orc, ny):
    st = perturbed_scene(mf, ny=ny, seed=80 + ny, blank_frac=0.01)
    wp = np.flatnonzero((st["tool_p"] == 0.0) & (st["blanked"] == 0.0) & (st["fixed"] == 0.0))
    out = wp[[0, len(wp) // 2, len(wp) - 1]]
    h = st["grid"][2]
    (x1, y1) = st["grid"][1]
    moved = dict(st, pos=st["pos"].copy())
    moved["pos"][out] = [(x1 + 40 * h, y1 + 3 * h), (x1 + 40.6 * h, y1 + 3.4 * h), (x1 + 90 * h, y1 + 70 * h)]
    ctx = load_product(mf, moved, flags=mf.OPT_KEEP_DERIVATIVES)
    for k in range(3):
        ctx.stage(k)
    assert ctx.status()["out_of_grid"] == 3
    by_id = np.argsort(ctx.get("id"))

    gone = dict(st, blanked=st["blanked"].copy())
    gone["blanked"][out] = 1.0
    o, near = load_oracle(orc, gone), load_product(mf, gone)
    near.stage(0)
    near.stage(1)
    o.L.orc_grid_update(o.s)
    o.L.orc_stage_predict(o.s)
    o.set_field("R", near.get("R"))
    o.L.orc_stage_interact(o.s)
    o.L.orc_stage_rates(o.s)
    o_by_id = np.argsort(o.get("idx"))  # (one sort: the index is the particle's number)
    live = (st["blanked"] == 0.0) & ~np.isin(np.arange(st["N"]), out)
    for f in RATES:
        assert rel_err(ctx.get(f)[by_id][live], o.get(f)[o_by_id][live]) <= 1e-12, f

    pos, vel, rho = (ctx.get(k)[by_id] for k in ("pos", "vel", "rho"))
    grad, mass, h_i = ctx.get("v_der")[by_id], st["phys"].mass, st["h"][0]
    fac = 0.454728408833987 / h_i**2
    for i, j in ((out[0], out[1]), (out[1], out[0])):
        x = pos[i] - pos[j]
        r = float(np.sqrt(np.float32(x @ x)))
        q = r / h_i
        dwr = -3.0 / h_i**2 * fac * (1 - 0.75 * q) if q <= 1 else -0.75 / h_i * fac * (2 - q) ** 2 / r
        term = mass / rho[j] * np.outer(vel[j] - vel[i], dwr * x).reshape(-1)
        assert np.abs(term).max() > 0.0
        assert rel_err(grad[i], term) <= 1e-12
    assert not grad[out[2]].any()
