"""Grids with more rows of cells than a float counts (2^24): the FP64 step's and the differentiable
step's pair sums on such a grid equal those of the same particles on an ordinary one.

Tolerance: 1e-12 of the field's largest value for the rates (the single-step bar of the FP64 pair sums,
whose order changes where a rounded cell bound does), 1e-9 for the forces after ten steps."""
import numpy as np
import pytest

from conftest import rel_err
from helpers import SCALAR, VEC2, VEC4, load_product, perturbed_scene

pytestmark = pytest.mark.gpu

RATES = ("pos_t", "vel_t", "S_t", "rho_t", "T_t")


def strip(mf):
    """The part of the cut scene around the tool's edge, twelve cells wide."""
    st = perturbed_scene(mf, ny=30, seed=5, tool_push_dx=3.0)
    h = st["grid"][2]
    x0 = st["pos"][st["tool_p"] == 0.0, 0].min()
    keep = np.abs(st["pos"][:, 0] - x0) < 6 * h
    for k in SCALAR + VEC2 + VEC4:
        if k in st:
            st[k] = st[k][keep]
    st["N"] = int(keep.sum())
    lo, hi = st["pos"].min(axis=0) - 2 * h, st["pos"].max(axis=0) + 2 * h
    st["grid"] = (tuple(lo), tuple(hi), h)
    return st


# the particles' rows around 2^24 and well above it
@pytest.mark.parametrize("rows", [2**24 - 12, 2**24 + 2**20])
def test_more_rows_than_a_float_counts(mf, rows):
    st = strip(mf)
    (x0, y0), hi, h = st["grid"]
    tall = dict(st, grid=((x0, y0 - rows * h), hi, h))
    near, far = load_product(mf, st), load_product(mf, tall)
    assert far.geometry()["ny"] > 2**24
    mean, dmean = near.tangent_mean_force_all(0, 10)
    tmean, tdmean = far.tangent_mean_force_all(0, 10)
    assert np.abs(mean).max() > 0.0
    assert rel_err(tmean, mean) <= 1e-9 and rel_err(tdmean, dmean) <= 1e-9
    for c in (near, far):
        for k in range(3):
            c.stage(k)
    a, b = np.argsort(near.get("id")), np.argsort(far.get("id"))
    for f in RATES:
        assert rel_err(far.get(f)[b], near.get(f)[a]) <= 1e-12, f
