"""The mixed form's pair sums take the cell size as a float, in the records' offsets as in the steps from
cell to cell: on two grids whose cell sizes round to the same float, with the same particles in every
cell, the rates are the same bit for bit. (Offsets from origins dx apart and steps of dx rounded
differ by the rounding, an error of one sign in every pair across a cell bound.)"""
import numpy as np
import pytest

from conftest import bits_equal
from helpers import load_product, perturbed_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("thermal_solver, lists", [(0, False), (0, True), (1, False)])
@pytest.mark.parametrize("ny", [12, 31, 43])
def test_cell_size_between_two_floats(mf, ny, thermal_solver, lists):
    st = perturbed_scene(mf, ny=ny, seed=70 + ny)
    bbmin, bbmax, h = st["grid"]
    size = np.float32(h * 1.001)
    between = float(size) + 0.45 * float(np.spacing(size))
    assert np.float32(between) == size and between != float(size)
    a, b = (load_product(mf, dict(st, grid=(bbmin, bbmax, x)), thermal_solver=thermal_solver,
                         precision=mf.PRECISION_MIXED, flags=mf.OPT_NEIGHBOUR_LISTS if lists else 0)
            for x in (float(size), between))
    for c in (a, b):
        c.step(1)
    assert np.array_equal(a.get("hash"), b.get("hash"))
    for f in ("pos_t", "vel_t", "S_t", "rho_t", "T_t"):
        assert bits_equal(a.get(f), b.get(f)), f
