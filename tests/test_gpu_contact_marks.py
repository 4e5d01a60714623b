"""Contact forces and normals carried by the particles that touch the tool only: a run must equal,
bit for bit, one whose normals are written back by the host before every step, which makes every
particle carry them. Contact particles come and go, and now and then the host swaps some with tool
particles, so that contact normals are left at array positions which tool particles take."""
import numpy as np
import pytest

from conftest import bits_equal
from helpers import perturbed_scene

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "S", "T", "fc", "ft", "n", "pos_t", "vel_t", "T_t", "blanked", "id")


def load(mf, st, grid_kind, precision):
    """The scene without host writes of the contact forces and normals (they start at zero)."""
    ctx = mf.Context(0)
    ctx.particles_create(st["pos"], st["vel"], st["rho"], st["h"], T=st["T"], fixed=st["fixed"],
                         tool_p=st["tool_p"], S=st["S"])
    for k in ("eps_pl", "eps_pl_dot"):
        ctx.set(k, st[k])
    ctx.grid_locked(grid_kind, *st["grid"])
    ctx.set_constants(st["phys"], st["corr"], st["joco"], st["trml_wp"], st["trml_tool"])
    ctx.set_options(0, 0, precision)
    ctx.tool_set(st["tool"])
    ctx.set_dt(st["dt"])
    return ctx


@pytest.mark.parametrize("grid_kind", [0, 1])
@pytest.mark.parametrize("precision", [0, 1])
def test_marked_particles_alone(mf, grid_kind, precision):
    st = perturbed_scene(mf, ny=12, seed=31, tool_push_dx=6.0)
    st["T"] += 50.0
    a, b = load(mf, st, grid_kind, precision), load(mf, st, grid_kind, precision)
    rng = np.random.default_rng(4)
    touched, taken = 0, []
    for k in range(60):
        # contact particles change places with tool particles, whose places others then take
        pos, tool, pid = a.get("pos"), a.get("tool_p") == 1.0, a.get("id")
        hit = (np.abs(a.get("fc")).sum(axis=1) > 0) & ~tool
        went = np.flatnonzero(np.isin(pid, taken))
        if k % 3 == 2 and len(went):
            i, j = went, rng.choice(np.flatnonzero(~tool & ~hit), len(went), replace=False)
            taken = []
        else:
            i = np.flatnonzero(hit)[: int(hit.sum()) // 2]
            j = rng.choice(np.flatnonzero(tool & ~np.isin(pid, taken)), len(i), replace=False)
            taken += list(pid[j])
        pos[np.concatenate([i, j])] = pos[np.concatenate([j, i])]
        a.set("pos", pos)
        b.set("pos", pos)
        a.step(1)
        b.set("n", b.get("n"))
        b.step(1)
        touched += int(np.count_nonzero(np.abs(b.get("fc")).sum(axis=1)))
        for f in FIELDS:
            assert bits_equal(a.get(f), b.get(f)), (k, f)
    assert touched > 200, touched
