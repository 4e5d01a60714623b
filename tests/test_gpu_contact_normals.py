"""Contact normals stay at their array positions while the particles, and with them the marks of
those that touch the tool, move: where a normal was left, it has to be found again, whatever happened
in between. Each run must equal, bit for bit, one whose normals are written back by the host before
every step, which marks every particle."""
import numpy as np
import pytest

from conftest import bits_equal
from helpers import perturbed_scene
from test_gpu_contact_marks import FIELDS, load

pytestmark = pytest.mark.gpu


def scene(mf):
    st = perturbed_scene(mf, ny=12, seed=33, tool_push_dx=6.0)
    st["T"] += 50.0
    return st


@pytest.mark.parametrize("grid_kind", [0, 1])
@pytest.mark.parametrize("precision", [0, 1])
def test_tool_removed_and_set_again(mf, grid_kind, precision):
    st = scene(mf)
    a, b = load(mf, st, grid_kind, precision), load(mf, st, grid_kind, precision)
    rng = np.random.default_rng(6)
    left = 0

    def both(k):
        a.step(1)
        b.set("n", b.get("n"))
        b.step(1)
        for f in FIELDS:
            assert bits_equal(a.get(f), b.get(f)), (k, f)

    for k in range(6):
        both((k, "contact"))
        hit = np.flatnonzero(np.abs(a.get("fc")).sum(axis=1) > 0)
        for c in (a, b):
            c.tool_set(None)
        # the particles of the contact go elsewhere: the sort takes their marks from the normals
        pos, wp = a.get("pos"), np.flatnonzero(a.get("tool_p") == 0.0)
        other = rng.choice(np.setdiff1d(wp, hit), len(hit), replace=False)
        pos[np.concatenate([hit, other])] = pos[np.concatenate([other, hit])]
        for c in (a, b):
            c.set("pos", pos)
        both((k, "no tool"))
        left += int(np.count_nonzero(np.abs(a.get("n")).sum(axis=1)))
        for c in (a, b):
            c.tool_set(st["tool"])
        both((k, "tool again"))
    assert left > 20, left


@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("stage", [1, 2])
def test_normals_written_between_stages(mf, stage, device):
    torch = pytest.importorskip("torch")
    st = scene(mf)
    a, b = load(mf, st, 0, 0), load(mf, st, 0, 0)
    rng = np.random.default_rng(7)
    n = rng.normal(0.0, 1.0, (st["N"], 2))
    on_device = torch.from_numpy(n).cuda()
    b.set("n", b.get("n"))
    for k in range(4):
        for c in (a, b):
            c.stage(k)
            if k == stage and device:
                c.set_device("n", on_device.data_ptr(), torch.cuda.current_stream().cuda_stream)
            elif k == stage:
                c.set("n", n)
    for k in range(3):
        for f in FIELDS:
            assert bits_equal(a.get(f), b.get(f)), (k, f)
        wp = a.get("tool_p") == 0.0
        out = wp & (np.abs(a.get("fc")).sum(axis=1) == 0) & (a.get("fixed") == 0.0)
        assert not a.get("n")[out].any()  # outside the tool: no normal
        b.set("n", b.get("n"))
        for c in (a, b):
            c.step(1)
