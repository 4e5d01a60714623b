"""The differentiable step's work memory: what a context keeps of it between calls is bounded."""
import pytest

pytestmark = pytest.mark.gpu


def free_bytes():
    torch = pytest.importorskip("torch")
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


# about 23 thousand particles, 0.17 GB for six directions; about 225 thousand, 1.5 GB
@pytest.mark.parametrize("ny, keeps", [(52, True), (160, False)])
def test_kept_memory(mf, ny, keeps):
    sc = mf.Scene.ref_cut(ny)
    ctx = mf.Context(0)
    ctx.upload_scene(sc, mf.GRID_GREEN)
    ctx.tangent_mean_force(0, 1, 5)  # (kernels loaded)
    ctx.upload_scene(sc, mf.GRID_GREEN)
    before = free_bytes()
    first = ctx.tangent_mean_force_all(0, 1)
    held = before - free_bytes()
    need = 6 * sc.N * 1000
    assert held > need if keeps else held <= 1 << 26, (held, need)
    again = ctx.tangent_mean_force_all(0, 1)
    assert all((a == b).all() for a, b in zip(first, again))
    assert before - free_bytes() == held
    ctx.close()
