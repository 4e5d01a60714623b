"""Batches with the PSE heat solver: each instance steps as a context of its own would, bit for bit,
whatever its lanes per particle, in both precisions and in the persistent form."""
import pytest

from helpers import load_product, perturbed_scene
from test_gpu_batch import assert_same

pytestmark = pytest.mark.gpu


# 2,724, 36,475 and 116,726 particles: four, two and one lanes per particle
@pytest.mark.parametrize("precision, persistent", [(0, False), (1, False), (1, True)])
def test_batch_equals_separate_contexts(mf, precision, persistent):
    sts = [perturbed_scene(mf, ny=ny, seed=90 + ny, blank_frac=0.01) for ny in (12, 42, 75)]
    batched, single = ([load_product(mf, st, thermal_solver=1, precision=precision) for st in sts] for _ in range(2))
    b = mf.Batch(batched, steps_per_launch=4)
    if persistent:
        b.set_form(mf.BATCH_PERSISTENT, 1, 4)
    assert b.fused
    b.step(2)
    for c in single:
        c.step(8)
    for x, y in zip(batched, single):
        assert_same(x, y)
    b.close()
