"""A batch built again after its instances' constants or options were changed: each instance steps as
a context of its own with them would, bit for bit."""
import pytest

from helpers import load_product
from test_gpu_batch import assert_same, scenes

pytestmark = pytest.mark.gpu


def two_sets(mf, precision):
    sts = scenes(mf)
    return sts, [[load_product(mf, st, precision=precision) for st in sts] for _ in range(2)]


@pytest.mark.parametrize("precision", [0, 1])
def test_constants_changed(mf, precision):
    sts, (batched, single) = two_sets(mf, precision)
    b = mf.Batch(batched, steps_per_launch=4)
    b.step(1)
    for c in single:
        c.step(4)
    for st, *pair in zip(sts, batched, single):
        corr, phys = mf.Corr.from_buffer_copy(st["corr"]), mf.Phys.from_buffer_copy(st["phys"])
        corr.alpha, corr.eta, corr.wdeltap = 1.3 * corr.alpha, 0.7 * corr.eta, 1.1 * corr.wdeltap
        phys.K = 0.9 * phys.K
        for c in pair:
            c.set_constants(phys, corr, st["joco"], st["trml_wp"], st["trml_tool"])
    b.set_form(mf.BATCH_PHASES, steps_per_launch=4)
    b.step(1)
    for c in single:
        c.step(4)
    for x, y in zip(batched, single):
        assert_same(x, y)
    b.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_one_instance_changes_precision(mf, precision):
    sts, (batched, single) = two_sets(mf, precision)
    b = mf.Batch(batched, steps_per_launch=4)
    b.step(1)
    for c in single:
        c.step(4)
    for c in (batched[1], single[1]):
        c.set_options(mf.THERMAL_BROOKSHAW, mf.JC_JOHNSON_COOK, 1 - precision)
    b.set_form(mf.BATCH_PHASES, steps_per_launch=4)
    assert not b.fused  # the batched kernels serve one precision
    b.step(1)
    for c in single:
        c.step(4)
    for x, y in zip(batched, single):
        assert_same(x, y)
    for c in (batched[1], single[1]):
        c.set_options(mf.THERMAL_BROOKSHAW, mf.JC_JOHNSON_COOK, precision)
    b.set_form(mf.BATCH_PHASES, steps_per_launch=4)
    assert b.fused
    b.step(1)
    for c in single:
        c.step(4)
    for x, y in zip(batched, single):
        assert_same(x, y)
    b.close()
