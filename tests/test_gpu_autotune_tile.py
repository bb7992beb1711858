"""The autotuner with frozen labels: the per-kernel steps do not take the march tile, so they have one time, and where
they win the batch keeps the tile it came with."""
import pytest

from test_gpu_batch import instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [0, 20])  # the labels freeze in the first candidate's untimed period, or before
@pytest.mark.parametrize("tile", [4 | (32 << 8), 5 | (16 << 8)])
def test_frozen_labels_keep_the_tile(tile, steps):
    from realmolecule_b200.batch import Batch
    b = Batch(instances(), precision="mixed", label_until=1, batch_tile=tile, fp32_rounding=1)  # no persistent form
    b.initialize()
    b.step(steps)
    rep = b.autotune()
    b.close()
    assert len(rep["tiles"]) == 6 and len({t["ms_per_step"] for t in rep["tiles"]}) == 1
    assert rep["config"]["batch_tile"] == tile and rep["config"]["batch_persistent"] == 0
    assert rep["tiles"][[t["batch_tile"] for t in rep["tiles"]].index(tile)]["ms_per_step"] > 0


def test_moving_labels_time_every_tile():
    from realmolecule_b200.batch import Batch
    b = Batch(instances(), precision="mixed", label_until=0, fp32_rounding=1)
    b.initialize()
    b.step(20)
    rep = b.autotune()
    b.close()
    assert len(rep["tiles"]) == 6 and len({t["ms_per_step"] for t in rep["tiles"]}) > 1
    best = min(t["ms_per_step"] for t in rep["tiles"])
    assert [t["ms_per_step"] for t in rep["tiles"] if t["batch_tile"] == rep["config"]["batch_tile"]] == [best]
