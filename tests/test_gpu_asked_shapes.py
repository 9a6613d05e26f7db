"""A launch shape that was asked for is the one that runs, on batches small
enough for wide teams too: a CTA of 256 threads holds the rods of two of 128,
so its shared memory is twice theirs. A batch that was never tuned takes its
own shape, and so may an autotuned one. No shape changes a result."""
import numpy as np
import pytest

from ropephysics_b200 import Batch, Material, Precision, Primitive, Rod, StepParams, World

pytestmark = pytest.mark.gpu
PARAMS = StepParams(dt=1.0 / 60, substeps=4)


def batch(rods=24, segments=64, self_collision=False):
    rod = Rod.straight(segments, 0.00625 * segments, Material(1e8, 0.3, 1100.0, 5e-3))
    world = World([Primitive.plane((0.0, 0.0, -0.03), (0.0, 0.0, 1.0), 0.4)], self_collision=self_collision)
    return Batch.create_mixed([rod] * rods, [world], [0] * rods)


@pytest.mark.parametrize("segments,self_collision", [(64, False), (64, True), (40, False), (128, True)])
def test_an_asked_shape_is_the_one_that_runs(segments, self_collision):
    with batch(24, segments, self_collision) as b:
        untuned, want = b.shared_bytes_per_block, None
        b.set_tuning(128, 1, 1)
        narrow = b.shared_bytes_per_block
        b.set_tuning(256, 1, 1)
        assert b.tuning == {"cta_threads": 256, "pairs_per_thread": 1, "steps_per_launch": 1}
        assert b.shared_bytes_per_block == 2 * narrow != untuned
        b.set_precision(Precision.COMPENSATED)  # planned anew, still as asked
        compensated = b.shared_bytes_per_block
        b.set_tuning(128, 1, 1)
        assert compensated == 2 * b.shared_bytes_per_block
        b.set_precision(0)
        for shape in ((256, 1, 1), (128, 2, 1)):
            with batch(24, segments, self_collision) as c, batch(24, segments, self_collision) as d:
                c.set_tuning(*shape)
                c.step_many(PARAMS, 3)
                d.step_many(PARAMS, 3)
                assert np.array_equal(c.download_positions(), d.download_positions())
                assert np.array_equal(c.download_frames(), d.download_frames())


def test_asking_first_for_the_default_numbers():
    """256 and 1 on a batch never tuned: the reported numbers stay, the shape becomes theirs."""
    with batch() as b, batch() as c:
        assert b.tuning["cta_threads"] == 256 and b.tuning["pairs_per_thread"] == 1
        b.set_tuning(256, 1, 1)
        c.set_tuning(128, 1, 1)
        assert b.shared_bytes_per_block == 2 * c.shared_bytes_per_block


def test_the_autotuner_may_keep_the_untuned_shape():
    """Whatever it keeps, the numbers it reports are in the documented range, and the state is untouched."""
    with batch() as b, batch() as c:
        untuned = b.shared_bytes_per_block
        tuning = b.autotune(PARAMS, max_steps_per_launch=2)
        assert tuning["cta_threads"] in (0, 128, 256) and tuning["pairs_per_thread"] in (1, 2)
        kept = b.shared_bytes_per_block
        c.set_tuning(128, 1, 1)
        one = c.shared_bytes_per_block
        assert kept in (untuned, one, 2 * one) or tuning["pairs_per_thread"] == 2
        b.step_many(PARAMS, 3)
        c.step_many(PARAMS, 3)
        assert np.array_equal(b.download_positions(), c.download_positions())
