"""Batches small enough for wide teams (about one thread per segment, CTAs of
128, 256 or 512 threads) against the narrow launch shapes, bit for bit: one
rod, teams of every size, mixed lengths of which only the longest are wide,
long self-colliding rods on 512 threads, and batches on both sides of the
limit."""
import numpy as np
import pytest

from ropephysics_b200 import Batch, Material, Precision, Primitive, Rod, StepParams, World
from ropephysics_b200.synth import helix

pytestmark = pytest.mark.gpu
MATERIAL = Material(1e8, 0.3, 1100.0, 5e-3)
LENGTHS = {
    "one": [64], "short": [5, 17, 31, 32, 33, 48, 49], "powers": [96, 97, 128, 192, 193, 256, 384, 385, 512, 513],
    "long": [900, 1500], "part": [40] * 500 + [200] * 60 + [470] * 30, "most": [64] * 592, "over": [64] * 700,
}


def batch(lengths, self_collision):
    shapes = {}
    for n in set(lengths):
        shapes[n] = Rod.centerline(helix(n, 0.00625 * n, 0.05, 0.0102), MATERIAL, frame_seed=(0.0, 0.0, 1.0))
        shapes[n].b_rest_darboux[:] = 0.0
    world = World([Primitive.plane((0.0, 0.0, -0.011), (0.0, 0.0, 1.0), 0.4),
                   Primitive.sphere((0.05, 0.0, -0.03), 0.03, 0.3)], self_collision=self_collision,
                  self_friction=0.3, hash_table_size=256)
    return Batch.create_mixed([shapes[n] for n in lengths], [world], [0] * len(lengths))


@pytest.mark.parametrize("name", sorted(LENGTHS))
@pytest.mark.parametrize("self_collision", [False, True])
@pytest.mark.parametrize("precision", [0, int(Precision.COMPENSATED)])
def test_wide_teams_equal_narrow(name, self_collision, precision):
    want = None
    for shape in (None, (128, 1, 1), (256, 2, 1)):
        with batch(LENGTHS[name], self_collision) as b:
            b.set_precision(precision)
            if shape:
                b.set_tuning(*shape)
            b.step_many(StepParams(dt=1.0 / 60, substeps=5, iterations=2), 3)
            got = (b.download_positions(), b.download_frames(), b.read_contact_states())
            assert b.error_count() == 0
        if want is None:
            want = got
        assert all(np.array_equal(g, w, equal_nan=True) for g, w in zip(got, want))
