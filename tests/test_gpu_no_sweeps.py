"""Steps of no constraint sweeps (iterations = 0) with self-collision: the
count and the pool run every substep with no sweep, and so no sweep's barrier,
between one substep's pool and the next one's centres. Pair lists, overflow and
positions equal the multi-kernel strategy's bit for bit, for coils whose teams
are one warp to sixteen, with contacts kept over one, two and three substeps."""
import numpy as np
import pytest

from ropephysics_b200 import Batch, Material, Precision, Primitive, Rod, StepParams, Strategy, World
from ropephysics_b200.synth import helix

pytestmark = pytest.mark.gpu
MATERIAL = Material(1e8, 0.3, 1100.0, 5e-3)


def outcome(rods, params, strategy, precision):
    world = World([Primitive.plane((0.0, 0.0, -0.03), (0.0, 0.0, 1.0), 0.4)], self_collision=True, self_friction=0.4,
                  hash_table_size=256)
    with Batch.create_mixed(rods, [world], [0] * len(rods), strategy) as b:
        b.set_precision(precision)
        got = []
        for _ in range(3):
            b.step_many(params, 2)
            got.append((b.download_positions(), b.download_frames(), b.self_contact_overflow(),
                        [b.read_self_contacts(r) for r in range(len(rods))]))
        assert b.error_count() == 0
        return got


@pytest.mark.parametrize("segments", [(64, 65, 33), (130, 200, 257), (385, 600, 500)])
@pytest.mark.parametrize("interval", [1, 2, 3])
@pytest.mark.parametrize("precision", [0, int(Precision.COMPENSATED)])
def test_no_sweeps_equal_serial(segments, interval, precision):
    rods = []
    for n, (radius, pitch) in zip(segments, ((0.03, 0.0098), (0.012, 0.004), (0.03, 0.0098))):
        rods.append(Rod.centerline(helix(n, 0.00625 * n, radius, pitch), MATERIAL, frame_seed=(0.0, 0.0, 1.0)))
    params = StepParams(dt=1.0 / 600, substeps=6, iterations=0, contact_interval=interval)
    got = outcome(rods, params, Strategy.BATCHED, precision)
    want = outcome(rods, params, Strategy.MULTI_KERNEL, precision)
    assert max(len(p) for p in want[0][3]) >= 32  # a pool of 64 segments holds 32
    for g, w in zip(got, want):
        assert np.array_equal(g[0], w[0]) and np.array_equal(g[1], w[1]) and g[2] == w[2]
        for a, b in zip(g[3], w[3]):
            assert np.array_equal(a, b)
