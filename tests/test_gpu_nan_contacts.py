"""A particle whose position is no longer a number: its segments touch what the
serial count says they touch. The rod lies at the origin, where the cell of such
a centre is, and its second velocity update makes one particle NaN (a step of no
sweeps keeps it to that one), so that the count of the last substep meets it
beyond, at and within the distances by which near pairs are ruled out."""
import numpy as np
import pytest

from ropephysics_b200 import Batch, Material, Rod, StepParams, Strategy, World

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("particle", [1, 4, 8, 12, 15, 16, 17, 18, 20, 23, 24])
def test_nan_particle_counts_as_serial(particle):
    rod = Rod.straight(24, 0.15, Material(1e8, 0.3, 1100.0, 5e-3))
    rod.v[particle] = np.nan
    world = World([], self_collision=True, hash_table_size=1 << 14)
    found = {}
    for strategy in (Strategy.BATCHED, Strategy.MULTI_KERNEL):
        with Batch.create_mixed([rod], [world], [0], strategy) as b:
            b.step_many(StepParams(dt=1.0 / 6000, substeps=2, iterations=0), 1)
            assert b.error_count() == 0
            found[strategy] = (b.read_self_contacts(0), b.self_contact_overflow())
    got, want = found[Strategy.BATCHED], found[Strategy.MULTI_KERNEL]
    assert len(want[0]) > 0
    assert np.array_equal(got[0], want[0]) and got[1] == want[1]
