"""Rods whose rest data are the same in every row read row 0 for all; a rod
with one row changed, in any of the arrays and at either end, must not: its
motion differs from the uniform rod's, and is the same from both kernels."""
import numpy as np
import pytest

from ropephysics_b200 import Batch, Material, Rod, StepParams, Strategy

pytestmark = pytest.mark.gpu


def straight(n):
    rod = Rod.straight(n, 0.4, Material(1e8, 0.3, 1100.0, 5e-3))
    rod.pin_particle(0)
    rod.ext_force[n // 2] = (0.3, -0.2, -0.4)
    rod.ext_torque[:] = (0.002, 0.001, -0.001)
    return rod


def motion(rod, strategy):
    with Batch.create(rod, 2, strategy) as b:
        b.step_many(StepParams(dt=1.0 / 60, substeps=10), 3)
        return b.download_positions(), b.download_frames()


@pytest.mark.parametrize("array", ["inv_inertia", "inertia", "s_rest", "s_compliance", "b_rest", "b_compliance",
                                   "b_rest_darboux"])
@pytest.mark.parametrize("row", [0, -1])
@pytest.mark.parametrize("n", [5, 64, 97])
def test_one_changed_row_counts(array, row, n):
    uniform, changed = straight(n), straight(n)
    rows = getattr(changed, array)
    rows[row] = rows[row] * 1.5 + (0.4 if array == "b_rest_darboux" else 0.0)
    got = [motion(r, s) for r in (uniform, changed) for s in (Strategy.BATCHED, Strategy.FUSED)]
    for batched, fused in ((got[0], got[1]), (got[2], got[3])):
        assert np.array_equal(batched[0], fused[0]) and np.array_equal(batched[1], fused[1])
    assert not np.array_equal(got[0][1], got[2][1])
