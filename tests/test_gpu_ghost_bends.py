"""The batched kernel's bend sweep of clamped rods: ghost frames at one end or
both, at lengths around a warp and a team, equal to the one-rod-per-CTA
kernel's, bit for bit."""
import numpy as np
import pytest

from ropephysics_b200 import Batch, Material, Precision, Rod, StepParams, Strategy

pytestmark = pytest.mark.gpu


def clamped(n, ends):
    rod = Rod.straight(n, 0.5, Material(1e8, 0.3, 1100.0, 5e-3))
    for tip in ends:
        rod.clamp_end(tip=tip)
    rod.ext_force[n // 2] = (0.01, 0.02, -0.05)
    return rod


@pytest.mark.parametrize("ends", [(False,), (True,), (False, True)])
@pytest.mark.parametrize("n", [2, 3, 4, 31, 32, 33, 63, 64, 65, 128, 129])
def test_ghost_bends_equal_fused(n, ends):
    got = []
    for strategy in (Strategy.BATCHED, Strategy.FUSED):
        for precision in (0, int(Precision.COMPENSATED)):
            with Batch.create(clamped(n, ends), 3, strategy) as b:
                b.set_precision(precision)
                b.step_many(StepParams(dt=1.0 / 60, substeps=8, iterations=2), 3)
                got.append((b.download_positions(), b.download_frames()))
    for batched, fused in ((got[0], got[2]), (got[1], got[3])):
        assert np.isfinite(batched[0]).all()
        assert np.array_equal(batched[0], fused[0]) and np.array_equal(batched[1], fused[1])
