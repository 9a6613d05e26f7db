"""One-warp rods that just filled a CTA's shared memory eight at a time: 32
segments and many free frames each, 28.5 KB of state a rod. The team's context
lies beside each rod's state, so eight of them no longer fit together; the
batch is planned with fewer to a CTA and steps as the multi-kernel strategy
does, bit for bit."""
import numpy as np
import pytest

from ropephysics_b200 import Batch, Material, Rod, StepParams, Strategy, World

pytestmark = pytest.mark.gpu


def framed(frames):
    """A straight rod of 32 segments with `frames` frames, the further ones free."""
    a = Rod.straight(32, 0.2, Material(1e8, 0.3, 1100.0, 5e-3))
    keys = ("x", "v", "inv_mass", "q", "inertia", "inv_inertia", "s_p0", "s_p1", "s_seg", "s_rest", "s_compliance",
            "b_a", "b_b", "b_rest", "b_compliance", "b_rest_darboux", "omega")
    cat = {k: np.array(getattr(a, k)) for k in keys}
    for k in ("q", "inertia", "inv_inertia", "omega"):
        cat[k] = np.concatenate([cat[k], np.repeat(cat[k][-1:], frames - 32, axis=0)])
    cat["omega"][32:] = np.random.default_rng(0).normal(size=(frames - 32, 3))
    return Rod.from_arrays(Material(1e8, 0.3, 1100.0, 5e-3), **cat)


@pytest.mark.parametrize("frames", [400, 841, 849])
def test_rods_that_filled_a_cta_still_run(frames):
    rods, params = [framed(frames)] * 20, StepParams(dt=1.0 / 60, substeps=4)
    got = []
    for strategy in (Strategy.BATCHED, Strategy.MULTI_KERNEL):
        with Batch.create_mixed(rods, [World([])], [0] * len(rods), strategy) as b:
            if strategy == Strategy.BATCHED:
                b.set_tuning(256, 1, 1)  # eight one-warp rods to a CTA, where they fit
            b.step_many(params, 3)
            assert b.error_count() == 0
            got.append((b.download_positions(), b.download_frames()))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
