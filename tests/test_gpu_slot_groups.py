"""World contact slots in shared memory where the rods' state and slots fill a
CTA's share of an SM and the teams' contexts come on top: a group gives up a rod
rather than its slots, so one CTA's shared memory still holds them (over 80 KB;
without the slots it is under 60). Rods on both sides of that range, lying on
their primitives, equal the multi-kernel strategy bit for bit, in the batch's own
buffers and in the static scratch."""
import ctypes as C

import numpy as np
import pytest

from ropephysics_b200 import Batch, Material, Primitive, Rod, StepParams, Strategy, World, _check, lib

pytestmark = pytest.mark.gpu


def world(prims, self_collision):
    return World([Primitive.plane((0.0, 0.0, -0.006), (0.0, 0.0, 1.0), 0.4)] +
                 [Primitive.sphere((0.05 * i, 0.004, -0.03), 0.03, 0.3) for i in range(1, prims)],
                 self_collision=self_collision, hash_table_size=256)


@pytest.mark.parametrize("segments,prims,self_collision,shared", [
    (59, 5, False, True), (60, 5, False, True), (61, 5, False, True), (64, 5, False, False),
    (60, 4, True, True), (61, 4, True, True), (109, 5, True, True), (64, 7, True, False)])
def test_slots_stay_in_shared_memory(segments, prims, self_collision, shared):
    rods = [Rod.straight(segments, 0.00625 * segments, Material(1e8, 0.3, 1100.0, 5e-3))] * 21
    params = StepParams(dt=1.0 / 60, substeps=5)
    got = []
    for strategy, static in ((Strategy.BATCHED, False), (Strategy.BATCHED, True), (Strategy.MULTI_KERNEL, False)):
        with Batch.create_mixed(rods, [world(prims, self_collision)], [0] * len(rods), strategy) as b:
            if strategy == Strategy.BATCHED:
                b.set_tuning(256, 1, 1)
                assert (b.shared_bytes_per_block > 80e3) == shared
            for _ in range(3):
                _check(lib().rp_batch_step_static_scratch(b._h, C.byref(params.to_c()))) if static else b.step(params)
            assert b.error_count() == 0
            got.append((b.download_positions(), b.download_frames(), b.read_contact_states()))
    assert got[0][2].any()
    for other in got[1:]:
        for g, w in zip(got[0], other):
            assert np.array_equal(g, w)
