"""Self-contact pools of every size, against the serial strategies: pair lists,
overflow, positions and frames equal bit for bit where the batched kernel
takes its pool from a few pairs (at most 32), from many, or -- more pairs than
segments -- from the hash, and projects it by one warp or by the team. Rods
around a warp and a team in length, chains and a rod of two chains, kept
contacts, several sweeps, both precisions."""
import numpy as np
import pytest

from ropephysics_b200 import Batch, Material, Precision, Primitive, Rod, StepParams, Strategy, World
from ropephysics_b200.synth import helix

pytestmark = pytest.mark.gpu
MATERIAL = Material(1e8, 0.3, 1100.0, 5e-3)


def coil(n, radius, pitch):
    rod = Rod.centerline(helix(n, 0.00625 * n, radius, pitch), MATERIAL, frame_seed=(0.0, 0.0, 1.0))
    rod.b_rest_darboux[:] = 0.0
    return rod


def two_chains(n):
    """Two parallel chains of n segments, 8 mm apart, as one rod."""
    a = Rod.straight(n, 0.00625 * n, MATERIAL)
    P, S = n + 1, n
    cat = {k: np.concatenate([getattr(a, k)] * 2) for k in
           ("x", "v", "inv_mass", "q", "inertia", "inv_inertia", "s_rest", "s_compliance", "b_rest", "b_compliance",
            "b_rest_darboux", "omega")}
    cat["x"] = np.concatenate([a.x, a.x + (0.0, 0.008, 0.003)])
    for k, step in (("s_p0", P), ("s_p1", P), ("s_seg", S), ("b_a", S), ("b_b", S)):
        v = getattr(a, k)
        cat[k] = np.concatenate([v, v + step])
    return Rod.from_arrays(MATERIAL, **cat)


def outcome(rods, world, params, steps, strategy, precision):
    with Batch.create_mixed(rods, [world], [0] * len(rods), strategy) as b:
        b.set_precision(precision)
        b.step_many(params, steps)
        pairs = [b.read_self_contacts(r) for r in range(len(rods))]
        assert b.error_count() == 0
        return b.download_positions(), b.download_frames(), pairs, b.self_contact_overflow()


def check(rods, params, steps=2, table=256, precision=0):
    world = World([Primitive.plane((0.0, 0.0, -0.03), (0.0, 0.0, 1.0), 0.4)], self_collision=True, self_friction=0.4,
                  hash_table_size=table)
    got = outcome(rods, world, params, steps, Strategy.BATCHED, precision)
    want = outcome(rods, world, params, steps, Strategy.MULTI_KERNEL, precision)
    for g, w in zip(got[2], want[2]):
        assert np.array_equal(g, w)
    assert got[3] == want[3]
    assert np.array_equal(got[0], want[0], equal_nan=True) and np.array_equal(got[1], want[1], equal_nan=True)
    return got


# radius and pitch: neighbouring turns just touching, turns well inside one
# another (more pairs than segments), and a loose coil with few contacts
COILS = {"touching": (0.03, 0.0098), "inside": (0.012, 0.004), "loose": (0.06, 0.012)}


@pytest.mark.parametrize("kind", sorted(COILS))
@pytest.mark.parametrize("n", [9, 16, 17, 31, 33, 64, 65, 130, 257, 600])
@pytest.mark.parametrize("precision", [0, int(Precision.COMPENSATED | Precision.FP64_CONE)])
def test_pools_equal_serial(kind, n, precision):
    rods = [coil(n, *COILS[kind]), coil(n + 1, *COILS[kind]), coil(max(8, n - 3), *COILS[kind])]
    got = check(rods, StepParams(dt=1.0 / 60, substeps=6), precision=precision)
    if n >= 130:
        found = max(len(p) for p in got[2])
        assert found > 32 or kind == "loose"
        assert (got[3] > 0) == (kind == "inside") or kind == "touching"


@pytest.mark.parametrize("interval,iterations", [(1, 3), (2, 1), (3, 2)])
def test_kept_contacts_and_sweeps_equal_serial(interval, iterations):
    rods = [coil(n, *COILS["touching"]) for n in (40, 97, 260)]
    check(rods, StepParams(dt=1.0 / 60, substeps=6, iterations=iterations, contact_interval=interval), steps=3)


@pytest.mark.parametrize("table", [1, 7, 64])
def test_small_hash_tables_equal_serial(table):
    check([coil(n, *COILS["touching"]) for n in (33, 120)], StepParams(dt=1.0 / 60, substeps=4), table=table)


@pytest.mark.parametrize("n", [16, 48, 90])
def test_general_topology_equal_serial(n):
    rods = [two_chains(n), two_chains(n + 3)]
    got = check(rods, StepParams(dt=1.0 / 3600, substeps=1), steps=1)  # the chains start in contact
    assert all(len(p) > 0 for p in got[2])
    check(rods, StepParams(dt=1.0 / 60, substeps=6))
