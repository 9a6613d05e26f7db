"""Self-contacts of rods that are not one chain, batched against the
multi-kernel strategy: pair lists, overflow, positions and frames equal bit
for bit. Segments of consecutive indices lie anywhere in such rods: strands of
a few segments of which some touch and the others are far away, strands that
end in a U-turn beside a far one, and one chain whose segments are listed in a
shuffled order. (Exact: the pair list is the same set in the same order.)"""
import numpy as np
import pytest

from ropephysics_b200 import Batch, Material, Primitive, Rod, StepParams, Strategy, World
from ropephysics_b200.synth import helix

pytestmark = pytest.mark.gpu
STEP = 0.00625
MATERIAL = Material(1e8, 0.3, 1100.0, 5e-3)


def line(n, at=(0.0, 0.0, 0.0)):
    return np.array(at) + np.outer(np.arange(n + 1) * STEP, (1.0, 0.0, 0.0))


def hairpin(n):
    """A strand of n segments whose last four turn back beside the ones before."""
    headings = np.zeros(n)
    headings[n - 4], headings[n - 3:] = 0.5 * np.pi, np.pi
    steps = STEP * np.stack([np.cos(headings), np.sin(headings), 0.0 * headings], axis=1)
    return np.concatenate([np.zeros((1, 3)), np.cumsum(steps, axis=0)])


def joined(strands):
    """One rod of several chains, given by their points."""
    rods = [Rod.centerline(s, MATERIAL, frame_seed=(0.0, 0.0, 1.0)) for s in strands]
    cat = {k: np.concatenate([getattr(r, k) for r in rods]) for k in
           ("x", "v", "inv_mass", "q", "inertia", "inv_inertia", "s_rest", "s_compliance", "b_rest", "b_compliance",
            "b_rest_darboux", "omega")}
    P = np.cumsum([0] + [len(r.x) for r in rods])
    S = np.cumsum([0] + [len(r.q) for r in rods])
    for k, at in (("s_p0", P), ("s_p1", P), ("s_seg", S), ("b_a", S), ("b_b", S)):
        cat[k] = np.concatenate([getattr(r, k) + o for r, o in zip(rods, at)])
    return Rod.from_arrays(MATERIAL, **cat)


def shuffled(n, seed):
    """A coil of n segments, its stretch constraints in a shuffled order."""
    rod = Rod.centerline(helix(n, STEP * n, 0.03, 0.0098), MATERIAL, frame_seed=(0.0, 0.0, 1.0))
    keys = ("x", "v", "inv_mass", "q", "inertia", "inv_inertia", "s_p0", "s_p1", "s_seg", "s_rest", "s_compliance",
            "b_a", "b_b", "b_rest", "b_compliance", "b_rest_darboux", "omega")
    a = {k: np.array(getattr(rod, k)) for k in keys}
    a["b_rest_darboux"][:] = 0.0
    order = np.random.default_rng(seed).permutation(n)
    for k in ("s_p0", "s_p1", "s_seg", "s_rest", "s_compliance"):
        a[k] = a[k][order]
    return Rod.from_arrays(MATERIAL, **a)


def bundle(n, strands, far):
    """Strands of n segments: the first two 8.5 mm apart, the others `far` from them and each other."""
    at = [(0.0, 0.0, 0.0), (0.0, 0.008, 0.003)] + [(0.0, far * (i + 1), 0.0) for i in range(strands - 2)]
    return joined([line(n, a) for a in at])


RODS = {
    "bundle4": lambda: bundle(4, 8, 0.5), "bundle8": lambda: bundle(8, 5, 0.5), "bundle7": lambda: bundle(7, 6, 0.2),
    **{f"hairpin{n}": (lambda n=n: joined([hairpin(n), line(n, (0.0, 0.5, 0.0))])) for n in (8, 16, 24, 32, 48, 64)},
    "shuffled40": lambda: shuffled(40, 1), "shuffled200": lambda: shuffled(200, 2), "shuffled600": lambda: shuffled(600, 3),
}


def outcome(rods, params, steps, strategy):
    world = World([Primitive.plane((0.0, 0.0, -0.03), (0.0, 0.0, 1.0), 0.4)], self_collision=True, self_friction=0.4,
                  hash_table_size=256)
    with Batch.create_mixed(rods, [world], [0] * len(rods), strategy) as b:
        b.step_many(params, steps)
        assert b.error_count() == 0
        return ([b.read_self_contacts(r) for r in range(len(rods))], b.self_contact_overflow(),
                b.download_positions(), b.download_frames())


@pytest.mark.parametrize("name", sorted(RODS))
@pytest.mark.parametrize("params,steps", [(StepParams(dt=1.0 / 3600, substeps=1), 1),
                                          (StepParams(dt=1.0 / 60, substeps=6), 2)])
def test_contacts_of_any_topology_equal_serial(name, params, steps):
    rods = [RODS[name](), RODS[name]()]
    got = outcome(rods, params, steps, Strategy.BATCHED)
    want = outcome(rods, params, steps, Strategy.MULTI_KERNEL)
    assert steps > 1 or all(len(p) > 0 for p in want[0])
    for g, w in zip(got[0], want[0]):
        assert np.array_equal(g, w)
    assert got[1] == want[1]
    assert np.array_equal(got[2], want[2], equal_nan=True) and np.array_equal(got[3], want[3], equal_nan=True)
