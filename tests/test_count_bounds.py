"""The box test of the batched self-contact count (`countSelfByBlocks`,
csrc/rp_batched.cu) bounds a block's pairs from the rod's longest segment and
the block's own box. In float32, on seeded rods near and far from the origin
with uneven segments, every pair the per-pair sphere test keeps lies in blocks
that the box test lets through."""
import numpy as np
import pytest

f32 = np.float32


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("far", [0.0, 40.0, 3000.0])
def test_box_test_keeps_what_the_sphere_test_keeps(seed, far):
    rng = np.random.default_rng(seed)
    n, radius = int(rng.integers(20, 200)), f32(rng.uniform(0.001, 0.02))
    steps = rng.normal(size=(n + 1, 3)) * rng.uniform(0.2, 1.8, (n + 1, 1)) * 0.006
    x = (np.cumsum(steps, axis=0) + far * rng.uniform(-1, 1, 3)).astype(f32)
    centre = (x[:-1] + x[1:]) * f32(0.5)
    d = x[1:] - x[:-1]
    length = np.sqrt((d * d).sum(1, dtype=f32)).astype(f32)
    half, two_r = f32(0.5) * length, f32(2.0) * radius
    cell = f32(length.max() + two_r)
    size = ((f32(1.0) + abs(centre[:, 0])) + abs(centre[:, 1])) + abs(centre[:, 2])
    blocks = (n + 7) // 8
    lo = np.array([centre[8 * b:8 * b + 8].min(0) for b in range(blocks)])
    hi = np.array([centre[8 * b:8 * b + 8].max(0) for b in range(blocks)])
    top = np.maximum(abs(lo), abs(hi))
    slack = f32(1e-6) * (((f32(1.0) + top[:, 0]) + top[:, 1]) + top[:, 2])
    kept = 0
    for j in range(n):
        gap = centre[j + 1:] - centre[j]
        plim = ((half[j] + half[j + 1:]) + two_r) * f32(1.001) + f32(1e-6) * size[j]
        near = ~((gap[:, 0] * gap[:, 0] + gap[:, 1] * gap[:, 1]) + gap[:, 2] * gap[:, 2] > plim * plim)
        J = j // 8
        for k in np.flatnonzero(near) + j + 1:
            K = k // 8
            g = np.maximum(f32(0), np.maximum(lo[K] - hi[J], lo[J] - hi[K]))
            lim = cell * f32(1.001) + slack[J]
            assert not (g[0] * g[0] + g[1] * g[1]) + g[2] * g[2] > (lim * lim) * f32(1.0001)
            kept += K > J + 1
    assert kept > 0 or far == 0.0


def turned_chain(rng, n, step, radius):
    """A chain of n segments turning by a random walk of curvature up to 1 / radius."""
    heading, x = np.array([1.0, 0.0, 0.0]), [np.zeros(3)]
    axis = rng.normal(size=3)
    for _ in range(n):
        axis = axis + 0.3 * rng.normal(size=3)
        turn = np.cross(heading, axis / np.linalg.norm(axis))
        heading = heading + turn * step / radius
        heading /= np.linalg.norm(heading)
        x.append(x[-1] + heading * step * rng.uniform(0.7, 1.0))
    return np.array(x)


@pytest.mark.parametrize("seed", range(8))
@pytest.mark.parametrize("gap", [1, 2, 3, 5, 7])
def test_cleared_segments_have_no_near_pair_in_reach(seed, gap):
    """The two distances by which the count rules out a segment's near pairs:
    no segment it clears has another gap + 1 to 23 segments on within reach, on
    chains from straight to curled up, with ends of every remainder."""
    rng = np.random.default_rng(100 * gap + seed)
    n, radius = int(rng.integers(gap + 2, 90)), f32(rng.uniform(0.001, 0.008))
    x = (turned_chain(rng, n, 0.006, rng.choice([0.004, 0.01, 0.03, 0.1, 10.0])) + rng.uniform(-2, 2, 3)).astype(f32)
    centre = (x[:-1] + x[1:]) * f32(0.5)
    d = x[1:] - x[:-1]
    longest = np.sqrt((d * d).sum(1, dtype=f32)).max()
    cell = f32(longest + f32(2.0) * radius)
    size = (f32(1.0) + abs(centre).sum(1, dtype=f32)).max()
    reach = f32(cell * f32(1.001) + f32(1e-6) * size)
    step, near, last = f32((cell - f32(2.0) * radius) * f32(1.0001)), gap + 1, n - 1

    def norm2(j, k):
        v = centre[k] - centre[j]
        return (v[0] * v[0] + v[1] * v[1]) + v[2] * v[2]
    cleared = 0
    for j in range(n):
        e8, e18 = min(j + 8, last), min(j + 18, last)
        need8 = (reach + f32(max(e8 - j - near, 4 if e8 < last else 0)) * step) * f32(1.002)
        need18 = (reach + f32(max(e18 - j - 13, 5 if e18 < last else 0)) * step) * f32(1.002)
        if (e8 - j < near or norm2(j, e8) > need8 * need8) and (e18 - j < 13 or norm2(j, e18) > need18 * need18):
            cleared += 1
            for k in range(j + near, min(j + 24, n)):
                assert norm2(j, k) > reach * reach * f32(1.0001)
    assert cleared > 0
