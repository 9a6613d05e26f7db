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
