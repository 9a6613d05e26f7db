"""The pairs that the batched self-contact count tests (`countSelfByBlocks`,
csrc/rp_batched.cu), replayed in float32 round by round: the pairs exactly `gap`
apart, the near rounds of the blocks that are not ruled out, and the far blocks
by the boxes of two blocks at a time. Every pair that the per-pair sphere test
of the serial query keeps must be among them, once, and be within the rod's
reach -- on chains from straight to folded, bundles of short strands, strands
that end in a U-turn beside far ones, chains in shuffled order and rods with a
NaN, for every gap on both sides of the near rule's limit and ends of every
remainder, near the origin and far from it."""
import numpy as np
import pytest

f32 = np.float32
INF = f32(3.0e38)


def norm2(v):
    return f32(f32(f32(v[0] * v[0]) + f32(v[1] * v[1])) + f32(v[2] * v[2]))


class Rod:
    """Centres, half lengths and what the centre pass makes of them (minima and
    maxima pass over NaN, as the kernel's do)."""

    def __init__(self, a, b, radius, chain):
        a, b = np.asarray(a, f32), np.asarray(b, f32)
        self.n, self.chain, self.radius = len(a), chain, f32(radius)
        d = b - a
        length = np.sqrt(np.array([norm2(v) for v in d], f32))
        self.c, self.half = (a + b) * f32(0.5), f32(0.5) * length
        self.l1 = ((f32(1.0) + abs(self.c[:, 0])) + abs(self.c[:, 1])) + abs(self.c[:, 2])
        self.cell = f32(np.fmax(f32(0.0), np.fmax.reduce(length)) + f32(2.0) * self.radius)
        size = np.fmax(f32(1.0), np.fmax.reduce(self.l1))
        self.reach = f32(self.cell * f32(1.001) + f32(1e-6) * size)
        self.reach2 = f32(f32(self.reach * self.reach) * f32(1.0001))
        blocks = range((self.n + 7) // 8)
        self.lo = np.array([np.fmin(INF, np.fmin.reduce(self.c[8 * B:8 * B + 8])) for B in blocks], f32)
        self.hi = np.array([np.fmax(-INF, np.fmax.reduce(self.c[8 * B:8 * B + 8])) for B in blocks], f32)

    def distance2(self, j, k):
        return norm2(self.c[k] - self.c[j])

    def sphere_keeps(self, j, k):  # querySelfSegment
        lim = f32(f32(f32(self.half[j] + self.half[k]) + f32(2.0) * self.radius) * f32(1.001)) + f32(1e-6) * self.l1[j]
        return not self.distance2(j, k) > f32(lim * lim)


def triangle(lane):
    """The lane's pair of a block with itself, by b - a descending."""
    e = lane
    for d in range(7, 0, -1):
        if e < 8 - d:
            return e, e + d
        e -= 8 - d
    return None


def cleared(rod, gap, j0):
    """Lanes of the chunk of 32 segments at j0 whose near pairs are ruled out."""
    near, last, step = gap + 1, rod.n - 1, f32(f32(rod.cell - f32(2.0) * rod.radius) * f32(1.0001))
    out, numbers = [], True
    for j in range(j0, j0 + 32):
        e8, e18, at = min(j + 8, last), min(j + 18, last), min(j, last)
        d8, d18 = rod.distance2(at, e8), rod.distance2(at, e18)
        need8 = f32((rod.reach + f32(max(e8 - j - near, 4 if e8 < last else 0)) * step) * f32(1.002))
        need18 = f32((rod.reach + f32(max(e18 - j - 13, 5 if e18 < last else 0)) * step) * f32(1.002))
        out.append((e8 - j < near or d8 > need8 * need8) and (e18 - j < 13 or d18 > need18 * need18))
        numbers = numbers and bool(d8 + d18 >= 0)
    return out if numbers else [False] * 32


def box_distance2(al, ah, bl, bh):
    return norm2([max(f32(0), f32(bl[i] - ah[i]), f32(al[i] - bh[i])) for i in range(3)])


def enumerated(rod, gap):
    """Every pair the count tests against the reach, in no particular order."""
    n, out = rod.n, []
    if n <= gap:
        return out
    blocks = (n + 7) // 8
    split = rod.chain and gap < 8
    near = gap + 1 if split else gap
    for j0 in range(0, n, 32):
        clear = [False] * 32
        if split:
            out += [(j, j + gap) for j in range(j0, j0 + 32) if j + gap < n]
            clear = cleared(rod, gap, j0)
        for J in range(j0 // 8, min(j0 // 8 + 4, blocks)):
            if all(clear[8 * J - j0:8 * J - j0 + 8]):
                continue
            for rnd in range(5):
                for lane in range(32):
                    pair = (lane & 7, 8 + (lane >> 3) + 4 * rnd) if rnd < 4 else triangle(lane)
                    if pair is None:
                        continue
                    j, k = 8 * J + pair[0], 8 * J + pair[1]
                    if k < n and k - j >= near:
                        out.append((j, k))
    for J0 in range(0, blocks, 2):
        J1 = min(J0 + 1, blocks - 1)
        lo, hi = np.fmin(rod.lo[J0], rod.lo[J1]), np.fmax(rod.hi[J0], rod.hi[J1])
        for K in range(J0 + 3, blocks):
            if box_distance2(lo, hi, rod.lo[K], rod.hi[K]) > rod.reach2:
                continue
            for J in (J0, J0 + 1):
                if K < J + 3 or box_distance2(rod.lo[J], rod.hi[J], rod.lo[K], rod.hi[K]) > rod.reach2:
                    continue
                out += [(j, k) for j in range(8 * J, 8 * J + 8) for k in range(8 * K, min(8 * K + 8, n)) if k - j >= near]
    return out


def check(rod, gap):
    got = enumerated(rod, gap)
    assert len(got) == len(set(got)), "a pair is tested twice"
    got = set(got)
    kept = 0
    for j in range(rod.n):
        for k in range(j + gap, rod.n):
            if not rod.sphere_keeps(j, k):
                continue
            if not np.isfinite(rod.distance2(j, k)) and k // 8 - j // 8 > 2:
                continue  # the boxes pass over a NaN
            kept += 1
            assert (j, k) in got, (j, k)
            assert not rod.distance2(j, k) > rod.reach2
    return kept


def walk(rng, n, turn, step=0.006):
    """A chain of n segments whose direction turns by up to `turn` a segment."""
    heading, x = np.array([1.0, 0.0, 0.0]), [np.zeros(3)]
    for _ in range(n):
        heading = heading + turn * rng.normal(size=3)
        heading /= np.linalg.norm(heading)
        x.append(x[-1] + heading * step * rng.uniform(0.7, 1.0))
    return np.array(x)


def strands(rng, lengths, far):
    """Strands of `lengths` segments: of every two, the second lies beside the first, the pairs `far` apart; a U-turn ends each."""
    a, b = [], []
    for i, n in enumerate(lengths):
        turn = np.zeros(n)
        turn[max(0, n - 4):] = 0.5 * np.pi
        turn[max(0, n - 3):] = np.pi
        d = 0.006 * np.stack([np.cos(turn), np.sin(turn), np.zeros(n)], 1)
        x = np.concatenate([np.zeros((1, 3)), np.cumsum(d, 0)]) + (0.0, (i // 2) * far, 0.008 * (i % 2))
        a.append(x[:-1])
        b.append(x[1:])
    return np.concatenate(a), np.concatenate(b)


GAPS = [2, 3, 5, 7, 8, 12, 24, 30]


@pytest.mark.parametrize("gap", GAPS)
@pytest.mark.parametrize("turn", [0.0, 0.15, 0.6, 3.0])
def test_chains(gap, turn):
    rng = np.random.default_rng(int(100 * turn) + gap)
    kept = 0
    for n, away in ((gap, 0.0), (gap + 1, 0.0), (9, 2.0), (16, 0.0), (33, 40.0), (50, 0.0), (71, 3000.0), (104, 2.0)):
        x = walk(rng, n, turn) + away * rng.uniform(-1, 1, 3)
        kept += check(Rod(x[:-1], x[1:], rng.uniform(0.002, 0.006), True), gap)
    assert kept > 0 or turn < 0.6


@pytest.mark.parametrize("gap", GAPS)
@pytest.mark.parametrize("lengths", [(4,) * 8, (7, 7, 7, 7, 7), (8, 8), (16, 16, 16), (48, 48), (5, 31, 12, 3)])
def test_strands(gap, lengths):
    a, b = strands(np.random.default_rng(gap), lengths, 0.5)
    check(Rod(a, b, 0.005, False), gap)


@pytest.mark.parametrize("lengths", [(4,) * 8, (48, 48, 48)])
def test_strands_taken_as_a_chain_lose_pairs(lengths):
    """The near rule is for chains: on strands it would rule out pairs in reach."""
    a, b = strands(np.random.default_rng(0), lengths, 0.5)
    with pytest.raises(AssertionError):
        check(Rod(a, b, 0.005, True), 3)


@pytest.mark.parametrize("gap", GAPS)
def test_shuffled_chains(gap):
    rng = np.random.default_rng(gap)
    kept = 0
    for n in (20, 75):
        x, order = walk(rng, n, 0.6), rng.permutation(n)
        kept += check(Rod(x[:-1][order], x[1:][order], 0.005, False), gap)
    assert kept > 0


@pytest.mark.parametrize("at", range(0, 40, 3))
@pytest.mark.filterwarnings("ignore:invalid value")
def test_a_nan_keeps_its_near_pairs(at):
    for turn in (0.0, 0.6):
        x = walk(np.random.default_rng(at), 40, turn)
        x[at] = np.nan
        assert check(Rod(x[:-1], x[1:], 0.005, True), 3) > 0
