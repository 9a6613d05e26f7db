// rp_batched.cu -- the persistent, length-sorted batched step.
//
// Work is a list of rod groups built on the host from rods sorted by length
// (longest first). A group is up to CTA/team rods that share a team size; the
// team size grows with the rod (about one thread per two segments, whole
// warps, 32..256), so a 64-segment rod is one warp and a 512-segment rod is
// eight; launches that leave half the GPU idle get about one thread per
// segment, up to 512 (planBatched). A persistent grid sized to the SMs' resident capacity pulls groups
// from a global counter, so long and short rods mix freely across SMs and the
// tail of the queue is short work.
//
// Inside a team the colour sweeps are separated by __syncwarp (one-warp teams)
// or a named barrier (bar.sync id, team) instead of a CTA-wide barrier, and
// the reference's self-collision pipeline (hash build, count pass, prefix sum,
// fill pass, sequential projection) is reorganised without changing its
// result:
//   * counting: the reference counts, for segment j, every later segment k
//     (k - j >= gap) in the hash buckets of the 27 cells around j whose
//     segments touch (separation < 0). A touching k sits in one bucket,
//     hash(cell(k)), so it is counted once per cell of the 27 whose hash is
//     that bucket. Touching pairs are found here by a broad phase over chain
//     blocks of 8 consecutive segments (box-distance culling with a bound no
//     tighter than the per-pair sphere test, then the per-pair test and the
//     shared narrow phase), each weighted by that multiplicity: the same
//     counts, without building the hash when nothing touches;
//   * when something touches, the pool is built from the touching pairs in
//     the reference's order: each entry's place is counted among its
//     segment's pairs. Only with more pairs than segments is the reference's
//     hash built (stable counting sort) and its fill pass run;
//   * the pool is projected level by level (contacts of a level share no
//     particle), which reproduces the sequential order's arithmetic, from
//     shared memory and by one warp while levels are narrow.
// Every per-element operation is the shared code in rp_step_common.cuh, so
// results are bit-identical to the plain kernel (contacts of a rod with itself
// use shared reciprocals here; rp_math.cuh names the one tie they round otherwise).
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "rp_bulk.cuh"
#include "rp_launch.h"
#include "rp_layout.h"
#include "rp_step_common.cuh"

namespace rp {

namespace {

__device__ __forceinline__ void teamSync(int team, int teamIdx) {
    if (team == 32) {
        __syncwarp();
    } else {
        asm volatile("bar.sync %0, %1;" ::"r"(teamIdx + 1), "r"(team) : "memory");
    }
}

// Minimum and maximum over a warp (NaN operands are passed over, as fminf does)
__device__ __forceinline__ float warpMax(float f) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(f));
    return r;
}
__device__ __forceinline__ float warpMin(float f) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(f));
    return r;
}

// A pointer into the kernel's shared memory, as one derived from the array
// itself: only through such does the compiler use shared-memory instructions
// (a pointer read back from memory is generic).
template <typename T>
__device__ __forceinline__ T* sharedMemory(T* p) {
    extern __shared__ __align__(16) unsigned char smem[];
    return reinterpret_cast<T*>(smem + (reinterpret_cast<const unsigned char*>(p) - smem));
}

__device__ __forceinline__ float4 driveVelocityB(const DDrive& d, double t) {
    const double s = double(d.amplitude) * double(d.omega) * cos(double(d.omega) * t + double(d.phase));
    return make_float4(float(s * double(d.ax)), float(s * double(d.ay)), float(s * double(d.az)), 0.0f);
}

// In-place exclusive scan of a[0..m) across the team; returns the total.
// `partial` holds one int per warp of the team. Integer, so deterministic.
__device__ int teamExclusiveScan(int32_t* a, int m, int lane, int team, int teamIdx, int32_t* partial) {
    const int per = (m + team - 1) / team;
    const int b = lane * per;
    const int e = min(m, b + per);
    int local = 0;
    for (int i = b; i < e; ++i) local += a[i];
    // inclusive scan of `local` within the warp
    const int wl = lane & 31;
    int inc = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (wl >= o) inc += y;
    }
    const int warp = lane >> 5, nwarps = team >> 5;
    if (wl == 31) partial[warp] = inc;
    teamSync(team, teamIdx);
    int before = 0, total = 0;
    for (int w = 0; w < nwarps; ++w) {
        const int pw = partial[w];
        if (w < warp) before += pw;
        total += pw;
    }
    int run = before + inc - local;
    for (int i = b; i < e; ++i) {
        const int v = a[i];
        a[i] = run;
        run += v;
    }
    teamSync(team, teamIdx);
    return total;
}

// Bits t = 9 (dz + 1) + 3 (dy + 1) + (dx + 1) of the 27 cells around
// cell(j) whose hash is k's bucket hash(cell(k)): the cells, in the
// reference's query order, at which its query meets k.
__device__ __forceinline__ unsigned bucketCells(float4 cj, float4 ck, float cell, int table) {
    bool ok = true;
    const Divisor d = divisor(cell, recip(cell, ok));
    ok = ok & (fmaxf(fmaxf(fabsf(cj.x), fabsf(cj.y)), fabsf(cj.z)) <= 0x1p60f) &
         (fmaxf(fmaxf(fabsf(ck.x), fabsf(ck.y)), fabsf(ck.z)) <= 0x1p60f);
    // cellCoord
    auto coord = [&](float v) { return static_cast<int>(floorf(ok ? quotient(v, d) : v / cell)); };
    const int cx = coord(cj.x), cy = coord(cj.y), cz = coord(cj.z);
    const unsigned hk = hashCell(coord(ck.x), coord(ck.y), coord(ck.z), table);
    const unsigned mask = unsigned(table) - 1u;
    unsigned m = 0u;
    if ((unsigned(table) & mask) == 0u) {  // hashCell masks its hash
        unsigned hx[3], hy[3], hz[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            hx[i] = unsigned(cx + i - 1) * 73856093u;
            hy[i] = unsigned(cy + i - 1) * 19349663u;
            hz[i] = (unsigned(cz + i - 1) * 83492791u) ^ hk;
        }
#pragma unroll
        for (int t = 0; t < 27; ++t)
            if (((hx[t % 3] ^ hy[t / 3 % 3] ^ hz[t / 9]) & mask) == 0u) m |= 1u << t;
        return m;
    }
    int t = 0;
    for (int dz = -1; dz <= 1; ++dz)
        for (int dy = -1; dy <= 1; ++dy)
            for (int dx = -1; dx <= 1; ++dx, ++t)
                if (hashCell(cx + dx, cy + dy, cz + dz, table) == hk) m |= 1u << t;
    return m;
}

constexpr int kMaxWarps = 16;  // of a CTA

// What a team needs about its rod beyond its shared-memory arrays: the fixed
// global pointers, the colour tables, the drive, the self-contact scratch.
// Lane 0 writes it once per rod into the rod's shared memory and every phase
// reads the fields it uses, so the substep loop carries only the current phase's values
// in registers (held in registers, these 64-bit pointers filled a third of
// the register file and pushed the constraint arithmetic into spills). The
// arrays in shared memory are not reached through it: pointers read back
// from memory lose their address space, and every access through them
// would be a generic load.
struct TeamCtx {
    RodGlobals G;                   // the rod's fixed global pointers (V.g)
    float4 rows[5];                 // its template rows where they are all equal
    RodView V;                      // copies of the view and scratch for the
    SelfScratch S;                  // separately compiled paths
    float4* velocity;               // the rod's velocities in global memory
    float4* omega;
    const int* sOrder;
    const int* bOrder;
    const int* sCol;
    const int* bCol;
    int32_t rod;                    // its index
    int32_t chain;                  // segment j joins particles j and j + 1
    int32_t sColors, bColors;
    int32_t nP, nSt;
    int32_t table, selfGap, selfCapacity;
    float selfFriction;
    double tRod;                    // the rod's simulated time (lane 0 advances it)
    int32_t driveP, wayP, wayStep;  // driven particle, waypoint particle and step
    int32_t stageFailed;            // a lane gave up waiting for the staged state
    uint64_t bar;                   // mbarrier of the rod's bulk stage-in

    // the particles of segments j and k
    __device__ void particles(int j, int k, int (&at)[4]) const {
        at[0] = chain ? j : G.sP0[j];
        at[1] = chain ? j + 1 : G.sP1[j];
        at[2] = chain ? k : G.sP0[k];
        at[3] = chain ? k + 1 : G.sP1[k];
    }
    // the rod's misc words (rp_layout.h)
    __device__ int32_t* misc() const { return S.live - 1; }
    __device__ int32_t* numLevels() const { return misc() + 3; }  // projection levels of the pool
    __device__ int32_t* partial() const { return misc() + 16; }   // scan partials, one per warp
    __device__ int32_t* touching() const { return misc() + 14; }  // a self-contact pair touches this substep
    __device__ int32_t* numPairs() const { return misc() + 15; }  // how many do
    // pair of every pool entry, (j << 16) | k, where the count's block bounds were
    __device__ int32_t* ids() const { return reinterpret_cast<int32_t*>(sharedMemory(S.blocks)); }
    // behind the rod's hash in global memory (DRod::hashOff)
    __device__ int32_t* cursor() const { return S.cellStart + (table + 1); }  // placement cursors
    __device__ int32_t* lvlOrder() const { return cursor() + (table + 1); }   // coloured mode only
    __device__ int32_t* lvlStart() const { return lvlOrder() + (selfCapacity + 1); }
    __device__ int32_t* lvlOf() const { return lvlStart() + (selfCapacity + 1); }
};

// A pair within reach: the shared narrow phase, and for a
// touching pair its bucket multiplicity, its count and its place in the pair
// list (which holds nSt pairs; beyond that the count alone is kept and the
// pool is built from the hash). Not inlined: few pairs get here, and its
// body is shared by every caller.
__device__ __noinline__ void countTouching(const TeamCtx& C, int j, int k, float cell) {
    const SelfScratch& S = C.S;
    const float4* const x = sharedMemory(C.V.x);
    int p[4];
    C.particles(j, k, p);
    const SegPair P = segmentPairNarrow(v3(x[p[0]]), v3(x[p[1]]), v3(x[p[2]]), v3(x[p[3]]), 2.0f * C.G.radius);
    if (P.separation >= 0.0f) return;
    const unsigned cells = bucketCells(S.centres[j], S.centres[k], cell, C.table);
    if (cells) {
        atomicAdd(&S.segCount[j], __popc(cells));
        *C.touching() = 1;
        const int at = atomicAdd(C.numPairs(), 1);
        if (at < C.nSt) {
            S.segStart[at] = (j << 16) | k;
            S.sorted[at] = int32_t(cells);  // for the pool; the hash path rebuilds it
        }
    }
}

// segCount[j] (zeroed by the caller) += the reference's count of segment j;
// every touching pair (j, k) is also appended to S.segStart as (j << 16) | k
// (*C.numPairs(), zeroed by the caller, counts them; entries past nSt are not
// stored).
// `reach` is the longest segment plus 2 r with the margins of the sphere test
// of querySelfSegment (1.001 and 1e-6 of the coordinates' size, here of the
// rod's largest), so a pair whose centres are farther apart fails that test;
// `cell` is the longest segment plus 2 r. Pairs of near indices are tested a
// segment per lane, or, on a chain, ruled out by two distances; the others by
// blocks of 8 segments: box distance, then, for blocks within reach, the 64
// pairs, two per lane. Box and centre distances are monotone in float, and the
// two distances bound a chain's centres by its longest segment, so no pair the
// sphere test keeps is missed (tests/test_count_enumeration.py replays the
// rounds). Pairs within reach wait in the warp's queue, and the narrow phase
// runs on 32 of them at once.
//
// Bound: issue slots. In free fall three of five rounds a block went to near
// pairs, which no rod passes that is not sharply bent. In settled rods two or
// three lanes of a round pass, and the narrow phase run for those alone took
// most of the count. 4096 uneven rods in free fall, 50 substeps, 6.55 -> 5.68 ms
// (the count 10.6 -> 6.3 thousand cycles a rod and substep); 256 settled rods of
// 16-512 2.02 -> 1.74 ms; 8 cables of 40-200, 20 substeps, 217 -> 157 us.
__device__ __forceinline__ void countSelfByBlocks(const TeamCtx& C, const SelfScratch& S, int nSt, int gap,
                                                  float cell, float reach, int lane, int team) {
    __shared__ int32_t queues[kMaxWarps][32];  // per warp: pairs that wait for the narrow phase
    if (nSt <= gap) return;
    const int wl = lane & 31, warp = lane >> 5, warps = team >> 5;
    const int nBlk = (nSt + 7) >> 3;
    // This lane's pair of the block with itself, for the near pairs: the 28
    // pairs (a, b), a < b, of a block ordered by b - a descending, so the
    // pairs with b - a >= gap are a prefix (28 of them for gap 1, 15 for 3).
    int ta = -1, tb = -1;
    {
        int e = wl;
        for (int d = 7; d >= 1; --d) {
            if (e < 8 - d) {
                ta = e;
                tb = e + d;
                break;
            }
            e -= 8 - d;
        }
    }
    // The per-pair test of every lane that has a pair. The pairs that pass wait
    // in the warp's queue for a full warp of them.
    const unsigned below = (1u << wl) - 1u;
    int32_t* const queue = queues[threadIdx.x >> 5];
    const float reach2 = reach * reach * 1.0001f;
    int waiting = 0;
    auto flush = [&]() {
        __syncwarp();
        if (wl < waiting) countTouching(C, queue[wl] >> 16, queue[wl] & 0xffff, cell);
        __syncwarp();
        waiting = 0;
    };
    auto testPairs = [&](bool have, int j, int k) {
        bool pass = false;
        if (have) pass = !(norm2(v3(S.centres[k]) - v3(S.centres[j])) > reach2);
        const unsigned m = __ballot_sync(0xffffffffu, pass);
        if (m) {
            if (waiting + __popc(m) > 32) flush();
            if (pass) queue[waiting + __popc(m & below)] = (j << 16) | k;
            waiting += __popc(m);
        }
    };
    // Near pairs: between a block J and itself, J + 1 and J + 2, at most 23
    // apart, 32 segments j at a time. Pairs exactly `gap` apart are tested as
    // they are, a segment per lane. The others need no test where the centres 8
    // and 18 segments on lie so far from j that those before and shortly
    // behind them, each at most the longest segment from the next, are out of
    // reach as well (the factor 1.002 is far above the rounding). That is so
    // on a chain only: segments of consecutive indices lie anywhere in other
    // rods, which test all near pairs, and so do rods with a gap above 7, past
    // what this covers.
    const bool split = C.chain && gap < 8;
    const int near = split ? gap + 1 : gap;
    const int last = nSt - 1;
    const float step = (cell - 2.0f * C.V.g->radius) * 1.0001f;  // the longest segment
    for (int j0 = 32 * warp; j0 < nSt; j0 += 32 * warps) {
        unsigned clear = 0u;
        if (split) {
            const int j = j0 + wl;
            testPairs(j + gap <= last, j, j + gap);
            const V3 cj = v3(S.centres[min(j, last)]);
            const int e8 = min(j + 8, last), e18 = min(j + 18, last);
            const float d8 = norm2(v3(S.centres[e8]) - cj), d18 = norm2(v3(S.centres[e18]) - cj);
            const float need8 = (reach + float(max(e8 - j - near, e8 < last ? 4 : 0)) * step) * 1.002f;
            const float need18 = (reach + float(max(e18 - j - 13, e18 < last ? 5 : 0)) * step) * 1.002f;
            clear = __ballot_sync(0xffffffffu, (e8 - j < near || d8 > need8 * need8) &&
                                                   (e18 - j < 13 || d18 > need18 * need18));
            // a centre that is no number says nothing of its neighbours' places
            // (the centres read here are all that the chunk's near pairs have)
            if (__any_sync(0xffffffffu, !(d8 + d18 >= 0.0f))) clear = 0u;
        }
        if (clear == 0xffffffffu) continue;
#pragma unroll 1
        for (int J = j0 >> 3; J < min((j0 >> 3) + 4, nBlk); ++J, clear >>= 8) {
            if ((clear & 0xffu) == 0xffu) continue;
            // J against J + 1 and J + 2 in two rounds of 32 each, J against
            // itself in one over the pairs with b - a >= near
#pragma unroll 1
            for (int round = 0; round < 5; ++round) {
                const int j = 8 * J + (round < 4 ? wl & 7 : ta);
                const int k = 8 * J + (round < 4 ? 8 + (wl >> 3) + 4 * round : tb);
                testPairs((round < 4 || ta >= 0) && k < nSt && k - j >= near, j, k);
            }
        }
    }
    // Far pairs: the boxes of two blocks J, J + 1 together against 32 blocks
    // K >= J + 3 at a time, then each of the two against the blocks that are left.
    for (int J0 = 2 * warp; J0 < nBlk; J0 += 2 * warps) {
        const int J1 = min(J0 + 1, nBlk - 1);
        const V3 l0 = v3(S.blocks[2 * J0]), h0 = v3(S.blocks[2 * J0 + 1]);
        const V3 l1 = v3(S.blocks[2 * J1]), h1 = v3(S.blocks[2 * J1 + 1]);
        const V3 lo{fminf(l0.x, l1.x), fminf(l0.y, l1.y), fminf(l0.z, l1.z)};
        const V3 hi{fmaxf(h0.x, h1.x), fmaxf(h0.y, h1.y), fmaxf(h0.z, h1.z)};
        auto apart = [](V3 al, V3 ah, V3 bl, V3 bh) {  // squared distance of two boxes
            const float gx = fmaxf(0.0f, fmaxf(bl.x - ah.x, al.x - bh.x));
            const float gy = fmaxf(0.0f, fmaxf(bl.y - ah.y, al.y - bh.y));
            const float gz = fmaxf(0.0f, fmaxf(bl.z - ah.z, al.z - bh.z));
            return gx * gx + gy * gy + gz * gz;
        };
        for (int K0 = J0 + 3; K0 < nBlk; K0 += 32) {
            const int K = K0 + wl;
            bool hit = false;
            if (K < nBlk) hit = !(apart(lo, hi, v3(S.blocks[2 * K]), v3(S.blocks[2 * K + 1])) > reach2);
            for (unsigned m = __ballot_sync(0xffffffffu, hit); m; m &= m - 1u) {
                const int Kh = K0 + __ffs(m) - 1;
                const V3 kl = v3(S.blocks[2 * Kh]), kh = v3(S.blocks[2 * Kh + 1]);
#pragma unroll 1
                for (int J = J0; J <= J0 + 1 && Kh >= J + 3; ++J) {
                    if (apart(J == J0 ? l0 : l1, J == J0 ? h0 : h1, kl, kh) > reach2) continue;
#pragma unroll 1
                    for (int h2 = 0; h2 < 2; ++h2) {
                        const int j = 8 * J + (wl & 7), k = 8 * Kh + (wl >> 3) + 4 * h2;
                        testPairs(k < nSt && k - j >= near, j, k);
                    }
                }
            }
        }
    }
    flush();
}

// Polls of the stage-in barrier before a lane gives up (each poll may wait a
// while in hardware): far beyond any real copy, so it ends only a broken one.
constexpr int kStageTries = 1 << 20;
// DArgs::errors bit of a rod whose state copy never completed
constexpr int32_t kErrorStage = 2;

static_assert(sizeof(TeamCtx) <= kContextBytes && alignof(TeamCtx) <= 16, "the layout's room for a team context");

// The order in which a filled pool is projected, by the team's first warp:
// levels such that contacts of one level share no particle and every earlier
// contact a contact shares a particle with lies in a lower level (level = 1 +
// the highest among those), so that projecting level by level computes what
// the serial pool order computes. S.segCount receives each contact's place in
// level-major order, then the end of every level; *C.numLevels() the count.
//
// Bound: the chain of levels through a chunk of 32 contacts, one shuffle per
// contact that a later one of the chunk depends on. Conflicts inside a chunk
// come from a mask of its lanes per particle, conflicts with earlier chunks
// from each particle's last level, both in the shared memory of the count's
// centres. The serial form, one thread over contacts in global memory, took
// 35 % of the step of 32 settled rods of 1500-2200 segments (474 contacts in
// 55 levels).
//
// An entry that was left unwritten (its id is -1 until the thread that writes
// the entry sets it) or that indexes outside the rod cuts the pool before it and
// is reported; it is never dereferenced.
__device__ __forceinline__ void orderPool(const TeamCtx& C, int live, int precision, int32_t* errorWord, int lane) {
    constexpr unsigned kAll = 0xffffffffu;
    const SelfScratch& S = C.S;
    const int nP = C.nP;
    int32_t* const last = reinterpret_cast<int32_t*>(sharedMemory(S.centres));  // per particle: its highest level + 1
    int32_t* const lanes = last + nP;                              // per particle: this chunk's lanes
    int32_t* const place = sharedMemory(S.segCount);
    const int32_t* const ids = C.ids();
    auto particles = [&](int c) {
        const int j = ids[c] >> 16, k = ids[c] & 0xffff;
        return C.chain ? make_int4(j, j + 1, k, k + 1) : *reinterpret_cast<const int4*>(S.pool[c].idx);
    };
    int kept = live;
    for (int c0 = 0; c0 < live; c0 += 32) {
        const int c = c0 + lane;
        bool ok = true;
        if (c < live) {
            const int4 at = particles(c);
            ok = min(min(at.x, at.y), min(at.z, at.w)) >= 0 && max(max(at.x, at.y), max(at.z, at.w)) < nP &&
                 ids[c] != -1;
            if (ok) {
                last[at.x] = last[at.y] = last[at.z] = last[at.w] = 0;
                lanes[at.x] = lanes[at.y] = lanes[at.z] = lanes[at.w] = 0;
            }
        }
        const unsigned bad = __ballot_sync(kAll, !ok);
        if (bad) {
            kept = c0 + __ffs(bad) - 1;
            break;
        }
    }
    __syncwarp();
    if (kept != live && lane == 0) {
        *S.live = kept;
        if (errorWord) atomicOr(errorWord, 1);
    }
    int32_t* const ends = place + kept;
    if (precision & kPrecisionColoredSelf) {
        // greedy colours instead (more than 32 of them: the levels)
        for (int i = lane; i < nP; i += 32) S.cellOf[i] = 0;
        __syncwarp();
        int n = 0;
        if (lane == 0) n = buildProjectionColors(S.pool, kept, S.cellOf, C.lvlOf(), C.lvlOrder(), C.lvlStart());
        n = __shfl_sync(kAll, n, 0);
        __syncwarp();
        if (n >= 0) {
            for (int i = lane; i < kept; i += 32) place[C.lvlOrder()[i]] = i;
            for (int l = lane; l < n; l += 32) ends[l] = C.lvlStart()[l + 1];
            if (lane == 0) *C.numLevels() = n;
            return;
        }
    }
    int levels = 0;
    for (int c0 = 0; c0 < kept; c0 += 32) {
        const int c = c0 + lane;
        const bool mine = c < kept;
        int4 at = make_int4(0, 0, 0, 0);
        int level = 0;
        if (mine) {
            at = particles(c);
            level = max(max(last[at.x], last[at.y]), max(last[at.z], last[at.w]));
            atomicOr(&lanes[at.x], 1 << lane);
            atomicOr(&lanes[at.y], 1 << lane);
            atomicOr(&lanes[at.z], 1 << lane);
            atomicOr(&lanes[at.w], 1 << lane);
        }
        __syncwarp();
        unsigned before = 0u;  // the chunk's earlier contacts this one shares a particle with
        if (mine)
            before = unsigned(lanes[at.x] | lanes[at.y] | lanes[at.z] | lanes[at.w]) & ((1u << lane) - 1u);
        for (unsigned need = __reduce_or_sync(kAll, before); need; need &= need - 1u) {
            const int l = __ffs(need) - 1;
            const int above = __shfl_sync(kAll, level, l) + 1;
            if ((before >> l) & 1u) level = max(level, above);
        }
        if (mine) {
            place[c] = level;
            lanes[at.x] = lanes[at.y] = lanes[at.z] = lanes[at.w] = 0;
            atomicMax(&last[at.x], level + 1);
            atomicMax(&last[at.y], level + 1);
            atomicMax(&last[at.z], level + 1);
            atomicMax(&last[at.w], level + 1);
        }
        levels = max(levels, __reduce_max_sync(kAll, mine ? level + 1 : 0));
        __syncwarp();
    }
    // counts per level, their running sum, and each contact's place: a
    // level's cursor ends at its last contact
    for (int l = lane; l < levels; l += 32) ends[l] = 0;
    __syncwarp();
    for (int c = lane; c < kept; c += 32) atomicAdd(&ends[place[c]], 1);
    __syncwarp();
    int sum = 0;
    for (int l0 = 0; l0 < levels; l0 += 32) {
        const int l = l0 + lane;
        const int n = l < levels ? ends[l] : 0;
        int inc = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kAll, inc, o);
            if (lane >= o) inc += y;
        }
        if (l < levels) ends[l] = sum + inc - n;
        sum += __shfl_sync(kAll, inc, 31);
    }
    __syncwarp();
    for (int c = lane; c < kept; c += 32) place[c] = atomicAdd(&ends[place[c]], 1);
    if (lane == 0) *C.numLevels() = levels;
}

// The pool fill of a substep on which some segment pair touches: the
// reference's hash (a stable counting sort) and its fill pass in bucket order.
// For pools that the pair list cannot give (more than nSt touching pairs).
__device__ __forceinline__ void fillSelfPool(const TeamCtx& C, float cell, int live, int lane, int team,
                                             int teamIdx) {
    const RodView& V = C.V;
    const SelfScratch& S = C.S;
    const int nSt = C.nSt, table = C.table;
    int32_t* const cursor = C.cursor();
    int32_t* const partial = C.partial();
    // ---- fill, in the reference's order: its hash buckets ----
    for (int t = lane; t <= table; t += team) S.cellStart[t] = 0;
    for (int c = lane; c < live; c += team) S.pool[c].seg = -1;
    teamSync(team, teamIdx);
    for (int j = lane; j < nSt; j += team) {
        const float4 c = S.centres[j];
        const int h0 = int(hashCell(cellCoord(c.x, cell), cellCoord(c.y, cell),
                                    cellCoord(c.z, cell), table));
        S.cellOf[j] = h0;
        atomicAdd(&S.cellStart[h0], 1);
    }
    teamSync(team, teamIdx);
    // counts -> starts: cellStart[t] = first slot of bucket t,
    // cellStart[table] = segment count (the reference's offsets)
    teamExclusiveScan(S.cellStart, table + 1, lane, team, teamIdx, partial);
    for (int t = lane; t < table; t += team) cursor[t] = S.cellStart[t];
    teamSync(team, teamIdx);
    // stable placement, one warp walking segments in order
    if (lane < 32) {
        for (int j0 = 0; j0 < nSt; j0 += 32) {
            const int j = j0 + lane;
            const bool valid = j < nSt;
            const int c = valid ? S.cellOf[j] : -1 - lane;
            const unsigned peers = __match_any_sync(0xffffffffu, c);
            const int rank = __popc(peers & ((1u << lane) - 1u));
            const int start = valid ? cursor[c] : 0;
            __syncwarp();
            if (valid) {
                S.sorted[start + rank] = j;
                if (rank == 0) cursor[c] = start + __popc(peers);
            }
            __syncwarp();
        }
    }
    teamSync(team, teamIdx);
    for (int j = lane; j < nSt; j += team)
        if (S.segCount[j] > 0 && S.segStart[j] < C.selfCapacity)
            querySelfSegment<true>(V, S, j, nSt, C.selfGap, table, C.selfCapacity, C.selfFriction, true);
}

// Most touching substeps have a handful of touching pairs; for those the
// pool is built from the count's pair list by the team's first warp, with
// no hash. The reference's query for segment j walks the 27 cells around
// cell(j) in order and, in each, the bucket of that cell's hash in segment
// order, so its pool holds one entry per touching pair (j, k) and per cell t
// whose hash is k's bucket, ordered by (j, t, k), and segment j's entries
// start after every entry of the segments before it. Each lane takes one
// pair, finds its cells, ranks each of its entries by counting the entries
// of every pair that order before it, and writes them with the query's own
// entry writer: the same pool, entry for entry. Lanes past the capacity
// write nothing, as the query does. Every lane of the warp calls this; it
// returns the reference's count of entries. The pair list is
// S.segStart[0..numPairs), numPairs <= 32, with the cells in S.sorted; S.segCount
// holds the pairs' cells afterwards.
__device__ __forceinline__ int poolFromPairs(const TeamCtx& C, int numPairs, int lane) {
    const SelfScratch& S = C.S;
    const float4* const x = sharedMemory(C.V.x);
    const float friction = C.selfFriction * C.G.frictionScale;
    int32_t* const ids = C.ids();
    const bool mine = lane < numPairs;
    int j = 0, k = 0;
    unsigned cells = 0u;
    if (mine) {
        const int pr = S.segStart[lane];
        j = pr >> 16;
        k = pr & 0xffff;
        cells = unsigned(S.sorted[lane]);
    }
    const int total = __reduce_add_sync(0xffffffffu, __popc(cells));
    __syncwarp();
    for (int c = lane; c < min(total, C.selfCapacity); c += 32) ids[c] = -1;  // not written yet
    if (mine) S.segCount[lane] = int32_t(cells);
    __syncwarp();
    if (mine) {
        int at[4];
        C.particles(j, k, at);
        const SegPair P = segmentPairNarrow(v3(x[at[0]]), v3(x[at[1]]), v3(x[at[2]]), v3(x[at[3]]), 2.0f * C.G.radius);
        // entries of the pairs of earlier segments
        int before = 0;
        for (int q = 0; q < numPairs; ++q)
            if ((S.segStart[q] >> 16) < j) before += __popc(unsigned(S.segCount[q]));
        for (unsigned rest = cells; rest; rest &= rest - 1u) {
            const int t = __ffs(rest) - 1;
            const unsigned below = (1u << t) - 1u;
            int rank = before;
            for (int q = 0; q < numPairs; ++q) {
                const int pq = S.segStart[q];
                if ((pq >> 16) != j) continue;
                const unsigned cq = unsigned(S.segCount[q]);
                rank += __popc(cq & below) + (((cq >> t) & 1u) && (pq & 0xffff) < k ? 1 : 0);
            }
            if (rank < C.selfCapacity) {
                writeSelfEntryAt(x, S.pool[rank], at, j, k, P, friction);
                ids[rank] = (j << 16) | k;
            }
        }
    }
    return total;
}

// The same pool from any number of listed pairs (at most nSt), by the whole
// team. Where a segment's entries start is the running sum of the counts;
// their order within the segment comes from the segment's own pairs, linked
// per segment (the order of a list is of no matter: ranks are sums over it).
// Lists and cells lie in the shared memory of the count's centres.
//
// Against the hash (build, placement by one warp, and the 27-cell query of
// every touching segment by one thread each), which bound the step of settled
// rods: with orderPool above and projectSelfCompact below, 32 settled rods of
// 1500-2200 segments at 20 substeps 32.4 -> 10.5 ms, 256 of 16-512 at 50
// substeps 8.53 -> 2.08 ms, and rods in free fall, which touch now and then,
// 4096 of 16-512, 7.65 -> 6.93 ms.
__device__ __forceinline__ int poolFromManyPairs(const TeamCtx& C, int numPairs, int lane, int team, int teamIdx) {
    const SelfScratch& S = C.S;
    const int nSt = C.nSt;
    const float4* const x = sharedMemory(C.V.x);
    const float friction = C.selfFriction * C.G.frictionScale;
    int32_t* const ids = C.ids();
    int32_t* const head = reinterpret_cast<int32_t*>(sharedMemory(S.centres));  // per segment: its last linked pair
    int32_t* const next = head + nSt;                             // per pair
    int32_t* const cellsOf = next + nSt;                          // per pair
    for (int p = lane; p < numPairs; p += team) {
        head[S.segStart[p] >> 16] = -1;
        cellsOf[p] = S.sorted[p];
    }
    const int total = teamExclusiveScan(S.segCount, nSt, lane, team, teamIdx, C.partial());
    for (int c = lane; c < min(total, C.selfCapacity); c += team) ids[c] = -1;  // not written yet
    for (int p = lane; p < numPairs; p += team) next[p] = atomicExch(&head[S.segStart[p] >> 16], p);
    teamSync(team, teamIdx);
    for (int p = lane; p < numPairs; p += team) {
        const int pr = S.segStart[p], j = pr >> 16, k = pr & 0xffff;
        const int before = S.segCount[j];
        if (before >= C.selfCapacity) continue;
        const unsigned cells = unsigned(cellsOf[p]);
        int at[4];
        C.particles(j, k, at);
        const SegPair P = segmentPairNarrow(v3(x[at[0]]), v3(x[at[1]]), v3(x[at[2]]), v3(x[at[3]]), 2.0f * C.G.radius);
        for (unsigned rest = cells; rest; rest &= rest - 1u) {
            const int t = __ffs(rest) - 1;
            const unsigned below = (1u << t) - 1u;
            int rank = before;
            for (int q = head[j]; q >= 0; q = next[q]) {
                const unsigned cq = unsigned(cellsOf[q]);
                rank += __popc(cq & below) + (((cq >> t) & 1u) && (S.segStart[q] & 0xffff) < k ? 1 : 0);
            }
            if (rank < C.selfCapacity) {
                writeSelfEntryAt(x, S.pool[rank], at, j, k, P, friction);
                ids[rank] = (j << 16) | k;
            }
        }
    }
    return total;
}

// The pool of a substep on which some pair touches, and its order. One call:
// each function called from the substep loop makes the loop's registers live
// across it.
__device__ __noinline__ void buildPool(const TeamCtx& C, float cell, int precision, int32_t* errorWord, int lane,
                                       int team, int teamIdx) {
    const SelfScratch& S = C.S;
    const int pairs = *C.numPairs(), nSt = C.nSt;
    int total = 0;
    if (pairs <= 32 && pairs <= nSt) {
        if (lane < 32) total = poolFromPairs(C, pairs, lane);
    } else if (pairs <= nSt) {
        total = poolFromManyPairs(C, pairs, lane, team, teamIdx);
    } else {
        for (int j = lane; j < nSt; j += team) S.segStart[j] = S.segCount[j];
        teamSync(team, teamIdx);
        total = teamExclusiveScan(S.segStart, nSt, lane, team, teamIdx, C.partial());
        fillSelfPool(C, cell, min(total, C.selfCapacity), lane, team, teamIdx);
        teamSync(team, teamIdx);
        for (int c = lane; c < min(total, C.selfCapacity); c += team) C.ids()[c] = S.pool[c].seg;
    }
    if (lane == 0) {
        *S.live = min(total, C.selfCapacity);
        if (total > C.selfCapacity) *S.overflow += total - C.selfCapacity;
    }
    teamSync(team, teamIdx);  // pool written, positions read: the prediction may start
    if (lane < 32) orderPool(C, *S.live, precision, errorWord, lane);
}

// Contact c of the pool into its place of the compact, level-major rows in
// shared memory: {particles}, {u, w}, {n.x, n.y}, {n.z, offset}, {lambdaN,
// applied}, each a row of `live` 8-byte words.
__device__ __forceinline__ void compactContact(const SelfScratch& S, int c, int live) {
    const DSelf& k = S.pool[c];
    float2* const rows = reinterpret_cast<float2*>(S.centres) + S.segCount[c];
    rows[0] = make_float2(__int_as_float(k.idx[0] | (k.idx[1] << 16)), __int_as_float(k.idx[2] | (k.idx[3] << 16)));
    rows[live] = make_float2(k.weight[1], -k.weight[3]);
    rows[2 * live] = make_float2(k.nx, k.ny);
    rows[3 * live] = make_float2(k.nz, k.offset);
    rows[4 * live] = make_float2(0.0f, 0.0f);
}

// The self-contact pool projected level by level: contacts of one level
// share no particle, and every earlier contact a contact shares a particle
// with sits in a lower level -- the serial pool order's result, bit for bit
// (but for the ties of rp_math.cuh's shared reciprocals).
// Not inlined: it runs only while contacts are live. Levels are short (nine
// contacts on average in settled rods) and there are many, so the chain of
// one contact's loads and arithmetic per level is what it takes: one warp
// does them without team barriers unless the levels are wider than a warp,
// from shared memory.
template <bool COMP>
__device__ __noinline__ void projectSelfCompact(const TeamCtx& C, int levels, int live, int lane, int team,
                                                int teamIdx) {
    extern __shared__ __align__(16) unsigned char smem[];
    const RodView& V = C.V;
    const SelfScratch& S = C.S;
    // the compiler reaches shared memory with shared-memory instructions only
    // through a pointer derived from the array itself
    auto shared = [&](const void* p) { return smem + (static_cast<const unsigned char*>(p) - smem); };
    float4* const x = reinterpret_cast<float4*>(shared(V.x));
    float4* const xPrev = reinterpret_cast<float4*>(shared(V.xPrev));
    float4* const xComp = COMP ? reinterpret_cast<float4*>(shared(V.xComp)) : nullptr;
    float2* const rows = reinterpret_cast<float2*>(shared(S.centres));
    const int32_t* const ends = reinterpret_cast<const int32_t*>(shared(S.segCount)) + live;
    const float friction = C.selfFriction * V.g->frictionScale;
    const bool oneWarp = live <= 32 * levels;
    const int stride = oneWarp ? 32 : team;
    if (lane < stride) {
        for (int l = 0, begin = 0; l < levels; ++l) {
            const int end = ends[l];
            for (int c = begin + lane; c < end; c += stride) {
                const float2 i = rows[c], uw = rows[live + c], nxy = rows[2 * live + c], nzo = rows[3 * live + c];
                float2 lam = rows[4 * live + c];
                const unsigned a = __float_as_uint(i.x), b = __float_as_uint(i.y);
                const int at[4] = {int(a & 0xffffu), int(a >> 16), int(b & 0xffffu), int(b >> 16)};
                const float weight[4] = {1.0f - uw.x, uw.x, -(1.0f - uw.y), -uw.y};
                const V3 n{nxy.x, nxy.y, nzo.x};
                const bool distinct = at[0] != at[1] && at[0] != at[2] && at[0] != at[3] && at[1] != at[2] &&
                                      at[1] != at[3] && at[2] != at[3];
                if (!distinct || !projectSelfDistinct<COMP>(x, xPrev, xComp, at, weight, n, nzo.y, friction,
                                                            lam.x, lam.y)) {
                    DSelf k;
                    for (int m = 0; m < 4; ++m) {
                        k.idx[m] = at[m];
                        k.weight[m] = weight[m];
                    }
                    k.nx = n.x;
                    k.ny = n.y;
                    k.nz = n.z;
                    k.offset = nzo.y;
                    k.friction = friction;
                    k.lambdaN = lam.x;
                    k.applied = lam.y;
                    projectSelf<COMP>(V, k);
                    lam = make_float2(k.lambdaN, k.applied);
                }
                rows[4 * live + c] = lam;
            }
            begin = end;
            if (oneWarp)
                __syncwarp();
            else
                teamSync(team, teamIdx);
        }
    }
    teamSync(team, teamIdx);
}

template <bool COMP, bool FP64, bool SELF>
__device__ void runRod(const DArgs& A, int r, unsigned char* base, int lane, int team, int teamIdx) {
    const DRod R = A.rods[r];
    const DTemplate T = A.tmpl[R.tmpl];
    const int nP = T.nP, nS = T.nS, nSt = T.nSt, nB = T.nB;

    const RodLayout L = rodLayout(nP, nS, nSt, nB, R.numPrims, R.selfCollision, R.hashTableSize,
                                  R.selfCapacity, 1, COMP ? 1 : 0, A.slotsShared);
    TeamCtx& C = *reinterpret_cast<TeamCtx*>(base + L.ctx);
    // The view of the rod's arrays lives in registers: its shared-memory
    // arrays are addressed from `base`, so the compiler reaches them with
    // shared-memory instructions through 32-bit addresses. The fixed global
    // pointers (loads, template, primitives) sit in the team's context,
    // reached through V.g.
    RodView V;
    V.g = &C.G;
    V.numPrims = R.numPrims;
    V.rowMask = T.evenOdd & 4 ? 0 : -1;
    V.softness = A.invH2 * A.complianceScale[r];
    V.q = reinterpret_cast<float4*>(base + L.q);
    V.qPrev = COMP ? A.gqPrev + R.sOff : reinterpret_cast<float4*>(base + L.qPrev);
    V.x = reinterpret_cast<float4*>(base + L.x);
    V.xPrev = reinterpret_cast<float4*>(base + L.xPrev);
    V.xComp = COMP ? reinterpret_cast<float4*>(base + L.xComp) : A.xComp + R.pOff;
    V.qComp = COMP ? reinterpret_cast<float4*>(base + L.qComp) : A.qComp + R.sOff;
    // velocities: none in shared memory (see the prediction below); the
    // state arrays in global memory hold them between steps
    V.v = nullptr;
    V.omega = nullptr;
    // multipliers: none at one iteration; else in global memory (L1/L2)
    V.lamS = A.iterations > 1 ? A.gLamS + R.stOff : nullptr;
    V.lamB = A.iterations > 1 ? A.gLamB + R.bOff : nullptr;
    V.slots = A.slotsShared ? reinterpret_cast<DSlot*>(base + L.slots) : A.gSlots + R.slotOff;
    SelfScratch S;
    S.centres = reinterpret_cast<float4*>(base + L.centres);
    S.segCount = reinterpret_cast<int32_t*>(base + L.selfInt);
    S.segStart = S.segCount + nSt;
    // touched only on substeps where a pair touches: global memory (L1/L2)
    S.cellOf = A.gSelfInt + 2 * int64_t(R.stOff);
    S.sorted = S.cellOf + nSt;
    S.cellStart = A.gHash + R.hashOff;  // then the cursors, then the levels
    S.pool = A.gPool + R.poolOff;
    int32_t* misc = reinterpret_cast<int32_t*>(base + L.misc);
    S.cellSize = reinterpret_cast<float*>(misc);
    S.live = misc + 1;
    S.overflow = misc + 2;
    S.blocks = S.centres + nSt;
    int32_t* numLevels = misc + 3;
    unsigned long long* primMask = reinterpret_cast<unsigned long long*>(misc + 12);
    int32_t* touching = misc + 14;
    int32_t* numPairs = misc + 15;
    float* red = reinterpret_cast<float*>(misc + 16);  // 8 floats per warp
    if (lane == 0) {
        RodGlobals& G = C.G;
        G.invMass = A.tInvMass + T.pOff;
        G.invInertia = A.tInvInertia + T.sOff;
        G.inertia = A.tInertia + T.sOff;
        G.sP0 = A.tSP0 + T.stOff;
        G.sP1 = A.tSP1 + T.stOff;
        G.sSeg = A.tSSeg + T.stOff;
        G.sComp = A.tSComp + T.stOff;
        G.bA = A.tBA + T.bOff;
        G.bB = A.tBB + T.bOff;
        G.bComp = A.tBComp + T.bOff;
        G.bRestD = A.tBRestD + T.bOff;
        G.prims = A.prims + R.primOff;
        if (V.rowMask == 0) {
            const float4* const from[5] = {G.invInertia, G.inertia, G.sComp, G.bComp, G.bRestD};
            for (int i = 0; i < 5; ++i) C.rows[i] = i < 3 || nB > 0 ? *from[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            G.invInertia = &C.rows[0];
            G.inertia = &C.rows[1];
            G.sComp = &C.rows[2];
            G.bComp = &C.rows[3];
            G.bRestD = &C.rows[4];
        }
        // lean layout: loads and kinematic velocities stay in global memory
        G.force = A.force + R.pOff;
        G.kin = A.kinVel + R.pOff;
        G.torque = A.torque + R.sOff;
        G.radius = R.radius;
        G.contactMargin = R.contactMargin;
        G.frictionScale = A.frictionScale[r];
        C.velocity = A.v + R.pOff;
        C.omega = A.omega + R.sOff;
        C.V = V;  // for the rarely run, separately compiled paths
        G.view = &C.V;
        C.S = S;
        C.nP = nP;
        C.nSt = nSt;
        C.table = R.hashTableSize;
        C.selfGap = R.selfGap;
        C.selfCapacity = R.selfCapacity;
        C.selfFriction = R.selfFriction;
        C.sOrder = A.tOrder + T.sOrderOff;
        C.bOrder = A.tOrder + T.bOrderOff;
        C.sCol = A.tColorStart + T.sColorOff;
        C.bCol = A.tColorStart + T.bColorOff;
        C.sColors = T.sColors;
        C.bColors = T.bColors;
        C.rod = r;
        C.chain = T.chain;
        *numLevels = 0;
        *primMask = ~0ull;
        // simulated time of this rod, advanced per step exactly as the
        // one-step-per-launch path advances rodTime[r]
        C.tRod = A.rodTime[r];
        C.driveP = -1;
        if (A.drives) {
            const int p = A.drives[r].particle;
            if (p >= 0 && p < nP) C.driveP = p;
        }
        C.wayP = -1;  // waypoint schedule: its particle and step count
        C.wayStep = 0;
        if (A.waypoints) {
            const DWaypoints& W = A.waypoints[r];
            if (W.particle >= 0 && W.particle < nP) {
                C.wayP = W.particle;
                C.wayStep = W.step;
            }
        }
    }
    teamSync(team, teamIdx);
    const int* const& sOrder = C.sOrder;
    const int* const& bOrder = C.bOrder;
    const int* const& sCol = C.sCol;
    const int* const& bCol = C.bCol;

    // ---- stage in: one bulk copy per state array, on the team's mbarrier ----
    const uint32_t pBytes = uint32_t(nP) * 16u, sBytes = uint32_t(nS) * 16u;
    if (lane == 0) {
        C.stageFailed = 0;
        mbarInit(&C.bar);
        mbarArriveExpectTx(&C.bar, pBytes + sBytes + (COMP ? pBytes + sBytes : 0u));
        bulkLoad(V.x, A.x + R.pOff, pBytes, &C.bar);
        bulkLoad(V.q, A.q + R.sOff, sBytes, &C.bar);
        if (COMP) {
            bulkLoad(V.xComp, A.xComp + R.pOff, pBytes, &C.bar);
            bulkLoad(V.qComp, A.qComp + R.sOff, sBytes, &C.bar);
        }
    }
    teamSync(team, teamIdx);  // the barrier is initialised before anyone polls it
    if (!mbarWaitBounded(&C.bar, 0, kStageTries)) atomicOr(&C.stageFailed, 1);
    teamSync(team, teamIdx);  // every lane is past the wait: the barrier can go
    if (lane == 0) mbarInvalidate(&C.bar);
    if (C.stageFailed) {  // team-uniform: read after the barrier
        if (lane == 0 && A.errors) atomicOr(A.errors + r, kErrorStage);
        fenceProxyAsyncShared();
        return;
    }

    // the inverse masses ride in the positions' fourth word: every phase that
    // needs one reads the position anyway
    for (int i = lane; i < nP; i += team) V.x[i].w = V.g->invMass[i];

    const V3 g{A.gx, A.gy, A.gz};
    const float h = A.h;
    const int interval = A.contactInterval;
    const bool self = SELF && R.selfCollision != 0;
    // bits 0 and 1: even/odd stretch and bend colours of a chain; bit 2: a chain
    const int order = T.chain ? (T.evenOdd & 3) | 4 : 0;

    const int stepsHere = A.stepsPerLaunch > 0 ? A.stepsPerLaunch : 1;
    for (int step = 0; step < stepsHere; ++step) {
        if (lane == 0) {
            if (C.driveP >= 0) V.g->kin[C.driveP] = driveVelocityB(A.drives[C.rod], C.tRod);
            if (C.wayP >= 0) V.g->kin[C.wayP] = waypointVelocity(A.waypoints[C.rod], C.wayStep + step);
        }
        teamSync(team, teamIdx);
        for (int sub = 0; sub < A.substeps; ++sub) {
            if (V.lamS) {  // team-uniform
                for (int k = lane; k < nSt; k += team) V.lamS[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                for (int k = lane; k < nB; k += team) V.lamB[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
            const bool regenerate = sub % interval == 0;
            unsigned long long maskNow = *primMask;  // this substep's primitive cull
            float cellNow = 0.0f, sizeNow = 1.0f;    // this substep's self-collision cell, coordinate size
            if (regenerate && (V.numPrims > 0 || self)) {
                // One pass for both contact kinds: segment centres and half
                // lengths, the longest segment (self-collision cell size), and the
                // rod's bounding box (primitive culling).
                //
                // Bound: issue slots (17 % of a step of rods in free fall). Two
                // segments a lane, so that a chain block of 8 takes two shuffle
                // steps per bound instead of three and its inner particles are
                // read once; the count bounds half lengths and coordinates by
                // the rod's largest instead of the block's; a chain's box for the cull is its centres' box
                // grown by half the longest segment; minima over the warp are one
                // float redux each. 4096 x 64 over a floor, 80 substeps, 1.27 ->
                // 1.19 ms; 4096 uneven rods with self-collision, 50 substeps, 6.93
                // -> 6.55 ms.
                float mx = 0.0f, size = 1.0f;
                V3 lo{3.0e38f, 3.0e38f, 3.0e38f}, hi{-3.0e38f, -3.0e38f, -3.0e38f};
                auto cover = [](V3& l, V3& h, V3 p) {
                    l = V3{fminf(l.x, p.x), fminf(l.y, p.y), fminf(l.z, p.z)};
                    h = V3{fmaxf(h.x, p.x), fmaxf(h.y, p.y), fmaxf(h.z, p.z)};
                };
                const bool chain = (order & 4) != 0;
                const bool boxOfCentres = self && chain;
                if (self) {
                    // whole warps per round (team is a multiple of 32), so the
                    // 4-lane shuffles bounding each chain block of 8 segments
                    // always have every lane present; the counts are zeroed
                    // here too, so the count needs no barrier of its own
                    for (int i0 = 0; 2 * i0 < nSt; i0 += team) {
                        const int j = 2 * (i0 + lane);
                        V3 bl{3.0e38f, 3.0e38f, 3.0e38f}, bh{-3.0e38f, -3.0e38f, -3.0e38f};
                        auto centre = [&](int k, V3 a, V3 b) {
                            const float len = norm(b - a);
                            const V3 c = (a + b) * 0.5f;
                            S.centres[k] = make_float4(c.x, c.y, c.z, 0.5f * len);
                            S.segCount[k] = 0;
                            mx = fmaxf(mx, len);
                            size = fmaxf(size, 1.0f + fabsf(c.x) + fabsf(c.y) + fabsf(c.z));
                            cover(bl, bh, c);
                        };
                        if (j < nSt) {
                            V3 a = v3(V.x[chain ? j : V.g->sP0[j]]), b = v3(V.x[chain ? j + 1 : V.g->sP1[j]]);
                            centre(j, a, b);
                            if (j + 1 < nSt) {
                                a = chain ? b : v3(V.x[V.g->sP0[j + 1]]);
                                b = v3(V.x[chain ? j + 2 : V.g->sP1[j + 1]]);
                                centre(j + 1, a, b);
                            }
                        }
                        lo = V3{fminf(lo.x, bl.x), fminf(lo.y, bl.y), fminf(lo.z, bl.z)};
                        hi = V3{fmaxf(hi.x, bh.x), fmaxf(hi.y, bh.y), fmaxf(hi.z, bh.z)};
#pragma unroll
                        for (int o = 1; o < 4; o <<= 1) {
                            bl.x = fminf(bl.x, __shfl_xor_sync(0xffffffffu, bl.x, o));
                            bl.y = fminf(bl.y, __shfl_xor_sync(0xffffffffu, bl.y, o));
                            bl.z = fminf(bl.z, __shfl_xor_sync(0xffffffffu, bl.z, o));
                            bh.x = fmaxf(bh.x, __shfl_xor_sync(0xffffffffu, bh.x, o));
                            bh.y = fmaxf(bh.y, __shfl_xor_sync(0xffffffffu, bh.y, o));
                            bh.z = fmaxf(bh.z, __shfl_xor_sync(0xffffffffu, bh.z, o));
                        }
                        if ((lane & 3) == 0 && j < nSt) {
                            S.blocks[2 * (j >> 3)] = f4(bl);
                            S.blocks[2 * (j >> 3) + 1] = f4(bh);
                        }
                    }
                    mx = warpMax(mx);
                    size = warpMax(size);
                }
                if (V.numPrims > 0) {
                    if (!boxOfCentres) {
                        lo = V3{3.0e38f, 3.0e38f, 3.0e38f};
                        hi = V3{-3.0e38f, -3.0e38f, -3.0e38f};
                        for (int i = lane; i < nP; i += team) cover(lo, hi, v3(V.x[i]));
                    }
                    lo = V3{warpMin(lo.x), warpMin(lo.y), warpMin(lo.z)};
                    hi = V3{warpMax(hi.x), warpMax(hi.y), warpMax(hi.z)};
                }
                if (team > 32 && (lane & 31) == 0) {
                    float4* const row = reinterpret_cast<float4*>(red + 8 * (lane >> 5));
                    row[0] = make_float4(mx, lo.x, lo.y, lo.z);
                    row[1] = make_float4(hi.x, hi.y, hi.z, size);
                }
                // reset before the barrier: the count below follows without one
                if (lane == 0) {
                    *touching = 0;
                    *numPairs = 0;
                }
                teamSync(team, teamIdx);  // centres, blocks, zeroed counts, rows visible
                // every lane reduces the rows in the same order (max and min
                // are exact), so every lane holds the same mask and cell size;
                // lane 0 also publishes them for the later phases
                for (int w = 0; team > 32 && w < (team >> 5); ++w) {
                    const float4* const row = reinterpret_cast<const float4*>(red + 8 * w);
                    const float4 a = row[0], b = row[1];
                    mx = fmaxf(mx, a.x);
                    size = fmaxf(size, b.w);
                    lo = V3{fminf(lo.x, a.y), fminf(lo.y, a.z), fminf(lo.z, a.w)};
                    hi = V3{fmaxf(hi.x, b.x), fmaxf(hi.y, b.y), fmaxf(hi.z, b.z)};
                }
                if (V.numPrims > 0) {
                    const float grow = boxOfCentres ? 0.5f * mx : 0.0f;
                    const V3 g3{grow, grow, grow};
                    maskNow = primitivesNearBox(V, lo - g3, hi + g3, lane & 31);
                    if (lane == 0) *primMask = maskNow;
                }
                cellNow = mx + 2.0f * V.g->radius;
                sizeNow = size;
                if (self && lane == 0) {
                    if (sub == 0) *S.overflow = 0;
                    *S.cellSize = cellNow;  // for the fill pass, after later barriers
                }
            }
            if (V.numPrims > 0 && maskNow != 0ull) {  // team-uniform; a fully culled world has no slot
                for (int i = lane; i < nP; i += team) generateSlotsMasked<COMP>(V, i, regenerate, maskNow);
            }
            if (self) {
                if (regenerate) {
                    const float cell = cellNow;
                    // ---- count: contacts per segment, by chain blocks ----
                    // chain-block bounds and zeroed counts come from the centre pass
                    // the pair list takes segStart, which the hash path rebuilds
                    countSelfByBlocks(C, S, nSt, C.selfGap, cell, cell * 1.001f + 1e-6f * sizeNow, lane, team);
                    teamSync(team, teamIdx);
                    // team-uniform: shared words read after the barrier
                    if (*touching) {
                        buildPool(C, cell, A.precision, A.errors ? A.errors + C.rod : nullptr, lane, team, teamIdx);
                    } else if (lane == 0) {
                        *S.live = 0;
                        *numLevels = 0;
                    }
                } else {
                    float2* const lam = reinterpret_cast<float2*>(S.centres) + 4 * *S.live;
                    for (int c = lane; c < *S.live; c += team) lam[c] = make_float2(0.0f, 0.0f);
                }
                // no barrier here: every read of positions above finished before
                // an earlier barrier, the prediction below touches neither the
                // pool nor its order, and what the first warp writes last
                // is read only after the prediction's barrier -- so the other
                // warps predict while it orders the pool
            }
            // the previous substep's velocity update runs here, fused with this
            // substep's prediction: nothing between them reads v or omega,
            // and each element's two updates stay with one thread, so the
            // velocities pass from the update to the prediction in registers;
            // the prediction's own velocity is never read (the next update
            // replaces it), so velocities are in memory only between steps
            for (int i = lane; i < nP; i += team) {
                const float4 vi = sub > 0 ? finishedVelocity<COMP>(V, i, h, A.linDecay) : C.velocity[i];
                predictParticleFrom<COMP>(V, i, h, g, vi, nullptr);
            }
            for (int j = lane; j < nS; j += team) {
                const float4 wj = sub > 0 ? finishedOmega<COMP>(V, j, h, A.angDecay) : C.omega[j];
                predictFrameFrom<COMP>(V, j, h, wj, nullptr);
            }
            teamSync(team, teamIdx);
            // the ordered pool into shared memory, over the count's centres and
            // counts: the barriers of the sweeps below come before its rows are
            // read and before the next substep's centre pass writes there again.
            // A step of no sweeps has no such barrier, and nothing reads the rows.
            if (self && regenerate && A.iterations > 0 && *numLevels > 0)
                for (int c = lane; c < *S.live; c += team) compactContact(S, c, *S.live);

            for (int it = 0; it < A.iterations; ++it) {
                // a chain coloured even/odd: constraint k of colour c is
                // k = 2 i + c with particles k, k+1 and frames k, k+1, so no
                // index is loaded; same constraints, same arithmetic
                if (order & 1) {
                    for (int c = 0; c < 2; ++c) {
                        for (int k = 2 * lane + c; k < nSt; k += 2 * team)
                            projectStretchAt<COMP>(V, k, k, k + 1, k);
                        teamSync(team, teamIdx);
                    }
                } else {
                    for (int c = 0; c < C.sColors; ++c) {
                        for (int ci = sCol[c] + lane; ci < sCol[c + 1]; ci += team)
                            projectStretchOne<COMP>(V, sOrder[ci]);
                        teamSync(team, teamIdx);
                    }
                }
                if ((order & 2) && nB < nSt) {
                    for (int c = 0; c < 2; ++c) {
                        for (int k = 2 * lane + c; k < nB; k += 2 * team)
                            projectBendAt<COMP>(V, k, k, k + 1);
                        teamSync(team, teamIdx);
                    }
                } else if (order & 2) {
                    // with ghost frames, whose bends follow the real ones: one
                    // call for both, or the warp that holds a ghost runs the
                    // whole projection twice (a 64-segment cantilever's step:
                    // 184 -> 123 us; the same loop for rods without ghosts
                    // would cost the 4096 x 64 grid 4 %)
                    for (int c = 0; c < 2; ++c) {
                        for (int k = 2 * lane + c; k < nB; k += 2 * team) {
                            const bool ghost = k >= nSt - 1;
                            const int a = ghost ? V.g->bA[k] : k;
                            const int b = ghost ? V.g->bB[k] : k + 1;
                            projectBendAt<COMP>(V, k, a, b);
                        }
                        teamSync(team, teamIdx);
                    }
                } else {
                    for (int c = 0; c < C.bColors; ++c) {
                        for (int ci = bCol[c] + lane; ci < bCol[c + 1]; ci += team)
                            projectBendOne<COMP>(V, bOrder[ci]);
                        teamSync(team, teamIdx);
                    }
                }
                const unsigned long long mask = V.numPrims > 0 ? *primMask : 0ull;
                if (mask != 0ull) {
                    for (int i = lane; i < nP; i += team) projectSlots<COMP, FP64>(V, i, mask);
                    teamSync(team, teamIdx);
                }
                if (self) {
                    const int nl = *numLevels;
                    if (nl > 0) projectSelfCompact<COMP>(C, nl, *S.live, lane, team, teamIdx);
                }
            }

        }
        // the step's last velocity update
        for (int i = lane; i < nP; i += team) C.velocity[i] = finishedVelocity<COMP>(V, i, h, A.linDecay);
        for (int j = lane; j < nS; j += team) C.omega[j] = finishedOmega<COMP>(V, j, h, A.angDecay);
        teamSync(team, teamIdx);

        // ---- per-step bookkeeping ----
        if (lane == 0) {
            if (self) A.selfOverflow[C.rod] += *S.overflow;
            if (A.hold) {
                DHold& H = A.hold[C.rod];
                if (H.particle >= 0 && H.particle < nP) {
                    H.steps += 1;
                    if (A.holdInterval > 0 && H.steps % A.holdInterval == 0) {
                        double z = double(V.x[H.particle].z);
                        if (COMP) z -= double(V.xComp[H.particle].z);
                        const double rise = z - H.startZ;
                        if (rise > H.maxRise) H.maxRise = rise;
                    }
                }
            }
        }
        if (lane == 0) C.tRod += double(A.dt);
    }  // steps of this launch

    // ---- stage out: bulk copies from shared memory, then the outputs ----
    const DRod& out = A.rods[C.rod];  // read again: not worth registers through the steps
    for (int i = lane; i < nP; i += team) V.x[i].w = 0.0f;  // the rows' pad in global memory
    // every lane's writes above reach the async proxy before lane 0 copies
    fenceProxyAsyncShared();
    teamSync(team, teamIdx);
    if (lane == 0) {
        bulkStore(A.x + out.pOff, V.x, pBytes);
        bulkStore(A.q + out.sOff, V.q, sBytes);
        if (COMP) {
            bulkStore(A.xComp + out.pOff, V.xComp, pBytes);
            bulkStore(A.qComp + out.sOff, V.qComp, sBytes);
        }
        bulkCommit();
    }
    if (V.numPrims > 0 && A.contactState) {
        const int slots = nP * V.numPrims;
        for (int s = lane; s < slots; s += team)
            A.contactState[out.slotOff + s] = ((*primMask >> (s % V.numPrims)) & 1ull) ? static_cast<uint8_t>(V.slots[s].state) : uint8_t(0);
    }
    if (self) {
        const int live = *S.live;
        for (int c = lane; c < live; c += team) A.selfPairs[out.poolOff + c] = S.pool[c].seg;
    }
    if (lane == 0) {
        if (self) A.selfCount[C.rod] = *S.live;
        A.rodTime[C.rod] = C.tRod;
        if (C.wayP >= 0) A.waypoints[C.rod].step = C.wayStep + stepsHere;
    }
    // the stores have read the rows, and every lane's accesses of this shared
    // memory come before the next rod's bulk copies overwrite it
    if (lane == 0) bulkWaitRead();
    fenceProxyAsyncShared();
}

// SELF: some rod of the launch collides with itself. Launches without run an
// instance without that code, which spills nothing where this one spills 212
// bytes (loads, reference order) at the 128 registers that two 256-thread CTAs
// leave: 4096 rods of 64 over a floor, 80 substeps, 1.25 -> 1.13 ms.
template <bool COMP, bool FP64, bool SELF>
__global__ void __launch_bounds__(512, 1) kBatchedStep(DArgs A, const int32_t* __restrict__ groups,
                                                       int numGroups, int32_t* queue) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int sGroup;
    const int tid = threadIdx.x;
    for (;;) {
        if (tid == 0) sGroup = atomicAdd(queue, 1);
        __syncthreads();
        const int gi = sGroup;
        __syncthreads();
        if (gi >= numGroups) break;
        const int first = groups[4 * gi], count = groups[4 * gi + 1], team = groups[4 * gi + 2];
        const int teamIdx = tid / team, lane = tid - teamIdx * team;
        if (teamIdx < count) {
            // this team's slice of the group's shared memory
            size_t off = 0;
            for (int k = 0; k < teamIdx; ++k) {
                const DRod Rk = A.rods[A.work[first + k]];
                const DTemplate Tk = A.tmpl[Rk.tmpl];
                off += size_t(rodLayout(Tk.nP, Tk.nS, Tk.nSt, Tk.nB, Rk.numPrims, Rk.selfCollision,
                                        Rk.hashTableSize, Rk.selfCapacity, 1, COMP ? 1 : 0, A.slotsShared)
                                  .bytes);
            }
            runRod<COMP, FP64, SELF>(A, A.work[first + teamIdx], smem + off, lane, team, teamIdx);
        }
        __syncthreads();
    }
    bulkWaitAll();  // this thread's state stores are complete before it exits
    // The last CTA out resets the queue for the next launch.
    if (tid == 0) {
        __threadfence();
        const int done = atomicAdd(queue + 1, 1);
        if (done == int(gridDim.x) - 1) {
            atomicExch(queue, 0);
            atomicExch(queue + 1, 0);
            __threadfence();
        }
    }
}

using Kernel = void (*)(DArgs, const int32_t*, int, int32_t*);

// The instance for a precision and for launches with or without
// self-collision.
Kernel instance(int precision, bool self) {
    const bool comp = (precision & 1) != 0, fp64 = (precision & 2) != 0;
    if (self) {
        if (comp) return fp64 ? kBatchedStep<true, true, true> : kBatchedStep<true, false, true>;
        return fp64 ? kBatchedStep<false, true, true> : kBatchedStep<false, false, true>;
    }
    if (comp) return fp64 ? kBatchedStep<true, true, false> : kBatchedStep<true, false, false>;
    return fp64 ? kBatchedStep<false, true, false> : kBatchedStep<false, false, false>;
}

}  // namespace

cudaError_t launchBatchedStep(const DArgs& a, const BatchedPlan& p, int precision, cudaStream_t s) {
    if (p.numGroups <= 0) return cudaSuccess;
    instance(precision, p.anySelf)<<<p.blocks, p.threads, p.smemBytes, s>>>(a, p.groups, p.numGroups, p.queue);
    return cudaGetLastError();
}

// The attribute belongs to the kernel, not to a batch: it only ever grows
// (per device), so a later, smaller plan never shrinks what an earlier batch
// launches with.
cudaError_t batchedReserveSmem(size_t bytes) {
    static std::mutex mu;
    static int reserved[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> g(mu);
    const int want = static_cast<int>(bytes);
    if (want <= reserved[dev]) return cudaSuccess;
    for (int i = 0; i < 8; ++i)
        if ((e = cudaFuncSetAttribute(instance(i & 3, (i & 4) != 0), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      want)) != cudaSuccess)
            return e;
    reserved[dev] = want;
    return cudaSuccess;
}

// The kernel's static shared memory (the warps' queues, the group word): the
// dynamic part of a plan may use the opt-in limit minus this.
size_t batchedStaticSmem() {
    size_t most = 0;
    cudaFuncAttributes a;
    for (int i = 0; i < 8; ++i)
        if (cudaFuncGetAttributes(&a, instance(i & 3, (i & 4) != 0)) == cudaSuccess)
            most = std::max(most, a.sharedSizeBytes);
    cudaGetLastError();
    return most;
}

cudaError_t batchedOccupancy(int threads, size_t smem, int precision, bool anySelf, int* perSm) {
    // the instance the launch will use: register counts differ between them
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(perSm, instance(precision, anySelf), threads, smem);
}

}  // namespace rp
