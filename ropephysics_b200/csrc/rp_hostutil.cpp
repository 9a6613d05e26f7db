// rp_hostutil.cpp -- host helpers shared by the batch (rp_batch.cpp) and the
// serving loop (rp_server.cpp): device checks, descriptor conversion to the
// device layout, and the length-sorted group plan of the batched kernel.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "rp_host.h"
#include "rp_launch.h"
#include "rp_layout.h"

namespace rpx {

namespace {
float4 f4(double a, double b, double c, double d = 0.0) {
    return make_float4(float(a), float(b), float(c), float(d));
}
}  // namespace

bool deviceUsable(std::string* why) {
    int n = 0;
    const cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n == 0) {
        if (why) {
            int rt = 0, dr = 0;
            cudaRuntimeGetVersion(&rt);
            cudaDriverGetVersion(&dr);
            *why = std::string("no usable CUDA device: error ") + std::to_string(int(e)) + " (" +
                   cudaGetErrorString(e) + "); runtime CUDA " + std::to_string(rt / 1000) + "." +
                   std::to_string((rt % 1000) / 10) + ", driver supports CUDA " +
                   std::to_string(dr / 1000) + "." + std::to_string((dr % 1000) / 10);
        }
        cudaGetLastError();
        return false;
    }
    return true;
}

size_t optinSmem(int device) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess) {
        cudaGetLastError();
        return 48 * 1024;
    }
    return size_t(v);
}

rp::DPrim toDPrim(const rp_primitive& p) {
    rp::DPrim d{};
    d.ax = float(p.a[0]);
    d.ay = float(p.a[1]);
    d.az = float(p.a[2]);
    d.radius = float(p.radius);
    d.bx = float(p.b[0]);
    d.by = float(p.b[1]);
    d.bz = float(p.b[2]);
    d.friction = float(p.friction);
    d.nx = float(p.normal[0]);
    d.ny = float(p.normal[1]);
    d.nz = float(p.normal[2]);
    d.typef = float(p.type);
    d.hx = float(p.half_extents[0]);
    d.hy = float(p.half_extents[1]);
    d.hz = float(p.half_extents[2]);
    d.qw = float(p.rotation[0]);
    d.qx = float(p.rotation[1]);
    d.qy = float(p.rotation[2]);
    d.qz = float(p.rotation[3]);
    return d;
}

std::string validateWorld(const rp_world& w) {
    if (w.num_primitives < 0 || (w.num_primitives > 0 && !w.primitives))
        return "world has primitives but a NULL array";
    if (w.num_primitives > 64) return "at most 64 primitives per world";
    for (int k = 0; k < w.num_primitives; ++k) {
        const rp_primitive& p = w.primitives[k];
        if (p.type < 0 || p.type > 3) return "primitive type must be 0..3";
        if ((p.type == 1 || p.type == 2) && !(p.radius >= 0)) return "negative primitive radius";
    }
    if (w.self_collision && (w.hash_table_size < 1 || w.hash_table_size > (1 << 20)))
        return "self-collision needs 1 <= hash_table_size <= 2^20";
    return "";
}

// Chain topology: stretch k = (k, k+1, frame k); bends 0..nSt-2 = (k, k+1);
// any further bends involve a ghost frame (index >= nSt).
int isChain(const rp_rod_desc* d) {
    if (d->num_particles != d->num_stretch + 1) return 0;
    for (int k = 0; k < d->num_stretch; ++k)
        if (d->s_p0[k] != k || d->s_p1[k] != k + 1 || d->s_seg[k] != k) return 0;
    if (d->num_bend < d->num_stretch - 1) return 0;
    for (int k = 0; k < d->num_stretch - 1; ++k)
        if (d->b_a[k] != k || d->b_b[k] != k + 1) return 0;
    for (int k = d->num_stretch - 1; k < d->num_bend; ++k)
        if (d->b_a[k] < d->num_stretch && d->b_b[k] < d->num_stretch) return 0;
    return 1;
}

void packParticles(const rp_rod_desc* d, float4* x, float4* v, float4* f, float4* k) {
    for (int i = 0; i < d->num_particles; ++i) {
        if (x) x[i] = f4(d->x[3 * i], d->x[3 * i + 1], d->x[3 * i + 2]);
        if (v) v[i] = d->v ? f4(d->v[3 * i], d->v[3 * i + 1], d->v[3 * i + 2]) : f4(0, 0, 0);
        if (f)
            f[i] = d->ext_force ? f4(d->ext_force[3 * i], d->ext_force[3 * i + 1], d->ext_force[3 * i + 2])
                                : f4(0, 0, 0);
        if (k)
            k[i] = d->kin_velocity
                       ? f4(d->kin_velocity[3 * i], d->kin_velocity[3 * i + 1], d->kin_velocity[3 * i + 2])
                       : f4(0, 0, 0);
    }
}

void packFrames(const rp_rod_desc* d, float4* q, float4* w, float4* t) {
    for (int j = 0; j < d->num_frames; ++j) {
        if (q) q[j] = f4(d->q[4 * j], d->q[4 * j + 1], d->q[4 * j + 2], d->q[4 * j + 3]);
        if (w) w[j] = d->omega ? f4(d->omega[3 * j], d->omega[3 * j + 1], d->omega[3 * j + 2]) : f4(0, 0, 0);
        if (t)
            t[j] = d->ext_torque ? f4(d->ext_torque[3 * j], d->ext_torque[3 * j + 1], d->ext_torque[3 * j + 2])
                                 : f4(0, 0, 0);
    }
}

// One rod shape's static device data (reference gpu_batch.cpp:193-230 converts
// the same quantities to float): masses, inertias, constraint topology and
// rest data, colour orders. Offsets in T are relative to this template.
void makeTemplate(const rp_rod_desc* d, TemplateHost& h) {
    rp::DTemplate& T = h.T;
    T = rp::DTemplate{};
    T.nP = d->num_particles;
    T.nS = d->num_frames;
    T.nSt = d->num_stretch;
    T.nB = d->num_bend;
    h.invMass.resize(T.nP);
    for (int i = 0; i < T.nP; ++i) h.invMass[i] = float(d->inv_mass[i]);
    h.invInertia.resize(T.nS);
    h.inertia.resize(T.nS);
    h.fixed.assign(T.nS, 0);
    for (int j = 0; j < T.nS; ++j) {
        const double* iI = d->inv_inertia + 3 * j;
        h.invInertia[j] = f4(iI[0], iI[1], iI[2]);
        h.inertia[j] = f4(d->inertia[3 * j], d->inertia[3 * j + 1], d->inertia[3 * j + 2]);
        h.fixed[j] = (iI[0] * iI[0] + iI[1] * iI[1] + iI[2] * iI[2]) == 0.0;
    }
    h.sP0.assign(d->s_p0, d->s_p0 + T.nSt);
    h.sP1.assign(d->s_p1, d->s_p1 + T.nSt);
    h.sSeg.assign(d->s_seg, d->s_seg + T.nSt);
    h.sComp.resize(T.nSt);
    for (int k = 0; k < T.nSt; ++k)
        h.sComp[k] = f4(d->s_compliance[3 * k], d->s_compliance[3 * k + 1], d->s_compliance[3 * k + 2],
                        d->s_rest[k]);
    h.bA.assign(d->b_a, d->b_a + T.nB);
    h.bB.assign(d->b_b, d->b_b + T.nB);
    h.bComp.resize(T.nB);
    h.bRestD.resize(T.nB);
    for (int k = 0; k < T.nB; ++k) {
        h.bComp[k] = f4(d->b_compliance[3 * k], d->b_compliance[3 * k + 1], d->b_compliance[3 * k + 2],
                        d->b_rest[k]);
        h.bRestD[k] = f4(d->b_rest_darboux[3 * k], d->b_rest_darboux[3 * k + 1], d->b_rest_darboux[3 * k + 2]);
    }
    std::vector<int> order, cs;
    h.order.clear();
    h.colorStart.clear();
    T.sColors = colorRod(d, false, order, cs);
    T.sOrderOff = 0;
    T.sColorOff = 0;
    h.order.insert(h.order.end(), order.begin(), order.end());
    h.colorStart.insert(h.colorStart.end(), cs.begin(), cs.end());
    T.bColors = colorRod(d, true, order, cs);
    T.bOrderOff = int(h.order.size());
    T.bColorOff = int(h.colorStart.size());
    h.order.insert(h.order.end(), order.begin(), order.end());
    h.colorStart.insert(h.colorStart.end(), cs.begin(), cs.end());
    T.chain = isChain(d);
    // two colours holding the even and the odd constraints in ascending order:
    // the kernel can then compute a constraint's index instead of loading it
    auto evenOdd = [](const std::vector<int>& ord, const std::vector<int>& starts, int n) {
        const int half = (n + 1) / 2;
        if (n < 2 || starts.size() != 3 || starts[0] != 0 || starts[1] != half || starts[2] != n) return false;
        for (int i = 0; i < n; ++i)
            if (ord[i] != (i < half ? 2 * i : 2 * (i - half) + 1)) return false;
        return true;
    };
    T.evenOdd = (evenOdd(std::vector<int>(h.order.begin(), h.order.begin() + d->num_stretch),
                         std::vector<int>(h.colorStart.begin(), h.colorStart.begin() + T.sColors + 1),
                         d->num_stretch)
                     ? 1
                     : 0) |
                (evenOdd(std::vector<int>(h.order.begin() + T.bOrderOff, h.order.end()),
                         std::vector<int>(h.colorStart.begin() + T.bColorOff, h.colorStart.end()), d->num_bend)
                     ? 2
                     : 0);
    auto same = [](const std::vector<float4>& v) {
        for (const float4& a : v)
            if (std::memcmp(&a, &v[0], sizeof(float4)) != 0) return false;
        return true;
    };
    if (same(h.invInertia) && same(h.inertia) && same(h.sComp) && same(h.bComp) && same(h.bRestD)) T.evenOdd |= 4;
}

namespace {

constexpr size_t kMisaligned = ~size_t(0);
constexpr int kNoWide = INT32_MAX;

// Threads of a rod's team: about one per two segments (a colour's constraints
// one to a lane), whole warps, 32..256. A rod longer than `wideFrom` gets about one
// per segment instead, a power of two, for launches that leave room (see
// planBatched): up to 512 where a lane still has more than one constraint of a
// colour or a self-contact count to share, else up to 256 (512 segments without
// self-collision: 152 us a step with 256 threads, 166 with 512).
int teamThreads(int nSt, bool self, int pairsPerThread, int wideFrom) {
    if (nSt > wideFrom) {
        const int most = self || nSt > 512 ? 512 : 256;
        int t = 32;
        while (t < most && 2 * nSt > 3 * t) t *= 2;
        return t;
    }
    int t = (nSt / 2 + pairsPerThread - 1) / pairsPerThread;
    t = (t + 31) / 32 * 32;
    return std::max(32, std::min(256, t));
}

// Length-sorted groups for the batched kernel (kMisaligned if a rod's layout
// would break the 16-byte alignment its rows and bulk copies need: refused
// on the host, never launched). `order` receives the rod ids
// longest first (stable), `groups` four ints per group: first index into
// `order`, rod count, team size, shared bytes. A group ends before the rod that
// would take it past `room` bytes. Returns the largest group's shared bytes.
size_t planGroups(const std::vector<int32_t>& rodIds, const rp::DRod* rods, const rp::DTemplate* tmpls,
                  int cta, int pairsPerThread, int wideFrom, bool comp, bool slotsShared, size_t room,
                  std::vector<int32_t>& order, std::vector<int32_t>& groups) {
    order = rodIds;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
        return tmpls[rods[x].tmpl].nSt > tmpls[rods[y].tmpl].nSt;
    });
    auto teamOf = [&](int r) {
        return std::min(cta, teamThreads(tmpls[rods[r].tmpl].nSt, rods[r].selfCollision != 0, pairsPerThread, wideFrom));
    };
    groups.clear();
    size_t maxSmem = 0;
    const int n = int(order.size());
    int i = 0;
    while (i < n) {
        const int team = teamOf(order[i]);
        const int perCta = std::min(8, cta / team);
        int cnt = 0;
        size_t smem = 0;
        while (i + cnt < n && cnt < perCta) {
            const rp::DRod& R = rods[order[i + cnt]];
            const rp::DTemplate& T = tmpls[R.tmpl];
            if (teamOf(order[i + cnt]) != team) break;
            const rp::RodLayout L = rp::rodLayout(T.nP, T.nS, T.nSt, T.nB, R.numPrims, R.selfCollision,
                                                  R.hashTableSize, R.selfCapacity, 1, comp ? 1 : 0,
                                                  slotsShared ? 1 : 0);
            if (!rp::rodLayoutAligned(L)) return kMisaligned;
            if (cnt > 0 && smem + size_t(L.bytes) > room) break;
            smem += size_t(L.bytes);
            ++cnt;
        }
        groups.push_back(i);
        groups.push_back(cnt);
        groups.push_back(team);
        groups.push_back(int32_t(smem));
        maxSmem = std::max(maxSmem, smem);
        i += cnt;
    }
    return maxSmem;
}

// Shared memory of a CTA if an SM is to hold `ctas` of them.
size_t smemPerCta(int device, int ctas) {
    int sm = 0, reserved = 0;
    if (cudaDeviceGetAttribute(&sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, device) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return size_t(std::max(0, sm / ctas - reserved));
}

// One launch shape: its groups, its shared memory, and how many of its CTAs
// an SM holds.
rp_status planShape(const std::vector<int32_t>& rodIds, const rp::DRod* rods, const rp::DTemplate* tmpls, int cta,
                    int pairsPerThread, int wideFrom, int precision, int device, bool mayShareSlots,
                    BatchedShape& out, int* perSm) {
    const size_t optin = optinSmem(device);
    const bool comp = (precision & RP_PRECISION_COMPENSATED) != 0;
    const size_t fixed = rp::batchedStaticSmem() + 64;  // the kernel's own shared memory
    out.cta = cta;
    out.slotsShared = 0;
    const size_t room = fixed < optin ? optin - fixed : 0;
    out.smem = planGroups(rodIds, rods, tmpls, cta, pairsPerThread, wideFrom, comp, false, room, out.order, out.groups);
    if (out.smem == kMisaligned)
        return fail(RP_ERR_INVALID, "internal: a rod's shared-memory layout is not 16-byte aligned");
    // World contact slots go into shared memory when the groups still fit as
    // many CTAs per SM with them (few contact primitives per rod, or short
    // rods); otherwise they stay in global memory. Where only the teams' contexts
    // take them past that, the groups give up a rod and keep the slots: 4096 rods
    // of 60 lying on their primitives (five a rod), 20 substeps, take 906 us with
    // eight to a CTA and the slots in global memory and 519 with seven. Far from
    // the primitives, where no slot is touched, it is 281 and 290 (2100 rods of
    // 61, a last wave more: 149 and 240).
    if (mayShareSlots) {
        std::vector<int32_t> order2, groups2;
        size_t smem2 = planGroups(rodIds, rods, tmpls, cta, pairsPerThread, wideFrom, comp, true, SIZE_MAX, order2,
                                  groups2);
        auto ctas = [&](size_t smem) {  // an SM holds
            int n = 0;
            if (smem + fixed > optin || rp::batchedReserveSmem(std::max<size_t>(smem, 1)) != cudaSuccess ||
                rp::batchedOccupancy(cta, smem, precision, out.anySelf, &n) != cudaSuccess)
                n = 0;
            cudaGetLastError();
            return n;
        };
        const int most = smem2 == kMisaligned ? 0 : ctas(out.smem);
        if (most >= 1 && ctas(smem2) < most) {
            size_t bare = 0;  // the largest group without its contexts
            for (size_t g = 0; g < groups2.size(); g += 4)
                bare = std::max(bare, size_t(groups2[g + 3]) - size_t(groups2[g + 1]) * rp::kContextBytes);
            const size_t each = smemPerCta(device, most);
            const size_t room2 = std::min(room, each > fixed ? each - fixed : 0);
            if (bare <= room2)
                smem2 = planGroups(rodIds, rods, tmpls, cta, pairsPerThread, wideFrom, comp, true, room2, order2,
                                   groups2);
        }
        if (most >= 1 && ctas(smem2) >= most) {
            out.smem = smem2;
            out.order.swap(order2);
            out.groups.swap(groups2);
            out.slotsShared = 1;
        }
    }
    if (out.smem + fixed > optin)
        return fail(RP_ERR_SHARED_MEMORY, "a rod group needs " + std::to_string(out.smem) +
                                              " bytes of shared memory; the device allows " +
                                              std::to_string(optin));
    if (rp::batchedReserveSmem(std::max<size_t>(out.smem, 1)) != cudaSuccess) {
        cudaGetLastError();
        return fail(RP_ERR_SHARED_MEMORY, "cannot opt into the batched shared memory");
    }
    if (rp::batchedOccupancy(cta, out.smem, precision, out.anySelf, perSm) != cudaSuccess || *perSm < 1) {
        cudaGetLastError();
        return fail(RP_ERR_SHARED_MEMORY, "batched kernel cannot be resident with this group size");
    }
    return RP_OK;
}

}  // namespace

// The launch of the batched kernel over `rodIds` with the asked CTA size and
// segment pairs per thread, or, with `mayWiden` (nobody asked for a shape), with
// wide teams where the launch leaves room for them.
//
// The default shape (256 threads, one pair per thread) gives a rod the threads
// its constraint colours need, which is best while the GPU is full. With fewer
// rods the step takes as long as its slowest rod, and the phases with one
// item per segment or more (prediction, contacts, the self-contact count) gain
// from twice the team. So as many of the longest rods as still leave every group
// of the launch resident at once, on half the GPU's threads, get about one
// thread per segment: all of them if that fits, else those longer than 64,
// 128, ... 448 segments. Beyond half, a batch alone still gains a little, but
// batches on other streams are kept out of the SMs (three batches of 296 rods of
// 200, 20 substeps: 93 us a step each against 130).
//
// Measured on a B200, 20 substeps, one batch alone (three at once, a step
// each): one rod of 64 126 -> 118 us (51 -> 44), 64 of 128 148 -> 124 (61 -> 52),
// 16 of 900 295 -> 222 (112 -> 84), 64 settled rods of 40-200 with
// self-collision 1271 -> 968 (447 -> 355).
rp_status planBatched(const std::vector<int32_t>& rodIds, const rp::DRod* rods, const rp::DTemplate* tmpls, int cta,
                      int pairsPerThread, bool mayWiden, int precision, int device, bool mayShareSlots,
                      BatchedShape& out) {
    int sms = 0, perSm = 0;
    out.anySelf = out.wide = false;
    for (int32_t r : rodIds) out.anySelf = out.anySelf || rods[r].selfCollision != 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (mayWiden) {
        int longest = 0;
        for (int32_t r : rodIds) longest = std::max(longest, tmpls[rods[r].tmpl].nSt);
        for (int wideFrom = 0; wideFrom < std::min(longest, 449); wideFrom += 64) {
            int64_t threads = 0;
            int most = 128;
            for (int32_t r : rodIds) {
                const int team = teamThreads(tmpls[rods[r].tmpl].nSt, rods[r].selfCollision != 0, 1, wideFrom);
                threads += team;
                most = std::max(most, team);
            }
            if (threads > int64_t(sms) * 256) continue;
            const int wideCta = most <= 128 ? 128 : most <= 256 ? 256 : 512;
            if (planShape(rodIds, rods, tmpls, wideCta, 1, wideFrom, precision, device, mayShareSlots, out, &perSm) ==
                    RP_OK &&
                int(out.groups.size() / 4) <= sms * perSm) {
                out.blocks = std::max(1, int(out.groups.size() / 4));
                out.wide = true;
                return RP_OK;
            }
        }
    }
    const rp_status st = planShape(rodIds, rods, tmpls, cta, pairsPerThread, kNoWide, precision, device, mayShareSlots,
                                   out, &perSm);
    if (st == RP_OK) out.blocks = std::max(1, std::min(int(out.groups.size() / 4), sms * perSm));
    return st;
}

}  // namespace rpx
