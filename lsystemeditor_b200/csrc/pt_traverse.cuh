// Traversal of a queue of rays by whole warps (closest hit or any hit; flat
// scenes, or the two-level BVH of instanced ones).
//
// Every lane owns one ray; the warp steps together:
//   fetch   when at least kFetchLanes lanes are idle they take the next
//           entries of the warp's chunk of the queue (one atomic per chunk);
//   node    every lane that has no triangles to test intersects the eight
//           children of its next node;
//   round   the (ray, triangle) pairs that the lanes hold are dealt out to
//           the lanes, 32 at a time: a lane tests whichever pair it gets, with
//           the owner's ray from shared memory, and the closest hit of each
//           owner is settled by a 64-bit minimum over (t, ~triangle id).  A
//           round runs when the pairs fill at least kRoundPairs lanes, or no
//           lane can do a node step.  Lanes with pairs left wait, so a ray
//           tests a node's triangles before its next node, as traceRay does.
//   pop     lanes without work take the next group from their stack, or finish;
//   steal   (flat scenes) once the queue is drained, idle lanes take the oldest
//           stack entry of busy lanes and traverse that part of their ray, so
//           that a launch does not wait for one lane's long ray.
//
// The hits do not depend on which parts are stolen when.  A ray in one piece
// visits its nodes in one order.  A ray in several culls by whatever its parts
// have found so far, and that changes its hit only where another hit, a rival,
// would cull the closest one's box: where the rival lies before the entry into
// that box, give or take the rounding of box and triangle tests (hitSlack).  So a
// split ray culls two slacks beyond its closest hit, which keeps every rival in
// sight, and one whose closest hit has such a rival is traced again in one piece.
// (A hit found before the ray was split has none; a shadow ray is settled by any
// hit below a fixed tMax.)  Without the second trace, 12 of 60 scenes of
// overlapping coplanar rectangles rendered differently from run to run, in up to
// 3% of their pixels.  Few rays need it (8 of the 403M of the large frame below,
// 159 of the 4.9M of a 256^2 frame of 20k triangles whose tubes share their ends:
// 1.13 -> 1.16 ms; 1024^2 waves 6.42 -> 6.54; the other timed frames within 0.5%).
//
// Why: in a free-running loop (a lane fetched and stepped on its own) 6 of 32
// lanes worked per executed instruction, a node's triangles were tested one
// after the other, and every finished ray was an atomic on one address.  It is
// bound by issue and by the latency of the node and triangle loads (20 of 32
// lanes, 64 - 68% of the issue slots, the ALU pipe at 53 - 59%; DRAM idles, the
// scene is in L2).  Registers matter more than warps: with spills at 64 registers
// it lost a quarter, so the per-ray words that only the ends of a ray need are in
// shared memory, and the closest-hit kernel leaves rays of quirk Q1 to k_route
// (the call costs it registers; the shadow kernel traces its own).
// Measured: closest hit of the large frame (972k triangles, 403M rays) 163 ->
// 79 ms (88 without stealing), of one 1024^2 wave (1.6M rays over 8 launches) 1.86
// -> 0.78 ms (1.33 without stealing: the launches of late bounces wait for their
// longest ray), shadow rays of a 513x511 32-spp emitter-MIS frame 3.73 -> 2.0 ms
// (2.45 without stealing).
#pragma once

#include "pt_trace.cuh"

#include <type_traits>

namespace pt {

#ifndef PT_TRACE_STACK
#define PT_TRACE_STACK 16
#endif
#ifndef PT_FETCH_LANES
#define PT_FETCH_LANES 8
#endif
#ifndef PT_ROUND_PAIRS
#define PT_ROUND_PAIRS 16
#endif
#ifndef PT_TRACE_CHUNK
// (smaller: the atomics, on one address, cost more; larger: warps end a launch
// apart; 1M camera rays 362 us at 128, 223 at 32)
#define PT_TRACE_CHUNK 32
#endif
constexpr int kTraceThreads = 128;
constexpr int kTraceStack = PT_TRACE_STACK;       // stack entries per lane in shared memory (the rest is local)
constexpr int kFetchLanes = PT_FETCH_LANES;
constexpr int kRoundPairs = PT_ROUND_PAIRS;
constexpr unsigned int kTraceChunk = PT_TRACE_CHUNK;

// A ray: its scene, origin, normalised direction and the parametric interval it is tested on.
struct LaneRay {
    const DevScene* S;
    float3 o;
    float3 dn;
    float tMin;
    float tMax;
};

struct TraceInstPart {
    float4 wo[32];    // world ray (o / d below are the object's while inside one)
    float4 wd[32];
    uint2 cur[32];    // instance being traversed, first shading record of its object
};
struct TraceFlatPart {
    float tMax[32];         // closest-hit rays
    // of a split ray
    unsigned int rival[32]; // bits of the smallest t of the hits behind the closest
    float entry[32];        // latest t at which it may enter the box of its closest hit; -1: found in order
};

// A warp's shared memory.
template <bool Inst> struct WarpTrace {
    float4 o[32];                 // ray origin, tMin
    float4 d[32];                 // ray direction; hitSlack once the ray is split, -0: not to be split again
    float4 res[32];               // u, v, triangle, instance of the best hit so far
    uint2 entry[32];              // queue entry, caller's word
    unsigned int lanes[32];       // lanes that traverse this ray
    unsigned long long key[32];   // closest t << 32 | ~(id of that hit); see warpTraversal
    uint2 stack[kTraceStack][32];
    uint2 give[32];               // stack entries handed to idle lanes
    uint16_t pair[32];            // owner lane | its ray << 5 | triangle bit << 10
    std::conditional_t<Inst, TraceInstPart, TraceFlatPart> in;
};

// The latest t at which a ray may enter a triangle's bounding box: per axis the
// near plane and its share of the slack.
__device__ __forceinline__ float boxEntry(float3 o, float3 d, const TriVerts& tv, float slack)
{
    const float3 r = f3(__fdividef(1.0f, d.x), __fdividef(1.0f, d.y), __fdividef(1.0f, d.z));
    const float unit = slack / fminf(fmaxf(fmaxf(fabsf(r.x), fabsf(r.y)), fabsf(r.z)), 65536.0f);
    auto axis = [unit](float a, float b, float c, float oo, float rr) {
        const float near = rr < 0.0f ? fmaxf(fmaxf(a, b), c) : fminf(fminf(a, b), c);
        return fmaf(unit, fabsf(rr), (near - oo) * rr);
    };
    return fmaxf(fmaxf(axis(tv.v0.x, tv.v1.x, tv.v2.x, o.x, r.x), axis(tv.v0.y, tv.v1.y, tv.v2.y, o.y, r.y)),
        axis(tv.v0.z, tv.v1.z, tv.v2.z, o.z, r.z));
}

//   load(k, ray, word) -> bool: reads queue entry k (word: kept for finish);
//     false when the entry was decided without the wide traversal.
//   finish(k, word, hit, t, u, v, tri, inst): the result of entry k (for AnyHit,
//     hit means occluded and the rest is unset).
// Multi: rays of several scenes (their node and triangle arrays differ per lane).
// Ties: of several hits at exactly the same t the highest original triangle id
// wins (instanced: the highest (instance, triangle)), as in traceRay.
template <bool AnyHit, bool Inst, bool Multi, class Load, class Finish>
__device__ __forceinline__ void warpTraversal(const DevScene& S0, unsigned int count, unsigned int* fetch,
    WarpTrace<Inst>& W, unsigned int* overflowCounter, Load load, Finish finish)
{
    constexpr unsigned int kAll = 0xFFFFFFFFu;
    constexpr bool kPerRay = Inst || Multi;
    constexpr bool kRivals = !AnyHit && !Inst;
    const unsigned int lane = threadIdx.x & 31u;
    const unsigned int below = (1u << lane) - 1u;
    uint2 spill[kTraversalStack];
    bool active = false, overflow = false;
    unsigned int ray = lane; // the ray (index into W) that this lane traverses
    float3 o = f3(0.0f, 0.0f, 0.0f), idir = o;
    float tMin = 0.0f, cull = 0.0f; // cull: closest hit so far (split ray: and two slacks)
    uint32_t octinv = 0;
    uint2 ngroup = make_uint2(0u, 0u), tgroup = make_uint2(0u, 0u);
    int sp = 0, sb = 0; // stack entries sb .. sp - 1
    const DevScene* S = &S0;
    const CwNode* nodes = Inst ? nullptr : S0.nodes;
    const TriVerts* tris = Inst ? nullptr : S0.tris;
    int level = 0, base = 0;
    // the warp's chunk of the queue; small queues are spread over all warps
    // (a warp's first chunk is its own; the counter hands out those behind them)
    const unsigned int warps = gridDim.x * (kTraceThreads / 32);
    const unsigned int chunk = min(kTraceChunk, max(1u, count / (warps * 2u)));
    unsigned int poolNext = (blockIdx.x * (kTraceThreads / 32) + (threadIdx.x >> 5)) * chunk;
    unsigned int poolEnd = min(poolNext + chunk, count);

    auto push = [&](uint2 g) -> bool {
        if (sp < kTraceStack) {
            W.stack[sp][lane] = g;
        } else if (sp < kTraceStack + kTraversalStack) {
            spill[sp - kTraceStack] = g;
        } else {
            return false;
        }
        ++sp;
        return true;
    };
    auto setRay = [&](float3 a, float3 d) {
        o = a;
        if constexpr (Inst) {
            d.x = fabsf(d.x) < 1.0e-20f ? copysignf(1.0e-20f, d.x) : d.x;
            d.y = fabsf(d.y) < 1.0e-20f ? copysignf(1.0e-20f, d.y) : d.y;
            d.z = fabsf(d.z) < 1.0e-20f ? copysignf(1.0e-20f, d.z) : d.z;
        }
        idir = f3(__frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z));
        octinv = 7u - ((d.x < 0.0f ? 4u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 1u : 0u));
    };
    // every slot's octant of the root group: only slot 0 exists
    auto rootGroup = [&]() { return make_uint2(0u, 0x80000000u | (1u << (7u - octinv))); };
    auto keyT = [&](unsigned int r) { return __uint_as_float(static_cast<uint32_t>(W.key[r] >> 32)); };
    // The loop is compiled twice: while the queue lasts, and once it is drained
    // (with one loop for both, the split rays' words cost the first 2%).
    auto run = [&](auto phase) {
        constexpr bool kDrained = decltype(phase)::value;
        for (;;) {
            const unsigned int idle = __ballot_sync(kAll, !active);
            if (!kDrained && __popc(idle) >= kFetchLanes) {
                if (poolNext >= poolEnd) {
                    unsigned int b = 0;
                    if (lane == 0) {
                        b = atomicAdd(fetch, chunk);
                    }
                    poolNext = __shfl_sync(kAll, b, 0) + warps * chunk;
                    poolEnd = min(poolNext + chunk, count);
                    if (poolNext >= count) {
                        return;
                    }
                }
                {
                    const unsigned int n = min(static_cast<unsigned int>(__popc(idle)), poolEnd - poolNext);
                    const unsigned int r = __popc(idle & below);
                    if (!active && r < n) {
                        const unsigned int k = poolNext + r;
                        LaneRay q;
                        uint32_t word = 0;
                        if (load(k, q, word)) {
                            W.entry[lane] = make_uint2(k, word);
                            W.lanes[lane] = 1u;
                            W.o[lane] = make_float4(q.o.x, q.o.y, q.o.z, q.tMin);
                            W.d[lane] = make_float4(q.dn.x, q.dn.y, q.dn.z, 0.0f);
                            if constexpr (Inst) {
                                W.in.wo[lane] = make_float4(q.o.x, q.o.y, q.o.z, 0.0f);
                                W.in.wd[lane] = make_float4(q.dn.x, q.dn.y, q.dn.z, 0.0f);
                            }
                            // (low word 0: a hit at exactly tMax does not count)
                            W.key[lane] = static_cast<unsigned long long>(__float_as_uint(q.tMax)) << 32;
                            W.res[lane] =
                                make_float4(0.0f, 0.0f, __uint_as_float(0xFFFFFFFFu), __uint_as_float(0xFFFFFFFFu));
                            setRay(q.o, q.dn);
                            tMin = q.tMin;
                            cull = q.tMax;
                            if constexpr (kRivals) {
                                W.in.tMax[lane] = q.tMax;
                            }
                            if constexpr (kPerRay) {
                                S = q.S;
                                // (a flat scene of an instanced batch starts inside its only object)
                                const bool flat = !Inst || S->instanceCount == 0;
                                nodes = flat ? S->nodes : S->tlasNodes;
                                tris = flat ? S->tris : S->tlasLeaves;
                                if constexpr (Inst) {
                                    W.in.cur[lane] = make_uint2(0xFFFFFFFFu, 0u);
                                    level = flat ? 1 : 0;
                                    base = 0;
                                }
                            }
                            sp = sb = 0;
                            ngroup = rootGroup();
                            tgroup = make_uint2(0u, 0u);
                            active = true;
                        }
                    }
                    poolNext += n;
                }
            }
            if constexpr (kDrained) {
                if (idle == kAll) {
                    return;
                }
                if constexpr (!Inst) {
                    const bool gives = active && sp > sb && sb < kTraceStack &&
                        (!kRivals || __float_as_uint(W.d[ray].w) != 0x80000000u);
                    const unsigned int victims = __ballot_sync(kAll, gives);
                    if (idle != 0u && victims != 0u) {
                        const unsigned int n = min(__popc(idle), __popc(victims));
                        const unsigned int r = __popc((active ? victims : idle) & below);
                        if (gives && r < n) {
                            W.pair[r] = static_cast<uint16_t>(lane | (ray << 5));
                            W.give[r] = W.stack[sb][lane];
                            ++sb;
                            atomicAdd(&W.lanes[ray], 1u);
                            if constexpr (kRivals) {
                                const float slack = hitSlack(nodes, o, idir); // (the same for every lane of the ray)
                                if (W.d[ray].w == 0.0f) { // (a ray in one piece has one lane)
                                    W.d[ray].w = slack;
                                    W.in.rival[ray] = 0x7F800000u;
                                    W.in.entry[ray] = -1.0f;
                                }
                                cull = fmaf(2.0f, slack, keyT(ray));
                            }
                        }
                        __syncwarp();
                        const bool takes = !active && r < n;
                        const unsigned int p = takes ? W.pair[r] : lane;
                        if constexpr (Multi) {
                            const unsigned long long np =
                                __shfl_sync(kAll, reinterpret_cast<unsigned long long>(nodes), p & 31u);
                            const unsigned long long tp =
                                __shfl_sync(kAll, reinterpret_cast<unsigned long long>(tris), p & 31u);
                            if (takes) {
                                nodes = reinterpret_cast<const CwNode*>(np);
                                tris = reinterpret_cast<const TriVerts*>(tp);
                            }
                        }
                        if (takes) {
                            ray = p >> 5;
                            const float4 ro = W.o[ray], rd = W.d[ray];
                            setRay(f3(ro.x, ro.y, ro.z), f3(rd.x, rd.y, rd.z));
                            tMin = ro.w;
                            cull = fmaf(2.0f, rd.w, keyT(ray));
                            ngroup = W.give[r];
                            tgroup = make_uint2(0u, 0u);
                            sp = sb = 0;
                            active = true;
                        }
                        __syncwarp(); // the pair list is rewritten by the triangle round
                    }
                }
            }
            // --- node step (lanes whose triangles are all tested) ---
            if (active && tgroup.y == 0u && (!Inst || ngroup.y > 0x00FFFFFFu)) {
                const uint32_t bit = 31u - __clz(ngroup.y);
                ngroup.y &= ~(1u << bit);
                const uint32_t slot = (bit - 24u) ^ octinv;
                const uint32_t child = ngroup.x + __popc(ngroup.y & 0xffu & ((1u << slot) - 1u));
                if (ngroup.y > 0x00FFFFFFu && !push(ngroup)) {
                    overflow = true;
                }
                uint32_t childBase, triBase, imask;
                const uint32_t hits =
                    intersectChildren(nodes, child, o, idir, octinv, tMin, cull, childBase, triBase, imask);
                ngroup = make_uint2(childBase, (hits & 0xFF000000u) | imask);
                tgroup = make_uint2(triBase, hits & 0x00FFFFFFu);
            }
            if constexpr (Inst) {
                if (level == 0 && tgroup.y != 0u) {
                    // an instance: descend into its object
                    const int kt = __ffs(tgroup.y) - 1;
                    tgroup.y &= tgroup.y - 1u;
                    const uint32_t inst = __float_as_uint(__ldg(&tris[tgroup.x + kt].v0.w));
                    bool saved = true;
                    if (ngroup.y > 0x00FFFFFFu) {
                        saved = push(ngroup);
                    }
                    if (saved && tgroup.y != 0u) {
                        saved = push(tgroup);
                    }
                    if (!saved) {
                        overflow = true; // the rest of this top-level group is dropped
                    }
                    const DevInstance& I = S->instances[inst];
                    const DevBlas B = S->blases[I.meta.x];
                    nodes = B.nodes;
                    tris = B.tris;
                    const float4 wo = W.in.wo[lane], wd = W.in.wd[lane];
                    const float3 od = xformVector(I.w2o, f3(wd.x, wd.y, wd.z));
                    setRay(xformPoint(I.w2o, f3(wo.x, wo.y, wo.z)), od);
                    W.o[lane] = make_float4(o.x, o.y, o.z, tMin);
                    W.d[lane] = make_float4(od.x, od.y, od.z, 0.0f);
                    W.in.cur[lane] = make_uint2(inst, B.triBase);
                    if constexpr (!AnyHit) {
                        // at an exact tie this instance's triangles win or lose as a whole
                        // (an instance is a single top-level leaf)
                        const uint32_t bi = __float_as_uint(W.res[lane].w);
                        const bool wins = bi != 0xFFFFFFFFu && inst > bi;
                        W.key[lane] = (static_cast<unsigned long long>(__float_as_uint(cull)) << 32) |
                            (wins ? 0xFFFFFFFFull : 0ull);
                    }
                    level = 1;
                    base = sp;
                    ngroup = B.nodeCount > 0 ? rootGroup() : make_uint2(0u, 0u);
                    tgroup = make_uint2(0u, 0u);
                }
            }
            // --- triangle round ---
            {
                const unsigned int c = min(__popc(tgroup.y), 7);
                const unsigned int b0 = __ballot_sync(kAll, (c & 1u) != 0u);
                const unsigned int b1 = __ballot_sync(kAll, (c & 2u) != 0u);
                const unsigned int b2 = __ballot_sync(kAll, (c & 4u) != 0u);
                const int total = __popc(b0) + 2 * __popc(b1) + 4 * __popc(b2);
                const bool canStep = active && tgroup.y == 0u;
                if (total >= kRoundPairs || (total > 0 && !__any_sync(kAll, canStep))) {
                    const unsigned int off = __popc(b0 & below) + 2 * __popc(b1 & below) + 4 * __popc(b2 & below);
                    const unsigned int end = min(off + c, 32u);
                    for (unsigned int j = off; j < end; ++j) {
                        const unsigned int kt = __ffs(tgroup.y) - 1;
                        tgroup.y &= tgroup.y - 1u;
                        W.pair[j] = static_cast<uint16_t>(lane | (ray << 5) | (kt << 10));
                    }
                    __syncwarp();
                    const bool mine = static_cast<int>(lane) < total;
                    const unsigned int p = mine ? W.pair[lane] : lane;
                    const unsigned int owner = p & 31u, oray = (p >> 5) & 31u;
                    const uint32_t tb = __shfl_sync(kAll, tgroup.x, owner);
                    const TriVerts* tp = tris;
                    if constexpr (kPerRay) {
                        tp = reinterpret_cast<const TriVerts*>(
                            __shfl_sync(kAll, reinterpret_cast<unsigned long long>(tris), owner));
                    }
                    bool hit = false;
                    float t = 0.0f, u = 0.0f, v = 0.0f, entry = -1.0f;
                    uint32_t id = 0;
                    unsigned long long nk = 0;
                    if (mine) {
                        const TriVerts tv = tp[tb + (p >> 10)];
                        const float4 ro = W.o[oray], rd = W.d[oray];
                        const float cl = keyT(oray);
                        // (rd.w: a split ray's rivals behind its closest hit count as hits; they do not change the key)
                        hit = intersectTriExact(f3(ro.x, ro.y, ro.z), f3(rd.x, rd.y, rd.z),
                            f3(tv.v0.x, tv.v0.y, tv.v0.z), f3(tv.v1.x, tv.v1.y, tv.v1.z),
                            f3(tv.v2.x, tv.v2.y, tv.v2.z), ro.w, kRivals && kDrained ? cl + rd.w : cl, t, u, v);
                        if constexpr (AnyHit) {
                            hit = hit && t < cl;
                        } else if (hit) {
                            id = __float_as_uint(tv.v0.w);
                            // (t >= tMin >= 0: the bits order like the values; -0 counts as 0)
                            nk = (static_cast<unsigned long long>(__float_as_uint(__fadd_rn(t, 0.0f))) << 32) | (~id);
                            if constexpr (kRivals) {
                                if (kDrained && rd.w > 0.0f) {
                                    entry = boxEntry(f3(ro.x, ro.y, ro.z), f3(rd.x, rd.y, rd.z), tv, rd.w);
                                    atomicMin(&W.in.rival[oray], __float_as_uint(fmaxf(__fadd_rn(t, 0.0f), cl)));
                                }
                            }
                        }
                    }
                    if (__any_sync(kAll, hit)) {
                        if constexpr (AnyHit) {
                            if (hit) {
                                W.res[oray].x = 1.0f;
                            }
                            __syncwarp();
                            if (active && W.res[ray].x != 0.0f) {
                                tgroup.y = 0u; // occluded: the ray ends below
                                ngroup.y = 0u;
                                sp = sb;
                            }
                        } else {
                            if (hit) {
                                atomicMin(&W.key[oray], nk);
                            }
                            __syncwarp();
                            if (hit && W.key[oray] == nk) {
                                if constexpr (Inst) {
                                    const uint2 cur = W.in.cur[oray];
                                    W.res[oray] =
                                        make_float4(u, v, __uint_as_float(cur.y + id), __uint_as_float(cur.x));
                                } else {
                                    W.res[oray] = make_float4(u, v, __uint_as_float(id), 0.0f);
                                }
                            }
                            if constexpr (kRivals) {
                                if (kDrained && hit && W.d[oray].w > 0.0f) {
                                    if (W.key[oray] == nk) {
                                        W.in.entry[oray] = entry;
                                    } else {
                                        atomicMin(&W.in.rival[oray], static_cast<uint32_t>(nk >> 32));
                                    }
                                }
                            }
                            if (active) {
                                cull = keyT(ray);
                                if (kRivals && kDrained) {
                                    cull = fmaf(2.0f, W.d[ray].w, cull);
                                }
                            }
                        }
                    }
                    __syncwarp(); // the pair list, keys and rays are rewritten after this
                }
            }
            // --- pop ---
            if (active && tgroup.y == 0u && ngroup.y <= 0x00FFFFFFu) {
                if constexpr (Inst) {
                    if (level == 1 && sp == base && sp > 0) { // (sb is 0: no stealing)
                        // the object is done: back to the top level in world space
                        level = 0;
                        nodes = S->tlasNodes;
                        tris = S->tlasLeaves;
                        const float4 wo = W.in.wo[lane], wd = W.in.wd[lane];
                        setRay(f3(wo.x, wo.y, wo.z), f3(wd.x, wd.y, wd.z));
                    }
                }
                if (sp == sb) {
                    // (the last lane of a ray finishes it)
                    bool again = false;
                    if (Inst || atomicSub(&W.lanes[ray], 1u) == 1u) {
                        if constexpr (kRivals) {
                            if (kDrained && W.d[ray].w > 0.0f && __uint_as_float(W.in.rival[ray]) <= W.in.entry[ray]) {
                                // from the root, in one piece
                                again = true;
                                const float4 ro = W.o[ray], rd = W.d[ray];
                                setRay(f3(ro.x, ro.y, ro.z), f3(rd.x, rd.y, rd.z));
                                cull = W.in.tMax[ray];
                                W.key[ray] = static_cast<unsigned long long>(__float_as_uint(cull)) << 32;
                                W.res[ray] = make_float4(0.0f, 0.0f, __uint_as_float(0xFFFFFFFFu), 0.0f);
                                W.d[ray].w = -0.0f;
                                W.lanes[ray] = 1u;
                                sp = sb = 0;
                                ngroup = rootGroup();
                            }
                        }
                        if (!again) {
                            const float4 rs = W.res[ray];
                            const uint2 en = W.entry[ray];
                            const bool h = AnyHit ? rs.x != 0.0f : __float_as_uint(rs.z) != 0xFFFFFFFFu;
                            finish(en.x, en.y, h, keyT(ray), rs.x, rs.y, __float_as_uint(rs.z), __float_as_uint(rs.w));
                        }
                    }
                    if (!again) {
                        if (overflow && overflowCounter != nullptr && !(AnyHit && W.res[ray].x != 0.0f)) {
                            // rays whose stack overflowed (an occluded any-hit ray is not counted)
                            atomicAdd(overflowCounter, 1u);
                        }
                        active = false;
                    }
                    overflow = false;
                } else {
                    --sp;
                    const uint2 g = sp < kTraceStack ? W.stack[sp][lane] : spill[sp - kTraceStack];
                    if (!Inst || g.y > 0x00FFFFFFu) {
                        ngroup = g;
                    } else {
                        tgroup = g; // the rest of a top-level leaf group
                    }
                }
            }
        }
    };
    if (poolNext < count) {
        run(std::false_type{});
    }
    run(std::true_type{});
}

} // namespace pt
