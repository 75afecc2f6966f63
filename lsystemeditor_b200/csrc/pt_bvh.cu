// GPU acceleration-structure build: LBVH -> compressed 8-wide BVH.
//
// Replaces the reference's host-side median-split builder
// (PathTracerLib/src/MeshAccel/MeshBvhBuilder.cpp:52-142, O(N log^2 N) on one
// core) with a fully parallel build:
//   1. per-triangle bounds + centroid, centroid bounds       (k_prepare)
//   2. 30-bit Morton codes of the centroids                   (k_morton)
//   3. radix sort of (code, index) pairs                      (CUB onesweep)
//   4. binary radix tree, Karras 2012 "Maximizing Parallelism in the
//      Construction of BVHs, Octrees, and k-d Trees"         (k_karras)
//   5. bottom-up bounds + leaf counts                         (k_refit)
//   6. treelet reordering of the binary tree for SAH cost,
//      after Karras & Aila 2013 "Fast Parallel Construction of
//      High-Quality Bounding Volume Hierarchies"             (k_treelet)
//   7. top-down collapse to 8-wide nodes with quantised child boxes and
//      octant-ordered child slots, Ylitie, Karras & Laine 2017 (k_collapse)
//
// Closest-hit results do not depend on the tree shape (any BVH whose boxes
// contain their triangles returns the same nearest hit), so the product
// builds whatever tree traverses fastest.
#include "pt_bvh.cuh"


#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdio>

namespace pt {

namespace {

constexpr int kBlock = 256;

__device__ __forceinline__ unsigned int floatToOrdered(float f)
{
    const unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float orderedToFloat(unsigned int u)
{
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

__device__ __forceinline__ float3 loadVertex(const float* pos, uint32_t tri, int k)
{
    const float* p = pos + 9ull * tri + 3 * k;
    return make_float3(p[0], p[1], p[2]);
}

// (1) triangle bounds, centroids and the centroid bounding box.
__global__ void k_prepare(const float* __restrict__ pos, uint32_t n, float4* __restrict__ triLo,
    float4* __restrict__ triHi, unsigned int* __restrict__ cbounds)
{
    float3 cmin = make_float3(FLT_MAX, FLT_MAX, FLT_MAX);
    float3 cmax = make_float3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float3 a = loadVertex(pos, i, 0), b = loadVertex(pos, i, 1), c = loadVertex(pos, i, 2);
        const float3 lo = make_float3(fminf(fminf(a.x, b.x), c.x), fminf(fminf(a.y, b.y), c.y), fminf(fminf(a.z, b.z), c.z));
        const float3 hi = make_float3(fmaxf(fmaxf(a.x, b.x), c.x), fmaxf(fmaxf(a.y, b.y), c.y), fmaxf(fmaxf(a.z, b.z), c.z));
        triLo[i] = make_float4(lo.x, lo.y, lo.z, 0.0f);
        triHi[i] = make_float4(hi.x, hi.y, hi.z, 0.0f);
        const float3 ce = make_float3((lo.x + hi.x) * 0.5f, (lo.y + hi.y) * 0.5f, (lo.z + hi.z) * 0.5f);
        cmin = make_float3(fminf(cmin.x, ce.x), fminf(cmin.y, ce.y), fminf(cmin.z, ce.z));
        cmax = make_float3(fmaxf(cmax.x, ce.x), fmaxf(cmax.y, ce.y), fmaxf(cmax.z, ce.z));
    }
    // warp and block reductions, then one atomic per block and bound (an atomic
    // per warp was 182k on six addresses for 972k triangles: 129 -> 13 us)
    for (int off = 16; off > 0; off >>= 1) {
        cmin.x = fminf(cmin.x, __shfl_xor_sync(0xffffffffu, cmin.x, off));
        cmin.y = fminf(cmin.y, __shfl_xor_sync(0xffffffffu, cmin.y, off));
        cmin.z = fminf(cmin.z, __shfl_xor_sync(0xffffffffu, cmin.z, off));
        cmax.x = fmaxf(cmax.x, __shfl_xor_sync(0xffffffffu, cmax.x, off));
        cmax.y = fmaxf(cmax.y, __shfl_xor_sync(0xffffffffu, cmax.y, off));
        cmax.z = fmaxf(cmax.z, __shfl_xor_sync(0xffffffffu, cmax.z, off));
    }
    __shared__ float sBound[6][kBlock / 32];
    if ((threadIdx.x & 31) == 0) {
        const int w = threadIdx.x >> 5;
        sBound[0][w] = cmin.x;
        sBound[1][w] = cmin.y;
        sBound[2][w] = cmin.z;
        sBound[3][w] = cmax.x;
        sBound[4][w] = cmax.y;
        sBound[5][w] = cmax.z;
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        float v = sBound[threadIdx.x][0];
        for (int w = 1; w < kBlock / 32; ++w) {
            v = threadIdx.x < 3 ? fminf(v, sBound[threadIdx.x][w]) : fmaxf(v, sBound[threadIdx.x][w]);
        }
        if (threadIdx.x < 3) {
            atomicMin(&cbounds[threadIdx.x], floatToOrdered(v));
        } else {
            atomicMax(&cbounds[threadIdx.x], floatToOrdered(v));
        }
    }
}

__device__ __forceinline__ uint32_t expandBits10(uint32_t v)
{
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}

// (2) Morton codes of the box centroids in the centroid bounds.
__global__ void k_morton(const float4* __restrict__ triLo, const float4* __restrict__ triHi, uint32_t n,
    const unsigned int* __restrict__ cbounds, uint32_t* __restrict__ keys, uint32_t* __restrict__ vals)
{
    const float3 lo = make_float3(orderedToFloat(cbounds[0]), orderedToFloat(cbounds[1]), orderedToFloat(cbounds[2]));
    const float3 hi = make_float3(orderedToFloat(cbounds[3]), orderedToFloat(cbounds[4]), orderedToFloat(cbounds[5]));
    const float3 ext = make_float3(hi.x - lo.x, hi.y - lo.y, hi.z - lo.z);
    const float3 inv = make_float3(ext.x > 0.0f ? 1.0f / ext.x : 0.0f, ext.y > 0.0f ? 1.0f / ext.y : 0.0f,
        ext.z > 0.0f ? 1.0f / ext.z : 0.0f);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 a = triLo[i], b = triHi[i];
        const float cx = ((a.x + b.x) * 0.5f - lo.x) * inv.x;
        const float cy = ((a.y + b.y) * 0.5f - lo.y) * inv.y;
        const float cz = ((a.z + b.z) * 0.5f - lo.z) * inv.z;
        const uint32_t x = min(max(__float2int_rd(cx * 1024.0f), 0), 1023);
        const uint32_t y = min(max(__float2int_rd(cy * 1024.0f), 0), 1023);
        const uint32_t z = min(max(__float2int_rd(cz * 1024.0f), 0), 1023);
        keys[i] = (expandBits10(x) << 2) | (expandBits10(y) << 1) | expandBits10(z);
        vals[i] = i;
    }
}

// Common-prefix length of sorted keys i, j with the position as tie-breaker.
__device__ __forceinline__ int delta(const uint32_t* __restrict__ k, int n, int i, int j)
{
    if (j < 0 || j >= n) {
        return -1;
    }
    const uint32_t a = k[i], b = k[j];
    if (a != b) {
        return __clz(a ^ b);
    }
    return 32 + __clz(static_cast<uint32_t>(i) ^ static_cast<uint32_t>(j));
}

// (4) Karras radix tree. Internal nodes 0..n-2, leaf j is node n-1+j.
__global__ void k_karras(const uint32_t* __restrict__ keys, int n, int2* __restrict__ child, int* __restrict__ parent)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n - 1; i += gridDim.x * blockDim.x) {
        const int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
        const int dmin = delta(keys, n, i, i - d);
        int lmax = 2;
        while (delta(keys, n, i, i + lmax * d) > dmin) {
            lmax <<= 1;
        }
        int l = 0;
        for (int t = lmax >> 1; t >= 1; t >>= 1) {
            if (delta(keys, n, i, i + (l + t) * d) > dmin) {
                l += t;
            }
        }
        const int j = i + l * d;
        const int dnode = delta(keys, n, i, j);
        int s = 0;
        int t = l;
        do {
            t = (t + 1) >> 1;
            if (delta(keys, n, i, i + (s + t) * d) > dnode) {
                s += t;
            }
        } while (t > 1);
        const int gamma = i + s * d + min(d, 0);
        const int left = (min(i, j) == gamma) ? (n - 1 + gamma) : gamma;
        const int right = (max(i, j) == gamma + 1) ? (n - 1 + gamma + 1) : gamma + 1;
        child[i] = make_int2(left, right);
        parent[left] = i;
        parent[right] = i;
    }
}

// (5) Bottom-up bounds. Node bounds: lo.xyz + leaf count (w, int bits), hi.xyz + area (w).
__global__ void k_refit(const uint32_t* __restrict__ sortedIdx, const float4* __restrict__ triLo,
    const float4* __restrict__ triHi, int n, const int2* __restrict__ child, const int* __restrict__ parent,
    float4* nodeLo, float4* nodeHi, int* visits)
{
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        int node = n - 1 + j;
        const uint32_t tri = sortedIdx[j];
        float4 lo = triLo[tri], hi = triHi[tri];
        lo.w = __int_as_float(1);
        hi.w = 2.0f * ((hi.x - lo.x) * (hi.y - lo.y) + (hi.y - lo.y) * (hi.z - lo.z) + (hi.z - lo.z) * (hi.x - lo.x));
        nodeLo[node] = lo;
        nodeHi[node] = hi;
        if (n == 1) {
            continue;
        }
        __threadfence();
        int p = parent[node];
        while (p >= 0) {
            if (atomicAdd(&visits[p], 1) == 0) {
                break; // the sibling's thread finishes this node
            }
            __threadfence();
            const int2 c = child[p];
            const float4 al = __ldcg(&nodeLo[c.x]), ah = __ldcg(&nodeHi[c.x]);
            const float4 bl = __ldcg(&nodeLo[c.y]), bh = __ldcg(&nodeHi[c.y]);
            float4 ml = make_float4(fminf(al.x, bl.x), fminf(al.y, bl.y), fminf(al.z, bl.z),
                __int_as_float(__float_as_int(al.w) + __float_as_int(bl.w)));
            float4 mh = make_float4(fmaxf(ah.x, bh.x), fmaxf(ah.y, bh.y), fmaxf(ah.z, bh.z), 0.0f);
            mh.w = 2.0f * ((mh.x - ml.x) * (mh.y - ml.y) + (mh.y - ml.y) * (mh.z - ml.z) + (mh.z - ml.z) * (mh.x - ml.x));
            __stcg(&nodeLo[p], ml);
            __stcg(&nodeHi[p], mh);
            __threadfence();
            p = parent[p];
        }
    }
}

__device__ __forceinline__ float boxArea(float3 lo, float3 hi)
{
    const float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
    return 2.0f * (dx * dy + dy * dz + dz * dx);
}

// (6) Treelet restructuring (Karras & Aila 2013): every node whose subtree
// holds at least `minLeaves` triangles forms a treelet of up to 7 leaves by
// repeatedly opening its largest-area leaf; the optimal binary topology over
// those leaves is found by dynamic programming over leaf subsets with the SAH
// cost, and the treelet is rewritten in place. Processed bottom-up, one
// treelet per warp, with visit counters like k_refit so that a node is
// optimised only after both subtrees are final.
//
// Bound by latency: a treelet is a chain of dependent loads, and the treelets
// towards the root are a chain themselves.  So lane k holds treelet leaf k (one
// round trip per opened leaf: its box, children and cost are loaded together),
// the subsets' boxes come from the seven leaf boxes in shared memory, and the
// partitions of the two largest subset sizes are spread over the lanes.  The
// first form (one lane forming the treelet, boxes read from L2 per subset, one
// lane per subset) took 4.96 ms for 972k triangles and 1.90 ms for 132k; this
// one 1.10 and 0.48 ms.  Same trees.
constexpr int kTreeletLeaves = 7;
constexpr int kSubsets = 1 << kTreeletLeaves;

struct TreeletScratch {
    float area[kSubsets];
    float cost[kSubsets];
    float4 leafLo[kTreeletLeaves]; // w: triangles (int bits)
    float4 leafHi[kTreeletLeaves];
    int leaf[kTreeletLeaves];
    int internal[kTreeletLeaves - 1];
    int kids[kTreeletLeaves - 1][2]; // of the rewritten internal nodes
    uint8_t mask[kTreeletLeaves - 1]; // their leaf subsets
    uint8_t split[kSubsets];
};

// Subsets of seven leaves by size: 2 (21 of them), 3 (35), 4 (35), 5 (21).
struct SubsetTable {
    uint8_t m[112];
};
constexpr SubsetTable makeSubsetTable()
{
    SubsetTable t{};
    int at = 0;
    for (int size = 2; size <= 5; ++size) {
        for (int m = 1; m < kSubsets; ++m) {
            int bits = 0;
            for (int k = 0; k < kTreeletLeaves; ++k) {
                bits += (m >> k) & 1;
            }
            if (bits == size) {
                t.m[at++] = static_cast<uint8_t>(m);
            }
        }
    }
    return t;
}
__device__ const SubsetTable kSubsetTable = makeSubsetTable();

__device__ __forceinline__ bool isLeafNode(int node, int n) { return node >= n - 1; }

// The subsets of a lane in the rounds of sizes 2, 3, 3, 4, 4, 5 (0: none).
struct LaneSubsets {
    uint8_t m[6];
};
__device__ __forceinline__ LaneSubsets laneSubsets()
{
    const int lane = threadIdx.x & 31;
    LaneSubsets l;
    l.m[0] = lane < 21 ? kSubsetTable.m[lane] : 0;
    l.m[1] = kSubsetTable.m[21 + lane];
    l.m[2] = lane < 3 ? kSubsetTable.m[21 + 32 + lane] : 0;
    l.m[3] = kSubsetTable.m[56 + lane];
    l.m[4] = lane < 3 ? kSubsetTable.m[56 + 32 + lane] : 0;
    l.m[5] = lane < 21 ? kSubsetTable.m[91 + lane] : 0;
    return l;
}

__device__ void treeletOptimize(int root, int n, int2* child, int* parent, float4* nodeLo, float4* nodeHi,
    float* subtreeCost, TreeletScratch& s, const LaneSubsets& mine, float costNode)
{
    constexpr unsigned int kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    // --- form the treelet: open the largest-area treelet leaf until 7 leaves ---
    int node = -1, internal = root;
    bool inner = false;
    float4 lo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hi = lo;
    int2 kids = make_int2(-1, -1);
    float cost = 0.0f;
    auto hold = [&](int x) {
        node = x;
        inner = !isLeafNode(x, n);
        lo = __ldcg(&nodeLo[x]);
        hi = __ldcg(&nodeHi[x]);
        cost = __ldcg(&subtreeCost[x]);
        if (inner) {
            kids = __ldcg(&child[x]);
        }
    };
    {
        const int2 c = __ldcg(&child[root]);
        if (lane < 2) {
            hold(lane == 0 ? c.x : c.y);
        }
    }
    int nl = 2, ni = 1;
    while (nl < kTreeletLeaves) {
        // (areas are not negative: their bits order like the values)
        const unsigned int key = inner && hi.w > -1.0f ? __float_as_uint(hi.w) + 1u : 0u;
        const unsigned int top = __reduce_max_sync(kAll, key);
        if (top == 0u) {
            break;
        }
        const int best = __ffs(__ballot_sync(kAll, key == top)) - 1;
        const int opened = __shfl_sync(kAll, node, best);
        const int kx = __shfl_sync(kAll, kids.x, best), ky = __shfl_sync(kAll, kids.y, best);
        if (lane == ni) {
            internal = opened;
        }
        if (lane == best || lane == nl) {
            hold(lane == best ? kx : ky);
        }
        ++ni;
        ++nl;
    }
    if (nl < 3) {
        return;
    }
    if (lane < nl) {
        s.leafLo[lane] = lo;
        s.leafHi[lane] = hi;
        s.leaf[lane] = node;
        s.cost[1 << lane] = cost; // a treelet leaf keeps its (already optimised) subtree
        if (lane < ni) {
            s.internal[lane] = internal;
        }
    }
    __syncwarp();
    const int subsets = 1 << nl;
    // --- area of every leaf subset: bits 2.. from the lane, bits 0 and 1 in turn ---
    {
        float3 bl = make_float3(FLT_MAX, FLT_MAX, FLT_MAX), bh = make_float3(-FLT_MAX, -FLT_MAX, -FLT_MAX);
        auto join = [&](float3& l, float3& h, int k) {
            const float4 a = s.leafLo[k], b = s.leafHi[k];
            l = make_float3(fminf(l.x, a.x), fminf(l.y, a.y), fminf(l.z, a.z));
            h = make_float3(fmaxf(h.x, b.x), fmaxf(h.y, b.y), fmaxf(h.z, b.z));
        };
        for (int k = 2; k < nl; ++k) {
            if ((lane >> (k - 2)) & 1) {
                join(bl, bh, k);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float3 l = bl, h = bh;
            if (j & 1) {
                join(l, h, 0);
            }
            if (j & 2) {
                join(l, h, 1);
            }
            const int m = 4 * lane + j;
            if (m > 0 && m < subsets) {
                s.area[m] = boxArea(l, h);
            }
        }
    }
    __syncwarp();
    // --- SAH-optimal topology by dynamic programming over subsets of growing size ---
    // A partition is named by its part with the lowest leaf; of equal costs the
    // largest such part is taken (parts are tried in falling order).
    auto settle = [&](int m, float best, int part) {
        s.cost[m] = costNode * s.area[m] + best;
        s.split[m] = static_cast<uint8_t>(part);
    };
#pragma unroll
    for (int r = 0; r < 6; ++r) {
        const int m = mine.m[r];
        if (m != 0 && m < subsets) {
            const int low = m & -m, rest = m ^ low;
            float best = FLT_MAX;
            int part = low;
            for (int q = (rest - 1) & rest;; q = (q - 1) & rest) {
                const float c = s.cost[low | q] + s.cost[rest ^ q];
                if (c < best) {
                    best = c;
                    part = low | q;
                }
                if (q == 0) {
                    break;
                }
            }
            settle(m, best, part);
        }
        if (r == 0 || r == 2 || r >= 4) {
            __syncwarp();
        }
    }
    if (nl >= 6) {
        // seven subsets of six leaves, 31 partitions each, four lanes to a subset
        const int m = (kSubsets - 1) ^ (1 << (lane >> 2));
        const bool on = lane < 28 && m < subsets;
        const int low = m & -m, rest = m ^ low;
        float best = FLT_MAX;
        int at = 64, part = low;
        if (on) {
            int q = rest;
            for (int i = 0; i < 31; ++i) {
                q = (q - 1) & rest;
                if ((i & 3) == (lane & 3)) {
                    const float c = s.cost[low | q] + s.cost[rest ^ q];
                    if (c < best) {
                        best = c;
                        at = i;
                        part = low | q;
                    }
                }
            }
        }
#pragma unroll
        for (int d = 1; d <= 2; d <<= 1) {
            const float c = __shfl_xor_sync(kAll, best, d);
            const int i = __shfl_xor_sync(kAll, at, d), pt = __shfl_xor_sync(kAll, part, d);
            if (c < best || (c == best && i < at)) {
                best = c;
                at = i;
                part = pt;
            }
        }
        if (on && (lane & 3) == 0) {
            settle(m, best, part);
        }
        __syncwarp();
    }
    if (nl == kTreeletLeaves) {
        // all seven leaves: 63 partitions over the warp
        constexpr int rest = kSubsets - 2;
        float best = FLT_MAX;
        int at = 64;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = lane + 32 * h;
            if (i < 63) {
                const int q = 2 * (62 - i);
                const float c = s.cost[1 | q] + s.cost[rest ^ q];
                if (c < best) {
                    best = c;
                    at = i;
                }
            }
        }
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const float c = __shfl_xor_sync(kAll, best, d);
            const int i = __shfl_xor_sync(kAll, at, d);
            if (c < best || (c == best && i < at)) {
                best = c;
                at = i;
            }
        }
        if (lane == 0) {
            settle(kSubsets - 1, best, at < 63 ? 1 | (2 * (62 - at)) : 1);
        }
        __syncwarp();
    }
    // --- rewrite the treelet in place, reusing its internal node ids ---
    if (lane == 0) {
        int stack[kTreeletLeaves];
        int sp = 0, next = 1;
        s.mask[0] = static_cast<uint8_t>(subsets - 1);
        stack[sp++] = 0;
        while (sp > 0) {
            const int e = stack[--sp];
            const int m = s.mask[e];
            const int parts[2] = {static_cast<int>(s.split[m]), m ^ static_cast<int>(s.split[m])};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if ((parts[h] & (parts[h] - 1)) == 0) {
                    s.kids[e][h] = s.leaf[__ffs(parts[h]) - 1];
                } else {
                    s.mask[next] = static_cast<uint8_t>(parts[h]);
                    s.kids[e][h] = s.internal[next];
                    stack[sp++] = next++;
                }
            }
        }
    }
    __syncwarp();
    if (lane < ni) {
        const int m = s.mask[lane];
        const int2 k = make_int2(s.kids[lane][0], s.kids[lane][1]);
        float4 l = make_float4(FLT_MAX, FLT_MAX, FLT_MAX, 0.0f), h = make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, s.area[m]);
        int tris = 0;
        for (int j = 0; j < nl; ++j) {
            if ((m >> j) & 1) {
                const float4 a = s.leafLo[j], b = s.leafHi[j];
                l = make_float4(fminf(l.x, a.x), fminf(l.y, a.y), fminf(l.z, a.z), 0.0f);
                h = make_float4(fmaxf(h.x, b.x), fmaxf(h.y, b.y), fmaxf(h.z, b.z), h.w);
                tris += __float_as_int(a.w);
            }
        }
        l.w = __int_as_float(tris);
        child[internal] = k;
        parent[k.x] = internal;
        parent[k.y] = internal;
        __stcg(&nodeLo[internal], l);
        __stcg(&nodeHi[internal], h);
        __stcg(&subtreeCost[internal], s.cost[m]);
        __threadfence();
    }
    __syncwarp();
}

// Bottom-up pass of the subtrees too small for treelets, one thread per leaf
// (as the refit): the SAH cost of every subtree with fewer than minLeaves
// triangles, and the list of the nodes where treelet work starts (at least
// minLeaves triangles, both children finished here).  The second thread to
// reach a node goes on; the first stops.
__global__ void k_treelet_leaves(int n, const int2* child, const int* parent, const float4* nodeLo,
    const float4* nodeHi, int* visits, float* subtreeCost, int minLeaves, float costTri, float costNode,
    int* frontier, unsigned int* frontierCount)
{
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const int leaf = n - 1 + j;
        __stcg(&subtreeCost[leaf], costTri * __ldcg(&nodeHi[leaf]).w);
        __threadfence();
        int p = __ldcg(&parent[leaf]);
        while (p >= 0) {
            if (atomicAdd(&visits[p], 1) == 0) {
                break;
            }
            __threadfence();
            if (__float_as_int(__ldcg(&nodeLo[p]).w) >= minLeaves) {
                frontier[atomicAdd(frontierCount, 1u)] = p;
                break;
            }
            const int2 c = __ldcg(&child[p]);
            __stcg(&subtreeCost[p],
                costNode * __ldcg(&nodeHi[p]).w + __ldcg(&subtreeCost[c.x]) + __ldcg(&subtreeCost[c.y]));
            __threadfence();
            p = __ldcg(&parent[p]);
        }
    }
}

// Treelet reordering (Karras & Aila 2013), one warp per node of the frontier
// list and then up the tree: a node is optimised by the second warp to reach it
// (its first arrival may have come from k_treelet_leaves, for a small child).
// Every node from the frontier up has at least minLeaves triangles.
#ifndef PT_TREELET_BLOCKS
#define PT_TREELET_BLOCKS 6
#endif
__global__ void __launch_bounds__(kBlock, PT_TREELET_BLOCKS) k_treelet(int n, int2* child, int* parent, float4* nodeLo,
    float4* nodeHi, int* visits, float* subtreeCost, float costNode, const int* frontier,
    const unsigned int* frontierCount)
{
    __shared__ TreeletScratch scratch[kBlock / 32];
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    TreeletScratch& s = scratch[threadIdx.x >> 5];
    const LaneSubsets mine = laneSubsets();
    const int count = static_cast<int>(*frontierCount);
    for (int f = warp; f < count; f += warps) {
        int p = frontier[f];
        for (;;) {
            treeletOptimize(p, n, child, parent, nodeLo, nodeHi, subtreeCost, s, mine, costNode);
            int arrived = 0;
            if (lane == 0) {
                p = __ldcg(&parent[p]);
                arrived = p >= 0 ? atomicAdd(&visits[p], 1) : 0;
                __threadfence();
            }
            p = __shfl_sync(0xffffffffu, p, 0);
            if (__shfl_sync(0xffffffffu, arrived, 0) == 0) {
                break; // the sibling's warp goes on, or this was the root
            }
        }
    }
}

// The treelet passes of a build: per pass, the small subtrees bottom-up (one
// thread per leaf), then the treelets from the frontier up (one warp per
// frontier node, a grid of resident warps).
static cudaError_t runTreelets(int N, int2* child, int* parent, float4* nodeLo, float4* nodeHi, int* visits,
    float* subCost, int* frontier, unsigned int* frontierCount, const BvhBuildOptions& opt, cudaStream_t stream)
{
    for (int pass = 0; pass < opt.treeletPasses; ++pass) {
        cudaError_t e = cudaMemsetAsync(visits, 0, sizeof(int) * (N - 1), stream);
        if (e == cudaSuccess) {
            e = cudaMemsetAsync(frontierCount, 0, sizeof(unsigned int), stream);
        }
        if (e != cudaSuccess) {
            return e;
        }
        k_treelet_leaves<<<(N + kBlock - 1) / kBlock, kBlock, 0, stream>>>(N, child, parent, nodeLo, nodeHi, visits, subCost,
            opt.treeletMinLeaves, opt.costTriangle, opt.costNode, frontier, frontierCount);
        int dev = 0, sms = 1;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        k_treelet<<<sms * PT_TREELET_BLOCKS, kBlock, 0, stream>>>(N, child, parent, nodeLo, nodeHi, visits, subCost, opt.costNode,
            frontier, frontierCount);
    }
    return cudaGetLastError();
}

// (7) Collapse to 8-wide compressed nodes, level by level: a task is a binary
// node and the slot of its compressed node; a level emits the next one's tasks.
struct CollapseArgs {
    int n;
    const int2* child;
    const float4* nodeLo;
    const float4* nodeHi;
    const uint32_t* sortedIdx;
    const float* pos;
    CwNode* cw;
    TriVerts* tris;
    unsigned int* counters; // [0] next node, [1] next triangle, [2], [3] tasks of even and odd levels
    int maxLeafSize;
};

// Smallest exponent e with extent <= 255 * 2^e (extent computed exactly in double).
// Finite boxes need at most 2^121; an infinite one gets 2^127, so that the biased
// exponent stays a byte (a larger one would run into the node's child mask).
__device__ __forceinline__ int quantExp(double extent)
{
    if (!(extent > 0.0)) {
        return -126;
    }
    if (extent > 2.0 * FLT_MAX) {
        return 127;
    }
    int e;
    frexp(extent / 255.0, &e); // extent/255 in [2^(e-1), 2^e)
    e -= 1;
    while (ldexp(255.0, e) < extent) {
        ++e;
    }
    return max(e, -126);
}

// Eight lanes per task, one per child.  Bound by latency: a level has few tasks
// at the top, and one thread per task walked its eight children one after the
// other (boxes, 64-entry cost table, quantisation in double, triangle records):
// 50 - 160 us per level, 11 levels for 972k triangles; now 330 us in all
// against 916.  The task count of a level stays on the device, so that the host
// asks only once per kCollapseAhead levels whether there are more.
constexpr int kCollapseThreads = 128;
constexpr int kCollapseAhead = 4;

__global__ void __launch_bounds__(kCollapseThreads) k_collapse(CollapseArgs a, const int2* __restrict__ tasks,
    int2* __restrict__ nextTasks, int level)
{
    constexpr unsigned int kAll = 0xffffffffu;
    __shared__ uint4 sNode[kCollapseThreads / 8][5];
    const int taskCount = static_cast<int>(a.counters[2 + (level & 1)]);
    unsigned int* nextCount = &a.counters[2 + ((level & 1) ^ 1)];
    const int lane = threadIdx.x & 31, k = lane & 7, first = lane & 24;
    const int group = (blockIdx.x * blockDim.x + threadIdx.x) >> 3, groups = (gridDim.x * blockDim.x) >> 3;
    uint4* words = sNode[threadIdx.x >> 3];
    uint8_t* bytes = reinterpret_cast<uint8_t*>(words);
    // (a warp's four groups loop together)
    for (int t0 = group - (lane >> 3); t0 < taskCount; t0 += groups) {
        const int ti = t0 + (lane >> 3);
        const bool valid = ti < taskCount;
        const int2 task = valid ? tasks[ti] : make_int2(0, 0);
        const int bnode = task.x;
        // --- children: open the largest-area candidate until 8 slots are used, first
        // those that are too big for a leaf, then the remaining internal ones ---
        int cand = -1, count = 0;
        bool inner = false;
        float4 cl = make_float4(0.0f, 0.0f, 0.0f, 0.0f), ch = cl;
        int2 kids = make_int2(-1, -1);
        auto hold = [&](int x) {
            cand = x;
            inner = !isLeafNode(x, a.n);
            cl = a.nodeLo[x];
            ch = a.nodeHi[x];
            count = __float_as_int(cl.w);
            if (inner) {
                kids = a.child[x];
            }
        };
        float4 nl4 = cl, nh4 = cl;
        int nc = 0;
        if (valid) {
            nl4 = a.nodeLo[bnode];
            nh4 = a.nodeHi[bnode];
            if (isLeafNode(bnode, a.n)) {
                nc = 1;
                if (k == 0) {
                    hold(bnode);
                }
            } else {
                const int2 c = a.child[bnode];
                nc = 2;
                if (k < 2) {
                    hold(k == 0 ? c.x : c.y);
                }
            }
        }
        for (int r = 0; r < 6; ++r) {
            // (areas are not negative: their bits order like the values)
            unsigned int key = 0u;
            if (inner && nc < 8 && ch.w > -1.0f) {
                key = (__float_as_uint(ch.w) + 1u) | (count > a.maxLeafSize ? 0x80000000u : 0u);
            }
            unsigned int top = key;
#pragma unroll
            for (int d = 1; d < 8; d <<= 1) {
                top = max(top, __shfl_xor_sync(kAll, top, d));
            }
            const unsigned int at = __ballot_sync(kAll, key == top) >> first;
            const int best = __ffs(at & 0xffu) - 1;
            const int kx = __shfl_sync(kAll, kids.x, first + best), ky = __shfl_sync(kAll, kids.y, first + best);
            if (top != 0u) {
                if (k == best || k == nc) {
                    hold(k == best ? kx : ky);
                }
                ++nc;
            }
        }
        // --- node bounds ---
        const float3 lo = make_float3(nl4.x, nl4.y, nl4.z);
        const float3 hi = make_float3(nh4.x, nh4.y, nh4.z);
        const float extLo = k == 0 ? lo.x : (k == 1 ? lo.y : lo.z), extHi = k == 0 ? hi.x : (k == 1 ? hi.y : hi.z);
        const int own = valid && k < 3 ? quantExp(static_cast<double>(extHi) - extLo) : 0;
        const int ex = __shfl_sync(kAll, own, first), ey = __shfl_sync(kAll, own, first + 1),
                  ez = __shfl_sync(kAll, own, first + 2);
        // --- octant-ordered slot assignment: slot s receives the child that is nearest
        // for rays whose direction signs are s (bit 2 = -x, bit 1 = -y, bit 0 = -z) ---
        const float3 nc3 = make_float3((lo.x + hi.x) * 0.5f, (lo.y + hi.y) * 0.5f, (lo.z + hi.z) * 0.5f);
        const float3 d3 = make_float3((cl.x + ch.x) * 0.5f - nc3.x, (cl.y + ch.y) * 0.5f - nc3.y,
            (cl.z + ch.z) * 0.5f - nc3.z);
        int slot = -1;
        unsigned int taken = 0u;
        for (int round = 0; round < 8; ++round) {
            // the cheapest free (child, slot) pair; of equal ones the first child's first slot
            float best = FLT_MAX;
            int bs = -1;
            if (slot < 0 && k < nc) {
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const float dx = (s & 4) ? -d3.x : d3.x;
                    const float dy = (s & 2) ? -d3.y : d3.y;
                    const float dz = (s & 1) ? -d3.z : d3.z;
                    const float c = dx + dy + dz;
                    if (((taken >> s) & 1u) == 0u && (c < best || bs < 0)) {
                        best = c;
                        bs = s;
                    }
                }
            }
            // (+ 0: -0 counts as 0; the key orders like the cost and is not 0)
            const unsigned int key = bs < 0 ? 0xffffffffu : min(floatToOrdered(best + 0.0f), 0xfffffffeu);
            unsigned int low = key;
#pragma unroll
            for (int d = 1; d < 8; d <<= 1) {
                low = min(low, __shfl_xor_sync(kAll, low, d));
            }
            const unsigned int at = __ballot_sync(kAll, key == low) >> first;
            const int win = __ffs(at & 0xffu) - 1;
            const int ws = __shfl_sync(kAll, bs, first + win);
            if (low != 0xffffffffu) {
                if (k == win) {
                    slot = ws;
                }
                taken |= 1u << ws;
            }
        }
        // --- internal children and leaf triangles, in slot order ---
        const bool used = valid && slot >= 0;
        const bool internal = used && count > a.maxLeafSize;
        unsigned int imask = internal ? 1u << slot : 0u;
        unsigned int counts = used && !internal ? static_cast<unsigned int>(count) << (2 * slot) : 0u; // two bits per slot
#pragma unroll
        for (int d = 1; d < 8; d <<= 1) {
            imask |= __shfl_xor_sync(kAll, imask, d);
            counts |= __shfl_xor_sync(kAll, counts, d);
        }
        auto triangles = [](unsigned int c) { return __popc(c & 0x5555u) + 2 * __popc(c & 0xAAAAu); };
        const unsigned int internals = __popc(imask), triTotal = triangles(counts);
        unsigned int childBase = 0u, triBase = 0u, taskBase = 0u;
        if (k == 0 && internals != 0u) {
            childBase = atomicAdd(&a.counters[0], internals);
            taskBase = atomicAdd(nextCount, internals);
        }
        if (k == 0 && triTotal != 0u) {
            triBase = atomicAdd(&a.counters[1], triTotal);
        }
        childBase = __shfl_sync(kAll, childBase, first);
        taskBase = __shfl_sync(kAll, taskBase, first);
        triBase = __shfl_sync(kAll, triBase, first);
        // --- the compressed node, put together in shared memory ---
        if (k < 5) {
            uint4 w = make_uint4(0u, 0u, 0u, 0u);
            if (k == 0) {
                w = make_uint4(__float_as_uint(lo.x), __float_as_uint(lo.y), __float_as_uint(lo.z),
                    static_cast<unsigned>(ex + 127) | (static_cast<unsigned>(ey + 127) << 8) |
                        (static_cast<unsigned>(ez + 127) << 16) | (imask << 24));
            } else if (k == 1) {
                w.x = childBase;
                w.y = triBase;
            }
            words[k] = w;
        }
        __syncwarp();
        if (used) {
            const float clv[3] = {cl.x, cl.y, cl.z};
            const float chv[3] = {ch.x, ch.y, ch.z};
            const float pv[3] = {lo.x, lo.y, lo.z};
            const int ev[3] = {ex, ey, ez};
#pragma unroll
            for (int ax = 0; ax < 3; ++ax) {
                const double inv = ldexp(1.0, -ev[ax]); // (a power of two: the product is the exact quotient)
                const double ql = floor((static_cast<double>(clv[ax]) - static_cast<double>(pv[ax])) * inv);
                const double qh = ceil((static_cast<double>(chv[ax]) - static_cast<double>(pv[ax])) * inv);
                bytes[32 + 8 * ax + slot] = static_cast<uint8_t>(fmin(fmax(ql, 0.0), 255.0));
                bytes[56 + 8 * ax + slot] = static_cast<uint8_t>(fmin(fmax(qh, 0.0), 255.0));
            }
            if (internal) {
                bytes[24 + slot] = static_cast<uint8_t>(0x20 | (24 + slot));
                const int rank = __popc(imask & ((1u << slot) - 1u));
                nextTasks[taskBase + rank] = make_int2(cand, static_cast<int>(childBase) + rank);
            } else {
                unsigned int triOff = triangles(counts & ((1u << (2 * slot)) - 1u));
                bytes[24 + slot] = static_cast<uint8_t>((((1 << count) - 1) << 5) | triOff);
                // gather the subtree's triangles (at most maxLeafSize leaves)
                int st[8];
                int sp = 0;
                st[sp++] = cand;
                while (sp > 0) {
                    const int x = st[--sp];
                    if (isLeafNode(x, a.n)) {
                        const uint32_t tri = a.sortedIdx[x - (a.n - 1)];
                        const float3 v0 = loadVertex(a.pos, tri, 0), v1 = loadVertex(a.pos, tri, 1),
                                     v2 = loadVertex(a.pos, tri, 2);
                        TriVerts tv;
                        tv.v0 = make_float4(v0.x, v0.y, v0.z, __uint_as_float(tri));
                        tv.v1 = make_float4(v1.x, v1.y, v1.z, 0.0f);
                        tv.v2 = make_float4(v2.x, v2.y, v2.z, 0.0f);
                        a.tris[triBase + triOff] = tv;
                        ++triOff;
                    } else {
                        const int2 cc = a.child[x];
                        st[sp++] = cc.y;
                        st[sp++] = cc.x;
                    }
                }
            }
        }
        __syncwarp();
        if (valid && k < 5) {
            a.cw[task.y].w[k] = words[k];
        }
        __syncwarp();
    }
}

inline int gridFor(long long n, int block = kBlock)
{
    long long g = (n + block - 1) / block;
    if (g < 1) {
        g = 1;
    }
    if (g > 148 * 32) {
        g = 148 * 32;
    }
    return static_cast<int>(g);
}

} // namespace

#define PT_TRY(call)                                                                                              \
    do {                                                                                                          \
        cudaError_t e_ = (call);                                                                                  \
        if (e_ != cudaSuccess) {                                                                                  \
            std::snprintf(err, errLen, "%s failed: %s", #call, cudaGetErrorString(e_));                          \
            return e_ == cudaErrorMemoryAllocation ? PT_ERR_OUT_OF_MEMORY : PT_ERR_CUDA;                          \
        }                                                                                                         \
    } while (0)

// All levels of the collapse, from the root task in taskA and counters[2] = 1.
static int runCollapse(const CollapseArgs& ca, int2* taskA, int2* taskB, cudaStream_t stream, char* err, size_t errLen)
{
    constexpr int kBlocks = 148 * 8;
    const int blocks = std::min<long long>(kBlocks, (static_cast<long long>(ca.n) + kCollapseThreads / 8 - 1) / (kCollapseThreads / 8));
    for (int level = 0; level < 256; ++level) {
        PT_TRY(cudaMemsetAsync(ca.counters + 2 + ((level & 1) ^ 1), 0, sizeof(unsigned int), stream));
        k_collapse<<<blocks, kCollapseThreads, 0, stream>>>(ca, (level & 1) ? taskB : taskA, (level & 1) ? taskA : taskB, level);
        if (level % kCollapseAhead == kCollapseAhead - 1) {
            unsigned int next = 0;
            PT_TRY(cudaMemcpyAsync(&next, ca.counters + 2 + ((level & 1) ^ 1), sizeof(unsigned int), cudaMemcpyDeviceToHost, stream));
            PT_TRY(cudaStreamSynchronize(stream));
            if (next == 0) {
                return PT_OK;
            }
        }
    }
    std::snprintf(err, errLen, "BVH collapse did not terminate");
    return PT_ERR_INTERNAL;
}

int buildBvh(const float* dPositions, uint32_t n, BvhBuffers& out, cudaStream_t stream, const BvhBuildOptions& opt,
    char* err, size_t errLen)
{
    out.nodeCount = out.triCount = 0;
    if (n == 0) {
        return PT_OK;
    }
    const int N = static_cast<int>(n);
    const int nodesBin = 2 * N - 1;
    DeviceArena& ar = out.scratch;
    ar.failed = false;
    float4* triLo = ar.get<float4>(0, n);
    float4* triHi = ar.get<float4>(1, n);
    unsigned int* cbounds = ar.get<unsigned int>(2, 8);
    uint32_t* keys = ar.get<uint32_t>(3, n);
    uint32_t* vals = ar.get<uint32_t>(4, n);
    uint32_t* keysSorted = ar.get<uint32_t>(5, n);
    uint32_t* valsSorted = ar.get<uint32_t>(6, n);
    int2* child = ar.get<int2>(7, static_cast<size_t>(N > 1 ? N - 1 : 1));
    int* parent = ar.get<int>(8, static_cast<size_t>(nodesBin));
    float4* nodeLo = ar.get<float4>(9, static_cast<size_t>(nodesBin));
    float4* nodeHi = ar.get<float4>(10, static_cast<size_t>(nodesBin));
    int* visits = ar.get<int>(11, static_cast<size_t>(N > 1 ? N - 1 : 1));
    float* subCost = ar.get<float>(12, static_cast<size_t>(nodesBin));
    if (!ar.ok()) {
        std::snprintf(err, errLen, "BVH scratch allocation failed (%u triangles)", n);
        return PT_ERR_OUT_OF_MEMORY;
    }

    // bounds sentinel: min slots get 0xFFFFFFFF, max slots 0
    const unsigned int init[8] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u, 0u, 0u};
    PT_TRY(cudaMemcpyAsync(cbounds, init, sizeof(init), cudaMemcpyHostToDevice, stream));
    k_prepare<<<std::min(gridFor(n), 148 * 8), kBlock, 0, stream>>>(dPositions, n, triLo, triHi, cbounds);
    k_morton<<<gridFor(n), kBlock, 0, stream>>>(triLo, triHi, n, cbounds, keys, vals);
    const size_t tempBytes = radixSortTempBytes(n);
    void* temp = ar.getBytes(13, tempBytes);
    if (!ar.ok()) {
        std::snprintf(err, errLen, "radix sort scratch allocation failed");
        return PT_ERR_OUT_OF_MEMORY;
    }
    PT_TRY(radixSortPairs(keys, vals, keysSorted, valsSorted, n, 30, temp, tempBytes, stream));
    PT_TRY(cudaMemsetAsync(parent, 0xff, sizeof(int) * nodesBin, stream));
    if (N > 1) {
        k_karras<<<gridFor(N - 1), kBlock, 0, stream>>>(keysSorted, N, child, parent);
        PT_TRY(cudaMemsetAsync(visits, 0, sizeof(int) * (N - 1), stream));
    }
    k_refit<<<gridFor(N), kBlock, 0, stream>>>(valsSorted, triLo, triHi, N, child, parent, nodeLo, nodeHi, visits);
    if (N > 1 && opt.treeletPasses > 0) {
        int* frontier = ar.get<int>(17, static_cast<size_t>(N - 1));
        unsigned int* frontierCount = ar.get<unsigned int>(18, 1);
        if (!ar.ok()) {
            std::snprintf(err, errLen, "treelet scratch allocation failed");
            return PT_ERR_OUT_OF_MEMORY;
        }
        PT_TRY(runTreelets(N, child, parent, nodeLo, nodeHi, visits, subCost, frontier, frontierCount, opt, stream));
    }
    PT_TRY(cudaGetLastError());

    // Collapse. Upper bounds: nodes <= n (every compressed node has >= 2 children or is the root),
    // triangles == n.
    const size_t maxNodes = static_cast<size_t>(n) + 1;
    if (!out.reserve(maxNodes, static_cast<size_t>(n))) {
        std::snprintf(err, errLen, "BVH output allocation failed (%u triangles)", n);
        out.release();
        return PT_ERR_OUT_OF_MEMORY;
    }
    int2* taskA = ar.get<int2>(14, maxNodes);
    int2* taskB = ar.get<int2>(15, maxNodes);
    unsigned int* counters = ar.get<unsigned int>(16, 4);
    if (!ar.ok()) {
        std::snprintf(err, errLen, "collapse scratch allocation failed");
        return PT_ERR_OUT_OF_MEMORY;
    }
    // counters: [0] next node (root = 0 already taken), [1] next triangle, [2] tasks of level 0
    const unsigned int cinit[4] = {1u, 0u, 1u, 0u};
    PT_TRY(cudaMemcpyAsync(counters, cinit, sizeof(cinit), cudaMemcpyHostToDevice, stream));
    const int rootBin = N > 1 ? 0 : 0; // internal root 0, or the single leaf node 0 (= n - 1) when n == 1
    const int2 rootTask = make_int2(N > 1 ? rootBin : 0, 0);
    PT_TRY(cudaMemcpyAsync(taskA, &rootTask, sizeof(int2), cudaMemcpyHostToDevice, stream));
    CollapseArgs ca{N, child, nodeLo, nodeHi, valsSorted, dPositions, out.nodes, out.tris, counters, opt.maxLeafSize};
    const int st = runCollapse(ca, taskA, taskB, stream, err, errLen);
    if (st != PT_OK) {
        return st;
    }
    unsigned int finalCounts[2] = {0, 0};
    PT_TRY(cudaMemcpyAsync(finalCounts, counters, sizeof(finalCounts), cudaMemcpyDeviceToHost, stream));
    PT_TRY(cudaStreamSynchronize(stream));
    out.nodeCount = finalCounts[0];
    out.triCount = finalCounts[1];
    if (out.triCount != n) {
        std::snprintf(err, errLen, "BVH collapse placed %u of %u triangles", out.triCount, n);
        return PT_ERR_INTERNAL;
    }
    return PT_OK;
}

} // namespace pt

namespace pt {

size_t bvhSortTempBytes(uint32_t n)
{
    return radixSortTempBytes(n);
}

// Same build as buildBvh, into caller-provided buffers: nothing is allocated.
int buildBvhInto(const float* dPositions, uint32_t n, const BvhScratch& sc, CwNode* outNodes, TriVerts* outTris,
    uint32_t* outNodeCount, cudaStream_t stream, const BvhBuildOptions& opt, char* err, size_t errLen)
{
    if (n == 0) {
        *outNodeCount = 0;
        return PT_OK;
    }
    const int N = static_cast<int>(n);
    const int nodesBin = 2 * N - 1;
    const unsigned int init[8] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u, 0u, 0u};
    PT_TRY(cudaMemcpyAsync(sc.cbounds, init, sizeof(init), cudaMemcpyHostToDevice, stream));
    k_prepare<<<std::min(gridFor(n), 148 * 8), kBlock, 0, stream>>>(dPositions, n, sc.triLo, sc.triHi, sc.cbounds);
    k_morton<<<gridFor(n), kBlock, 0, stream>>>(sc.triLo, sc.triHi, n, sc.cbounds, sc.keys, sc.vals);
    const size_t tempBytes = radixSortTempBytes(n);
    if (tempBytes > sc.sortTempBytes) {
        std::snprintf(err, errLen, "radix sort needs %zu scratch bytes, %zu reserved", tempBytes, sc.sortTempBytes);
        return PT_ERR_INVALID_ARGUMENT;
    }
    PT_TRY(radixSortPairs(sc.keys, sc.vals, sc.keysSorted, sc.valsSorted, n, 30, sc.sortTemp, tempBytes, stream));
    PT_TRY(cudaMemsetAsync(sc.parent, 0xff, sizeof(int) * nodesBin, stream));
    if (N > 1) {
        k_karras<<<gridFor(N - 1), kBlock, 0, stream>>>(sc.keysSorted, N, sc.child, sc.parent);
        PT_TRY(cudaMemsetAsync(sc.visits, 0, sizeof(int) * (N - 1), stream));
    }
    k_refit<<<gridFor(N), kBlock, 0, stream>>>(sc.valsSorted, sc.triLo, sc.triHi, N, sc.child, sc.parent, sc.nodeLo,
        sc.nodeHi, sc.visits);
    if (N > 1 && opt.treeletPasses > 0) {
        PT_TRY(runTreelets(N, sc.child, sc.parent, sc.nodeLo, sc.nodeHi, sc.visits, sc.subCost, sc.frontier,
            sc.frontierCount, opt, stream));
    }
    PT_TRY(cudaGetLastError());
    const unsigned int cinit[4] = {1u, 0u, 1u, 0u};
    PT_TRY(cudaMemcpyAsync(sc.counters, cinit, sizeof(cinit), cudaMemcpyHostToDevice, stream));
    const int2 rootTask = make_int2(0, 0);
    PT_TRY(cudaMemcpyAsync(sc.taskA, &rootTask, sizeof(int2), cudaMemcpyHostToDevice, stream));
    CollapseArgs ca{N, sc.child, sc.nodeLo, sc.nodeHi, sc.valsSorted, dPositions, outNodes, outTris, sc.counters,
        opt.maxLeafSize};
    const int st = runCollapse(ca, sc.taskA, sc.taskB, stream, err, errLen);
    if (st != PT_OK) {
        return st;
    }
    unsigned int finalCounts[2] = {0, 0};
    PT_TRY(cudaMemcpyAsync(finalCounts, sc.counters, sizeof(finalCounts), cudaMemcpyDeviceToHost, stream));
    PT_TRY(cudaStreamSynchronize(stream));
    if (finalCounts[1] != n) {
        std::snprintf(err, errLen, "BVH collapse placed %u of %u triangles", finalCounts[1], n);
        return PT_ERR_INTERNAL;
    }
    *outNodeCount = finalCounts[0];
    return PT_OK;
}

} // namespace pt
