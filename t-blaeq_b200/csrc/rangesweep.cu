// Exact range batches: upper test, sweep, gather (see rangesweep.cuh).
#include "rangesweep.cuh"

#include <algorithm>
#include <type_traits>

#include "knnsweep.cuh"

namespace tblaeq {

namespace {

constexpr uint32_t FULL = 0xffffffffu;

// The level-synchronous kernels' radius test (kPredRangeRadius): box gap accumulated with fma in
// dimension order against the subtree radius. Out of line, like the point test below: both are rare
// (radiusQuick and the float points decide nearly everything), and inlined their registers would
// count against the loops around them.
__device__ __noinline__ bool radiusMeets(const double* y, const double* box, int D, double rad) {
    double dist = 0.0;
    for (int d = 0; d < D; ++d) {
        const double v = __ldg(y + d), l = __ldg(box + d), h = __ldg(box + D + d);
        double diff = 0.0;
        if (v < l) {
            diff = l - v;
        } else if (v > h) {
            diff = v - h;
        }
        dist = __fma_rn(diff, diff, dist);
    }
    return dist <= __dmul_rn(rad, rad);
}

__device__ __noinline__ bool pointInside(const double* y, const double* box, int D) {
    bool in = true;
    for (int d = 0; d < D; ++d) in = in && __ldg(box + d) <= __ldg(y + d) && __ldg(y + d) <= __ldg(box + D + d);
    return in;
}

// The same test in float, where its rounding cannot matter: 1 = survives, 0 = does not, -1 = too near
// the radius to tell (the FP64 test decides). `margin` bounds the error of the gap's length from
// rounding the box outward and the centre to nearest; the sums' relative error is within kRel.
constexpr float kRel = 1.00001f;
template <int DP, class Lo, class Hi>
__device__ __forceinline__ int radiusQuick(const float* y, Lo&& lo, Hi&& hi, float rad, float margin) {
    float g = 0.f;
#pragma unroll
    for (int d = 0; d < DP; d += 4) {
        const float4 c = *reinterpret_cast<const float4*>(y + d);  // shared or global memory
        const float4 l = lo(d), h = hi(d);
        const float e0 = fmaxf(fmaxf(l.x - c.x, c.x - h.x), 0.f), e1 = fmaxf(fmaxf(l.y - c.y, c.y - h.y), 0.f);
        const float e2 = fmaxf(fmaxf(l.z - c.z, c.z - h.z), 0.f), e3 = fmaxf(fmaxf(l.w - c.w, c.w - h.w), 0.f);
        g = fmaf(e0, e0, g);
        g = fmaf(e1, e1, g);
        g = fmaf(e2, e2, g);
        g = fmaf(e3, e3, g);
    }
    const float far = rad + margin, near = rad / kRel - margin;  // rad is rounded up
    if (g > far * far * kRel) return 0;
    if (near > 0.f && g * kRel <= near * near) return 1;
    return -1;
}

// Boxes on the grid: kRangeGrid steps over the data's extent per dimension, lower corners rounded down,
// upper corners up (both the same monotone function of the coordinate, so boxes that meet still meet),
// two 15-bit coordinates to a word. With the guard bit set above the larger operand, one subtraction
// compares two dimensions: the bit survives where upper >= lower. Against 2 D float comparisons the
// pair test takes D subtractions, half the shared-memory reads and a third of the registers.
constexpr uint32_t kGuard = 0x80008000u;

// ---- upper meshes -----------------------------------------------------------------------------------
constexpr uint32_t kUpperChunk = 4;                             // upper units of a block
constexpr uint32_t kUpperNodes = kUpperChunk * kRangeUpperUnit;  // and their nodes

template <int DP>
constexpr int upperWarps() {
    return DP <= 16 ? 4 : 2;  // static shared memory
}

// Blocks of kUpperChunk upper units (siblings of the last upper mesh, kRangeUpperUnit at most) by a range
// of query words. The block stages its nodes' boxes, centres and radii, and their parents'; a warp
// takes one word at a time, a query a lane, and tests it against every node: box tests node by
// node (the ballot is the node's word), then the radius tests of the pairs that passed, 32 at a time.
// Ancestors are tested once per unit, and counted by the first unit below each. Batches of few words
// give every warp a unit instead of a word. With the nodes read from memory by every warp the
// launch spent its time on chains of loads: 78 us for 4,096 queries x 2,100 nodes.
template <int DP>
__global__ void __launch_bounds__(upperWarps<DP>() * 32) rangeUpperKernel(RangeSweepArgs a, uint32_t wordsPerBlock,
                                                                            uint32_t wordBlocks, int byUnit) {
    constexpr int WARPS = upperWarps<DP>();
    constexpr int THREADS = WARPS * 32;
    constexpr int ROW = 3 * DP + 4;  // a staged node: lo, hi, centre, radius
    __shared__ uint32_t sCount[2 * kRangeMaxHeight];  // survivors and their children, by mesh
    __shared__ __align__(16) float sNode[kUpperNodes][ROW];
    __shared__ __align__(16) float sParent[kUpperChunk][ROW];
    __shared__ uint32_t sKids[kUpperNodes];
    __shared__ float sT[WARPS][2 * DP][33], sMargin[WARPS][32];  // a word's boxes, a dimension a row
    __shared__ uint16_t sPairs[WARPS][32 * kUpperNodes];
    __shared__ uint32_t sWord[WARPS][kUpperNodes];
    const int D = a.D, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int last = a.height - 3;  // the mesh whose bits are kept
    // One grid axis for both: the y axis ends at 65,535 blocks, and an index of small fan-outs has more chunks.
    const uint32_t chunk = blockIdx.x / wordBlocks, wordBlock = blockIdx.x - chunk * wordBlocks;
    const uint32_t unit0 = chunk * kUpperChunk;
    const uint32_t nUnits = last >= 0 ? min(kUpperChunk, a.nUpper - unit0) : 0u;
    if (tid < 2 * static_cast<int>(kRangeMaxHeight)) sCount[tid] = 0;
    auto stage = [&](float* to, int m, uint32_t g, int piece) {
        const RangeSweepLevel& L = a.level[m];
        if (piece < DP / 2)
            reinterpret_cast<float4*>(to)[piece] = __ldg(reinterpret_cast<const float4*>(L.box + static_cast<size_t>(g) * 2 * DP) + piece);
        else if (piece < 3 * DP / 4)
            reinterpret_cast<float4*>(to)[piece] =
                __ldg(reinterpret_cast<const float4*>(L.xF + static_cast<size_t>(g) * DP) + (piece - DP / 2));
        else
            to[3 * DP] = __ldg(L.radF + g);
    };
    constexpr int PIECES = 3 * DP / 4 + 1;
    for (uint32_t i = tid; i < nUnits * kRangeUpperUnit * PIECES; i += THREADS) {
        const uint32_t n = i / PIECES, at = n % kRangeUpperUnit;
        const RangeUnit un = a.upper[unit0 + n / kRangeUpperUnit];
        if (at >= un.count) continue;
        stage(sNode[n], last, un.first + at, i % PIECES);
        if (i % PIECES == 0) sKids[n] = a.level[last].nodes[un.first + at].cnt;
    }
    if (last > 0)
        for (uint32_t i = tid; i < nUnits * PIECES; i += THREADS)
            stage(sParent[i / PIECES], last - 1, a.upper[unit0 + i / PIECES].node, i % PIECES);
    if (blockIdx.x == 0 && tid == 0) {
        a.hdr[0] = a.nq;
        a.hdr[1] = a.nq * a.level[0].count;
    }
    __syncthreads();
    const uint32_t w1 = min(a.words, (wordBlock + 1) * wordsPerBlock);
    for (uint32_t w = wordBlock * wordsPerBlock + (byUnit ? 0 : warp); w < w1; w += byUnit ? 1 : WARPS) {
        const uint32_t q = w * 32 + lane, n = min(32u, a.nq - w * 32);
        const bool qv = q < a.nq;
        const bool writes = chunk == 0 && (!byUnit || warp == 0);
        // The word's boxes as floats: outward for the box tests, inward for the points'. Padding
        // dimensions hold [-1, 1] around the data's 0.
        __syncwarp();
#pragma unroll 4
        for (uint32_t i = lane; i < n * 2 * DP; i += 32) {
            const uint32_t k = i / (2 * DP), r = i % (2 * DP), d = r % DP;
            const bool upper = r >= DP;
            float out = upper ? 1.f : -1.f, in = out;
            if (d < static_cast<uint32_t>(D)) {
                const double v = __ldg(a.boxes + static_cast<size_t>(w * 32 + k) * 2 * D + (upper ? D : 0) + d);
                out = upper ? __double2float_ru(v) : __double2float_rd(v);
                in = upper ? __double2float_rd(v) : __double2float_ru(v);
            }
            sT[warp][r][k] = out;
            if (writes) {
                a.boxF[static_cast<size_t>(w * 32 + k) * 4 * DP + r] = out;
                a.boxF[static_cast<size_t>(w * 32 + k) * 4 * DP + 2 * DP + r] = in;
            }
        }
        __syncwarp();
        float lo[DP], hi[DP], most = 0.f;
#pragma unroll
        for (int d = 0; d < DP; ++d) {
            lo[d] = qv ? sT[warp][d][lane] : 1.f;
            hi[d] = qv ? sT[warp][DP + d][lane] : -1.f;
            most = fmaxf(most, fmaxf(fabsf(lo[d]), fabsf(hi[d])));
        }
        sMargin[warp][lane] = (most + a.maxAbs) * a.marginScale;
        if (writes && qv) {
            a.margin[q] = sMargin[warp][lane];
            const double* box = a.boxes + static_cast<size_t>(q) * 2 * D;
            uint32_t* grid = a.boxGrid + static_cast<size_t>(q) * DP;
#pragma unroll
            for (int d = 0; d < DP; d += 2) {
                uint32_t l[2], h[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const bool on = d + i < D;
                    l[i] = on ? rangeGridLower(__ldg(box + d + i), a.gridMin[d + i], a.gridScale[d + i]) : 0u;
                    h[i] = on ? rangeGridUpper(__ldg(box + D + d + i), a.gridMin[d + i], a.gridScale[d + i]) : 0u;
                }
                grid[d / 2] = kGuard | h[0] | (h[1] << 16);
                grid[DP / 2 + d / 2] = l[0] | (l[1] << 16);
            }
        }
        if (last < 0) {  // two meshes: the clusters hang below one virtual root
            const uint32_t all = __ballot_sync(FULL, qv);
            if (writes && lane == 0) a.bits[w] = all;
            continue;
        }
        __syncwarp();
        auto boxMeets = [&](const float* b, bool on) {
#pragma unroll
            for (int d = 0; d < DP; d += 4) {
                const float4 l = *reinterpret_cast<const float4*>(b + d), h = *reinterpret_cast<const float4*>(b + DP + d);
                on = on && l.x <= hi[d] && l.y <= hi[d + 1] && l.z <= hi[d + 2] && l.w <= hi[d + 3] && h.x >= lo[d] &&
                     h.y >= lo[d + 1] && h.z >= lo[d + 2] && h.w >= lo[d + 3];
            }
            return on;
        };
        // Radius test of a staged node (g of mesh m) and the word's query k.
        auto radius = [&](const float* node, int m, uint32_t g, uint32_t k) {
            const float(*t)[33] = sT[warp];
            const int quick = radiusQuick<DP>(
                node + 2 * DP, [&](int d) { return make_float4(t[d][k], t[d + 1][k], t[d + 2][k], t[d + 3][k]); },
                [&](int d) { return make_float4(t[DP + d][k], t[DP + d + 1][k], t[DP + d + 2][k], t[DP + d + 3][k]); },
                node[3 * DP], sMargin[warp][k]);
            return quick >= 0 ? quick != 0
                              : radiusMeets(a.level[m].x + static_cast<size_t>(g) * D,
                                            a.boxes + static_cast<size_t>(w * 32 + k) * 2 * D, D, a.level[m].nodes[g].rad);
        };
        uint32_t word = 0;  // lane i: node i's
        for (uint32_t v = byUnit ? warp : 0; v < nUnits; v += byUnit ? WARPS : 1) {
            const RangeUnit un = a.upper[unit0 + v];
            uint32_t alive = __ballot_sync(FULL, qv);
            for (int t = 0; t < last && alive; ++t) {
                uint32_t k = un.node;  // the parent, a node of mesh last - 1; its ancestor at mesh t
                for (int up = last - 1; up > t; --up) k = __ldg(a.level[up].parent + k);
                bool on = (alive >> lane) & 1u;
                if (t == last - 1) {
                    on = boxMeets(sParent[v], on);
                    if (on) on = radius(sParent[v], t, k, lane);
                } else if (on) {
                    // (higher ancestors, of indexes of five meshes and more, are few: the exact test alone;
                    // a node whose box misses the query has no survivor below it either way)
                    const float* b = a.level[t].box + static_cast<size_t>(k) * 2 * DP;
#pragma unroll
                    for (int d = 0; d < DP; ++d) on = on && __ldg(b + d) <= hi[d] && __ldg(b + DP + d) >= lo[d];
                    if (on)
                        on = radiusMeets(a.level[t].x + static_cast<size_t>(k) * D, a.boxes + static_cast<size_t>(q) * 2 * D, D,
                                         a.level[t].nodes[k].rad);
                }
                alive = __ballot_sync(FULL, on);
                if (lane == 0 && alive && ((un.pad >> t) & 1u)) {
                    atomicAdd(&sCount[2 * t], __popc(alive));
                    atomicAdd(&sCount[2 * t + 1], __popc(alive) * a.level[t].nodes[k].cnt);
                }
            }
            if (alive == 0) continue;
            for (uint32_t i = 0; i < un.count; ++i) {
                const uint32_t node = v * kRangeUpperUnit + i;
                const uint32_t b = __ballot_sync(FULL, boxMeets(sNode[node], (alive >> lane) & 1u));
                if (static_cast<uint32_t>(lane) == node) word = b;
            }
        }
        // This warp's node of each lane, if any.
        const uint32_t v = lane / kRangeUpperUnit;
        RangeUnit un{0, 0, 0, 0};
        if (v < nUnits && (!byUnit || v % WARPS == static_cast<uint32_t>(warp))) un = a.upper[unit0 + v];
        const bool mine = lane % kRangeUpperUnit < un.count;
        const uint32_t kids = mine ? sKids[lane] : 0u;
        if (kids == 0) word = 0;
        uint32_t inc = __popc(word);
        const uint32_t own = inc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(FULL, inc, o);
            if (lane >= o) inc += t;
        }
        const uint32_t nPairs = __shfl_sync(FULL, inc, 31);
        if (nPairs) {
            uint32_t at = inc - own;
            sWord[warp][lane] = word;
            for (uint32_t left = word; left; left &= left - 1)
                sPairs[warp][at++] = static_cast<uint16_t>(lane * 32 + __ffs(left) - 1);
            __syncwarp();
            for (uint32_t i0 = 0; i0 < nPairs; i0 += 32) {
                const uint32_t i = i0 + lane;
                const uint32_t it = i < nPairs ? sPairs[warp][i] : 0u, node = it >> 5;
                const uint32_t g = __shfl_sync(FULL, un.first, node) + node % kRangeUpperUnit;
                if (i < nPairs && !radius(sNode[node], last, g, it & 31u)) atomicAnd(&sWord[warp][node], ~(1u << (it & 31u)));
            }
            __syncwarp();
            word = sWord[warp][lane];
        }
        if (mine) {
            if (word) {
                atomicAdd(&sCount[2 * last], __popc(word));
                atomicAdd(&sCount[2 * last + 1], __popc(word) * kids);
            }
            a.bits[static_cast<size_t>(un.first + lane % kRangeUpperUnit) * a.words + w] = word;
        }
    }
    __syncthreads();
    if (tid < 2 * (last + 1) && sCount[tid]) atomicAdd(a.hdr + 2 + tid, sCount[tid]);
}

// ---- sweep ----------------------------------------------------------------------------------------
constexpr uint32_t kBlockWords = kRangeTaskQueries / 32;  // most query words of a task

// ROWS: a cluster's hits leave in the order of its rows, as the level-synchronous path returns them at
// dimensions where it tests no point groups; elsewhere in point-group order.
template <int DP, bool ROWS>
struct SweepShape {
    static constexpr int kWarps = DP > 8 ? 2 : 4;             // static shared memory
    static constexpr int kBlocks = 7;                         // resident, for the register allocation
    static constexpr uint32_t kHits = ROWS ? kRangeRowsCluster : 128;  // hits a warp holds before it writes them out
};

// One warp per task. Bound by the latency of a task's loads (unit, bits, boxes, then for the few pairs
// that meet: node, groups, points), so resident warps count: registers are held to seven blocks an SM
// and the rare exact tests are out of line. 24M (query, cluster) pairs of 4,096 boxes (N = 10M, D = 8):
// 143 us; with 2 D float comparisons a pair 180 us.
//
// Once a task has had kHeavyPairs (query, cluster) pairs and three quarters of the blocks' first warps have none any
// more, the rest of it is left to a second launch (SLICES) in a few queries each: boxes that lie together meet
// the same few units with all of their queries, and one warp a task took 6.0 ms (4,096 boxes of +-8% at one
// place, N = 10M, D = 8; the level-synchronous launches 1.2), in slices 0.78.
constexpr uint32_t kHeavyPairs = 64;
template <int DP, bool ROWS, bool SLICES>
__global__ void __launch_bounds__(SweepShape<DP, ROWS>::kWarps * 32, SweepShape<DP, ROWS>::kBlocks) rangeSweepKernel(RangeSweepArgs a, uint32_t nTasks,
                                                                                    uint32_t qPer, uint32_t parts) {
    constexpr int WARPS = SweepShape<DP, ROWS>::kWarps;
    constexpr uint32_t kHits = SweepShape<DP, ROWS>::kHits;
    __shared__ uint16_t sList[WARPS][kBlockWords * 32];
    __shared__ uint16_t sItem[WARPS][32 * kRangeUnit];
    __shared__ __align__(16) float sBox[WARPS][32][2 * DP];
    __shared__ __align__(16) uint32_t sGrid[WARPS][32][DP];  // the same boxes on the grid
    __shared__ float sMargin[WARPS][32];
    __shared__ uint32_t sHit[WARPS][kHits];
    // ROWS: the hits of the (query, cluster) pair at hand, a bit per row of the cluster.
    __shared__ uint32_t sPair[WARPS][ROWS ? kRangeRowsCluster / 32 : 1];
    if constexpr (SLICES) {
        waitForEarlierLaunch();
        if (*a.sliceCnt == 0) return;
    } else if (a.sliced) {
        letNextLaunchStart();
    }
    if (ROWS && (threadIdx.x & 31) < kRangeRowsCluster / 32) sPair[threadIdx.x >> 5][threadIdx.x & 31] = 0;
    __syncwarp();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t lanesLt = (1u << lane) - 1u;
    const uint32_t warps = gridDim.x * WARPS;
    const int D = a.D, H = a.height;
    const RangeSweepLevel& C = a.level[H - 2];
    const int hLast = H - 1;  // header of the clusters that survive
    uint32_t nEntries = 0, nItems = 0, nKept = 0, nTested = 0;

    for (uint32_t task = blockIdx.x * WARPS + w; SLICES || task < nTasks;) {
        uint32_t sliceFrom = 0, sliceN = 0;
        if constexpr (SLICES) {  // the next slice
            uint32_t t = 0;
            if (lane == 0) t = atomicAdd(a.sliceTicket, 1u);
            t = __shfl_sync(FULL, t, 0);
            if (t >= min(*a.sliceCnt, kRangeSlices)) break;
            const uint2 e = a.slices[t];
            task = e.x;
            sliceFrom = e.y & 0xffffu;
            sliceN = e.y >> 16;
        }
        const uint32_t qb = task / (a.nUnits * parts), up = task - qb * a.nUnits * parts;
        const uint32_t u = up / parts, part = up - u * parts;
        // The next task: the first ones are dealt out, the rest claimed.
        uint32_t next = 0;
        if (!SLICES && lane == 0) next = warps + atomicAdd(a.ticket, 1u);
        const RangeUnit un = a.units[u];
        // The task's queries: qPer of them (a power of two) from qb * qPer on; list entries count from qBase.
        const uint32_t qBase = qb * qPer / 32 * 32, wi = qBase / 32 + lane;
        uint32_t word = (wi < a.words && static_cast<uint32_t>(lane) * 32 < qPer)
                            ? a.bits[static_cast<size_t>(un.node) * a.words + wi]
                            : 0u;
        if (qPer < 32) word &= ((1u << qPer) - 1u) << (qb * qPer - qBase);
        uint32_t nLive = __popc(word);
        {
            uint32_t inc = nLive;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(FULL, inc, o);
                if (lane >= o) inc += t;
            }
            uint32_t at = inc - nLive;
            while (word) {
                sList[w][at++] = static_cast<uint16_t>(lane * 32 + __ffs(word) - 1);
                word &= word - 1;
            }
            nLive = __shfl_sync(FULL, inc, 31);
        }
        next = __shfl_sync(FULL, next, 0);
        __syncwarp();
        if (nLive) {
            const uint32_t c = un.first + lane;
            const bool cv = static_cast<uint32_t>(lane) >= un.count * part / parts &&
                            static_cast<uint32_t>(lane) < un.count * (part + 1) / parts && C.nodes[c].cnt > 0;
            // The cluster's box on the grid: lower corners, then upper corners with their guard bits.
            uint32_t clo[DP / 2], chi[DP / 2];
            {
                const uint4* b = reinterpret_cast<const uint4*>(a.clusterGrid + static_cast<size_t>(cv ? c : un.first) * DP);
#pragma unroll
                for (int d = 0; d < DP; d += 4) {
                    const uint4 v = __ldg(b + d / 4);
                    (d < DP / 2 ? clo[d] : chi[d - DP / 2]) = v.x;
                    (d + 1 < DP / 2 ? clo[d + 1] : chi[d + 1 - DP / 2]) = v.y;
                    (d + 2 < DP / 2 ? clo[d + 2] : chi[d + 2 - DP / 2]) = v.z;
                    (d + 3 < DP / 2 ? clo[d + 3] : chi[d + 3 - DP / 2]) = v.w;
                }
            }
            uint32_t taskPairs = 0;
            for (uint32_t from = SLICES ? sliceFrom : 0u; from < (SLICES ? sliceFrom + sliceN : nLive); from += 32) {
                const uint32_t nB = SLICES ? sliceN : min(32u, nLive - from);
                const uint32_t myQ = qBase + (static_cast<uint32_t>(lane) < nB ? sList[w][from + lane] : sList[w][from]);
                __syncwarp();
                for (uint32_t i = lane; i < nB * (DP / 2); i += 32) {  // the outward box, in pieces of 16 bytes
                    const uint32_t k = i / (DP / 2), piece = i % (DP / 2);
                    reinterpret_cast<float4*>(sBox[w][k])[piece] =
                        __ldg(reinterpret_cast<const float4*>(a.boxF + static_cast<size_t>(qBase + sList[w][from + k]) * 4 * DP) + piece);
                }
                for (uint32_t i = lane; i < nB * (DP / 4); i += 32) {
                    const uint32_t k = i / (DP / 4), piece = i % (DP / 4);
                    reinterpret_cast<uint4*>(sGrid[w][k])[piece] =
                        __ldg(reinterpret_cast<const uint4*>(a.boxGrid + static_cast<size_t>(qBase + sList[w][from + k]) * DP) + piece);
                }
                sMargin[w][lane] = a.margin[myQ];
                __syncwarp();
                // Lanes are clusters; every query's box is a broadcast.
                uint32_t bits = 0;
                for (uint32_t k = 0; k < nB; ++k) {
                    const uint32_t* b = sGrid[w][k];  // upper corners with guard bits, then lower corners
                    uint32_t ok = kGuard;
#pragma unroll
                    for (int d = 0; d < DP / 2; d += 2) {
                        const uint2 h = *reinterpret_cast<const uint2*>(b + d), l = *reinterpret_cast<const uint2*>(b + DP / 2 + d);
                        ok &= (h.x - clo[d]) & (h.y - clo[d + 1]);
                        ok &= (chi[d] - l.x) & (chi[d + 1] - l.y);
                    }
                    const uint32_t m = __ballot_sync(FULL, cv && ok == kGuard);
                    if (static_cast<uint32_t>(lane) == k) bits = m;
                }
                // (query, cluster) pairs in order, 32 at a time: float box, then radius.
                uint32_t inc = __popc(bits);
                const uint32_t own = inc;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t t = __shfl_up_sync(FULL, inc, o);
                    if (lane >= o) inc += t;
                }
                const uint32_t nPairs = __shfl_sync(FULL, inc, 31);
                if (nPairs == 0) continue;
                taskPairs += nPairs;
                if (!SLICES && taskPairs > kHeavyPairs && a.sliced && *static_cast<volatile uint32_t*>(a.idle) > gridDim.x / 4 * 3) {
                    const uint32_t per = min(32u, max(1u, 16u * kHeavyPairs / nPairs)), cnt = (nB + per - 1u) / per;
                    uint32_t at = 0;
                    if (lane == 0) at = atomicAdd(a.sliceCnt, cnt);
                    at = __shfl_sync(FULL, at, 0);
                    const bool fits = at < kRangeSlices && cnt <= kRangeSlices - at;  // else no queries, and the warp's own
                    const uint32_t left = nB > lane * per ? nB - lane * per : 0u;
                    if (static_cast<uint32_t>(lane) < cnt && at < kRangeSlices && static_cast<uint32_t>(lane) < kRangeSlices - at)
                        a.slices[at + lane] = make_uint2(task, (from + lane * per) | (fits ? min(per, left) << 16 : 0u));
                    if (fits) continue;
                }
                {
                    uint32_t at = inc - own;
                    while (bits) {
                        sItem[w][at++] = static_cast<uint16_t>(lane * 32 + __ffs(bits) - 1);
                        bits &= bits - 1;
                    }
                }
                __syncwarp();
                // Hits of the query being written (batch index hitQ) and its runs so far.
                uint32_t hitQ = 0xffffffffu, nHit = 0, run = 0;
                auto flush = [&]() {
                    if (nHit == 0) return;
                    __syncwarp();
                    const uint32_t q = __shfl_sync(FULL, myQ, hitQ);
                    uint32_t pos = 0;
                    if (lane == 0) {
                        pos = atomicAdd(a.rawCnt, nHit);
                        const uint32_t slot = atomicAdd(a.qsegs + q, 1u);
                        atomicAdd(a.qcount + q, nHit);
                        if (slot < a.segSlots)
                            a.segs[static_cast<size_t>(q) * a.segSlots + slot] =
                                RangeSegment{(static_cast<uint64_t>(up) << 32) | run, pos, nHit};
                        else
                            atomicOr(a.status, kStatusOverflowItems);
                        if (pos + nHit < pos)  // past 2^32 hits the count no longer tells how many
                            atomicOr(a.status, kStatusOverflowSum);
                        else if (pos + nHit > a.rawCap)
                            atomicOr(a.status, kStatusOverflowEntries);
                    }
                    pos = __shfl_sync(FULL, pos, 0);
                    for (uint32_t i = lane; i < nHit; i += 32)
                        if (pos < a.rawCap && i < a.rawCap - pos) a.raw[pos + i] = sHit[w][i];
                    __syncwarp();
                    nHit = 0;
                    ++run;
                };
                // ROWS: the pair's hits so far join the query's, in row order.
                uint32_t nPair = 0, pairId = 0xffffffffu, pairBase = 0;
                auto closePair = [&]() {
                    if (!ROWS || nPair == 0) return;
                    if (nHit + nPair > kHits) flush();
                    __syncwarp();
                    uint32_t rows = 0;
                    if (static_cast<uint32_t>(lane) < kRangeRowsCluster / 32) {
                        rows = sPair[w][lane];
                        sPair[w][lane] = 0;
                    }
                    uint32_t end = __popc(rows);
                    const uint32_t mine = end;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t t = __shfl_up_sync(FULL, end, o);
                        if (lane >= o) end += t;
                    }
                    for (uint32_t at = nHit + end - mine; rows; rows &= rows - 1)
                        sHit[w][at++] = pairBase + lane * 32 + __ffs(rows) - 1;
                    nHit += nPair;
                    __syncwarp();
                    nPair = 0;
                };
                for (uint32_t i0 = 0; i0 < nPairs; i0 += 32) {
                    const uint32_t i = i0 + lane;
                    const bool pv = i < nPairs;
                    const uint32_t item = pv ? sItem[w][i] : 0u;
                    const uint32_t k = item >> 5, cl = un.first + (item & 31u);
                    const uint32_t q = __shfl_sync(FULL, myQ, k);
                    bool keep = false;
                    NodeRec gr{0.0, 0u, 0u}, cr{0.0, 0u, 0u};
                    if (pv) {
                        cr = C.nodes[cl];
                        const float* b = sBox[w][k];
                        const float4* cb = reinterpret_cast<const float4*>(C.box + static_cast<size_t>(cl) * 2 * DP);
                        keep = true;
#pragma unroll
                        for (int d = 0; d < DP; d += 4) {
                            const float4 cl4 = __ldg(cb + d / 4), ch4 = __ldg(cb + DP / 4 + d / 4);
                            const float4 l = *reinterpret_cast<const float4*>(b + d);
                            const float4 h = *reinterpret_cast<const float4*>(b + DP + d);
                            keep = keep && cl4.x <= h.x && cl4.y <= h.y && cl4.z <= h.z && cl4.w <= h.w && ch4.x >= l.x &&
                                   ch4.y >= l.y && ch4.z >= l.z && ch4.w >= l.w;
                        }
                        if (keep) {
                        const int quick = radiusQuick<DP>(
                            C.xF + static_cast<size_t>(cl) * DP, [&](int d) { return *reinterpret_cast<const float4*>(b + d); },
                            [&](int d) { return *reinterpret_cast<const float4*>(b + DP + d); }, __ldg(C.radF + cl), sMargin[w][k]);
                        keep = quick >= 0 ? quick != 0
                                          : radiusMeets(C.x + static_cast<size_t>(cl) * D,
                                                        a.boxes + static_cast<size_t>(q) * 2 * D, D, cr.rad);
                        }
                        if (keep) {
                            gr = a.clusterGroups[cl];
                            ++nEntries;
                            nItems += a.countRec[cl].cnt;
                        }
                    }
                    // The survivors' groups, laid end to end.
                    uint32_t ginc = keep ? gr.cnt : 0u;
                    const uint32_t gown = ginc;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t t = __shfl_up_sync(FULL, ginc, o);
                        if (lane >= o) ginc += t;
                    }
                    const uint32_t gpre = ginc - gown;
                    const uint32_t nGroups = __shfl_sync(FULL, ginc, 31);
                    for (uint32_t g0 = 0; g0 < nGroups; g0 += 32) {
                        const uint32_t gi = g0 + lane;
                        // The pair whose groups hold gi: the last lane with gpre <= gi among those with groups,
                        // found by bisection over the inclusive sums.
                        int at = 0;
#pragma unroll
                        for (int step = 16; step > 0; step >>= 1) {
                            const uint32_t t = __shfl_sync(FULL, ginc, at + step - 1);
                            if (t <= gi) at += step;
                        }
                        at = min(at, 31);
                        const uint32_t pk = __shfl_sync(FULL, k, at);
                        const uint32_t gFirst = __shfl_sync(FULL, gr.cbeg, at), gp = __shfl_sync(FULL, gpre, at);
                        const bool gv = gi < nGroups;
                        const uint32_t g = gv ? gFirst + (gi - gp) : 0u;
                        bool meets = gv;
                        NodeRec pr{0.0, 0u, 0u};
                        if (gv) {
                            const float4* gb = reinterpret_cast<const float4*>(a.groupBox + static_cast<size_t>(g) * 2 * DP);
                            const float* b = sBox[w][pk];
#pragma unroll
                            for (int d = 0; d < DP; d += 4) {
                                const float4 gl = __ldg(gb + d / 4), gh = __ldg(gb + DP / 4 + d / 4);
                                const float4 l = *reinterpret_cast<const float4*>(b + d);
                                const float4 h = *reinterpret_cast<const float4*>(b + DP + d);
                                meets = meets && gl.x <= h.x && gl.y <= h.y && gl.z <= h.z && gl.w <= h.w && gh.x >= l.x &&
                                        gh.y >= l.y && gh.z >= l.z && gh.w >= l.w;
                            }
                            if (meets) pr = a.groupRec[g];
                        }
                        uint32_t mask = __ballot_sync(FULL, meets);
                        if (meets) {
                            ++nKept;
                            nTested += pr.cnt;
                        }
                        // Points of the kept groups, a point per lane; where registers allow, the next group's load
                        // while one is tested (at D = 8 they cost more resident warps than the overlap gains).
                        constexpr bool kAhead = DP <= 4;
                        float4 pt[DP / 4], ahead[DP / 4];
                        uint32_t rowOf = 0, rowOfAhead = 0;  // ROWS: the point's row
                        auto fetch = [&](int s, float4 (&to)[DP / 4], uint32_t& r) {
                            const uint32_t first = __shfl_sync(FULL, pr.cbeg, s), cnt = __shfl_sync(FULL, pr.cnt, s);
                            if (static_cast<uint32_t>(lane) < cnt) {
                                const float4* p4 = reinterpret_cast<const float4*>(a.pointsF + static_cast<size_t>(first + lane) * DP);
#pragma unroll
                                for (int d = 0; d < DP / 4; ++d) to[d] = __ldg(p4 + d);
                                if constexpr (ROWS) r = __ldg(a.perm + first + lane);
                            }
                        };
                        int s = __ffs(mask) - 1;
                        if (kAhead && mask) fetch(s, pt, rowOf);
                        while (mask) {
                            if (!kAhead) fetch(s, pt, rowOf);
                            mask &= mask - 1;
                            const int nextS = __ffs(mask) - 1;
                            if (kAhead && mask) fetch(nextS, ahead, rowOfAhead);
                            const uint32_t qk = __shfl_sync(FULL, pk, s);
                            const uint32_t first = __shfl_sync(FULL, pr.cbeg, s), cnt = __shfl_sync(FULL, pr.cnt, s);
                            const uint32_t row = first + lane;
                            bool in = false;
                            if (static_cast<uint32_t>(lane) < cnt) {
                                const float* b = sBox[w][qk];
                                const uint32_t qq = qBase + sList[w][from + qk];
                                const float4* inner = reinterpret_cast<const float4*>(a.boxF + (static_cast<size_t>(qq) * 4 + 2) * DP);
                                bool out = false;
                                in = true;
#pragma unroll
                                for (int d = 0; d < DP; d += 4) {
                                    const float4 v = pt[d / 4];
                                    const float4 l = *reinterpret_cast<const float4*>(b + d);
                                    const float4 h = *reinterpret_cast<const float4*>(b + DP + d);
                                    const float4 li = __ldg(inner + d / 4), hin = __ldg(inner + DP / 4 + d / 4);
                                    in = in && v.x > li.x && v.y > li.y && v.z > li.z && v.w > li.w && v.x < hin.x &&
                                         v.y < hin.y && v.z < hin.z && v.w < hin.w;
                                    out = out || v.x < l.x || v.y < l.y || v.z < l.z || v.w < l.w || v.x > h.x || v.y > h.y ||
                                          v.z > h.z || v.w > h.w;
                                }
                                if (!in && !out)  // a coordinate within float rounding of a face
                                    in = pointInside(a.pointsD + static_cast<size_t>(ROWS ? rowOf : row) * D,
                                                     a.boxes + static_cast<size_t>(qq) * 2 * D, D);
                            }
                            const uint32_t hb = __ballot_sync(FULL, in);
                            if (hb) {  // warp-uniform
                                if constexpr (ROWS) {
                                    const uint32_t id = i0 + __shfl_sync(FULL, at, s);
                                    if (id != pairId) {
                                        closePair();
                                        pairId = id;
                                        pairBase = __shfl_sync(FULL, cr.cbeg, static_cast<int>(id - i0));
                                    }
                                }
                                if (qk != hitQ) {
                                    flush();
                                    hitQ = qk;
                                    run = 0;
                                } else if (!ROWS && nHit + 32 > kHits) {
                                    flush();
                                }
                                if constexpr (ROWS) {
                                    const uint32_t r = rowOf - pairBase;
                                    if (in) atomicOr(&sPair[w][r >> 5], 1u << (r & 31u));
                                } else {
                                    if (in) sHit[w][nHit + __popc(hb & lanesLt)] = row;
                                    nHit += __popc(hb);
                                }
                                if constexpr (ROWS) nPair += __popc(hb);
                            }
                            if constexpr (kAhead) {
#pragma unroll
                                for (int d = 0; d < DP / 4; ++d) pt[d] = ahead[d];
                                rowOf = rowOfAhead;
                            }
                            s = nextS;
                        }
                    }
                }
                closePair();
                flush();
            }
        }
        __syncwarp();
        task = next;
    }
    if (!SLICES && threadIdx.x == 0 && a.sliced) atomicAdd(a.idle, 1u);
    nEntries = __reduce_add_sync(FULL, nEntries);
    nItems = __reduce_add_sync(FULL, nItems);
    nKept = __reduce_add_sync(FULL, nKept);
    nTested = __reduce_add_sync(FULL, nTested);
    if (lane == 0 && nEntries) {
        atomicAdd(a.hdr + 2 * hLast, nEntries);
        atomicAdd(a.hdr + 2 * hLast + 1, nItems);
        atomicAdd(a.hdr + 2 * (H + 3), nKept);
        atomicAdd(a.hdr + 2 * (H + 3) + 1, nTested);
    }
}

// ---- gather ---------------------------------------------------------------------------------------

// One block per (query, share of its results). Orders the query's segments by key (counting for a few,
// a bitonic network for many), then every thread finds its results' segments by bisection.
template <int THREADS>
__global__ void __launch_bounds__(THREADS) rangeGatherKernel(RangeSweepArgs a, uint32_t shares, uint32_t slotCap,
                                                                   int scanned) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t* sKey = reinterpret_cast<uint64_t*>(smem);
    uint32_t* sSlot = reinterpret_cast<uint32_t*>(sKey + slotCap);
    uint32_t* sEnd = sSlot + slotCap;  // inclusive lengths, in order (a segment's first hit then replaces its slot)
    __shared__ unsigned long long sBase;
    __shared__ unsigned long long sWarp[THREADS / 32];
    __shared__ uint32_t sCarry, sW32[THREADS / 32];
    const uint32_t q = blockIdx.x / shares, share = blockIdx.x - q * shares;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (*a.status) return;
    // Results of the queries before this one.
    unsigned long long sum = 0;
    for (uint32_t i = tid; !scanned && i < q; i += THREADS) sum += a.qcount[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(FULL, sum, o);
    if (lane == 0) sWarp[warp] = sum;
    __syncthreads();
    if (tid == 0) {
        unsigned long long t = 0;
        for (int i = 0; i < THREADS / 32; ++i) t += sWarp[i];
        if (scanned) t = a.offsets[q];
        sBase = t;
        if (share == 0) {
            if (!scanned) a.offsets[q] = t;
            if (q == a.nq - 1) {
                if (!scanned) a.offsets[a.nq] = t + a.qcount[q];
                a.hdr[2 * a.height] = static_cast<uint32_t>(t + a.qcount[q]);
                if (t + a.qcount[q] > a.resultCap) atomicOr(a.status, kStatusOverflowEntries);
            }
        }
        sCarry = 0;
    }
    __syncthreads();
    const uint32_t total = a.qcount[q];
    const uint32_t n = min(a.qsegs[q], min(a.segSlots, slotCap));
    const unsigned long long base = sBase;
    if (total == 0 || base + total > a.resultCap) return;
    const uint32_t per = max(8u * THREADS, (total + shares - 1) / shares);
    const uint32_t r0 = share * per < total ? share * per : total, r1 = min(total, r0 + per);
    if (r0 >= r1) return;
    const RangeSegment* segs = a.segs + static_cast<size_t>(q) * a.segSlots;
    if (n == 1) {
        if (tid == 0) {
            sSlot[0] = segs[0].pos;
            sEnd[0] = segs[0].len;
        }
        __syncthreads();
    } else {
        uint32_t size = 1;
        while (size < n) size <<= 1;
        for (uint32_t i = tid; i < size; i += THREADS) {
            sKey[i] = i < n ? segs[i].key : ~0ull;
            sSlot[i] = i;
        }
        __syncthreads();
        if (n <= THREADS) {
            uint32_t place = 0;
            if (static_cast<uint32_t>(tid) < n) {
                const uint64_t k = sKey[tid];
                for (uint32_t i = 0; i < n; ++i) place += sKey[i] < k ? 1u : 0u;
            }
            __syncthreads();
            if (static_cast<uint32_t>(tid) < n) sSlot[place] = tid;
        } else {
            for (uint32_t s = 2; s <= size; s <<= 1)
                for (uint32_t stride = s >> 1; stride > 0; stride >>= 1) {
                    for (uint32_t t = tid; t < size / 2; t += THREADS) {
                        const uint32_t lo = 2 * t - (t & (stride - 1)), hi = lo + stride;
                        const bool asc = (lo & s) == 0;
                        if (asc == (sKey[lo] > sKey[hi])) {
                            const uint64_t k = sKey[lo];
                            sKey[lo] = sKey[hi];
                            sKey[hi] = k;
                            const uint32_t v = sSlot[lo];
                            sSlot[lo] = sSlot[hi];
                            sSlot[hi] = v;
                        }
                    }
                    __syncthreads();
                }
        }
        __syncthreads();
        for (uint32_t i0 = 0; i0 < n; i0 += THREADS) {
            const uint32_t i = i0 + tid;
            uint32_t inc = i < n ? segs[sSlot[i]].len : 0u;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(FULL, inc, o);
                if (lane >= o) inc += t;
            }
            if (lane == 31) sW32[warp] = inc;
            __syncthreads();
            uint32_t before = sCarry;
            for (int x = 0; x < warp; ++x) before += sW32[x];
            if (i < n) {
                sEnd[i] = before + inc;
                sSlot[i] = segs[sSlot[i]].pos;
            }
            __syncthreads();
            if (tid == THREADS - 1) sCarry = before + inc;
            __syncthreads();
        }
    }
    for (uint32_t r = r0 + tid; r < r1; r += THREADS) {
        uint32_t lo = 0, hi = n - 1;  // the first segment that ends past r
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (sEnd[mid] > r) hi = mid; else lo = mid + 1;
        }
        const uint32_t row = a.raw[sSlot[lo] + (r - (lo ? sEnd[lo - 1] : 0u))];
        a.ids[base + r] = a.map[a.rowOrder ? row : __ldg(a.perm + row)];
        if (a.vals) {
            const double* y = a.pointsD + static_cast<size_t>(row) * a.D;
            double* out = a.vals + (base + r) * a.D;
            for (int d = 0; d < a.D; ++d) out[d] = __ldg(y + d);
        }
    }
}

int residentBlocks(const void* kern, int threads) {
    int dev = 0, sms = 0, perSm = 0;
    TBLAEQ_CUDA(cudaGetDevice(&dev));
    TBLAEQ_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    TBLAEQ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kern, threads, 0));
    return std::max(1, sms * std::max(1, perSm));
}

template <int DP, bool ROWS>
void launchPadded(const RangeSweepArgs& a, cudaStream_t s) {
    // A word per warp, several in turn only where that still leaves eight blocks an SM; in batches too
    // small to fill the GPU that way, a unit per warp and a word per block.
    const uint32_t chunks = std::max(1u, (a.nUpper + kUpperChunk - 1) / kUpperChunk);
    constexpr uint32_t uw = upperWarps<DP>();
    const uint64_t wordSteps = (a.words + uw - 1) / uw;
    const bool byUnit = chunks * wordSteps < 592;
    const uint32_t steps = static_cast<uint32_t>(std::max<uint64_t>(1, std::min<uint64_t>(16, chunks * wordSteps / 1184)));
    const uint32_t perBlock = byUnit ? 1 : steps * uw;
    const uint32_t wordBlocks = (a.words + perBlock - 1) / perBlock;  // (useRangeSweep bounds nodes x words)
    rangeUpperKernel<DP><<<chunks * wordBlocks, uw * 32, 0, s>>>(a, perBlock, wordBlocks, byUnit ? 1 : 0);
    TBLAEQ_LAUNCHED();
    constexpr int WARPS = SweepShape<DP, ROWS>::kWarps;
    static const int full = residentBlocks(reinterpret_cast<const void*>(rangeSweepKernel<DP, ROWS, false>), WARPS * 32);
    const RangeSweepTasks t = rangeSweepTasks(a.nUnits, a.nq);
    const uint32_t nTasks = static_cast<uint32_t>(t.count);
    const uint32_t blocks = std::min<uint32_t>(static_cast<uint32_t>(full), (nTasks + WARPS - 1) / WARPS);
    // (Tasks of fewer queries are short enough: the second launch costs about 5 us where it has nothing to do.)
    RangeSweepArgs b = a;
    b.sliced = std::min(a.nq, t.qPer) >= 128;
    rangeSweepKernel<DP, ROWS, false><<<std::max(1u, blocks), WARPS * 32, 0, s>>>(b, nTasks, t.qPer, t.parts);
    TBLAEQ_LAUNCHED();
    if (b.sliced) {
        launchEarly(rangeSweepKernel<DP, ROWS, true>, std::max(1, full / 2), WARPS * 32, s, b, nTasks, t.qPer, t.parts);
    }
    // A few queries may hold many results each, and every block of a query orders all of its segments: large
    // blocks share a query then, about as many as are resident at once, at least 4,096 results each. 20 boxes
    // with 6.4M results (N = 1M, D = 2): the gather takes 132 us; 590 us with 236 shares of 128 threads,
    // 180 us with 88 of 512. 300 boxes with 14.9M: 520 us for the batch with four shares, 630 with one.
    const bool few = a.nq <= 592;
    const uint32_t shares = few ? std::max(4u, 592u / a.nq) : std::max<uint32_t>(1u, 4736u / a.nq);
    // Each block sums the counts before its query, unless that many reads would cost more than a scan.
    const bool scanned = a.nq > 8192;
    if (scanned) launchExclusiveScan(a.qcount, a.offsets, a.nq, s);
    const uint32_t slotCap = std::min(a.segSlots, kRangeSegments);
    uint32_t pow2 = 1;
    while (pow2 < slotCap) pow2 <<= 1;
    if (few)
        rangeGatherKernel<512><<<a.nq * shares, 512, pow2 * 16, s>>>(a, shares, pow2, scanned ? 1 : 0);
    else
        rangeGatherKernel<128><<<a.nq * shares, 128, pow2 * 16, s>>>(a, shares, pow2, scanned ? 1 : 0);
    TBLAEQ_LAUNCHED();
}

}  // namespace

uint64_t rangeSweepBitBytes(uint64_t lastUpper, uint64_t nq) { return lastUpper * ((nq + 31) / 32) * 4; }

void launchRangeSweep(const RangeSweepArgs& a, cudaStream_t s) {
    switch (a.D) {  // the dimensions whose point groups the level-synchronous path tests too
        case 4: if (!a.rowOrder) return launchPadded<4, false>(a, s); break;
        case 8: if (!a.rowOrder) return launchPadded<8, false>(a, s); break;
        case 16: if (!a.rowOrder) return launchPadded<16, false>(a, s); break;
        default: break;
    }
    switch (paddedDims(static_cast<uint64_t>(a.D))) {
        case 4: return launchPadded<4, true>(a, s);
        case 8: return launchPadded<8, true>(a, s);
        case 12: return launchPadded<12, true>(a, s);
        case 16: return launchPadded<16, true>(a, s);
        case 20: return launchPadded<20, true>(a, s);
        case 24: return launchPadded<24, true>(a, s);
        case 28: return launchPadded<28, true>(a, s);
        case 32: return launchPadded<32, true>(a, s);
        default: throw std::invalid_argument("range sweep: D must be in [1, 32]");
    }
}

}  // namespace tblaeq
