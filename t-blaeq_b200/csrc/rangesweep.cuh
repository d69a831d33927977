// Exact range batches in three launches (four with slices): upper test, sweep, gather.
//
//   upper   a warp per word of 32 queries, a query a lane, over staged units of at most eight sibling
//           nodes of the mesh above the finest clusters: bit (node, query) = the node and its ancestors
//           survive for the query;
//   sweep   one warp per (unit, up to 1,024 queries), a unit being at most 32 sibling clusters: lanes are
//           clusters while their boxes are tested against the queries whose bit is set, then
//           (query, cluster) pairs, then (query, group) pairs, then points. Hits go out as segments:
//           runs of points of one query and one unit, in traversal order;
//   gather  per query, its segments in the order of their units, as ids (and coordinates).
//
// Against one launch per level this keeps nothing between the levels in memory: no frontier with its
// coordinates, no look-back, no per-level tail. Every (query, node) pair is decided as there: float box, FP64
// radius (in float first, outside a margin), float point with the FP64 test near a face. So the same
// nodes survive at every level, the counts per level are the same, and so are the results and their
// order (depth-first: queries, then the clusters in traversal order, then the points: in point-group
// order at D = 4, 8 and 16, in row order elsewhere).
//
// Measured on B200 against the level-synchronous launches, device time of one batch: 4,096 boxes, N = 10M,
// D = 8: 620 -> 220 us; 37 boxes there: 105 -> 46 us; 100 boxes, N = 500k, D = 5: 110 -> 60 us; one box:
// 60 -> 28 us; 301 boxes with 1.0M results and their coordinates, N = 1.5M, D = 3: 180 -> 140 us.
#pragma once

#include <cstdint>

#include "common.cuh"
#include "traverse.cuh"

namespace tblaeq {

constexpr uint32_t kRangeUnit = 32;        // clusters per unit
constexpr uint32_t kRangeSegments = 2048;  // segments of a query the gather can order
constexpr uint32_t kRangeMaxHeight = 16;
// Most points of a cluster at dimensions whose hits leave in row order (sorted per cluster on chip).
constexpr uint32_t kRangeRowsCluster = 512;

// At most kRangeUnit consecutive children (finest clusters) of one node of the mesh above.
struct RangeUnit {
    uint32_t node, first, count;
    uint32_t pad;  // upper units: bit t = the first unit below its ancestor of mesh t
};
constexpr uint32_t kRangeUpperUnit = 8;    // nodes of an upper unit

// Steps of a box coordinate on the grid of the data's extent (see rangesweep.cu); the host lays out the
// clusters' boxes with the same functions.
constexpr double kRangeGrid = 32767.0;
__host__ __device__ inline double rangeGridStep(double v, double lo, double scale) {
#ifdef __CUDA_ARCH__
    return __dmul_rn(__dsub_rn(v, lo), scale);
#else
    return (v - lo) * scale;
#endif
}
__host__ __device__ inline uint32_t rangeGridLower(double v, double lo, double scale) {
    const double s = rangeGridStep(v, lo, scale);  // not a number: 0, which every cluster's box meets
    return s >= kRangeGrid ? static_cast<uint32_t>(kRangeGrid) : s > 0.0 ? static_cast<uint32_t>(s) : 0u;
}
__host__ __device__ inline uint32_t rangeGridUpper(double v, double lo, double scale) {
    const double s = rangeGridStep(v, lo, scale);
    if (!(s < kRangeGrid)) return static_cast<uint32_t>(kRangeGrid);
    if (!(s > 0.0)) return 0u;
    const uint32_t f = static_cast<uint32_t>(s);
    return f + (static_cast<double>(f) < s ? 1u : 0u);
}

// Tasks of the sweep: `parts` parts of a unit's clusters by blocks of qPer queries. Large batches take whole
// units and as many queries as leave several tasks for every resident warp; small ones split both, so that
// a query that holds a whole unit is not one warp's serial work (1.0M results of 301 boxes, D = 3: the
// sweep takes 179 us with whole units, 92 us in parts).
constexpr uint32_t kRangeTaskQueries = 1024;
constexpr uint64_t kRangeTasksMax = 1ull << 31;  // the tasks' numbers, and the ticket that runs past them, have 32 bits
struct RangeSweepTasks {
    uint32_t parts, qPer;
    uint64_t count;
};
inline RangeSweepTasks rangeSweepTasks(uint64_t nUnits, uint64_t nq) {
    RangeSweepTasks t{};
    const uint64_t pairs = nUnits * nq;
    t.parts = pairs >= (4u << 20) ? 1u : pairs >= (1u << 20) ? 2u : 4u;
    t.qPer = kRangeTaskQueries;
    while (t.qPer > 4 && nUnits * t.parts * ((nq + t.qPer - 1) / t.qPer) < 12288) t.qPer >>= 1;
    t.count = nUnits * t.parts * ((nq + t.qPer - 1) / t.qPer);
    return t;
}

// Whether the level-synchronous launches serve a batch sooner than the sweep: on indexes of small fan-outs,
// whose units are mostly empty lanes and whose last upper mesh is most of the hierarchy. `top`, `upper` and
// `clusters` are the nodes of mesh 0, the last upper mesh and the finest clusters. Three cases, each on
// an index of many units and fewer than twelve clusters a node, measured as sweep / levels in us:
// - few queries: 0.8 ns a task against about 40 us of saved launches and, a query, 0.01 ns a node of mesh 0
//   and 0.3 us. One box: fan-outs 2, N = 1M, D = 8: 801 / 96; fan-outs 4, D = 5, N = 2M: 411 / 79; fan-outs
//   6, N = 1M: 125 / 100. 100 boxes there: 108 / 167 with fan-outs 6, 170 / 186 with 4.
// - fan-outs below four: 8,000 boxes, fan-outs 2, N = 1M: 12,028 / 9,612; fan-outs 3, N = 3M: 8,444 / 5,489;
//   fan-outs 4, N = 1M: 2,122 / 2,388.
// - five meshes and more, below eight: fan-outs 5, N = 1M: 100 boxes 136 / 174, 1,000 398 / 293, 8,000 2,400 / 1,080.
inline bool rangeSweepNarrow(uint64_t height, uint64_t top, uint64_t upper, uint64_t clusters, uint64_t nUnits, uint64_t nq) {
    if (height <= 2 || nUnits <= 16384 || clusters >= 12 * upper) return false;
    return rangeSweepTasks(nUnits, nq).count > 50000 + nq * (375 + 12 * top / 1000) ||
           (clusters < 4 * upper && (nUnits > 65536 || nq >= 2048)) || (height >= 5 && clusters < 8 * upper && nq >= 512);
}

constexpr uint32_t kRangeSlices = 1u << 18;  // slices of a launch; batches beyond are not sliced

struct RangeSegment {
    uint64_t key;  // unit, then the run's number within it
    uint32_t pos;  // first hit
    uint32_t len;
};

struct RangeSweepLevel {
    const float* box;       // two padded rows: lo, hi, rounded outward
    const double* x;        // decoded centres
    const float* xF;        // the same, padded float rows
    const float* radF;      // subtree radius, rounded up
    const NodeRec* nodes;   // subtree radius, first child, child count
    const uint32_t* parent; // position in the mesh above (null for mesh 0)
    uint32_t count;
};

struct RangeSweepArgs {
    int D, height;
    uint32_t nq, words;
    const double* boxes;    // nq x (lo[D] hi[D])
    float* boxF;            // nq x 4 padded rows: outward lo, hi, inward lo, hi
    float* margin;          // nq: see radiusQuick
    uint32_t* boxGrid;      // nq x paddedDims: upper corners (guard bits set), lower corners, two to a word
    const uint32_t* clusterGrid;  // per finest cluster: lower corners, upper corners (guard bits set)
    double gridMin[32], gridScale[32];
    float maxAbs;           // largest |coordinate| of the data, rounded up
    float marginScale;      // margin = (largest |box coordinate| + maxAbs) * marginScale
    RangeSweepLevel level[kRangeMaxHeight];  // meshes 0 .. height-2
    const RangeUnit* units; // in traversal order
    uint32_t nUnits;
    const RangeUnit* upper; // siblings of mesh height-3 (node: their parent)
    uint32_t nUpper;
    int rowOrder;           // pointsD (and the hits) are in row order, not in point-group order
    const NodeRec* clusterGroups;
    const NodeRec* groupRec;
    const float* groupBox;
    const NodeRec* countRec;  // what a surviving cluster adds to the finest level's count
    const float* pointsF;
    const double* pointsD;
    const uint32_t* perm;
    const uint64_t* map;
    uint32_t* bits;         // last upper mesh (or one virtual root) x words
    uint32_t* raw;          // hits: rows of the points
    uint32_t rawCap;
    RangeSegment* segs;     // nq x segSlots
    uint32_t segSlots;
    int sliced;             // set at the launch: batches of many pairs are left as slices
    uint2* slices;          // kRangeSlices of (task, first list entry | queries << 16)
    // Zeroed before the launch:
    uint32_t* sliceCnt;
    uint32_t* sliceTicket;
    uint32_t* idle;         // blocks of the sweep whose first warp has no task any more
    uint32_t* ticket;
    uint32_t* rawCnt;
    uint32_t* qsegs;        // segments per query
    uint32_t* qcount;       // hits per query
    uint32_t* hdr;          // the engine's level headers
    uint32_t* status;
    // Results
    uint64_t* offsets;
    uint64_t* ids;
    double* vals;
    uint32_t resultCap;
};

// kStatusOverflowItems here: a query has more segments than segSlots; kStatusOverflowSum: more than 2^32
// hits (rawCnt and the headers tell the other capacities).
void launchRangeSweep(const RangeSweepArgs& a, cudaStream_t s);
// (query, unit block) tasks etc. are sized inside; bytes of `bits` for nq queries:
uint64_t rangeSweepBitBytes(uint64_t lastUpper, uint64_t nq);

}  // namespace tblaeq
