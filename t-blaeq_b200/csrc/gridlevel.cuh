// One level of the per-level plugin (IQueryStrategy::runLevel) for grids of moderate size.
//
// The grid's entries are kept by the reference's predicate -- range: box distance against the radius;
// KNN: the STEP set -- and every kept entry's children are written out in order. STEP needs no sort:
// an entry belongs to the part that sets the running bound when the children of the entries before
// it (by lower bound, then by place) number less than K, which is a sum over the grid, and every later
// entry is taken by its bound alone. Four launches (range: three) and one wait replace the sort's
// tile and merge launches, STEP in one CTA, and two persistent expands with their look-back. The query
// travels in the launch arguments. One KNN call (launches, wait and all): 7 entries 97 -> 38 us, 156
// entries 109 -> 38 us, 3,645 entries with 38,400 outputs 145 -> 64 us.
#pragma once

#include <cstdint>

#include "common.cuh"
#include "traverse.cuh"

namespace tblaeq {

// Largest grid of this path: the sums take p^2 / 2 comparisons (16,384 entries: 134M) and one CTA scans
// the kept counts. Larger grids sort, and from half of that on those whose K reaches far into the grid, as the
// sums end at K: above an eighth of its children (estimated from the meshes' sizes). Counted / sorted, a call:
// 8,000 entries, K = all 1M children: 150 / 192 us; 16,129 entries, K = 3% 196 / 197, all 322 / 225; 15,625
// entries, K = 2% 485 / 507, half 614 / 544. (At D = 32, where the sorted path's expands carry long rows, 507 / 714
// for all of 16,129 entries.)
constexpr uint64_t kGridLevelMax = 16384;
inline bool gridLevelCounts(uint64_t p, uint64_t D, bool knn, uint64_t K, uint64_t nodes, uint64_t children) {
    if (p == 0 || p > kGridLevelMax) return false;
    return !knn || p <= kGridLevelMax / 2 || D >= 16 || static_cast<double>(K) * static_cast<double>(nodes) * 8.0 <=
                                                 static_cast<double>(p) * static_cast<double>(children);
}

struct GridLevelArgs {
    const uint64_t* ids;
    const double* vals;
    uint32_t p;
    int D;
    int knn;
    double q[64];            // range: lo[D] hi[D]; KNN: the point
    uint64_t K;
    const NodeRec* nodes;    // by original id: the reference's radius, first child row, children
    const double* rows;
    int rowsOnHost;
    const uint64_t* map;
    // Scratch (p entries each; prefix p + 1)
    uint64_t* keys;
    double* reach;
    uint32_t* cnt;
    uint8_t* first;
    uint32_t* prefix;
    unsigned long long* bound;  // [0] bits of the running bound, [1] outputs; zeroed here
    uint64_t* outIds;
    double* outVals;
    uint32_t outCap;
};

size_t gridLevelScratchBytes(uint64_t p);
void gridLevelScratch(GridLevelArgs& a, void* scratch);
void launchGridLevel(const GridLevelArgs& a, cudaStream_t s);

}  // namespace tblaeq
