// Exact KNN batches as a probe and one sweep over the finest clusters.
//
// Two facts carry the design. (1) The K-th distance within the few clusters whose centres lie nearest
// the query is within a few percent of the true K-th distance (measured over the synthetic indexes,
// D = 3..16, K = 10..100: 1.00-1.06 of it with 17 clusters), so one bound per query, taken from them,
// leaves almost nothing for a second one to prune. (2) Testing every (query, cluster) pair against
// that bound is cheap when it is dense: a pair is one product on the matrix units, with no list, sort
// or atomic.
//
//   probe   one CTA per query walks down from the root with a beam, takes the points of its
//           best-ranked clusters and selects their K-th distance (tau);
//   bound   a warp holds 32 clusters and walks 256 queries: bit (cluster, query) = the cluster's
//           sphere reaches within tau of the query;
//   sweep   one warp per cluster gathers the queries whose bit is set, 32 at a time, tests them
//           against the cluster's point groups (boxes), and the groups' points against the queries
//           whose box test passed, one point per lane, or above eight dimensions against all 32 as
//           a product. Clusters that many queries reach go to a second launch in slices of their
//           queries (batches above 512, up to eight dimensions);
//   finish  per query, the K smallest candidates by (FP64 squared distance, id).
//
// The tests run in single precision with a margin that covers every rounding (sweepPrepareKernel in
// knnsweep.cu), so they only ever let too much through; a point that passes is measured in FP64 from
// the decoded coordinates (fma in dimension order) before it becomes a candidate. The candidates
// are therefore exactly the points whose FP64 squared distance lies within tau^2 (1 + 1e-9).
//
// Measured on B200 against the level-synchronous walk (beam, wave 1, node-major completion in two
// refinement stages; about 90 launches), device time of one batch: 4,096 queries, K = 20 / 100, N = 10M,
// D = 8: 11.4 -> 0.86 ms; 300 queries there: 3.0 -> 0.20 ms; one query: 0.38 -> 0.08 ms; 1,000 queries,
// N = 5M, D = 16, scored: 40 -> 2.15 ms.
#pragma once

#include <cstdint>

#include "common.cuh"
#include "traverse.cuh"

namespace tblaeq {

// Floats per row of the padded float copies (points, boxes, centres): D rounded up to 16 bytes.
constexpr uint32_t paddedDims(uint64_t D) { return static_cast<uint32_t>((D + 3) / 4 * 4); }

// Largest |coordinate| (data or query) the float tests take: squared distances stay finite.
constexpr double kSweepMaxAbs = 1e18;
// Batches and clusters of more queries are sliced (sweepClusters). Up to it a cluster is one warp's work, 1.4 ms
// at worst (512 queries at one place, K = 100, N = 1M, D = 3), as long as the level-synchronous walk takes.
constexpr uint32_t kSweepSliced = 512;
// Points a probe reads at most (its selection stage), and so the largest K it can bound.
constexpr uint32_t kProbePoints = 4096;
constexpr uint32_t kSweepMaxHeight = 16;
// Most times 4 K + 64 candidate slots a query that batches keep for the ones after them (a power of four): with a
// scorer and small K single queries need more than 64 (N = 100M, D = 8), and a second run on every batch.
constexpr uint32_t kSweepFactorMax = 256;
// An index of at most this many times 4 K + 64 points is swept also without a bound.
constexpr uint32_t kSweepWhole = 64;

struct KnnSweepLevel {
    const float* x;        // centres, paddedDims floats per node
    const float* rad;      // subtree radius, rounded up
    const NodeRec* nodes;  // first child and child count
    const uint32_t* leaf;  // finest points below
    uint32_t count;
};

struct KnnSweepArgs {
    int D, height;
    uint32_t nq;
    const double* points;   // nq x D
    const uint32_t* K;
    double maxAbs;          // largest |coordinate| of the data
    uint64_t nPoints;
    KnnSweepLevel level[kSweepMaxHeight];  // meshes 0 .. height-2
    // Finest points in point-group order, and the groups.
    const float* pointsF;
    const double* pointsD;
    const uint32_t* perm;
    int rowOrder;           // pointsD is in row order (row perm[i] holds point i), not in point-group order
    const uint64_t* map;
    const NodeRec* clusterGroups;
    const NodeRec* groupRec;
    const float* groupBox;
    // Per query: float coordinates (dead queries far away), margin, bound.
    float* qF;              // nq x paddedDims
    float* margin;          // nq
    double* tau;            // nq
    float* tauF;            // nq: tau + margin, rounded up
    float* thrF;            // nq: squared, with the arithmetic's relative margin
    uint64_t* outOff;       // nq + 1: results (min(K, nPoints) each)
    uint64_t* candOff;      // nq + 1: candidate slots
    uint32_t* candCnt;      // nq
    uint64_t candCap;       // slots in all
    uint32_t candFactor;       // slots per query: candFactor * (4 K + 64),
    const uint32_t* candWant;  // or this where it is more (nq, or null)
    uint64_t* candId;
    double* candD2;
    uint32_t beam;
    double waveFactor;      // wave scale / points per cluster (see BatchEngine::setWaveScale)
    // Cluster-level probe entries for a scorer: entries [entOff[q], + entCnt[q]) of query and node.
    uint32_t* entOff;
    uint32_t* entCnt;
    uint32_t* entQ;
    uint32_t* entNode;
    const double* score;
    uint32_t entCap;
    // Bit per (cluster, query of the block), `words` words a cluster.
    uint32_t* bits;
    uint32_t words;
    uint32_t qBegin, qEnd;  // the block
    uint32_t* live;         // clusters with a bit set (blocks of at most 256 queries)
    uint32_t* liveCnt;
    uint32_t* ticket;
    // Clusters that many queries reach (cluster, first of 32 words, queries there), at most one entry per 32
    // words of every cluster: see sweepClusters.
    int sliced;             // blocks above kSweepSliced queries, up to eight (padded) dimensions
    uint4* heavy;
    uint32_t* heavyCnt;
    uint32_t* heavyTicket;
    unsigned long long* reached;  // bits set
    uint32_t* hdr;          // the engine's level headers: (entries, items) of levels 0 .. height + 1
    unsigned long long* total; // results of the batch
    unsigned long long* work;  // [0] points the probe measured, [1] points the sweep tested
    uint32_t* status;
};

// kStatusOverflowItems here: a query has more candidates than slots; counting goes on to the end of the
// batch. Bits of KnnSweepArgs::status beyond DeviceStatus: this batch needs the level-synchronous path (a
// coordinate beyond kSweepMaxAbs or not finite, a K beyond the probe's stage, or fewer candidates than
// neighbours).
constexpr uint32_t kStatusKnnFallback = 1u << 5;

void launchKnnSweepPrepare(const KnnSweepArgs& a, cudaStream_t s);
enum KnnProbePhase { kProbeWhole = 0, kProbeEntries = 1, kProbeBound = 2 };
void launchKnnProbe(const KnnSweepArgs& a, KnnProbePhase phase, cudaStream_t s);
void launchKnnSweepBound(const KnnSweepArgs& a, cudaStream_t s);
void launchKnnSweepPoints(const KnnSweepArgs& a, cudaStream_t s);

}  // namespace tblaeq
