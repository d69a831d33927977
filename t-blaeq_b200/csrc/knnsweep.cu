// Exact KNN: probe, dense cluster bound and point sweep (see knnsweep.cuh).
#include "knnsweep.cuh"

#include <algorithm>
#include <type_traits>

namespace tblaeq {

namespace {

constexpr uint32_t FULL = 0xffffffffu;
constexpr float kRel = 1.00001f;  // the float sums' relative error: (D + 3) 2^-24 < 2.1e-6 for D <= 32
// What underflow can take from a float square, and from its root: D + 3 roundings of at most the smallest
// normal float each, under 1e-36.
constexpr double kTiny2 = 1e-36, kTiny = 1e-18;

__device__ __forceinline__ uint32_t floatKey(float f) {  // order-preserving bits
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// ---- prepare: float queries, result and candidate slots ------------------------------------------
// One block scans K (results are min(K, points) per query, known before any search); all blocks convert
// the queries. margin[q] bounds the distance error of rounding the query's and a data point's
// coordinates to float: sqrt(D) 2^-24 (|q| + |x|) each way, doubled.
__global__ void __launch_bounds__(1024) sweepPrepareKernel(KnnSweepArgs a, uint32_t DP) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (uint32_t q = blockIdx.x * blockDim.x + tid; q < a.nq; q += gridDim.x * blockDim.x) {
        double m = 0.0;
        bool ok = true;
        const uint32_t K = a.K[q];
        for (int d = 0; d < a.D; ++d) {
            const double p = a.points[static_cast<size_t>(q) * a.D + d];
            ok = ok && fabs(p) <= kSweepMaxAbs;  // false for NaN
            m = fmax(m, fabs(p));
        }
        if (!ok || K > kProbePoints / 2) atomicOr(a.status, kStatusKnnFallback);
        for (uint32_t d = 0; d < DP; ++d)
            a.qF[static_cast<size_t>(q) * DP + d] =
                d >= static_cast<uint32_t>(a.D) ? 0.f
                : K == 0                        ? static_cast<float>(kSweepMaxAbs)
                                                : static_cast<float>(a.points[static_cast<size_t>(q) * a.D + d]);
        a.margin[q] = __double2float_ru(sqrt(static_cast<double>(a.D)) * (m + a.maxAbs) * 1.2e-7);
        a.candCnt[q] = 0;
    }
    if (blockIdx.x) return;
    __shared__ unsigned long long sCarryR, sCarryC, sR[32], sC[32];
    if (tid == 0) {
        sCarryR = sCarryC = 0;
        *a.liveCnt = 0;
        *a.ticket = 0;
        *a.heavyCnt = 0;
        *a.heavyTicket = 0;
        *a.reached = 0;
        a.work[0] = a.work[1] = 0;
    }
    __syncthreads();
    for (uint32_t base = 0; base < a.nq; base += blockDim.x) {
        const uint32_t q = base + tid;
        const uint32_t K = q < a.nq ? a.K[q] : 0u;
        const unsigned long long r = min(static_cast<unsigned long long>(K), static_cast<unsigned long long>(a.nPoints));
        unsigned long long c = q < a.nq ? a.candFactor * (4ull * r + 64ull) : 0ull;
        if (a.candWant && q < a.nq) c = max(c, static_cast<unsigned long long>(a.candWant[q]));
        unsigned long long ir = r, ic = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(FULL, ir, o), u = __shfl_up_sync(FULL, ic, o);
            if (lane >= static_cast<uint32_t>(o)) {
                ir += t;
                ic += u;
            }
        }
        if (lane == 31) {
            sR[warp] = ir;
            sC[warp] = ic;
        }
        __syncthreads();
        unsigned long long br = sCarryR, bc = sCarryC;
        for (uint32_t w = 0; w < warp; ++w) {
            br += sR[w];
            bc += sC[w];
        }
        if (q < a.nq) {
            a.outOff[q] = br + ir - r;
            a.candOff[q] = bc + ic - c;
        }
        __syncthreads();
        if (tid == blockDim.x - 1) {
            sCarryR = br + ir;
            sCarryC = bc + ic;
        }
        __syncthreads();
    }
    if (tid == 0) {
        a.outOff[a.nq] = sCarryR;
        *a.total = sCarryR;
        a.candOff[a.nq] = sCarryC;
        a.hdr[0] = a.nq;
        a.hdr[1] = a.nq * a.level[0].count;
    }
}

// ---- probe ----------------------------------------------------------------------------------------
constexpr int kProbeThreads = 256;
constexpr int kProbeWarps = kProbeThreads / 32;
constexpr uint32_t kProbeBins = 2048;  // of an 11-bit digit

__device__ __forceinline__ uint64_t shflXor64(uint64_t v, int o) { return __shfl_xor_sync(FULL, v, o); }

// The warp's 32 smallest keys so far, ascending over the lanes.
struct WarpBest {
    uint64_t best = ~0ull;
    // Sorts v over the lanes and keeps the 32 smallest of both (bitonic networks).
    __device__ __forceinline__ void add(uint64_t v, int lane) {
        const uint64_t worst = __shfl_sync(FULL, best, 31);
        if (__ballot_sync(FULL, v < worst) == 0) return;
#pragma unroll
        for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                const uint64_t o = shflXor64(v, stride);
                const bool up = ((lane & size) == 0) == ((lane & stride) == 0);
                v = (up == (o < v)) ? o : v;
            }
        }
        merge(v, lane);
    }
    // v ascending over the lanes.
    __device__ __forceinline__ void merge(uint64_t v, int lane) {
        const uint64_t r = __shfl_sync(FULL, v, 31 - lane);
        best = min(best, r);
#pragma unroll
        for (int stride = 16; stride > 0; stride >>= 1) {
            const uint64_t o = shflXor64(best, stride);
            const bool low = (lane & stride) == 0;
            best = (low == (o < best)) ? o : best;
        }
    }
};

// Distance between two padded float rows; b may lie in global memory.
template <int DP>
__device__ __forceinline__ float rowDist2(const float (&p)[DP], const float* x) {
    float2 s = make_float2(0.f, 0.f);
#pragma unroll
    for (int d = 0; d < DP; d += 4) {
        const float4 c = __ldg(reinterpret_cast<const float4*>(x + d));
        const float2 e = __fadd2_rn(make_float2(p[d], p[d + 1]), make_float2(-c.x, -c.y));
        const float2 f = __fadd2_rn(make_float2(p[d + 2], p[d + 3]), make_float2(-c.z, -c.w));
        s = __ffma2_rn(e, e, s);
        s = __ffma2_rn(f, f, s);
    }
    return s.x + s.y;
}

// FP64 squared distance of a decoded point (the products the traversal rebuilds), fma in dimension
// order: the value KNN results report.
__device__ __forceinline__ double pointDist2(const double* p, const double* y, int D) {
    double s = 0.0;
    if ((D & 1) == 0) {  // rows start on 16-byte boundaries
        for (int d = 0; d < D; d += 2) {
            const double2 v = __ldg(reinterpret_cast<const double2*>(y + d));
            const double e = p[d] - v.x;
            s = __fma_rn(e, e, s);
            const double f = p[d + 1] - v.y;
            s = __fma_rn(f, f, s);
        }
    } else {
        for (int d = 0; d < D; ++d) {
            const double e = p[d] - __ldg(y + d);
            s = __fma_rn(e, e, s);
        }
    }
    return s;
}

// One CTA per query. Every warp keeps the 32 best of the nodes it ranked in registers; the eight lists
// merge through shared memory, pairwise, once per level. The chain of levels is what bounds it (a few
// thousand nodes and points per query, latency between the levels; an instruction in 55% of the issue
// slots at five CTAs an SM, and six with fewer registers measured 234 us), so each CTA is small. 4,096
// queries (N = 10M, D = 8): 226 us, 28 us for one; 250 and 31 us while every point searched its range, a
// warp merged all lists in turn and the selection counted four eight-bit digits.
template <int DP>
__global__ void __launch_bounds__(kProbeThreads) knnProbeKernel(const __grid_constant__ KnnSweepArgs a, int phase) {
    __shared__ uint64_t sMerge[kProbeWarps][32];
    __shared__ uint32_t sBeg[32], sPre[33];
    __shared__ float sKeys[kProbePoints];
    __shared__ __align__(16) uint32_t sHist[kProbeBins];
    __shared__ uint32_t sWarp[kProbeWarps];
    __shared__ uint32_t sSel[2], sTauUb;
    __shared__ uint64_t sScored[32];
    const uint32_t q = blockIdx.x;
    const uint32_t K = a.K[q];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int H = a.height;
    // (The same answer for every thread: a block below may raise the bit while this one starts.)
    if (__syncthreads_or(tid == 0 && (*a.status & kStatusKnnFallback))) return;
    if (K == 0) {
        if (tid == 0) {
            a.tau[q] = -1.0;
            a.tauF[q] = 0.f;
            a.thrF[q] = -1.f;
            if (phase != kProbeBound && a.entCnt) a.entCnt[q] = 0;
        }
        return;
    }
    float p[DP];
#pragma unroll
    for (int d = 0; d < DP; ++d) p[d] = a.qF[static_cast<size_t>(q) * DP + d];
    const float margin = a.margin[q];
    if (tid == 0) sTauUb = __float_as_uint(INFINITY);
    __syncthreads();

    const uint32_t M = static_cast<uint32_t>(
        fmin(32.0, fmax(2.0, ceil(a.waveFactor * static_cast<double>(K)) + 1.0)));
    uint32_t nList = 0;  // ranges in sBeg / sPre
    auto itemOf = [&](uint32_t i) {  // row i of the ranges laid end to end
        uint32_t lo = 0, hi = nList - 1;
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1) >> 1;
            if (sPre[mid] <= i) lo = mid; else hi = mid - 1;
        }
        return sBeg[lo] + (i - sPre[lo]);
    };
    // Leaves the 32 best of the items 0 .. total-1 in sMerge[0], ascending; keyOf(i) returns the
    // item's order key and node, and may lower the bound `ub`.
    auto rank = [&](uint32_t total, auto&& keyOf) {
        WarpBest best;
        for (uint32_t i0 = warp * 32; i0 < total; i0 += kProbeThreads) {
            const uint32_t i = i0 + lane;
            uint64_t key = ~0ull;
            uint32_t ub = 0xffffffffu;
            if (i < total) key = keyOf(i, ub);
            ub = __reduce_min_sync(FULL, ub);
            if (lane == 0 && ub != 0xffffffffu) atomicMin(&sTauUb, ub);
            best.add(key, lane);
        }
        sMerge[warp][lane] = best.best;
        __syncthreads();
#pragma unroll
        for (int half = kProbeWarps / 2; half > 0; half >>= 1) {
            if (warp < half) {
                best.merge(sMerge[warp + half][lane], lane);
                sMerge[warp][lane] = best.best;
            }
            __syncthreads();
        }
    };
    // Node j of mesh m: its centre's distance, less the subtree radius (the sphere's lower bound) when
    // bySphere. A node with K points below it bounds the K-th distance by its far side.
    auto nodeKey = [&](int m, uint32_t j, bool bySphere, uint32_t& ub) -> uint64_t {
        const KnnSweepLevel& L = a.level[m];
        const float d = sqrtf(rowDist2<DP>(p, L.x + static_cast<size_t>(j) * DP));
        const float r = __ldg(L.rad + j);
        if (__ldg(L.leaf + j) >= K) ub = __float_as_uint((d + r) * kRel + margin);
        if (L.nodes[j].cnt == 0) return ~0ull;
        return (static_cast<uint64_t>(floatKey(bySphere ? d - r : d)) << 32) | j;
    };
    // The ranges recs[] of the first `keep` nodes of sMerge[0] become the list; returns their rows.
    auto expand = [&](const NodeRec* recs, uint32_t keep, int headerLevel) {
        if (warp == 0) {
            const uint64_t key = sMerge[0][lane];
            const bool v = static_cast<uint32_t>(lane) < keep && key != ~0ull;
            const NodeRec nr = v ? recs[static_cast<uint32_t>(key)] : NodeRec{0.0, 0u, 0u};
            uint32_t inc = nr.cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(FULL, inc, o);
                if (lane >= o) inc += t;
            }
            sBeg[lane] = nr.cbeg;
            sPre[lane] = inc - nr.cnt;
            if (lane == 31) sPre[32] = inc;
            const uint32_t n = __popc(__ballot_sync(FULL, v));
            if (lane == 31) {
                sSel[0] = n;
                if (headerLevel > 0) {  // entries kept and their children
                    atomicAdd(a.hdr + 2 * headerLevel, n);
                    atomicAdd(a.hdr + 2 * headerLevel + 1, inc);
                }
            }
        }
        __syncthreads();
        nList = sSel[0];
        const uint32_t rows = sPre[32];
        __syncthreads();
        return rows;
    };

    uint32_t total = a.level[0].count;
    if (phase != kProbeBound) {
        for (int m = 0; m + 2 < H; ++m) {
            rank(total, [&](uint32_t i, uint32_t& ub) { return nodeKey(m, m ? itemOf(i) : i, true, ub); });
            total = expand(a.level[m].nodes, a.beam, m + 1);
        }
    }
    if (phase == kProbeEntries) {
        // Hand the clusters under the beam to the scorer.
        __shared__ uint32_t sBase;
        if (tid == 0) {
            sBase = atomicAdd(a.hdr + 2 * (H - 1), total);
            a.entOff[q] = sBase;
            a.entCnt[q] = total;
            if (static_cast<uint64_t>(sBase) + total > a.entCap) atomicOr(a.status, kStatusOverflowEntries);
            a.tau[q] = static_cast<double>(__uint_as_float(sTauUb));
        }
        __syncthreads();
        // Every slot the scorer reads (those below the capacity) is written, also when the entries
        // outgrow the capacity and the batch will rerun.
        const uint32_t base = sBase;
        const uint32_t room = base < a.entCap ? min(total, a.entCap - base) : 0u;
        for (uint32_t i = tid; i < room; i += kProbeThreads) {
            const uint32_t j = H > 2 ? itemOf(i) : i;
            a.entQ[base + i] = q;
            a.entNode[base + i] = j;
        }
        return;
    }
    uint32_t rows;
    if (phase == kProbeBound) {
        if (tid == 0) sTauUb = __float_as_uint(__double2float_ru(a.tau[q]));
        __syncthreads();
        // The M best-scored clusters (smaller = read earlier), filled up to 32 with the nearest centres
        // of the others, so that a scorer that ranks badly cannot leave the bound loose; of their point
        // groups the 32 whose boxes' centres lie nearest are read (all of them when K asks for more).
        const uint32_t base = a.entOff[q];
        const uint32_t n = static_cast<uint64_t>(base) + a.entCnt[q] <= a.entCap ? a.entCnt[q] : 0u;
        rank(n, [&](uint32_t i, uint32_t&) -> uint64_t {
            const uint32_t j = a.entNode[base + i];
            if (a.level[H - 2].nodes[j].cnt == 0) return ~0ull;
            return (static_cast<uint64_t>(floatKey(static_cast<float>(a.score[base + i]))) << 32) | j;
        });
        if (warp == 0) sScored[lane] = static_cast<uint32_t>(lane) < M ? sMerge[0][lane] : ~0ull;
        __syncthreads();
        rank(n, [&](uint32_t i, uint32_t& ub) -> uint64_t {
            const uint32_t j = a.entNode[base + i];
            const uint64_t key = nodeKey(H - 2, j, false, ub);
            for (uint32_t t = 0; t < M; ++t)
                if (sScored[t] != ~0ull && static_cast<uint32_t>(sScored[t]) == j) return ~0ull;
            return key;
        });
        if (warp == 0) {
            const uint64_t own = sScored[lane];
            const uint32_t nS = __popc(__ballot_sync(FULL, own != ~0ull));
            const uint64_t fill = sMerge[0][static_cast<uint32_t>(lane) >= nS ? lane - nS : 0];
            __syncwarp();
            sMerge[0][lane] = static_cast<uint32_t>(lane) < nS ? own : fill;
        }
        __syncthreads();
        const uint64_t mine = sMerge[0][lane];
        const uint32_t groups = expand(a.clusterGroups, 32, 0);
        rank(groups, [&](uint32_t i, uint32_t&) -> uint64_t {
            const uint32_t g = itemOf(i);
            const float* b = a.groupBox + static_cast<size_t>(g) * 2 * DP;
            float s = 0.f;
#pragma unroll
            for (int d = 0; d < DP; ++d) {
                const float e = 0.5f * (__ldg(b + d) + __ldg(b + DP + d)) - p[d];
                s = fmaf(e, e, s);
            }
            return (static_cast<uint64_t>(floatKey(s)) << 32) | g;
        });
        rows = expand(a.groupRec, 32, 0);
        if (rows < 2 * K) {
            if (warp == 0) sMerge[0][lane] = mine;
            __syncthreads();
            rows = expand(a.level[H - 2].nodes, 32, 0);
        }
    } else {
        rank(total, [&](uint32_t i, uint32_t& ub) { return nodeKey(H - 2, H > 2 ? itemOf(i) : i, false, ub); });
        if (tid == 0) atomicAdd(a.hdr + 2 * (H - 1), total);
        // A wide read: twelve times the clusters the scored one takes (float tests of points that lie near
        // the query anyway are cheap, and the bound they give is what the sweep costs by). N = 10M, D = 8, 4,096
        // queries, K = 20 / 100: as many as the scored one 932 us and 24.5k points a query, twice 894 and 23.6k,
        // four times 895, twelve times 900 and 23.8k; 300 queries, K = 1 to 256: 243, 221, 227, 221 us.
        const uint32_t wide = static_cast<uint32_t>(
            fmin(32.0, fmax(2.0, ceil(12.0 * a.waveFactor * static_cast<double>(K)) + 1.0)));
        rows = expand(a.level[H - 2].nodes, wide, 0);
    }
    // The K-th smallest distance among the points read.
    const uint32_t n = min(rows, kProbePoints);
    if (tid == 0) {
        atomicAdd(a.hdr + 2 * (H - 1) + 1, rows);
        atomicAdd(a.hdr + 2 * H, n);
        atomicAdd(a.work, static_cast<unsigned long long>(n));
    }
    // A warp per range of rows (a cluster or a group), four rows of a lane in flight.
    for (uint32_t r = warp; r < nList; r += kProbeWarps) {
        const uint32_t at = sPre[r];
        if (at >= n) break;
        const uint32_t cnt = min(sPre[r + 1], n) - at;
        const float* rowsF = a.pointsF + static_cast<size_t>(sBeg[r]) * DP;
#pragma unroll 4
        for (uint32_t i = lane; i < cnt; i += 32) sKeys[at + i] = rowDist2<DP>(p, rowsF + static_cast<size_t>(i) * DP);
    }
    if (tid == 0) {
        sSel[0] = 0;  // digits chosen so far
        sSel[1] = K;  // rank among the keys that have them
    }
    // A bound just above the K-th smallest: the upper 22 bits of its key (2^-14 of the squared distance),
    // by two counts of 11-bit digits (non-negative floats order like integers). Eight-bit digits put
    // nearly all keys of the first count into one or two bins, whose atomics then queue up.
    if (n >= K) {
        for (int shift = 20; shift >= 9; shift -= 11) {
            for (uint32_t i = tid; i < kProbeBins / 4; i += kProbeThreads)
                reinterpret_cast<uint4*>(sHist)[i] = make_uint4(0u, 0u, 0u, 0u);
            __syncthreads();
            const uint32_t chosen = sSel[0], need = sSel[1];
            for (uint32_t i = tid; i < n; i += kProbeThreads) {
                const uint32_t key = __float_as_uint(sKeys[i]);
                if (shift == 20 || (key >> 20) == chosen) atomicAdd(&sHist[(key >> shift) & (kProbeBins - 1)], 1u);
            }
            __syncthreads();
            constexpr int kOwn = kProbeBins / kProbeThreads;
            uint32_t c[kOwn], sum = 0;
#pragma unroll
            for (int i = 0; i < kOwn; i += 4) {
                const uint4 h = *reinterpret_cast<const uint4*>(&sHist[tid * kOwn + i]);
                c[i] = h.x;
                c[i + 1] = h.y;
                c[i + 2] = h.z;
                c[i + 3] = h.w;
                sum += h.x + h.y + h.z + h.w;
            }
            uint32_t inc = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(FULL, inc, o);
                if (lane >= o) inc += t;
            }
            if (lane == 31) sWarp[warp] = inc;
            __syncthreads();
            for (int w = 0; w < warp; ++w) inc += sWarp[w];
            uint32_t before = inc - sum;
            if (before < need && need <= inc) {  // one thread
#pragma unroll
                for (int i = 0; i < kOwn; ++i) {
                    if (before < need && need <= before + c[i]) {
                        sSel[0] = (chosen << 11) | static_cast<uint32_t>(tid * kOwn + i);
                        sSel[1] = need - before;
                    }
                    before += c[i];
                }
            }
            __syncthreads();
        }
    }
    if (tid == 0) {
        double tau = static_cast<double>(__uint_as_float(sTauUb));
        if (n >= K)
            tau = fmin(tau, sqrt(static_cast<double>(__uint_as_float((sSel[0] << 9) | 0x1ffu))) * static_cast<double>(kRel) +
                                static_cast<double>(margin));
        // Both come from float squares, which lose up to kTiny2 where they are denormal (coordinates of
        // 1e-19 and less), and the finish compares FP64 distances with tau.
        tau += kTiny;
        // Without a bound (K beyond the points read, and no node holds K) every point is a candidate: the
        // walk's case, unless slots that stay for the next batches hold them all (41 queries of K = 600,
        // fan-outs 4 and 3, N = 60,000: 1.8 ms against the walk's 5; N = 600,000: 18 ms against 11).
        const uint64_t r = min(static_cast<uint64_t>(K), a.nPoints);
        if (isinf(tau) && a.nPoints > kSweepWhole * (4 * r + 64)) atomicOr(a.status, kStatusKnnFallback);
        const double t = (tau + static_cast<double>(margin)) * (1.0 + 1e-7);
        a.tau[q] = tau;
        a.tauF[q] = __double2float_ru(t);
        const double s = t * static_cast<double>(kRel);
        a.thrF[q] = __double2float_ru(s * s + kTiny2);
    }
}

// ---- dense bound ----------------------------------------------------------------------------------
constexpr int kBoundThreads = 256;
constexpr int kBoundWords = 8;          // query words of one CTA
constexpr float kFarthest = 1.2e19f;    // above every distance between coordinates of at most kSweepMaxAbs, D <= 32
constexpr float kBoundSlack = 1.6e-5f;  // error of a bound product relative to |x|^2 + |p|^2 + r^2 + T^2, see below

// d = a (16 x 8) * b (8 x 8) + c, TF32 operands (the low 13 bits of a float are not read), FP32 sums.
__device__ __forceinline__ void mmaTf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, float c0, float c1,
                                       float c2, float c3) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}

// x = hi + lo: TF32 operands whose sum keeps 21 bits of x.
__device__ __forceinline__ float tf32Hi(float x) { return __uint_as_float(__float_as_uint(x) & 0xffffe000u); }

// 4 x 4 bytes across the four lanes of a quad: lane j gets byte j of lanes 0 .. 3, lane 0's lowest.
__device__ __forceinline__ uint32_t quadTranspose(uint32_t v, int j) {
    uint32_t o = __shfl_xor_sync(FULL, v, 1);
    v = __byte_perm(v, o, (j & 1) ? 0x3715 : 0x6240);
    o = __shfl_xor_sync(FULL, v, 2);
    return __byte_perm(v, o, (j & 2) ? 0x3276 : 0x5410);
}

// Which queries' bounds T reach which clusters (centre x, radius r): |x - p| <= T + r, written as
//     x.p + T r - (|x|^2 - r^2) / 2 - (|p|^2 - T^2) / 2 >= 0
// with x and p relative to a centre of the CTA's clusters, so that one product per pair on the matrix
// units remains, whose sign is the answer. Factors are split in two TF32 parts (hi hi + hi lo + lo hi);
// an eighth-K step of its own carries T r and the two sums. With 21 bits a factor, products lose less
// than 2^-18 of |x| |p| and T r, and the at most 13 steps' FP32 sums less than 2^-18 of all terms' sizes
// (together under 8e-6 of |x|^2 + |p|^2 + r^2 + T^2); kBoundSlack, twice that, is added to the sums, so a
// bit is only ever set too much (1e-35 covers what underflow loses). A warp holds 32 clusters as fragments and walks the CTA's queries, whose
// fragments are split once into shared memory, in an order that leaves each lane whole bytes of the words.
//
// 4,096 queries x 100,000 clusters, D = 8: 166 us (2.5e12 pairs/s), bound by the rate of the warp-wide
// products; as differences on the float pipe, a cluster per thread, 366 us, and 97 -> 48 us for 1,000 x
// 50,000 at D = 16, 42 -> 22 us for 300 x 100,000 at D = 8. (The walk's bound levels,
// filters and transposes took 3.4 ms for the first.)
template <int DP>
__global__ void __launch_bounds__(kBoundThreads) knnBoundBitsKernel(const __grid_constant__ KnnSweepArgs a, uint32_t iters) {
    constexpr int STEPS = (DP + 7) / 8;
    constexpr int W = STEPS <= 2 ? kBoundWords : kBoundWords / 2;  // words staged at once (48 KB of shared memory)
    __shared__ __align__(16) float4 sB[W][4][STEPS][32];  // hi, hi, lo, lo of a lane's two dimensions
    __shared__ __align__(8) float2 sE[W][4][32];
    __shared__ unsigned long long sReached;
    if (*a.status & ~kStatusOverflowItems) return;
    uint32_t reached = 0;  // pairs whose bit is set
    if (threadIdx.x == 0) sReached = 0;
    const KnnSweepLevel& L = a.level[a.height - 2];
    const uint32_t w0 = blockIdx.y * kBoundWords;
    const uint32_t left = a.qEnd - a.qBegin > w0 * 32 ? a.qEnd - a.qBegin - w0 * 32 : 0u;  // queries from w0 on
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int quad = lane >> 2, j = lane & 3;
    const uint32_t c0 = blockIdx.x * iters * kBoundThreads, c1 = min(L.count, c0 + iters * kBoundThreads);
    // The CTA's centre: its first cluster's (the origin where an empty cluster has none).
    auto centre = [&](int d) {
        const float x = __ldg(L.x + static_cast<size_t>(c0) * DP + d);
        return fabsf(x) <= static_cast<float>(kSweepMaxAbs) ? x : 0.f;
    };

    for (uint32_t wb = 0; wb < kBoundWords && wb * 32 < left; wb += W) {
        if (wb) __syncthreads();
        if (tid < W * 32) {
            // Bit b, lane byte j and tile t of query i's place in its word: the accumulators' layout.
            const uint32_t i = tid & 31, w = tid >> 5, t = (i >> 1) & 3, n = 2 * (i >> 3) + (i & 1);
            const uint32_t at = (wb + w) * 32 + i;
            const bool v = at < left;
            const uint32_t q = a.qBegin + w0 * 32 + (v ? at : 0);
            float n2 = 0.f;
#pragma unroll
            for (int s = 0; s < STEPS; ++s)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    float2 p = make_float2(0.f, 0.f);
                    if (v && 8 * s + 2 * k < DP) {
                        p = __ldg(reinterpret_cast<const float2*>(a.qF + static_cast<size_t>(q) * DP + 8 * s + 2 * k));
                        p.x -= centre(8 * s + 2 * k);
                        p.y -= centre(8 * s + 2 * k + 1);
                    }
                    n2 = fmaf(p.x, p.x, fmaf(p.y, p.y, n2));
                    const float hx = tf32Hi(p.x), hy = tf32Hi(p.y);
                    sB[w][t][s][n * 4 + k] = make_float4(hx, hy, p.x - hx, p.y - hy);
                }
            const float T = v ? fminf(a.tauF[q] * kRel, kFarthest) : 0.f;
            const float sum = v ? 0.5f * (T * T - n2) + kBoundSlack * (T * T + n2) + 1e-35f : -1e38f;
            const float hT = tf32Hi(T), hS = tf32Hi(sum);
            sE[w][t][n * 4 + 0] = make_float2(hT, sum - hS);  // against r hi, 1
            sE[w][t][n * 4 + 1] = make_float2(hT, 1.f);       // r lo, sum hi
            sE[w][t][n * 4 + 2] = make_float2(T - hT, 1.f);   // r hi, sum lo
            sE[w][t][n * 4 + 3] = make_float2(hS, 0.f);       // 1, 0
        }
        __syncthreads();
        for (uint32_t it = 0; it < iters; ++it) {
            const uint32_t base = c0 + it * kBoundThreads + warp * 32;
            if (base >= c1) break;  // warp-uniform
            uint32_t hi[2][STEPS][4], lo[2][STEPS][4], ext[2][4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const uint32_t c = base + quad + 8 * h;
                const bool v = c < c1 && L.nodes[c].cnt > 0;
                const int m = h >> 1, e = h & 1;
                float n2 = 0.f;
#pragma unroll
                for (int s = 0; s < STEPS; ++s) {
                    float2 x = make_float2(0.f, 0.f);
                    if (v && 8 * s + 2 * j < DP) {
                        x = __ldg(reinterpret_cast<const float2*>(L.x + static_cast<size_t>(c) * DP + 8 * s + 2 * j));
                        x.x -= centre(8 * s + 2 * j);
                        x.y -= centre(8 * s + 2 * j + 1);
                    }
                    n2 = fmaf(x.x, x.x, fmaf(x.y, x.y, n2));
                    const float hx = tf32Hi(x.x), hy = tf32Hi(x.y);
                    hi[m][s][e] = __float_as_uint(hx);
                    hi[m][s][2 + e] = __float_as_uint(hy);
                    lo[m][s][e] = __float_as_uint(x.x - hx);
                    lo[m][s][2 + e] = __float_as_uint(x.y - hy);
                }
                n2 += __shfl_xor_sync(FULL, n2, 1);
                n2 += __shfl_xor_sync(FULL, n2, 2);
                const float r = v ? __ldg(L.rad + c) * kRel : 0.f;
                const float sum = 0.5f * (r * r - n2) + kBoundSlack * (r * r + n2);
                const float hR = tf32Hi(r), hS = tf32Hi(sum);
                ext[m][e] = __float_as_uint(j == 1 ? r - hR : j == 3 ? 1.f : hR);
                ext[m][2 + e] = __float_as_uint(j == 0 ? 1.f : j == 1 ? hS : j == 2 ? sum - hS : 0.f);
            }
            const uint32_t c = base + quad + 8 * j;  // the cluster whose words this lane ends up with
            const bool valid = c < c1 && L.nodes[c].cnt > 0;
            uint32_t word[W], any = 0;
#pragma unroll
            for (int w = 0; w < W; ++w) {
                word[w] = 0;
                if ((wb + w) * 32 >= left) continue;  // uniform
                uint32_t far[4] = {0u, 0u, 0u, 0u};  // signs, a byte of the word per cluster row
#pragma unroll
                for (int t = 3; t >= 0; --t) {
                    float d[2][4];
                    const float2 e = sE[w][t][lane];
#pragma unroll
                    for (int m = 0; m < 2; ++m)
                        mmaTf32(d[m], ext[m], __float_as_uint(e.x), __float_as_uint(e.y), 0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int s = 0; s < STEPS; ++s) {
                        const float4 b = sB[w][t][s][lane];
                        const uint32_t bx = __float_as_uint(b.x), by = __float_as_uint(b.y);
                        const uint32_t bz = __float_as_uint(b.z), bw = __float_as_uint(b.w);
#pragma unroll
                        for (int m = 0; m < 2; ++m) {
                            mmaTf32(d[m], lo[m][s], bx, by, d[m][0], d[m][1], d[m][2], d[m][3]);
                            mmaTf32(d[m], hi[m][s], bz, bw, d[m][0], d[m][1], d[m][2], d[m][3]);
                            mmaTf32(d[m], hi[m][s], bx, by, d[m][0], d[m][1], d[m][2], d[m][3]);
                        }
                    }
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        far[h] = __funnelshift_l(__float_as_uint(d[h >> 1][2 * (h & 1) + 1]), far[h], 1);
                        far[h] = __funnelshift_l(__float_as_uint(d[h >> 1][2 * (h & 1)]), far[h], 1);
                    }
                }
                const uint32_t bytes = __byte_perm(__byte_perm(far[0], far[1], 0x0040), __byte_perm(far[2], far[3], 0x0040), 0x5410);
                const uint32_t near = quadTranspose(~bytes, j);
                word[w] = valid ? near : 0u;
                any |= word[w];
                reached += __popc(word[w]);
            }
            if (c < c1) {
                uint32_t* out = a.bits + static_cast<size_t>(c) * a.words + w0 + wb;
                if (a.words == 1) {
                    out[0] = word[0];
                } else {  // rows of a multiple of four words
#pragma unroll
                    for (int w = 0; w < W; w += 4)
                        if (w0 + wb + w < a.words) *reinterpret_cast<uint4*>(out + w) = make_uint4(word[w], word[w + 1], word[w + 2], word[w + 3]);
                }
            }
            if (gridDim.y == 1) {
                // Listed when the first queries that reach it are found: with the words in two turns, the second
                // turn lists what the first left out.
                const bool seen = wb && valid && a.words > 1 &&
                                  [&] {
                                      const uint4 f = *reinterpret_cast<const uint4*>(a.bits + static_cast<size_t>(c) * a.words);
                                      return (f.x | f.y | f.z | f.w) != 0;
                                  }();
                const uint32_t b = __ballot_sync(FULL, any != 0 && !seen);
                if (b) {
                    uint32_t at = 0;
                    if (lane == 0) at = atomicAdd(a.liveCnt, __popc(b));
                    at = __shfl_sync(FULL, at, 0);
                    if (any != 0 && !seen) a.live[at + __popc(b & ((1u << lane) - 1u))] = c;
                }
            }
        }
    }
    if (!a.sliced) return;
    reached = __reduce_add_sync(FULL, reached);
    if (lane == 0) atomicAdd(&sReached, static_cast<unsigned long long>(reached));
    __syncthreads();
    if (tid == 0 && sReached) atomicAdd(a.reached, sReached);
}

// ---- sweep ----------------------------------------------------------------------------------------
constexpr int kSweepThreads = 128;
constexpr int kSweepWarps = kSweepThreads / 32;
constexpr uint32_t kSweepList = 1024 + 32;
constexpr uint32_t kSweepGroups = 8;  // group boxes staged at once

// A point that passed the float filter: measured in FP64, and a candidate when it lies within the bound.
__device__ __forceinline__ bool measureInline(const KnnSweepArgs& a, uint32_t row, uint32_t q) {
    const uint32_t pr = __ldg(a.perm + row);
    const double d2 = pointDist2(a.points + static_cast<size_t>(q) * a.D,
                                 a.pointsD + static_cast<size_t>(a.rowOrder ? pr : row) * a.D, a.D);
    const double tau = a.tau[q];
    if (!(d2 <= tau * tau * (1.0 + 1e-9))) return false;
    const uint64_t pos = a.candOff[q] + atomicAdd(&a.candCnt[q], 1u);
    if (pos < a.candOff[q + 1] && pos < a.candCap) {
        a.candId[pos] = a.map[pr];
        a.candD2[pos] = d2;
        return true;
    }
    atomicOr(a.status, kStatusOverflowItems);
    return false;
}

// Out of line where the registers around it are short (a few in ten thousand tested points come here).
__device__ __noinline__ bool measure(const KnnSweepArgs& a, uint32_t row, uint32_t q) { return measureInline(a, row, q); }

// Deals the clusters to the warps and hands each cluster's queries (the set bits of its row) to
// batch(cluster, first list entry, n <= 32).
//
// SLICED: in batches above kSweepSliced queries, 32 words of a cluster with more than that many, in a cluster
// of more than twice what a warp would have if all were dealt out evenly, are left to a second launch
// (sweepSlices). A batch whose queries lie together, or far outside the data, reaches a hundred clusters with
// nearly all of its queries; one warp for each of those took 11.9 ms (4,096 queries, K = 100, N = 1M, D = 3;
// the level-synchronous walk 4.9) where spread queries take 0.36. In slices it takes 0.76; the second launch
// (placed early, see launchEarly) costs 2 to 5 us where there are none. (Taken by the same launch's warps as they run out of clusters it took
// 18 ms: most have left when the first slice appears.)
template <bool SLICED, class Batch>
__device__ __forceinline__ void sweepClusters(const KnnSweepArgs& a, uint32_t* list, Batch&& batch) {
    const int lane = threadIdx.x & 31;
    const bool listed = a.qEnd - a.qBegin <= kBoundWords * 32;
    const uint32_t nClusters = listed ? *a.liveCnt : a.level[a.height - 2].count;
    // Clusters per ticket: several where there are many, so the ticket's atomic does not bound the sweep.
    const uint32_t chunk = max(1u, min(8u, nClusters / (gridDim.x * kSweepWarps * 8u)));
    uint32_t k = 0, kEnd = 0;
    while (true) {
        if (k == kEnd) {
            if (lane == 0) k = atomicAdd(a.ticket, chunk);
            k = __shfl_sync(FULL, k, 0);
            if (k >= nClusters) break;
            kEnd = min(nClusters, k + chunk);
        }
        const uint32_t c = listed ? a.live[k] : k;
        ++k;
        const uint32_t* row = a.bits + static_cast<size_t>(c) * a.words;
        uint32_t n = 0;
        for (uint32_t w0 = 0; w0 < a.words; w0 += 32) {
            uint32_t word = (w0 + lane < a.words) ? row[w0 + lane] : 0u;
            uint32_t inc = __popc(word);
            const uint32_t own = inc;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(FULL, inc, o);
                if (lane >= o) inc += t;
            }
            const uint32_t add = __shfl_sync(FULL, inc, 31);
            if (add == 0) continue;
            if (SLICED && add > kSweepSliced && a.sliced &&
                static_cast<uint64_t>(add) * ((a.words + 31u) / 32u) * kSweepWarps * gridDim.x > 2ull * *a.reached) {
                if (lane == 0) a.heavy[atomicAdd(a.heavyCnt, 1u)] = make_uint4(c, w0, add, 0u);
                continue;
            }
            uint32_t at = n + inc - own;
            const uint32_t q0 = a.qBegin + (w0 + lane) * 32;
            while (word) {
                list[at++] = q0 + __ffs(word) - 1;
                word &= word - 1;
            }
            __syncwarp();
            n += add;
            uint32_t from = 0;
            const bool last = w0 + 32 >= a.words;
            for (; from + 32 <= n; from += 32) batch(c, from, 32);
            if (last) break;
            // The rest waits for the next words.
            const uint32_t rest = n - from;
            const uint32_t keep = static_cast<uint32_t>(lane) < rest ? list[from + lane] : 0u;
            __syncwarp();
            if (static_cast<uint32_t>(lane) < rest) list[lane] = keep;
            __syncwarp();
            n = rest;
        }
        const uint32_t full = n / 32 * 32;
        if (n > full) batch(c, full, n - full);
        __syncwarp();
    }
}

// What sweepClusters left, in slices of one to sixteen words with about kSweepSlice queries, a warp each.
constexpr uint32_t kSweepSlice = 64;
template <class Batch>
__device__ __forceinline__ void sweepSlices(const KnnSweepArgs& a, uint32_t* list, Batch&& batch) {
    const uint32_t lane = threadIdx.x & 31, total = *a.heavyCnt * 32u;
    while (total) {
        uint32_t t = 0;
        if (lane == 0) t = atomicAdd(a.heavyTicket, 1u);
        t = __shfl_sync(FULL, t, 0);
        if (t >= total) break;
        const uint4 e = a.heavy[t / 32u];  // cluster, first word, queries
        const uint32_t per = (32u * kSweepSlice + e.z - 1u) / e.z, w0 = e.y + t % 32u * per;
        const uint32_t w1 = min(min(e.y + 32u, a.words), w0 + per);
        if (t % 32u * per >= 32u || w0 >= w1) continue;  // the entry has fewer slices
        uint32_t word = w0 + lane < w1 ? a.bits[static_cast<size_t>(e.x) * a.words + w0 + lane] : 0u;
        uint32_t inc = __popc(word);
        const uint32_t own = inc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(FULL, inc, o);
            if (lane >= static_cast<uint32_t>(o)) inc += v;
        }
        const uint32_t n = __shfl_sync(FULL, inc, 31);
        const uint32_t q0 = a.qBegin + (w0 + lane) * 32;
        for (uint32_t at = inc - own; word; word &= word - 1) list[at++] = q0 + __ffs(word) - 1;
        __syncwarp();
        for (uint32_t from = 0; from < n; from += 32) batch(e.x, from, min(32u, n - from));
        __syncwarp();
    }
}

// Copies the boxes of ng groups from g on to shared memory.
template <int DP>
__device__ __forceinline__ void stageBoxes(const KnnSweepArgs& a, float (*box)[2 * DP], uint32_t g, uint32_t ng) {
    const float4* src = reinterpret_cast<const float4*>(a.groupBox + static_cast<size_t>(g) * 2 * DP);
    for (uint32_t i = threadIdx.x & 31; i < ng * (2 * DP / 4); i += 32) reinterpret_cast<float4*>(&box[0][0])[i] = __ldg(src + i);
}

// max(a, b, c) in one instruction (sm_100 three-input max.f32).
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Squared distance from p to a staged box, two dimensions an instruction where there is one.
template <int DP>
__device__ __forceinline__ float boxGap2(const float* b, const float (&p)[DP]) {
    float2 gap = make_float2(0.f, 0.f);
#pragma unroll
    for (int d = 0; d < DP; d += 4) {
        const float4 lo = *reinterpret_cast<const float4*>(b + d);
        const float4 hi = *reinterpret_cast<const float4*>(b + DP + d);
        const float2 q0 = make_float2(p[d], p[d + 1]), q1 = make_float2(p[d + 2], p[d + 3]);
        const float2 m0 = make_float2(-p[d], -p[d + 1]), m1 = make_float2(-p[d + 2], -p[d + 3]);
        const float2 l0 = __fadd2_rn(make_float2(lo.x, lo.y), m0), h0 = __fadd2_rn(q0, make_float2(-hi.x, -hi.y));
        const float2 l1 = __fadd2_rn(make_float2(lo.z, lo.w), m1), h1 = __fadd2_rn(q1, make_float2(-hi.z, -hi.w));
        const float2 e0 = make_float2(max3f(l0.x, h0.x, 0.f), max3f(l0.y, h0.y, 0.f));
        const float2 e1 = make_float2(max3f(l1.x, h1.x, 0.f), max3f(l1.y, h1.y, 0.f));
        gap = __ffma2_rn(e0, e0, gap);
        gap = __ffma2_rn(e1, e1, gap);
    }
    return gap.x + gap.y;
}

// One warp per cluster. Lanes are queries while boxes are tested and points while distances are: a
// group's points stay in registers and every query whose box test passed is broadcast from shared
// memory, so no lane idles for another query's sake. Bound by the float pipe and the latency of a
// cluster's first loads. 84M (query, point) tests of 4,096 queries, N = 10M, D = 8: 383 us (422 us before
// the box test took three-input maxima and packed pairs; the walk's point passes: 2.9 ms for 187M).
template <int DP, bool SLICES>
__global__ void __launch_bounds__(kSweepThreads) knnSweepKernel(const __grid_constant__ KnnSweepArgs a) {
    __shared__ uint32_t sList[kSweepWarps][kSweepList];
    __shared__ __align__(16) float sP[kSweepWarps][32][DP];
    if constexpr (SLICES)
        waitForEarlierLaunch();
    else if (a.sliced)
        letNextLaunchStart();
    __shared__ float sThr[kSweepWarps][32];
    __shared__ uint32_t sId[kSweepWarps][32];
    __shared__ __align__(16) float sBox[kSweepWarps][kSweepGroups][2 * DP];
    if (*a.status & ~kStatusOverflowItems) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned long long tested = 0;
    uint32_t kept = 0;              // this lane's candidates
    uint32_t staged = 0xffffffffu;  // first group whose box is in sBox

    // A batch of n <= 32 queries of the list against the cluster's groups.
    auto batch = [&](uint32_t c, uint32_t from, uint32_t n) {
        const NodeRec cg = a.clusterGroups[c];
        const bool v = static_cast<uint32_t>(lane) < n;
        const uint32_t q = v ? sList[w][from + lane] : 0u;
        float p[DP];
#pragma unroll
        for (int d = 0; d < DP; d += 4) {
            const float4 t = v ? __ldg(reinterpret_cast<const float4*>(a.qF + static_cast<size_t>(q) * DP + d))
                               : make_float4(0.f, 0.f, 0.f, 0.f);
            p[d] = t.x;
            p[d + 1] = t.y;
            p[d + 2] = t.z;
            p[d + 3] = t.w;
        }
        const float thr = v ? a.thrF[q] : -1.f;
        __syncwarp();
#pragma unroll
        for (int d = 0; d < DP; d += 4)
            *reinterpret_cast<float4*>(&sP[w][lane][d]) = make_float4(p[d], p[d + 1], p[d + 2], p[d + 3]);
        sThr[w][lane] = thr;
        sId[w][lane] = q;
        for (uint32_t g0 = 0; g0 < cg.cnt; g0 += kSweepGroups) {
            const uint32_t ng = min(kSweepGroups, cg.cnt - g0);
            __syncwarp();
            if (staged != cg.cbeg + g0) {
                staged = cg.cbeg + g0;
                stageBoxes<DP>(a, sBox[w], staged, ng);
            }
            __syncwarp();
            for (uint32_t g = 0; g < ng; ++g) {
                uint32_t mask = __ballot_sync(FULL, boxGap2<DP>(sBox[w][g], p) <= thr);
                if (mask == 0) continue;
                const NodeRec gr = a.groupRec[cg.cbeg + g0 + g];
                const bool pv = static_cast<uint32_t>(lane) < gr.cnt;
                const uint32_t row = gr.cbeg + (pv ? lane : 0u);
                tested += static_cast<unsigned long long>(__popc(mask)) * gr.cnt;
                float2 x[DP / 2];
#pragma unroll
                for (int d = 0; d < DP / 2; d += 2) {
                    const float4 t = __ldg(reinterpret_cast<const float4*>(a.pointsF + static_cast<size_t>(row) * DP) + d / 2);
                    x[d] = make_float2(-t.x, -t.y);
                    x[d + 1] = make_float2(-t.z, -t.w);
                }
                while (mask) {
                    const int s = __ffs(mask) - 1;
                    mask &= mask - 1;
                    float2 acc = make_float2(0.f, 0.f);
#pragma unroll
                    for (int d = 0; d < DP / 2; d += 2) {
                        const float4 t = *reinterpret_cast<const float4*>(&sP[w][s][2 * d]);
                        const float2 e = __fadd2_rn(x[d], make_float2(t.x, t.y));
                        const float2 f = __fadd2_rn(x[d + 1], make_float2(t.z, t.w));
                        acc = __ffma2_rn(e, e, acc);
                        acc = __ffma2_rn(f, f, acc);
                    }
                    const bool hit = pv && acc.x + acc.y <= sThr[w][s];
                    if (__ballot_sync(FULL, hit) == 0) continue;
                    if (hit && measureInline(a, row, sId[w][s])) ++kept;
                }
            }
        }
    };

    if constexpr (SLICES)
        sweepSlices(a, sList[w], batch);
    else
        sweepClusters<true>(a, sList[w], batch);
    if (lane == 0 && tested) atomicAdd(a.work + 1, tested);
    kept = __reduce_add_sync(FULL, kept);
    if (lane == 0 && kept) atomicAdd(a.hdr + 2 * (a.height + 1), kept);
}

// One warp per cluster: its queries, 32 at a time, against its points, 16 at a time, as a product on the
// matrix units. With y and p relative to the cluster's centre, |y - p|^2 <= thr is
//     y.p >= |y|^2 / 2 + (|p|^2 - thr) / 2,
// so the query's side seeds the accumulator and a comparison per pair remains. TF32 drops 13 bits of
// each factor: y.p is off by at most 2^-9 |y| |p|, and the query's side is lowered by that (with the
// cluster's radius for |y|), so the filter only lets too much through; measure() decides. The boxes of
// the cluster's point groups are tested first, a query a lane: a group no query of the batch reaches
// is not read.
//
// Taken above eight (padded) dimensions. On the float pipe (a point per lane, queries broadcast from shared
// memory) the broadcasts bound it there: 1,000 queries, N = 5M, D = 16, 811M needed pairs: 2.53 ms at 85%
// of the shared-memory pipe and 1,681M instructions, here 1.73 ms and 762M, bound by latency: four
// blocks an SM (128 registers, which DP = 12 and 16 exceed by 380 bytes of spills), an instruction in 40%
// of the issue slots. At D = 8, where a box test
// leaves about four of a batch's queries, the product does eight times the needed pairs and is slower
// (868 against 422 us).
template <int DP>
__global__ void __launch_bounds__(kSweepThreads, DP <= 16 ? 4 : 2) knnSweepMmaKernel(const __grid_constant__ KnnSweepArgs a) {
    constexpr int STEPS = (DP + 7) / 8;
    __shared__ uint32_t sList[kSweepWarps][kSweepList];
    __shared__ __align__(16) float sBox[kSweepWarps][kSweepGroups][2 * DP];
    if (*a.status & ~kStatusOverflowItems) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int quad = lane >> 2, kc = 2 * (lane & 3);  // fragment row, first of the lane's two dimensions in a step
    const KnnSweepLevel& L = a.level[a.height - 2];
    unsigned long long tested = 0;
    uint32_t kept = 0;               // this lane's candidates
    uint32_t staged = 0xffffffffu;  // first group whose box is in sBox

    // The lane's pair of dimensions of a padded float row, step s (zero past the row).
    auto pairAt = [&](const float* row, int s) {
        return (8 * s + kc < DP) ? __ldg(reinterpret_cast<const float2*>(row + 8 * s + kc)) : make_float2(0.f, 0.f);
    };

    // A batch of n <= 32 queries of the list against cluster c.
    auto batch = [&](uint32_t c, uint32_t from, uint32_t n) {
        const float* centre = L.x + static_cast<size_t>(c) * DP;
        const float rad = __ldg(L.rad + c);
        const uint32_t nt = (n + 7) / 8;
        float2 ctr[STEPS];
#pragma unroll
        for (int s = 0; s < STEPS; ++s) ctr[s] = pairAt(centre, s);
        // Queries: fragments (tile t, column quad), and what seeds the accumulators.
        uint32_t b[4][STEPS][2];
        float seed[4][2];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            seed[t][0] = seed[t][1] = -INFINITY;
            if (static_cast<uint32_t>(t) >= nt) continue;  // warp-uniform
            const uint32_t i = t * 8 + quad;
            const bool v = i < n;
            const uint32_t q = sList[w][from + (v ? i : 0)];
            const float* row = a.qF + static_cast<size_t>(q) * DP;
            float n2 = 0.f;
#pragma unroll
            for (int s = 0; s < STEPS; ++s) {
                const float2 p = pairAt(row, s);
                const float x = p.x - ctr[s].x, y = p.y - ctr[s].y;
                n2 = fmaf(x, x, fmaf(y, y, n2));
                b[t][s][0] = __float_as_uint(x);
                b[t][s][1] = __float_as_uint(y);
            }
            n2 += __shfl_xor_sync(FULL, n2, 1);
            n2 += __shfl_xor_sync(FULL, n2, 2);
            const float thr = a.thrF[q];
            const float slack = 0.0021f * rad * sqrtf(n2) + 4e-6f * (n2 + rad * rad);
            const float mine = v ? 0.5f * (thr * kRel - n2) + slack : -INFINITY;
            seed[t][0] = __shfl_sync(FULL, mine, kc * 4);
            seed[t][1] = __shfl_sync(FULL, mine, kc * 4 + 4);
        }
        // A group's points, all loaded at once (two tiles of sixteen rows) while the group before is tested.
        float2 y[4][STEPS];
        auto fetch = [&](uint32_t first, uint32_t cnt) {
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const uint32_t r = quad + 8 * h;
                const float* row = a.pointsF + static_cast<size_t>(first + (r < cnt ? r : 0)) * DP;
#pragma unroll
                for (int s = 0; s < STEPS; ++s) y[h][s] = pairAt(row, s);
            }
        };
        // Tests the fetched group; fetches the next (cnt2 points from first2 on) once its own are in use.
        auto points = [&](uint32_t first, uint32_t cnt, uint32_t first2, uint32_t cnt2) {
            const uint32_t end = first + cnt;
            uint32_t f[2][STEPS][4];
            float h[2][2];
#pragma unroll
            for (int tile = 0; tile < 2; ++tile)
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    float n2 = 0.f;
#pragma unroll
                    for (int s = 0; s < STEPS; ++s) {
                        const float x0 = y[2 * tile + half][s].x - ctr[s].x, x1 = y[2 * tile + half][s].y - ctr[s].y;
                        n2 = fmaf(x0, x0, fmaf(x1, x1, n2));
                        f[tile][s][half] = __float_as_uint(x0);
                        f[tile][s][2 + half] = __float_as_uint(x1);
                    }
                    n2 += __shfl_xor_sync(FULL, n2, 1);
                    n2 += __shfl_xor_sync(FULL, n2, 2);
                    h[tile][half] = 0.5f * n2;
                }
            if (cnt2) fetch(first2, cnt2);
#pragma unroll
            for (int tile = 0; tile < 2; ++tile) {
                if (static_cast<uint32_t>(tile) * 16 >= cnt) break;  // warp-uniform
                bool any = false;
                float d[4][4];
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    if (static_cast<uint32_t>(t) >= nt) continue;  // warp-uniform
                    mmaTf32(d[t], f[tile][0], b[t][0][0], b[t][0][1], seed[t][0], seed[t][1], seed[t][0], seed[t][1]);
#pragma unroll
                    for (int s = 1; s < STEPS; ++s)
                        mmaTf32(d[t], f[tile][s], b[t][s][0], b[t][s][1], d[t][0], d[t][1], d[t][2], d[t][3]);
                    any = any || d[t][0] >= h[tile][0] || d[t][1] >= h[tile][0] || d[t][2] >= h[tile][1] || d[t][3] >= h[tile][1];
                }
                if (__ballot_sync(FULL, any) == 0) continue;
                if (any) {
#pragma unroll
                    for (int t = 0; t < 4; ++t)
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const uint32_t r = first + 16 * tile + quad + (j & 2) * 4, i = t * 8 + kc + (j & 1);
                            if (i < n && r < end && d[t][j] >= h[tile][j >> 1] && measure(a, r, sList[w][from + i])) ++kept;
                        }
                }
                __syncwarp();
            }
        };
        // Lanes are queries while the groups' boxes are tested.
        const NodeRec cg = a.clusterGroups[c];
        const bool v = static_cast<uint32_t>(lane) < n;
        const uint32_t q = sList[w][from + (v ? lane : 0)];
        const float thr = v ? a.thrF[q] : -1.f;
        for (uint32_t g0 = 0; g0 < cg.cnt; g0 += kSweepGroups) {
            const uint32_t ng = min(kSweepGroups, cg.cnt - g0);
            __syncwarp();
            if (staged != cg.cbeg + g0) {
                staged = cg.cbeg + g0;
                stageBoxes<DP>(a, sBox[w], staged, ng);
            }
            const NodeRec gr = a.groupRec[cg.cbeg + g0 + min(static_cast<uint32_t>(lane), ng - 1)];
            __syncwarp();
            uint32_t mine = 0;  // lane g: group g's queries
            {
                float p[DP];
#pragma unroll
                for (int d = 0; d < DP; d += 4) {
                    const float4 t = __ldg(reinterpret_cast<const float4*>(a.qF + static_cast<size_t>(q) * DP + d));
                    p[d] = t.x;
                    p[d + 1] = t.y;
                    p[d + 2] = t.z;
                    p[d + 3] = t.w;
                }
                for (uint32_t g = 0; g < ng; ++g) {
                    const uint32_t m = __ballot_sync(FULL, boxGap2<DP>(sBox[w][g], p) <= thr);
                    if (static_cast<uint32_t>(lane) == g) mine = m;
                }
            }
            uint32_t some = __ballot_sync(FULL, mine != 0);
            if (some == 0) continue;
            tested += static_cast<unsigned long long>(__reduce_add_sync(FULL, __popc(mine) * gr.cnt));
            int g = __ffs(some) - 1;
            uint32_t first = __shfl_sync(FULL, gr.cbeg, g), cnt = __shfl_sync(FULL, gr.cnt, g);
            fetch(first, cnt);
            while (some) {
                some &= some - 1;
                g = some ? __ffs(some) - 1 : 0;
                const uint32_t first2 = __shfl_sync(FULL, gr.cbeg, g), cnt2 = some ? __shfl_sync(FULL, gr.cnt, g) : 0u;
                points(first, cnt, first2, cnt2);
                first = first2;
                cnt = cnt2;
            }
        }
    };

    // (Not in slices: a product takes less time a query. 4,096 queries at one place, K = 100, N = 500k, D = 12: 14 ms,
    // the level-synchronous walk 17.)
    sweepClusters<false>(a, sList[w], batch);
    if (lane == 0 && tested) atomicAdd(a.work + 1, tested);
    kept = __reduce_add_sync(FULL, kept);
    if (lane == 0 && kept) atomicAdd(a.hdr + 2 * (a.height + 1), kept);
}

int residentBlocks(const void* kern, int threads) {
    int dev = 0, sms = 0, perSm = 0;
    TBLAEQ_CUDA(cudaGetDevice(&dev));
    TBLAEQ_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    TBLAEQ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kern, threads, 0));
    return std::max(1, sms * std::max(1, perSm));
}

// Calls f with the padded dimension as a compile-time constant.
template <class F>
void withPadded(int D, F&& f) {
    switch (paddedDims(static_cast<uint64_t>(D))) {
        case 4: return f(std::integral_constant<int, 4>{});
        case 8: return f(std::integral_constant<int, 8>{});
        case 12: return f(std::integral_constant<int, 12>{});
        case 16: return f(std::integral_constant<int, 16>{});
        case 20: return f(std::integral_constant<int, 20>{});
        case 24: return f(std::integral_constant<int, 24>{});
        case 28: return f(std::integral_constant<int, 28>{});
        case 32: return f(std::integral_constant<int, 32>{});
        default: throw std::invalid_argument("KNN sweep: D must be in [1, 32]");
    }
}

}  // namespace

void launchKnnSweepPrepare(const KnnSweepArgs& a, cudaStream_t s) {
    const unsigned blocks = std::min<unsigned>(148u, (a.nq + 1023u) / 1024u);
    sweepPrepareKernel<<<std::max(1u, blocks), 1024, 0, s>>>(a, paddedDims(static_cast<uint64_t>(a.D)));
    TBLAEQ_LAUNCHED();
}

void launchKnnProbe(const KnnSweepArgs& a, KnnProbePhase phase, cudaStream_t s) {
    if (a.nq == 0) return;
    withPadded(a.D, [&](auto dp) {
        knnProbeKernel<decltype(dp)::value><<<a.nq, kProbeThreads, 0, s>>>(a, static_cast<int>(phase));
        TBLAEQ_LAUNCHED();
    });
}

void launchKnnSweepBound(const KnnSweepArgs& a, cudaStream_t s) {
    // 256 clusters a turn, and up to eight turns a CTA while a few CTAs per SM remain: a CTA's queries are
    // split once, which is a fifth of a single turn.
    const uint32_t turns = (a.level[a.height - 2].count + kBoundThreads - 1) / kBoundThreads;
    const uint32_t gy = (a.words + kBoundWords - 1) / kBoundWords;
    const uint32_t iters = std::max<uint32_t>(1, std::min<uint64_t>(8, static_cast<uint64_t>(turns) * gy / (148 * 8)));
    const dim3 grid((turns + iters - 1) / iters, gy);
    withPadded(a.D, [&](auto dp) {
        knnBoundBitsKernel<decltype(dp)::value><<<grid, kBoundThreads, 0, s>>>(a, iters);
        TBLAEQ_LAUNCHED();
    });
}

void launchKnnSweepPoints(const KnnSweepArgs& a, cudaStream_t s) {
    withPadded(a.D, [&](auto dp) {
        constexpr int DP = decltype(dp)::value;
        void (*kern)(const KnnSweepArgs);
        if constexpr (DP > 8)
            kern = knnSweepMmaKernel<DP>;
        else
            kern = knnSweepKernel<DP, false>;
        static const int grid = residentBlocks(reinterpret_cast<const void*>(kern), kSweepThreads);
        kern<<<grid, kSweepThreads, 0, s>>>(a);
        TBLAEQ_LAUNCHED();
        if constexpr (DP <= 8) {
            if (!a.sliced) return;
            launchEarly(knnSweepKernel<DP, true>, std::max(1, grid / 2), kSweepThreads, s, a);
        }
    });
}

}  // namespace tblaeq
