// Per-level plugin step without a sort (see gridlevel.cuh).
#include "gridlevel.cuh"

#include <algorithm>

#include "knn.cuh"

namespace tblaeq {

namespace {

constexpr uint32_t FULL = 0xffffffffu;

// Range: kept children per entry. KNN: lower bound (root rounded down, as the reference's), reach and children.
__global__ void __launch_bounds__(128) gridBoundKernel(GridLevelArgs a) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) a.bound[0] = a.bound[1] = 0;
    if (i >= a.p) return;
    const NodeRec nr = a.nodes[a.ids[i]];
    const double* x = a.vals + static_cast<size_t>(i) * a.D;
    double dist = 0.0;
    if (a.knn) {
        for (int d = 0; d < a.D; ++d) {
            const double diff = a.q[d] - x[d];
            dist = __fma_rn(diff, diff, dist);
        }
        const double lb = __dsqrt_rd(dist) - nr.rad;
        a.keys[i] = orderKey(lb);
        a.reach[i] = lb + 2.0 * nr.rad;
        a.cnt[i] = nr.cnt;
    } else {
        for (int d = 0; d < a.D; ++d) {
            const double y = x[d], l = a.q[d], h = a.q[a.D + d];
            double diff = 0.0;
            if (y < l) {
                diff = l - y;
            } else if (y > h) {
                diff = y - h;
            }
            dist = __fma_rn(diff, diff, dist);
        }
        a.cnt[i] = dist <= __dmul_rn(nr.rad, nr.rad) ? nr.cnt : 0u;
    }
}

// One warp per entry: whether the children of the entries before it number less than K. Most warps stop
// at the first chunk that passes K.
__global__ void __launch_bounds__(256) gridStepKernel(GridLevelArgs a) {
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) / 32u, lane = threadIdx.x & 31u;
    if (i >= a.p) return;
    const uint64_t key = a.keys[i];
    unsigned long long before = 0;
    for (uint32_t j0 = 0; j0 < a.p && before < a.K; j0 += 256) {
        unsigned long long s = 0;
#pragma unroll
        for (uint32_t t = 0; t < 8; ++t) {
            const uint32_t j = j0 + t * 32 + lane;
            if (j < a.p) {
                const uint64_t k = a.keys[j];
                if (k < key || (k == key && j < i)) s += a.cnt[j];
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(FULL, s, o);
        before += s;
    }
    if (lane) return;
    const bool first = before < a.K;
    a.first[i] = first ? 1 : 0;
    const double r = a.reach[i];
    if (first && r > 0.0) atomicMax(a.bound, static_cast<unsigned long long>(__double_as_longlong(r)));
}

// One CTA: exclusive prefix of the kept entries' children. KNN keeps the first part and every entry
// whose lower bound is within the running bound.
__global__ void __launch_bounds__(1024) gridScanKernel(GridLevelArgs a) {
    __shared__ unsigned long long sCarry, sWarp[32];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint64_t limit = a.knn ? orderKey(__longlong_as_double(static_cast<long long>(a.bound[0]))) : 0;
    if (tid == 0) sCarry = 0;
    __syncthreads();
    for (uint32_t base = 0; base < a.p; base += 4096) {
        const uint32_t i0 = base + tid * 4;
        uint32_t c[4];
        unsigned long long v = 0;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const uint32_t i = i0 + t;
            c[t] = i < a.p && (!a.knn || a.first[i] || a.keys[i] <= limit) ? a.cnt[i] : 0u;
            v += c[t];
        }
        unsigned long long inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(FULL, inc, o);
            if (lane >= static_cast<uint32_t>(o)) inc += t;
        }
        if (lane == 31) sWarp[warp] = inc;
        __syncthreads();
        unsigned long long run = sCarry + inc - v;
        for (uint32_t w = 0; w < warp; ++w) run += sWarp[w];
        const unsigned long long end = run + v;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            if (i0 + t < a.p) a.prefix[i0 + t] = static_cast<uint32_t>(run);
            run += c[t];
        }
        __syncthreads();
        if (tid == 1023) sCarry = end;
        __syncthreads();
    }
    if (tid == 0) {
        a.prefix[a.p] = static_cast<uint32_t>(sCarry);
        a.bound[1] = sCarry;
    }
}

// One thread per output: its entry by bisection over the prefix, the child's id through the map and its
// coordinates rebuilt with one rounded multiply per dimension.
__global__ void __launch_bounds__(256) gridWriteKernel(GridLevelArgs a) {
    const unsigned long long total = a.bound[1];
    if (total > a.outCap) return;  // the host reports it
    for (uint32_t o = blockIdx.x * blockDim.x + threadIdx.x; o < total; o += gridDim.x * blockDim.x) {
        uint32_t lo = 0, hi = a.p - 1;  // the last entry with prefix <= o that has children kept
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1) >> 1;
            if (__ldg(a.prefix + mid) <= o) lo = mid; else hi = mid - 1;
        }
        const NodeRec nr = a.nodes[a.ids[lo]];
        const size_t j = static_cast<size_t>(nr.cbeg) + (o - __ldg(a.prefix + lo));
        a.outIds[o] = a.map[j];
        const double* row = a.rows + j * a.D;
        const double* x = a.vals + static_cast<size_t>(lo) * a.D;
        double* out = a.outVals + static_cast<size_t>(o) * a.D;
        for (int d = 0; d < a.D; ++d) out[d] = __dmul_rn(a.rowsOnHost ? row[d] : __ldg(row + d), x[d]);
    }
}

size_t align256(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }

}  // namespace

size_t gridLevelScratchBytes(uint64_t p) {
    return 2 * align256(p * 8) + align256(p * 4) + align256(p) + align256((p + 1) * 4) + 256;
}

void gridLevelScratch(GridLevelArgs& a, void* scratch) {
    char* b = static_cast<char*>(scratch);
    a.bound = reinterpret_cast<unsigned long long*>(b);
    b += 256;
    a.keys = reinterpret_cast<uint64_t*>(b);
    b += align256(a.p * 8ull);
    a.reach = reinterpret_cast<double*>(b);
    b += align256(a.p * 8ull);
    a.cnt = reinterpret_cast<uint32_t*>(b);
    b += align256(a.p * 4ull);
    a.first = reinterpret_cast<uint8_t*>(b);
    b += align256(a.p);
    a.prefix = reinterpret_cast<uint32_t*>(b);
}

void launchGridLevel(const GridLevelArgs& a, cudaStream_t s) {
    gridBoundKernel<<<(a.p + 127) / 128, 128, 0, s>>>(a);
    TBLAEQ_LAUNCHED();
    if (a.knn) {
        gridStepKernel<<<(a.p + 7) / 8, 256, 0, s>>>(a);
        TBLAEQ_LAUNCHED();
    }
    gridScanKernel<<<1, 1024, 0, s>>>(a);
    TBLAEQ_LAUNCHED();
    const uint64_t most = std::min<uint64_t>(a.outCap, 148ull * 8 * 256);
    gridWriteKernel<<<static_cast<unsigned>(std::max<uint64_t>(1, (most + 255) / 256)), 256, 0, s>>>(a);
    TBLAEQ_LAUNCHED();
}

}  // namespace tblaeq
