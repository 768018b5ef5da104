// Adaptive-partitioning MI (MCPNet's default MI method), GPU form of
//   rank transform            splash::kernel::Rank<T, size_t, 0, false> as called by
//                             apps/pipeline/mcpnet_helper.hpp:122-131 (descending; the splash
//                             source is absent: tied values share the lowest rank here)
//   cumulative histograms     IntegralCumulativeHistogramKernel
//                             include/mcp/correlation/AdaptivePartitioningMI.hpp:414-438
//   per-pair MI               AdaptivePartitionRankMIKernel2::operator() (:535-648) over the
//                             symmetric InnerProduct (mcpnet_helper.hpp:152-163)
//
// Layout (all per gene, rows of n): xr = ranks (uint16), order = sample indices
// sorted by rank (uint16), cH = cumulative rank histogram, m + 1 entries
// (uint16; cH[k] = samples with rank < k).  m <= 16384.
//
// ap_mi_kernel: persistent blocks take the next X gene i from a global
// counter; X's ranks sit in shared memory, each with its quartile of the rank range;
// each warp takes the next Y gene j >= i:
//   * one pass over the samples in y-rank order counts the 4 x 4 grid of x and y quartiles (packed
//     byte counters).  That decides the root window (always split) and its four children, which for
//     unrelated genes is all: no grouped copy of the ranks, no further scan.
//   * a child that splits again is walked as the reference's window quadtree: x ranks
//     grouped by y rank, xg[k] = xr[order_Y[k]] (warp-private shared), and a window's
//     four sub-window counts from one warp-strided scan of its y band
//   * the chi-square split test `fl(S / e) > 7.815` is decided exactly in
//     128-bit integers (S and e are exact in double, so only the rounding of
//     the quotient matters, and it is reproduced against the midpoint of
//     7.815 and its successor)
//   * the depth-first order of the reference (a LIFO of pushed windows) is
//     kept; leaves are queued in that order, over several genes j, and
//     evaluated 32 at a time, one per lane (nxy * log2(nxy / (nx*ny)) in double).  A lane
//     then adds up one pair's leaves in queue order, so every sum has the reference's order.
// FP64 is a narrow pipe here (a warp instruction takes 16 clocks of an SM, however few lanes are
// active) and bound the kernel when every pair evaluated its own four-odd leaves and sums.
// The only source of difference from the reference is log2 (CUDA's vs the
// C library's, each within an ulp).
// Measured (4,096 x 1,024 / 20,000 x 2,000): 28.8 / 879 ms when every pair scanned the root and its children one
// by one and evaluated its own leaves, 8.9 / 359 ms now; at 64 registers (4 blocks per SM: instruction
// fetch and latencies bound it; 80 registers and 3 blocks ran 9.9 / 451 ms).
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "internal.h"

namespace mcpg {
namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int AP_MAX_M = 16384;
constexpr int AP_STACK = 64;   // the LIFO holds at most 3 * depth + 1 <= 46 windows for m <= 16384
constexpr int AP_LEAVES = 40;   // queue: flushed from 32 on, a step queues at most 4 more
constexpr int AP_WARPS = 8;

__device__ __forceinline__ uint32_t order_key_desc(float f) {
    uint32_t u = __float_as_uint(f);
    if ((u & 0x7fffffffu) == 0) u = 0;                      // -0 == +0
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);          // ascending order key
    return ~u;                                               // descending
}

// splitmix64 of (seed, gene, sample): U[0, amp) noise, the reference's tie breaker
// (mi.cpp:121-131 adds U[0, 1e-5) with its own generator).
__device__ __forceinline__ float noise_at(uint64_t seed, int64_t g, int64_t s, float amp) {
    uint64_t z = seed + 0x9E3779B97F4A7C15ull * (uint64_t)(g * 1000003 + s + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (float)((double)(z >> 40) * (1.0 / 16777216.0)) * amp;
}

// One gene per block iteration: bitonic sort of (descending key, sample) in
// shared memory, rank = first sorted position of the value's tie group.
__global__ void __launch_bounds__(1024, 1) ap_rank_kernel(const float* X, int64_t n, int64_t m, int64_t ldx, float amp,
                                                       uint64_t seed, int32_t* R, int64_t ldr, int* flag) {
    extern __shared__ unsigned long long ap_keys[];
    int64_t mp = 1;
    while (mp < m) mp <<= 1;
    for (int64_t g = blockIdx.x; g < n; g += gridDim.x) {
        bool bad = false;
        for (int64_t s = threadIdx.x; s < mp; s += blockDim.x) {
            unsigned long long k = ~0ull;
            if (s < m) {
                float v = X[g * ldx + s];
                if (amp > 0.0f) v = v + noise_at(seed, g, s, amp);
                bad |= (__float_as_uint(v) & 0x7fffffffu) > 0x7f800000u;
                k = ((unsigned long long)order_key_desc(v) << 32) | (unsigned long long)s;
            }
            ap_keys[s] = k;
        }
        if (bad) atomicOr(flag, 1);
        __syncthreads();
        for (int64_t k = 2; k <= mp; k <<= 1)
            for (int64_t j = k >> 1; j > 0; j >>= 1) {
                for (int64_t i = threadIdx.x; i < mp; i += blockDim.x) {
                    const int64_t ixj = i ^ j;
                    if (ixj > i) {
                        const unsigned long long a = ap_keys[i], b = ap_keys[ixj];
                        if ((a > b) == ((i & k) == 0)) {
                            ap_keys[i] = b;
                            ap_keys[ixj] = a;
                        }
                    }
                }
                __syncthreads();
            }
        for (int64_t p = threadIdx.x; p < m; p += blockDim.x) {
            const unsigned long long k = ap_keys[p];
            const unsigned long long hi = k & 0xffffffff00000000ull;
            int64_t lo = 0, up = p;  // first position whose value equals this one
            while (lo < up) {
                const int64_t mid = (lo + up) >> 1;
                if ((ap_keys[mid] & 0xffffffff00000000ull) < hi) lo = mid + 1; else up = mid;
            }
            R[g * ldr + (int64_t)(k & 0xffffffffull)] = (int32_t)lo;
        }
        __syncthreads();
    }
}

// Ranks -> uint16 ranks, the cumulative histogram and the samples ordered by rank.
__global__ void __launch_bounds__(1024) ap_prep_kernel(const int32_t* R, int64_t n, int64_t m, int64_t ldr,
                                                       uint16_t* xr, uint16_t* order, uint16_t* cH, int64_t ldc,
                                                       int* flag) {
    extern __shared__ uint32_t ap_cnt[];  // m + 1 counts, then m + 1 fill cursors
    uint32_t* fillc = ap_cnt + (m + 1);
    __shared__ uint32_t wsum[32];
    for (int64_t g = blockIdx.x; g < n; g += gridDim.x) {
        for (int64_t k = threadIdx.x; k <= m; k += blockDim.x) ap_cnt[k] = fillc[k] = 0;
        __syncthreads();
        bool bad = false;
        for (int64_t s = threadIdx.x; s < m; s += blockDim.x) {
            const int32_t r = R[g * ldr + s];
            if (r < 0 || r >= m) { bad = true; continue; }
            atomicAdd(&ap_cnt[r], 1u);
            xr[g * m + s] = (uint16_t)r;
        }
        if (bad) atomicOr(flag, 1);
        __syncthreads();
        // exclusive scan of ap_cnt[0..m] in place: each thread owns a contiguous chunk
        const int64_t chunk = ceil_div(m + 1, blockDim.x);
        const int64_t c0 = threadIdx.x * chunk;
        const int64_t c1 = c0 + chunk < m + 1 ? c0 + chunk : m + 1;
        uint32_t local = 0;
        for (int64_t k = c0; k < c1; ++k) local += ap_cnt[k];
        uint32_t x = local;
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[w] = x;
        __syncthreads();
        if (w == 0) {
            uint32_t t = lane < (int)(blockDim.x >> 5) ? wsum[lane] : 0;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, t, o);
                if (lane >= o) t += y;
            }
            wsum[lane] = t;
        }
        __syncthreads();
        uint32_t run = (w > 0 ? wsum[w - 1] : 0) + x - local;
        for (int64_t k = c0; k < c1; ++k) {
            const uint32_t v = ap_cnt[k];
            ap_cnt[k] = run;
            run += v;
        }
        __syncthreads();
        for (int64_t k = threadIdx.x; k <= m; k += blockDim.x) cH[g * ldc + k] = (uint16_t)ap_cnt[k];
        for (int64_t s = threadIdx.x; s < m; s += blockDim.x) {
            const int32_t r = R[g * ldr + s];
            if (r < 0 || r >= m) continue;
            const uint32_t pos = ap_cnt[r] + atomicAdd(&fillc[r], 1u);  // order within a tie is irrelevant
            order[g * m + pos] = (uint16_t)s;
        }
        __syncthreads();
    }
}

struct ApWin {
    uint16_t x1, y1, x2, y2;  // exclusive upper bounds
    uint32_t npts;
};

// fl((sum_q (c_q - n/4)^2) / (n/4)) > 7.815 in IEEE double, decided exactly for n = sum_q c_q <= 16384:
// with A = sum_q (4 c_q - n)^2 = 16 sum_q c_q^2 - 4 n^2 (< 2^32) the quotient is A / (4n); 7.815 =
// K * 2^-50 and the rounding boundary above it is (2K + 1) * 2^-51, so the test is A * 2^49 > (2K + 1) n
// (never equal: 2K + 1 is odd and n < 2^49), that is A > floor((2K + 1) n / 2^49).
__device__ __forceinline__ bool chi_square_above(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, uint32_t n) {
    constexpr unsigned long long B = 2 * 8798907771975107ull + 1;  // K = 7.815 * 2^50, exact
    const uint32_t A = 16u * (c0 * c0 + c1 * c1 + c2 * c2 + c3 * c3) - 4u * n * n;
    const unsigned long long t = (B >> 32) * n + (((B & 0xffffffffull) * n) >> 32);
    return A > (uint32_t)(t >> 17);
}

struct ApArgs {
    const uint16_t* xr;
    const uint16_t* order;
    const uint16_t* cH;
    int64_t ldc;
    int64_t n, m;
    float* MI;
    int64_t ldmi;
    unsigned* next_i;
    int* flag;
    int warp_bytes;  // shared bytes per warp
};

// A warp's leaf queue over up to 32 pairs: lane s holds pair slot s, its running sum and its leaves' range
// [beg, end) in the queue.  Evaluates all n <= AP_LEAVES queued leaves and adds each lane's range to sum, in
// queue order.  Not inlined: the instructions of the double logarithm, at each place that queues leaves,
// are more than the instruction cache holds.
__device__ __noinline__ double ap_flush(const uint32_t* nxy, const uint32_t* nxny, double* term, int n, int beg,
                                        int end, double sum) {
    __syncwarp();
    for (int k = threadIdx.x & 31; k < n; k += 32) {
        const double c = (double)nxy[k];
        term[k] = c * log2(c / (double)nxny[k]);
    }
    __syncwarp();
    const int most = (int)__reduce_max_sync(FULL, (unsigned)(end - beg));
    for (int r = 0; r < most; ++r)
        if (beg + r < end) sum += term[beg + r];
    __syncwarp();
    return sum;
}

// UN: samples per lane whose loads and sums a window scan keeps in flight, MINB: blocks per SM (launch_ap_mi).
template <int UN, int MINB>
__global__ void __launch_bounds__(AP_WARPS * 32, MINB) ap_mi_kernel(ApArgs a) {
    extern __shared__ __align__(16) unsigned char ap_smem[];
    __shared__ int s_i;
    __shared__ int s_next_j;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int m = (int)a.m;
    const int xr_bytes = (int)(((int64_t)m * 2 + 15) / 16 * 16);
    uint16_t* xr = (uint16_t*)ap_smem;  // rank | quartile << 14
    unsigned char* wbase = ap_smem + xr_bytes + w * a.warp_bytes;
    ApWin* stack = (ApWin*)wbase;
    double* term = (double*)(wbase + AP_STACK * sizeof(ApWin));
    uint32_t* lnxy = (uint32_t*)(term + AP_LEAVES);
    uint32_t* lnxny = lnxy + AP_LEAVES;
    uint16_t* xg = (uint16_t*)(lnxny + AP_LEAVES);
    int nq = 0, beg = 0, end = 0;  // queued leaves; this lane's slot's range
    double sum = 0.0;
    auto flush = [&]() {
        sum = ap_flush(lnxy, lnxny, term, nq, beg, end, sum);
        beg = end = nq = 0;
    };
    const double logm = log2((double)m);
    // the grid's boundaries: the midpoints of the root window and of its children
    const int half = m >> 1, lo4 = half >> 1, hi4 = (half + m) >> 1;

    for (;;) {
        if (threadIdx.x == 0) {
            s_i = (int)atomicAdd(a.next_i, 1u);
            s_next_j = s_i;
        }
        __syncthreads();
        const int i = s_i;
        if (i >= a.n) break;
        for (int s = threadIdx.x; s < m; s += blockDim.x) {
            const int r = a.xr[(int64_t)i * m + s];
            xr[s] = (uint16_t)(r | (((r >= lo4) + (r >= half) + (r >= hi4)) << 14));
        }
        __syncthreads();
        const uint16_t* cX = a.cH + (int64_t)i * a.ldc;
        const int nx_lo = cX[half], nx_hi = (int)cX[m] - nx_lo;
        int slot = 0, jmine = 0;
        bool broken_mine = false;
        bool more = true;
        while (more) {
            int j = 0;
            if (lane == 0) j = atomicAdd(&s_next_j, 1);
            j = __shfl_sync(FULL, j, 0);
            more = j < a.n;
            if (slot == 32 || !more) {  // the batch's pairs are complete
                flush();
                if (lane < slot) {
                    float v = (float)(sum / (double)m + logm);
                    if (broken_mine) {
                        v = __int_as_float(0x7fc00000);
                        atomicOr(a.flag, 2);
                    }
                    a.MI[(int64_t)i * a.ldmi + jmine] = v;
                    a.MI[(int64_t)jmine * a.ldmi + i] = v;
                }
                slot = 0;
                if (!more) break;
            }
            if (lane == slot) {
                sum = 0.0;
                beg = end = nq;
                jmine = j;
                broken_mine = false;
            }
            const uint16_t* oY = a.order + (int64_t)j * m;
            const uint16_t* cY = a.cH + (int64_t)j * a.ldc;
            // y boundaries as positions in rank order
            int bnd = 0;
            if (lane < 5) bnd = cY[lane == 0 ? 0 : lane == 1 ? lo4 : lane == 2 ? half : lane == 3 ? hi4 : m];
            int bpos[5];
#pragma unroll
            for (int e = 0; e < 5; ++e) bpos[e] = __shfl_sync(FULL, bnd, e);
            uint32_t g[4][4];  // [y quartile][x quartile]
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                uint32_t acc = 0;  // four byte counters, widened before a lane has added 255 samples
                uint32_t wide = 0, wide2 = 0;
                int k = bpos[e] + lane;
                int left = 255;
                for (; k + 96 < bpos[e + 1]; k += 128) {
                    const uint32_t o0 = oY[k], o1 = oY[k + 32], o2 = oY[k + 64], o3 = oY[k + 96];
                    const uint32_t v0 = xr[o0], v1 = xr[o1], v2 = xr[o2], v3 = xr[o3];
                    acc += (1u << ((v0 >> 11) & 24u)) + (1u << ((v1 >> 11) & 24u));
                    acc += (1u << ((v2 >> 11) & 24u)) + (1u << ((v3 >> 11) & 24u));
                    left -= 4;
                    if (left < 4) {  // widen before a byte can overflow
                        wide += (acc & 0xffu) + ((acc & 0xff00u) << 8);
                        wide2 += ((acc >> 16) & 0xffu) + ((acc >> 24) << 16);
                        acc = 0;
                        left = 255;
                    }
                }
                for (; k < bpos[e + 1]; k += 32) acc += 1u << (((uint32_t)xr[oY[k]] >> 11) & 24u);
                wide += (acc & 0xffu) + ((acc & 0xff00u) << 8);
                wide2 += ((acc >> 16) & 0xffu) + ((acc >> 24) << 16);
                wide = __reduce_add_sync(FULL, wide);  // 16-bit halves: at most m <= 16384 each
                wide2 = __reduce_add_sync(FULL, wide2);
                g[e][0] = wide & 0xffffu;
                g[e][1] = wide >> 16;
                g[e][2] = wide2 & 0xffffu;
                g[e][3] = wide2 >> 16;
            }
            // the root's children in the reference's order, one per lane 0..3: (x low, y low), (high, low),
            // (low, high), (high, high)
            const bool xh = lane & 1, yh = lane & 2;
            const uint32_t c0 = yh ? (xh ? g[2][2] : g[2][0]) : (xh ? g[0][2] : g[0][0]);
            const uint32_t c1 = yh ? (xh ? g[2][3] : g[2][1]) : (xh ? g[0][3] : g[0][1]);
            const uint32_t c2 = yh ? (xh ? g[3][2] : g[3][0]) : (xh ? g[1][2] : g[1][0]);
            const uint32_t c3 = yh ? (xh ? g[3][3] : g[3][1]) : (xh ? g[1][3] : g[1][1]);
            const uint32_t cc = c0 + c1 + c2 + c3;
            const uint32_t area = (uint32_t)(xh ? nx_hi : nx_lo) *
                                  (uint32_t)(yh ? bpos[4] - bpos[2] : bpos[2] - bpos[0]);
            const bool wide_enough = 1 < (xh ? m - half : half) || 1 < (yh ? m - half : half);
            const bool splittable = lane < 4 && wide_enough && cc > 2;
            const bool leaf_now = lane < 4 && !splittable && cc > 0;
            const unsigned msplit = __ballot_sync(FULL, splittable), mleaf = __ballot_sync(FULL, leaf_now);
            const unsigned magain = __ballot_sync(FULL, splittable && chi_square_above(c0, c1, c2, c3, cc));
            // leaves of the root's own step first, then the children from the last to the first
            const int at = leaf_now ? __popc(mleaf & ((1u << lane) - 1u)) : __popc(mleaf) + __popc(msplit >> (lane + 1));
            if (leaf_now || (splittable && !magain)) {
                lnxy[nq + at] = cc;
                lnxny[nq + at] = area;
            }
            nq += __popc(mleaf) + (magain ? 0 : __popc(msplit));
            if (lane == slot) end = nq;
            if (!magain) {
                ++slot;
                if (nq >= 32) flush();
                continue;
            }
#pragma unroll(UN < 4 ? 4 : UN)
            for (int k = lane; k < m; k += 32) xg[k] = xr[oY[k]] & 0x3fffu;
            __syncwarp();
            bool broken = false;
            int64_t guard = 0;
#pragma unroll 1
            for (int c = 3; c >= 0; --c) {
                if (!((msplit >> c) & 1u)) continue;
                const uint32_t ccc = __shfl_sync(FULL, cc, c), ar = __shfl_sync(FULL, area, c);
                if (!((magain >> c) & 1u)) {
                    if (lane == 0) {
                        lnxy[nq] = ccc;
                        lnxny[nq] = ar;
                    }
                    ++nq;
                    if (lane == slot) end = nq;
                    continue;
                }
                if (lane == 0)
                    stack[0] = ApWin{(uint16_t)((c & 1) ? half : 0), (uint16_t)((c >> 1) ? half : 0),
                                     (uint16_t)((c & 1) ? m : half), (uint16_t)((c >> 1) ? m : half), ccc};
                __syncwarp();
                int top = 1;
                bool from_grid = true;
#pragma unroll 1
                while (top > 0) {
                    if (++guard > 16ll * m + 64) {  // cannot happen: every pushed window is smaller than its parent
                        broken = true;
                        break;
                    }
                    if (nq >= 32) flush();
                    const ApWin wv = stack[top - 1];
                    __syncwarp();
                    const int mx = (wv.x1 + wv.x2) >> 1, my = (wv.y1 + wv.y2) >> 1;
                    uint32_t d0, d1, d2, d3;
                    if (from_grid) {  // the child itself: its counts and its split are known
                        d0 = __shfl_sync(FULL, c0, c);
                        d1 = __shfl_sync(FULL, c1, c);
                        d2 = __shfl_sync(FULL, c2, c);
                        d3 = __shfl_sync(FULL, c3, c);
                    } else {
                        const unsigned wl = mx - wv.x1, wa = wv.x2 - wv.x1;
                        const int b1 = cY[my];
                        // per y half: samples left of mx, and in the window
                        auto scan = [&](int from, int to, uint32_t& low, uint32_t& high) {
                            uint32_t l = 0, all = 0;
                            int k = from + lane;
                            if (UN > 2) {
                                uint32_t lu[UN] = {}, au[UN] = {};
#pragma unroll 1
                                for (; k + 32 * (UN - 1) < to; k += 32 * UN) {
                                    unsigned x[UN];
#pragma unroll
                                    for (int u = 0; u < UN; ++u) x[u] = (unsigned)xg[k + 32 * u] - wv.x1;
#pragma unroll
                                    for (int u = 0; u < UN; ++u) {
                                        lu[u] += x[u] < wl;
                                        au[u] += x[u] < wa;
                                    }
                                }
#pragma unroll
                                for (int u = 0; u < UN; ++u) {
                                    l += lu[u];
                                    all += au[u];
                                }
                            }
#pragma unroll 2
                            for (; k < to; k += 32) {
                                const unsigned x = (unsigned)xg[k] - wv.x1;
                                l += x < wl;
                                all += x < wa;
                            }
                            low = __reduce_add_sync(FULL, l);
                            high = __reduce_add_sync(FULL, all) - low;
                        };
                        scan(cY[wv.y1], b1, d0, d1);
                        scan(b1, cY[wv.y2], d2, d3);
                    }
                    --top;
                    if (from_grid || chi_square_above(d0, d1, d2, d3, wv.npts)) {
                        from_grid = false;
                        const int sx1[4] = {wv.x1, mx, wv.x1, mx}, sx2[4] = {mx, wv.x2, mx, wv.x2};
                        const int sy1[4] = {wv.y1, wv.y1, my, my}, sy2[4] = {my, my, wv.y2, wv.y2};
                        const uint32_t sc[4] = {d0, d1, d2, d3};
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const bool split = ((sx1[u] + 1) < sx2[u] || (sy1[u] + 1) < sy2[u]) && sc[u] > 2;
                            if (split) {
                                if (top >= AP_STACK) {
                                    broken = true;
                                    continue;
                                }
                                if (lane == 0)
                                    stack[top] = ApWin{(uint16_t)sx1[u], (uint16_t)sy1[u], (uint16_t)sx2[u],
                                                       (uint16_t)sy2[u], sc[u]};
                                ++top;
                            } else if (sc[u] > 0) {
                                if (lane == 0) {
                                    lnxy[nq] = sc[u];
                                    lnxny[nq] = (uint32_t)(cX[sx2[u]] - cX[sx1[u]]) * (uint32_t)(cY[sy2[u]] - cY[sy1[u]]);
                                }
                                ++nq;
                            }
                        }
                    } else {
                        if (lane == 0) {
                            lnxy[nq] = wv.npts;
                            lnxny[nq] = (uint32_t)(cX[wv.x2] - cX[wv.x1]) * (uint32_t)(cY[wv.y2] - cY[wv.y1]);
                        }
                        ++nq;
                    }
                    if (lane == slot) end = nq;
                    __syncwarp();
                    if (broken) break;
                }
                if (broken) break;
            }
            if (broken && lane == slot) broken_mine = true;
            __syncwarp();
            ++slot;
            if (nq >= 32) flush();
        }
        __syncthreads();
    }
}

}  // namespace

int64_t ap_max_samples() { return AP_MAX_M; }

cudaError_t launch_ap_ranks(const float* X, int64_t n, int64_t m, int64_t ldx, float noise, uint64_t seed,
                            int32_t* R, int64_t ldr, int* flag, cudaStream_t st, int64_t* launches) {
    if (n <= 0 || m <= 0) return cudaSuccess;
    if (m > AP_MAX_M) return cudaErrorNotSupported;
    int64_t mp = 1;
    while (mp < m) mp <<= 1;
    const size_t smem = (size_t)mp * 8;
    cudaError_t e = cudaFuncSetAttribute(ap_rank_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int threads = mp >= 1024 ? 1024 : (int)(mp < 32 ? 32 : mp);
    const int64_t grid = n < 152 * 2 ? n : 152 * 2;
    ap_rank_kernel<<<(unsigned)grid, threads, smem, st>>>(X, n, m, ldx, noise, seed, R, ldr, flag);
    if (launches) ++*launches;
    return cudaGetLastError();
}

cudaError_t launch_ap_prep(const int32_t* R, int64_t n, int64_t m, int64_t ldr, uint16_t* xr, uint16_t* order,
                           uint16_t* cH, int64_t ldc, int* flag, cudaStream_t st, int64_t* launches) {
    if (n <= 0 || m <= 0) return cudaSuccess;
    if (m > AP_MAX_M) return cudaErrorNotSupported;
    const size_t smem = (size_t)(m + 1) * 2 * sizeof(uint32_t);
    cudaError_t e = cudaFuncSetAttribute(ap_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int64_t grid = n < 152 * 4 ? n : 152 * 4;
    ap_prep_kernel<<<(unsigned)grid, 512, smem, st>>>(R, n, m, ldr, xr, order, cH, ldc, flag);
    if (launches) ++*launches;
    return cudaGetLastError();
}

cudaError_t launch_ap_mi(const uint16_t* xr, const uint16_t* order, const uint16_t* cH, int64_t ldc, int64_t n,
                         int64_t m, float* MI, int64_t ldmi, unsigned* next_i, int* flag, cudaStream_t st,
                         int64_t* launches) {
    if (n <= 0 || m <= 0) return cudaSuccess;
    if (m > AP_MAX_M) return cudaErrorNotSupported;
    ApArgs a;
    a.xr = xr;
    a.order = order;
    a.cH = cH;
    a.ldc = ldc;
    a.n = n;
    a.m = m;
    a.MI = MI;
    a.ldmi = ldmi;
    a.next_i = next_i;
    a.flag = flag;
    a.warp_bytes = (int)(AP_STACK * sizeof(ApWin) + AP_LEAVES * (sizeof(double) + 2 * sizeof(uint32_t)) +
                         ((int64_t)m * 2 + 15) / 16 * 16);
    int dev = 0, sms = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    const size_t xr_bytes = (size_t)((m * 2 + 15) / 16 * 16);
    // warps per block: up to AP_WARPS, as many as the shared memory holds (m = 16384: 5)
    int64_t warps = ((int64_t)optin - 1024 - (int64_t)xr_bytes) / a.warp_bytes;
    if (warps > AP_WARPS) warps = AP_WARPS;
    if (warps < 1) return cudaErrorNotSupported;
    const size_t smem = xr_bytes + (size_t)warps * a.warp_bytes;
    // With many genes and up to about 2,500 samples four blocks of 64 registers share an SM, and their warps hide a
    // scan's latencies.  Where the ranks or the genes leave it fewer, a scan has to keep more in flight itself: tied
    // values, 100 x 16,384 13.9 -> 8.5 ms, 100 x 8,192 4.9 -> 3.5 ms.
    auto* const kernel = n > 2 * sms && 4 * (smem + 1024) <= 228 * 1024 ? ap_mi_kernel<2, 4> : ap_mi_kernel<8, 2>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, (int)warps * 32, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorNotSupported;
    e = cudaMemsetAsync(next_i, 0, sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    int64_t grid = (int64_t)sms * per_sm;
    if (grid > n) grid = n;
    kernel<<<(unsigned)grid, (unsigned)(warps * 32), smem, st>>>(a);
    if (launches) ++*launches;
    return cudaGetLastError();
}

}  // namespace mcpg
