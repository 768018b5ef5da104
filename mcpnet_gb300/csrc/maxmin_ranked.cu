// Max-min products with the candidates k visited in descending order of one operand.
//
//   C[i][j] = max_k min(O[i][k], X[j][k])
//
// For an output (i, j) only the k with O[i][k] > C[i][j] matter, and on similarity
// matrices they are few: with independent rows the maximum sits near the
// sqrt(k)-th largest value of each row.  So each owner row i gets the list of its
// largest entries, (value, k) in descending order, and a warp walks that list for 128
// columns j at once: acc = max(acc, min(value, X[j][k])).  When every lane's acc has
// reached the next value of the list, no later k can raise it: the outputs are final.
// A selection has no rounding, so the bits are those of the exhaustive product.
//
// The walk reads X transposed, XT[k][j], 512 contiguous bytes per (k, warp): it is bound
// by L2-to-SM bandwidth (4 bytes per candidate), and visits a few percent of the
// n^3 candidates.  Column blocks are the slow grid axis, so the k x 128 slab that the
// resident CTAs read stays in L2.
//
// A symmetric product (O == X) needs each pair once, and the pair is cheaper from the
// row whose large values are smaller (the capacity is limited by that row: few of its
// entries exceed it, while a strongly connected row has many).  Rows are ordered by
// the strength of their 2 sqrt(k)-th largest value, weakest first, and the walk runs on
// the upper triangle of the product in that order, in a scratch matrix P that the last
// kernel reads back in gene order (with the MCP ratio fused).
//
// Outputs whose list ends too early go to a pending list and are completed one warp each
// from the other row's list, and where that is not enough from both whole rows.  If
// more outputs stay open than the pending list holds (data without such structure: many
// ties, closures), or an operand holds a NaN, a device-side count tells the exhaustive kernel
// (maxmin.cu), which is always enqueued behind and otherwise returns at once, to run.  No
// host synchronisation: the sequence stays asynchronous.
//
// Measured on MI-like matrices (symmetric product with ratio, whole call; exhaustive form ->
// this one): 20,000 genes 338 -> 18.8 ms (walk 13.5, lists 2.1, finish 1.6, transpose 1.1 ms); M1..M3
// with ratios at 2,000 genes 1.79 -> 0.46 ms; 300 genes, one product, 71 -> 49 us.  ncu at 8,192 genes: the
// walk keeps L1 and L2 at 77 % of their throughput, 97 % of its L1 misses hit L2.
#include <float.h>
#include <math.h>

#include <algorithm>

#include "common.cuh"
#include "internal.h"

namespace mcpg {
namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int LIST_TPB = 512;
constexpr int LIST_MAX = 1024;   // longest list (sort buffer)
constexpr int BATCH = 8;         // list entries between two exit tests
constexpr int COLS = 128;        // columns of a warp: a float4 per lane
constexpr int OWN = 8;           // owners (warps) of a CTA

// Order-preserving map of the float bits to signed integers (-0 below +0).
__device__ __forceinline__ int okey(float f) {
    const int u = __float_as_int(f);
    return u ^ ((u >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float okey_value(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }

// Whether the ranked form gave up: too many pending outputs, or a NaN operand (the exhaustive
// kernel behind it runs on the same condition).
__device__ __forceinline__ bool gave_up(const RankedArgs& a) {
    return *(const volatile unsigned long long*)a.pending_n > (unsigned long long)a.pending_cap || *a.nan != 0 ||
           (a.full_n && *(const volatile unsigned long long*)a.full_n > a.full_cap);
}
// The operands as choose_kernel assigned them: *flip == 1 makes X's rows the owners.
template <bool FLIP>
__device__ __forceinline__ RankedArgs oriented(RankedArgs a) {
    if (FLIP) {
        if (*a.flip == 1) {
            const float* o = a.O; a.O = a.X; a.X = o;
            const int64_t l = a.ldo; a.ldo = a.ldx; a.ldx = l;
            const int r = a.owners; a.owners = a.cols; a.cols = r;
            const int d = a.direct; a.direct = a.mirror; a.mirror = d;
        }
        a.ldt = (int64_t)(a.cols + COLS - 1) / COLS * COLS;
    }
    return a;
}
// The owners and columns of this CTA; FLIP: a one-dimensional grid that covers either assignment.
template <bool FLIP>
__device__ __forceinline__ bool tile_at(const RankedArgs& a, int& o0, int& p0) {
    if (FLIP) {
        const int nb = (a.owners + OWN - 1) / OWN;
        o0 = (int)(blockIdx.x % nb) * OWN;
        p0 = (int)(blockIdx.x / nb) * COLS;
        return p0 < a.cols;
    }
    o0 = blockIdx.x * OWN;
    p0 = blockIdx.y * COLS;
    return true;
}
dim3 tile_grid(const RankedArgs& a) {
    if (!a.flip) return dim3((unsigned)ceil_div(a.owners, OWN), (unsigned)ceil_div(a.cols, COLS));
    const int64_t t0 = ceil_div(a.owners, OWN) * ceil_div(a.cols, COLS), t1 = ceil_div(a.cols, OWN) * ceil_div(a.owners, COLS);
    return dim3((unsigned)std::max(t0, t1));
}
// 16 bytes through the read-only path; volatile keeps a batch's loads together and in front
// of their uses.
__device__ __forceinline__ float4 ldg4(const float* p) {
    float4 v;
    asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// One CTA per owner row (LOOP: per several): the row's keys sit in registers (EPT per thread); a bisection on the
// key counts entries above a pivot until between want and cap are, they are compacted
// and sorted (bitonic, key then index).  bound[i] = an upper bound of every entry not
// listed (-inf when all are).  Entries are padded to a multiple of BATCH with -inf.
template <int EPT, bool LOOP>
__global__ void __launch_bounds__(LIST_TPB, EPT <= 16 ? 3 : 1) lists_kernel(const float* __restrict__ O, int64_t ldo, int rows, int k,
                                                         int want, int cap, int strength_at, int skip_diag,
                                                         RankedLists L, unsigned long long* any_nan,
                                                         const unsigned long long* only_above,
                                                         unsigned long long only_cap, const RankedOther alt) {
    if (only_above && *only_above <= only_cap) return;  // uniform: no barrier is passed yet
    if (alt.flip && *alt.flip) {
        if (*alt.flip == 2) return;
        O = alt.O; ldo = alt.ldo; rows = alt.rows;
    }
    __shared__ unsigned long long buf[LIST_MAX];
    __shared__ int wcount[LIST_TPB / 32];
    __shared__ int fill;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int i = blockIdx.x;
    if (i >= rows) return;
    do {
        const float* row = O + (int64_t)i * ldo;
        int key[EPT];
        bool nan = false;
        int mn = INT_MAX, mx = INT_MIN;
#pragma unroll
        for (int e = 0; e < EPT; ++e) {
            const int c = tid + e * LIST_TPB;
            key[e] = INT_MIN;  // below okey(-inf): never counted
            if (c < k && !(skip_diag && c == i)) {
                const float v = row[c];
                nan |= (v != v);
                key[e] = okey(v);
                mn = min(mn, key[e]);
                mx = max(mx, key[e]);
            }
        }
        if (nan) *any_nan = 1;  // NaN has no place in the order: the exhaustive kernel takes the product
        auto block_sum = [&](int v) {
            v = __reduce_add_sync(FULL, v);
            __syncthreads();
            if (lane == 0) wcount[warp] = v;
            __syncthreads();
            int s = lane < LIST_TPB / 32 ? wcount[lane] : 0;
            return __reduce_add_sync(FULL, s);
        };
        auto above = [&](int pivot) {
            int c = 0;
#pragma unroll
            for (int e = 0; e < EPT; ++e) c += key[e] > pivot;
            return block_sum(c);
        };
        {
            mn = __reduce_min_sync(FULL, mn);
            mx = __reduce_max_sync(FULL, mx);
            __shared__ int smn[LIST_TPB / 32], smx[LIST_TPB / 32];
            if (lane == 0) { smn[warp] = mn; smx[warp] = mx; }
            __syncthreads();
            mn = __reduce_min_sync(FULL, lane < LIST_TPB / 32 ? smn[lane] : INT_MAX);
            mx = __reduce_max_sync(FULL, lane < LIST_TPB / 32 ? smx[lane] : INT_MIN);
        }
        // invariant: above(lo) > cap, above(hi) < want
        int pivot, n_above;
        const int avail = k - (skip_diag && i < k);  // entries that may be listed
        if (avail <= cap) {
            pivot = INT_MIN;  // everything is listed
            n_above = avail;
        } else {
            long long lo = (long long)mn - 1, hi = mx;
            pivot = mx;
            n_above = 0;
            while (hi - lo > 1) {
                const int mid = (int)(lo + (hi - lo) / 2);
                const int c = above(mid);
                if (c > cap) lo = mid;
                else {
                    hi = mid;
                    pivot = mid;
                    n_above = c;
                    if (c >= want) break;
                }
            }
        }
        // entries above the pivot, then entries equal to it as far as the list has room
        if (tid == 0) fill = 0;
        __syncthreads();
        for (int pass = 0; pass < 2; ++pass) {
            if (pass == 1 && (avail <= cap || n_above >= want)) break;
#pragma unroll
            for (int e = 0; e < EPT; ++e) {
                const bool take = key[e] != INT_MIN && (pass == 0 ? key[e] > pivot : key[e] == pivot);
                const unsigned b = __ballot_sync(FULL, take);
                if (!b) continue;
                int base = 0;
                if (lane == 0) base = atomicAdd(&fill, __popc(b));
                base = __shfl_sync(FULL, base, 0);
                const int at = base + __popc(b & ((1u << lane) - 1u));
                if (take && at < cap)
                    buf[at] = ((unsigned long long)((unsigned)key[e] ^ 0x80000000u) << 32) | (unsigned)(tid + e * LIST_TPB);
            }
            __syncthreads();
        }
        const int count = min(fill, cap);
        int p2 = 32;
        while (p2 < count) p2 <<= 1;
        for (int t = count + tid; t < p2; t += LIST_TPB) buf[t] = 0;
        __syncthreads();
        if (p2 == LIST_TPB) {
            // one entry per thread: partners less than a warp apart exchange by shuffle, without a barrier (shorter
            // lists leave warps idle here and sort faster below: 44 against 54 us for 2,000 rows)
            unsigned long long v = buf[tid];
            for (int s = 2; s <= LIST_TPB; s <<= 1) {
                const bool down = (tid & s) == 0;
                for (int j = s >> 1; j > 0; j >>= 1) {
                    unsigned long long u;
                    if (j >= 32) {
                        __syncthreads();
                        buf[tid] = v;
                        __syncthreads();
                        u = buf[tid ^ j];
                    } else {
                        u = __shfl_xor_sync(FULL, v, j);
                    }
                    const bool first = (tid & j) == 0;  // the lower position keeps the larger where descending
                    v = (first == down) ? (u > v ? u : v) : (u < v ? u : v);
                }
            }
            __syncthreads();
            buf[tid] = v;
            __syncthreads();
        } else {
            for (int s = 2; s <= p2; s <<= 1)
                for (int j = s >> 1; j > 0; j >>= 1) {
                    for (int t = tid; t < p2 / 2; t += LIST_TPB) {
                        const int x = ((t & ~(j - 1)) << 1) | (t & (j - 1)), y = x | j;
                        const unsigned long long a = buf[x], b = buf[y];
                        if ((a < b) == ((x & s) == 0)) {
                            buf[x] = b;
                            buf[y] = a;
                        }
                    }
                    __syncthreads();
                }
        }
        const int padded = (count + BATCH - 1) / BATCH * BATCH;
        uint2* out = L.entries + (int64_t)i * L.pitch;
        for (int t = tid; t < padded; t += LIST_TPB) {
            uint2 e = make_uint2(0xff800000u, 0u);  // -inf
            if (t < count) {
                const unsigned long long v = buf[t];
                e.x = __float_as_uint(okey_value((int)((unsigned)(v >> 32) ^ 0x80000000u)));
                e.y = (unsigned)v;
            }
            out[t] = e;
        }
        if (tid == 0) {
            const bool all = count == avail;
            L.count[i] = count;
            L.bound[i] = all ? -INFINITY : okey_value(pivot);
            L.strength[i] = strength_at < count ? (int)((unsigned)(buf[strength_at] >> 32) ^ 0x80000000u)
                                                : (all ? INT_MIN : pivot);
        }
        i += gridDim.x;
    } while (LOOP && i < rows);
}

// rank[i] = position of row i by ascending strength (ties by index), perm = its inverse.
__global__ void __launch_bounds__(256) order_kernel(const int* __restrict__ strength, int n, int* __restrict__ rank,
                                                    int* __restrict__ perm) {
    const int i = (blockIdx.x * 256 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= n) return;
    const int s = strength[i];
    int c = 0;
    for (int j = lane; j < n; j += 32) {
        const int t = strength[j];
        c += (t < s) || (t == s && j < i);
    }
    c = __reduce_add_sync(FULL, c);
    if (lane == 0) {
        rank[i] = c;
        perm[c] = i;
    }
}

// XT[k][p] = X[perm ? perm[p] : p][k] (skip_diag: -inf for k equal to the row); columns p in [rows, ldt) are +inf (they never keep a
// warp from its exit).
__global__ void __launch_bounds__(256) transpose_kernel(const float* __restrict__ X, int64_t ldx, int rows, int k,
                                                        int skip_diag, const int* __restrict__ perm, float* __restrict__ XT,
                                                        int64_t ldt, unsigned long long* any_nan) {
    __shared__ float tile[32][33];
    const int p0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
    for (int r = ty; r < 32; r += 8) {
        const int p = p0 + r, c = k0 + tx;
        float v = INFINITY;
        if (p < rows && c < k) {
            const int i = perm ? perm[p] : p;
            v = skip_diag && c == i ? -INFINITY : X[(int64_t)i * ldx + c];
        }
        if (v != v) *any_nan = 1;
        tile[r][tx] = v;
    }
    __syncthreads();
#pragma unroll
    for (int r = ty; r < 32; r += 8)
        if (k0 + r < k) XT[(int64_t)(k0 + r) * ldt + p0 + tx] = tile[tx][r];
}

// The same of the operand that does not own, after choose_kernel (32 x 32 tiles, each CTA several).
__global__ void __launch_bounds__(256) transpose_chosen_kernel(const RankedArgs a0, float* __restrict__ XT,
                                                               unsigned long long* any_nan) {
    __shared__ float tile[32][33];
    if (*a0.flip == 2) return;
    const RankedArgs a = oriented<true>(a0);
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int nb = (int)(a.ldt / 32), tiles = nb * ((a.k + 31) / 32);
    for (int b = blockIdx.x; b < tiles; b += gridDim.x) {
        const int p0 = b % nb * 32, k0 = b / nb * 32;
#pragma unroll
        for (int r = ty; r < 32; r += 8) {
            const int p = p0 + r, c = k0 + tx;
            const float v = p < a.cols && c < a.k ? a.X[(int64_t)p * a.ldx + c] : INFINITY;
            if (v != v) *any_nan = 1;
            tile[r][tx] = v;
        }
        __syncthreads();
#pragma unroll
        for (int r = ty; r < 32; r += 8)
            if (k0 + r < a.k) XT[(int64_t)(k0 + r) * a.ldt + p0 + tx] = tile[tx][r];
        __syncthreads();
    }
}

// Which operand's rows own the lists: a CTA per sampled output counts the candidates above it in either row.  An
// output whose owner's list of `cap` entries ends before them pends.  *flip = 1: the samples that pend with O's rows as
// owners are near what the product may leave pending (`most`), and with X's rows at most half as many do;
// 2: for a quarter of the samples neither row's list is long enough, more than any product can finish, or with either
// owner far more would pend than may: the exhaustive kernel is told to run at once.  M1 (x) A at 2,000 genes takes 0.20
// ms; from M1's rows it gave up after the walk, 1.07 ms (0.82 exhaustive).  The samples take 5 to 8 us.
// sum: zeroed; 16 bits each for the samples that pend with O as owner, with X, with both, and for those done (one
// atomic: the last CTA has the totals from its result).
constexpr int SAMPLES = 64, CHOOSE_TPB = 512;
__global__ void __launch_bounds__(CHOOSE_TPB) choose_kernel(const RankedArgs a, int cap, int most, int* flip,
                                                           unsigned long long* sum) {
    __shared__ int part[2][CHOOSE_TPB / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned x = (blockIdx.x + 1u) * 2654435761u, y = (x ^ (x >> 15)) * 2246822519u;
    const float* ro = a.O + (int64_t)(x % (unsigned)a.owners) * a.ldo;
    const float* rx = a.X + (int64_t)((y ^ (y >> 13)) % (unsigned)a.cols) * a.ldx;
    int m = INT_MIN;
#pragma unroll 4
    for (int c = threadIdx.x; c < a.k; c += CHOOSE_TPB) m = max(m, okey(fmin2(__ldg(ro + c), __ldg(rx + c))));
    m = __reduce_max_sync(FULL, m);
    if (lane == 0) part[0][w] = m;
    __syncthreads();
    m = __reduce_max_sync(FULL, lane < CHOOSE_TPB / 32 ? part[0][lane] : INT_MIN);
    __syncthreads();
    int no = 0, nx = 0;
#pragma unroll 4
    for (int c = threadIdx.x; c < a.k; c += CHOOSE_TPB) {
        no += okey(__ldg(ro + c)) > m;
        nx += okey(__ldg(rx + c)) > m;
    }
    no = __reduce_add_sync(FULL, no);
    nx = __reduce_add_sync(FULL, nx);
    if (lane == 0) {
        part[0][w] = no;
        part[1][w] = nx;
    }
    __syncthreads();
    if (w != 0) return;
    no = __reduce_add_sync(FULL, lane < CHOOSE_TPB / 32 ? part[0][lane] : 0);
    nx = __reduce_add_sync(FULL, lane < CHOOSE_TPB / 32 ? part[1][lane] : 0);
    if (lane != 0) return;
    const unsigned long long one = (unsigned long long)(no > cap) | (unsigned long long)(nx > cap) << 16 |
                                   (unsigned long long)(no > cap && nx > cap) << 32 | 1ull << 48;
    const unsigned long long all = atomicAdd(sum, one) + one;
    if ((all >> 48) != SAMPLES) return;
    const int po = (int)(all & 0xffff), px = (int)(all >> 16 & 0xffff), both = (int)(all >> 32 & 0xffff);
    if (both > SAMPLES / 4 || min(po, px) > 2 * most + 4) {
        *flip = 2;
        *a.pending_n = (unsigned long long)a.pending_cap + 1;
    } else if (po > most && 2 * px <= po) {
        *flip = 1;
    }
}

// One warp per (owner, 128 columns).  SYM: owners and columns in strength order, columns
// at or after the owner only.
template <bool SYM, bool FLIP = false>
__global__ void __launch_bounds__(OWN * 32) walk_kernel(const RankedArgs a0) {
    __shared__ float tile[OWN][COLS + 4];
    if (__syncthreads_or(threadIdx.x == 0 && gave_up(a0))) return;
    const RankedArgs a = oriented<FLIP>(a0);
    int o0, p0;
    if (!tile_at<FLIP>(a, o0, p0)) return;
    if (SYM && p0 + COLS <= o0) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int o = o0 + w, p = p0 + lane * 4;
    if (o < a.owners && !(SYM && p0 + COLS <= o)) {
        const int i = SYM ? a.perm[o] : o;
        const uint4* list = reinterpret_cast<const uint4*>(a.L.entries + (int64_t)i * a.L.pitch);
        const int count = a.L.count[i];
        const float bound = a.L.bound[i];
        const float* col = a.XT + p;
        // columns before the owner belong to other warps
        const bool live0 = !SYM || p >= o, live1 = !SYM || p + 1 >= o, live2 = !SYM || p + 2 >= o,
                   live3 = !SYM || p + 3 >= o;
        float4 acc = make_float4(live0 ? -INFINITY : INFINITY, live1 ? -INFINITY : INFINITY,
                                 live2 ? -INFINITY : INFINITY, live3 ? -INFINITY : INFINITY);
        bool open = count == 0;
        for (int t = 0; t < count; t += BATCH) {
            uint4 e[BATCH / 2];
            float4 b[BATCH];
#pragma unroll
            for (int u = 0; u < BATCH / 2; ++u) e[u] = __ldg(list + t / 2 + u);
#pragma unroll
            for (int u = 0; u < BATCH / 2; ++u) {
                b[2 * u] = ldg4(col + (int64_t)e[u].y * a.ldt);
                b[2 * u + 1] = ldg4(col + (int64_t)e[u].w * a.ldt);
            }
            // the largest entry not yet visited
            const float next = t + BATCH < count ? __uint_as_float(__ldg(&list[t / 2 + BATCH / 2].x)) : bound;
#pragma unroll
            for (int u = 0; u < BATCH / 2; ++u) {
                const float v0 = __uint_as_float(e[u].x), v1 = __uint_as_float(e[u].z);
                acc.x = fmax3(acc.x, fmin2(v0, b[2 * u].x), fmin2(v1, b[2 * u + 1].x));
                acc.y = fmax3(acc.y, fmin2(v0, b[2 * u].y), fmin2(v1, b[2 * u + 1].y));
                acc.z = fmax3(acc.z, fmin2(v0, b[2 * u].z), fmin2(v1, b[2 * u + 1].z));
                acc.w = fmax3(acc.w, fmin2(v0, b[2 * u].w), fmin2(v1, b[2 * u + 1].w));
            }
            const int kn = okey(next);
            open = okey(acc.x) < kn || okey(acc.y) < kn || okey(acc.z) < kn || okey(acc.w) < kn;
            if (!__any_sync(FULL, open)) break;
        }
        if (__any_sync(FULL, open)) {
            const int kn = okey(bound);
            const bool u0 = p < a.cols && okey(acc.x) < kn, u1 = p + 1 < a.cols && okey(acc.y) < kn;
            const bool u2 = p + 2 < a.cols && okey(acc.z) < kn, u3 = p + 3 < a.cols && okey(acc.w) < kn;
            const unsigned below = (1u << lane) - 1u;
            const unsigned m0 = __ballot_sync(FULL, u0), m1 = __ballot_sync(FULL, u1), m2 = __ballot_sync(FULL, u2),
                           m3 = __ballot_sync(FULL, u3);
            unsigned long long base = 0;
            const int total = __popc(m0) + __popc(m1) + __popc(m2) + __popc(m3);
            if (lane == 0 && total) base = atomicAdd(a.pending_n, (unsigned long long)total);
            base = __shfl_sync(FULL, base, 0);
            auto put = [&](bool u, unsigned long long at, int pp, float m) {
                if (u && at < (unsigned long long)a.pending_cap) a.pending[at] = RankedPending{o, pp, m};
            };
            put(u0, base + __popc(m0 & below), p, acc.x);
            base += __popc(m0);
            put(u1, base + __popc(m1 & below), p + 1, acc.y);
            base += __popc(m1);
            put(u2, base + __popc(m2 & below), p + 2, acc.z);
            base += __popc(m2);
            put(u3, base + __popc(m3 & below), p + 3, acc.w);
        }
        if (a.direct) {
            float* dst = a.P + (int64_t)o * a.ldp + p;
            if (live0) *reinterpret_cast<float4*>(dst) = acc;  // ldp covers the last column block
            else {
                if (live1) dst[1] = acc.y;
                if (live2) dst[2] = acc.z;
                if (live3) dst[3] = acc.w;
            }
        }
        if (a.mirror) *reinterpret_cast<float4*>(&tile[w][lane * 4]) = acc;
    }
    if (a.mirror) {
        __syncthreads();
        // P[p][o0 .. o0 + 7]: two float4 per row p
        const int r = threadIdx.x >> 1, h = (threadIdx.x & 1) * 4;
        const int pp = p0 + r;
        if (pp < a.cols) {
            float* dst = a.P + (int64_t)pp * a.ldp + o0 + h;
            const int last = o0 + h + 3;
            if (last < a.owners && (!SYM || pp >= last)) {
                *reinterpret_cast<float4*>(dst) = make_float4(tile[h][r], tile[h + 1][r], tile[h + 2][r], tile[h + 3][r]);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (o0 + h + q < a.owners && (!SYM || pp >= o0 + h + q)) dst[q] = tile[h + q][r];
            }
        }
    }
}

// One warp per pending output: the other row's list (SYM, or where it was built), then both whole rows.
template <bool SYM, bool FLIP = false>
__global__ void __launch_bounds__(256) pending_kernel(const RankedArgs a0) {
    const RankedArgs a = oriented<FLIP>(a0);
    const int lane = threadIdx.x & 31;
    // full_n rises while this runs: one lane's reading decides for the warp, whose votes need all lanes
    if (__any_sync(FULL, lane == 0 && gave_up(a))) return;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t count = (int64_t)*a.pending_n;
    const bool other = !SYM && a.LX.entries && count > (int64_t)a.lx_above;
    for (int64_t x = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; x < count; x += nw) {
        const RankedPending d = a.pending[x];
        const int i = SYM ? a.perm[d.o] : d.o, j = a.perm ? a.perm[d.p] : d.p;
        const float* ro = a.O + (int64_t)i * a.ldo;
        const float* rx = a.X + (int64_t)j * a.ldx;
        float acc = d.m;
        float bound = a.L.bound[i];
        bool open = true;
        if (SYM || other) {
            const RankedLists& L = SYM ? a.L : a.LX;
            const uint2* list = L.entries + (int64_t)j * L.pitch;
            const int c = L.count[j];
            const float bj = L.bound[j];
            for (int t = 0; t < c && open; t += 32) {
                if (t + lane < c) {
                    const uint2 e = __ldg(list + t + lane);
                    acc = fmax2(acc, fmin2(__uint_as_float(e.x), __ldg(ro + e.y)));
                }
                const float next = t + 32 < c ? __uint_as_float(__ldg(&list[t + 32].x)) : bj;
                open = !__any_sync(FULL, okey(acc) >= okey(next));
            }
            bound = fminf(bound, bj);
            if (open) open = !__any_sync(FULL, okey(acc) >= okey(bound));
        }
        if (open && other) {  // both whole rows: only so many of these (without lists no more than lx_above pend)
            unsigned long long seen = 0;
            if (lane == 0) seen = atomicAdd(a.full_n, 1ull);
            if (__shfl_sync(FULL, seen, 0) >= a.full_cap) return;
        }
        const int kb = okey(bound);
        for (int t = 0; t < a.k && open; t += 128) {
            const int c = t + lane * 4;
            if (c + 3 < a.k) {
                const float4 u = __ldg(reinterpret_cast<const float4*>(ro + c));
                const float4 v = __ldg(reinterpret_cast<const float4*>(rx + c));
                acc = fmax3(acc, fmin2(u.x, v.x), fmin2(u.y, v.y));
                acc = fmax3(acc, fmin2(u.z, v.z), fmin2(u.w, v.w));
            } else {
                for (int q = c; q < a.k; ++q) acc = fmax2(acc, fmin2(ro[q], rx[q]));
            }
            open = !__any_sync(FULL, okey(acc) >= kb);
        }
        const int best = __reduce_max_sync(FULL, okey(acc));
        if (lane == 0) {
            const float v = okey_value(best);
            if (a.direct) a.P[(int64_t)d.o * a.ldp + d.p] = v;
            if (a.mirror) a.P[(int64_t)d.p * a.ldp + d.o] = v;
        }
    }
}

__device__ __forceinline__ float ratio_value(float a, float m) {  // ratio_kernel, combine.hpp:210-222
    return (fabsf(a) < FLT_EPSILON) ? 0.0f : (fabsf(m) < FLT_EPSILON) ? FLT_MAX : __fdiv_rn(a, m);
}

// C[i][j] = P[rrank ? rrank[i] : i][crank ? crank[j] : j], R = ratio(E, C).
template <bool GATHER>
__global__ void __launch_bounds__(512) finish_kernel(const RankedArgs a, const int* __restrict__ rrank,
                                                     const int* __restrict__ crank, int rows, int cols,
                                                     float* __restrict__ C, int64_t ldc, const float* __restrict__ E,
                                                     int64_t lde, float* __restrict__ R, int64_t ldr) {
    extern __shared__ float prow[];
    if (__syncthreads_or(threadIdx.x == 0 && gave_up(a))) return;
    for (int i = blockIdx.x; i < rows; i += gridDim.x) {
        const float* src = a.P + (int64_t)(rrank ? rrank[i] : i) * a.ldp;
        if (GATHER) {
            __syncthreads();
            for (int j = threadIdx.x * 4; j < cols; j += 512 * 4)  // ldp is a multiple of 128
                *reinterpret_cast<float4*>(prow + j) = *reinterpret_cast<const float4*>(src + j);
            __syncthreads();
        }
        for (int j0 = threadIdx.x; j0 < cols; j0 += 4 * 512) {  // four columns' loads in flight
            int c[4];
            float e[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int j = j0 + u * 512;
                c[u] = GATHER && j < cols ? crank[j] : j;
                e[u] = R && j < cols ? E[i * lde + j] : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int j = j0 + u * 512;
                if (j >= cols) break;
                const float v = GATHER ? prow[c[u]] : src[j];
                if (C) C[i * ldc + j] = v;
                if (R) R[i * ldr + j] = ratio_value(e[u], v);
            }
        }
    }
}

// ---------------- witnesses ----------------
// K[i][j] = the first k with min(O[i][k], X[j][k]) == C[i][j] (-1 where C is -inf).  With the product in
// P, those k are the listed ones whose both entries reach P: the lists are walked once more, down to
// entries below P.  Zeros of either sign are equal here, as in the exhaustive kernel.  Two products with
// witnesses at 4,096 genes: 36.0 ms (exhaustive, compare and select per candidate) -> 2.2 ms.
constexpr int WITNESS_SCAN = 512, WITNESS_MANY = 16;
template <bool SYM, bool FLIP = false>
__global__ void __launch_bounds__(OWN * 32) witness_walk_kernel(const RankedArgs a0, int* __restrict__ PK,
                                                                unsigned long long* open_n) {
    __shared__ int tile[OWN][COLS + 4];
    if (__syncthreads_or(threadIdx.x == 0 &&
                         (gave_up(a0) || *(const volatile unsigned long long*)open_n > (unsigned long long)a0.pending_cap)))
        return;
    const RankedArgs a = oriented<FLIP>(a0);
    int o0, p0;
    if (!tile_at<FLIP>(a, o0, p0)) return;
    if (SYM && p0 + COLS <= o0) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int o = o0 + w, p = p0 + lane * 4;
    if (o < a.owners && !(SYM && p0 + COLS <= o)) {
        const int i = SYM ? a.perm[o] : o;
        const uint4* list = reinterpret_cast<const uint4*>(a.L.entries + (int64_t)i * a.L.pitch);
        const int count = a.L.count[i];
        const float bound = a.L.bound[i];
        const float* col = a.XT + p;
        float c[4];
        int k[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const bool live = p + q < a.cols && (!SYM || p + q >= o);
            c[q] = live ? (a.direct ? a.P[(int64_t)o * a.ldp + p + q] : a.P[(int64_t)(p + q) * a.ldp + o]) : INFINITY;
            k[q] = INT_MAX;
            if (c[q] == -INFINITY || !live) {  // no candidate attains it / not an output
                c[q] = INFINITY;
                k[q] = -1;
            }
        }
        auto wanted = [&](float next) {
            bool b = false;
#pragma unroll
            for (int q = 0; q < 4; ++q) b |= k[q] != -1 && next >= c[q];
            return __any_sync(FULL, b);
        };
        bool more = wanted(INFINITY);
        for (int t = 0; t < count && more; t += BATCH) {
            uint4 e[BATCH / 2];
            float4 b[BATCH];
#pragma unroll
            for (int u = 0; u < BATCH / 2; ++u) e[u] = __ldg(list + t / 2 + u);
#pragma unroll
            for (int u = 0; u < BATCH / 2; ++u) {
                b[2 * u] = ldg4(col + (int64_t)e[u].y * a.ldt);
                b[2 * u + 1] = ldg4(col + (int64_t)e[u].w * a.ldt);
            }
            const float next = t + BATCH < count ? __uint_as_float(__ldg(&list[t / 2 + BATCH / 2].x)) : bound;
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const float v = __uint_as_float(u & 1 ? e[u / 2].z : e[u / 2].x);
                const int ku = (int)(u & 1 ? e[u / 2].w : e[u / 2].y);
                if (fmin2(v, b[u].x) >= c[0]) k[0] = min(k[0], ku);
                if (fmin2(v, b[u].y) >= c[1]) k[1] = min(k[1], ku);
                if (fmin2(v, b[u].z) >= c[2]) k[2] = min(k[2], ku);
                if (fmin2(v, b[u].w) >= c[3]) k[3] = min(k[3], ku);
            }
            more = wanted(next);
        }
        // entries beyond the list may attain it too
        bool late[4];
        int total = 0;
        unsigned m[4];
        auto count_late = [&]() {
            total = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                m[q] = __ballot_sync(FULL, late[q]);
                total += __popc(m[q]);
            }
        };
#pragma unroll
        for (int q = 0; q < 4; ++q) late[q] = more && k[q] != -1 && bound >= c[q];
        count_late();
        // Many at once are mostly ties, which some early k attains: the warp scans in ascending k until one is left (the
        // pending list holds two per warp), and stops where the first 32 settle less than an eighth (outputs whose
        // lists were too short).  Left to the
        // pending list, ties overflowed it, and the exhaustive kernel ran after all (2,000 genes with five values 1.90
        // ms, 1.60 exhaustive).
        const int late0 = total;
        for (int t = 0; late0 >= WITNESS_MANY && t < min(a.k, WITNESS_SCAN) && total > 1; t += BATCH) {
            float v[BATCH];
            float4 b[BATCH];
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const int y = min(t + u, a.k - 1);
                v[u] = __ldg(a.O + (int64_t)i * a.ldo + y);
                b[u] = ldg4(col + (int64_t)y * a.ldt);
            }
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const int y = min(t + u, a.k - 1);
                if (late[0] && fmin2(v[u], b[u].x) >= c[0]) k[0] = min(k[0], y);
                if (late[1] && fmin2(v[u], b[u].y) >= c[1]) k[1] = min(k[1], y);
                if (late[2] && fmin2(v[u], b[u].z) >= c[2]) k[2] = min(k[2], y);
                if (late[3] && fmin2(v[u], b[u].w) >= c[3]) k[3] = min(k[3], y);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) late[q] = late[q] && k[q] >= t + BATCH;
            count_late();
            if (t == 32 - BATCH && total > late0 - late0 / 8) break;
        }
        if (total) {
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(open_n, (unsigned long long)total);
            base = __shfl_sync(FULL, base, 0);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const unsigned long long at = base + __popc(m[q] & ((1u << lane) - 1u));
                if (late[q]) {
                    if (at < (unsigned long long)a.pending_cap) a.pending[at] = RankedPending{o, p + q, c[q]};
                }
                base += __popc(m[q]);
            }
        }
        if (a.direct) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (p + q < a.cols && (!SYM || p + q >= o)) PK[(int64_t)o * a.ldp + p + q] = k[q];
        }
        *reinterpret_cast<int4*>(&tile[w][lane * 4]) = make_int4(k[0], k[1], k[2], k[3]);
    }
    if (a.mirror) {
        __syncthreads();
        const int r = threadIdx.x >> 1, h = (threadIdx.x & 1) * 4;
        const int pp = p0 + r;
        if (pp < a.cols)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (o0 + h + q < a.owners && (!SYM || pp >= o0 + h + q)) PK[(int64_t)pp * a.ldp + o0 + h + q] = tile[h + q][r];
    }
}

// The pending witnesses: one warp each, ascending k, 128 at a time, up to the first that attains C.
// More of them than the list holds: the first ones are done here, the rest (open_n above the capacity)
// make the exhaustive kernel run.
template <bool SYM, bool FLIP = false>
__global__ void __launch_bounds__(256) witness_pending_kernel(const RankedArgs a0, int* __restrict__ PK,
                                                              const unsigned long long* open_n) {
    const RankedArgs a = oriented<FLIP>(a0);
    if (gave_up(a) || *open_n > (unsigned long long)a.pending_cap) return;
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t count = (int64_t)*open_n;
    for (int64_t x = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; x < count; x += nw) {
        const RankedPending d = a.pending[x];
        const int i = SYM ? a.perm[d.o] : d.o, j = a.perm ? a.perm[d.p] : d.p;
        const float* ro = a.O + (int64_t)i * a.ldo;
        const float* rx = a.X + (int64_t)j * a.ldx;
        int k = INT_MAX;
        for (int t = 0; t < a.k && k == INT_MAX; t += 128) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int y = t + lane * 4 + q;
                if (y < a.k && fmin2(__ldg(ro + y), __ldg(rx + y)) >= d.m) k = min(k, y);
            }
            k = (int)__reduce_min_sync(FULL, (unsigned)k);
        }
        if (lane == 0) {
            if (a.direct) PK[(int64_t)d.o * a.ldp + d.p] = k;
            if (a.mirror) PK[(int64_t)d.p * a.ldp + d.o] = k;
        }
    }
}

// C and K in gene order; a zero takes the sign it has at its witness.
template <bool GATHER>
__global__ void __launch_bounds__(256) witness_finish_kernel(const RankedArgs a, const int* __restrict__ PK,
                                                             const unsigned long long* open_n,
                                                             const int* __restrict__ rank, int rows, int cols,
                                                             float* __restrict__ C, int64_t ldc, int* __restrict__ K,
                                                             int64_t ldk) {
    if (gave_up(a) || *open_n > (unsigned long long)a.pending_cap) return;
    for (int i = blockIdx.x; i < rows; i += gridDim.x) {
        const int64_t r = (int64_t)(GATHER ? rank[i] : i) * a.ldp;
        for (int j = threadIdx.x; j < cols; j += 256) {
            const int64_t at = r + (GATHER ? rank[j] : j);
            float c = a.P[at];
            const int k = PK[at];
            if (c == 0.0f && k >= 0) c = fmin2(a.O[(int64_t)i * a.ldo + k], a.X[(int64_t)j * a.ldx + k]);
            C[(int64_t)i * ldc + j] = c;
            K[(int64_t)i * ldk + j] = k;
        }
    }
}

// ---------------- DPI ----------------
// (x, z) goes when some y outside {x, z} has min(A[x][y], A[z][y]) >= threshold(A[x][z]) (dpi_kernel,
// dpi.hpp:56-68): the same walk with the diagonal left out of the lists and of XT, and an
// output settled as soon as its maximum reaches the threshold or no later entry can.  On MI
// matrices nearly every pair is decided by its first few entries.  P receives a value
// on the right side of both orientations' thresholds.  Measured (whole call, tolerance 0.1; the tiled
// first-phase form -> this one): 20,000 genes 69.4 -> 11.8 ms (walk 6.4, lists 2.1, finish 1.2 ms; 14.8 ms
// with the thresholds' products in FP64 and gathered for both orientations), 2,000 genes 355 -> 174 us.
// The threshold (float)(e * tm) with the product in double, mostly without the FP64 pipe (16 clocks of an SM
// per warp instruction): e times tm as a pair of floats, exact to 2^-45.  Where the rounding to float is
// that far from a tie, it is the reference's; else, and outside the range the pair is good for, the double
// product runs.
struct DpiMult {
    double tm;
    float hi, lo;
    bool pair;
};
DpiMult dpi_mult(double tm) {
    DpiMult m;
    m.tm = tm;
    m.hi = (float)tm;
    m.pair = isfinite(m.hi);
    m.lo = m.pair ? (float)(tm - (double)m.hi) : 0.0f;
    return m;
}
__device__ __forceinline__ float dpi_threshold(float e, const DpiMult& m) {
    if (m.pair) {
        const float ph = __fmul_rn(e, m.hi);
        const float lo = __fmaf_rn(e, m.lo, __fmaf_rn(e, m.hi, -ph));
        const float r = __fadd_rn(ph, lo);
        const float err = __fadd_rn(__fsub_rn(ph, r), lo);
        const uint32_t u = __float_as_uint(r) & 0x7fffffffu;
        const float ulp = __uint_as_float(((u >> 23) - 23u) << 23);
        if (u > 0x0d000000u && u < 0x7e000000u && (u & 0x7fffffu) && fabsf(err) < __fmul_rn(0.4999f, ulp)) return r;
        if (e == 0.0f) return ph;
    }
    return (float)((double)e * m.tm);
}
__device__ __forceinline__ bool dpi_open(float acc, float next, float t0, float t1) {
    return (acc < t0 && next >= t0) || (acc < t1 && next >= t1);
}

// *asym = 1 when some A[i][j] != A[j][i] (64 x 64 tiles on and above the diagonal).
__global__ void __launch_bounds__(256) symmetry_kernel(const float* __restrict__ A, int64_t lda, int n,
                                                       unsigned long long* asym) {
    __shared__ float tile[64][65];
    const int bi = blockIdx.y * 64, bj = blockIdx.x * 64;
    if (bj < bi || *(volatile unsigned long long*)asym) return;
    const int tx = threadIdx.x & 63, ty = threadIdx.x >> 6;
#pragma unroll
    for (int r = ty; r < 64; r += 4)
        tile[r][tx] = bi + r < n && bj + tx < n ? A[(int64_t)(bi + r) * lda + bj + tx] : 0.0f;
    __syncthreads();
    bool differ = false;
#pragma unroll
    for (int r = ty; r < 64; r += 4) {
        const float v = bj + r < n && bi + tx < n ? A[(int64_t)(bj + r) * lda + bi + tx] : 0.0f;
        differ |= v != tile[tx][r];
    }
    if (differ) *asym = 1;
}

__global__ void __launch_bounds__(OWN * 32) dpi_walk_kernel(const RankedArgs a, const DpiMult tm,
                                                           const unsigned long long* asym) {
    __shared__ float tile[OWN][COLS + 4];
    if (__syncthreads_or(threadIdx.x == 0 && gave_up(a))) return;
    const int o0 = blockIdx.x * OWN, p0 = blockIdx.y * COLS;
    if (p0 + COLS <= o0) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int o = o0 + w, p = p0 + lane * 4;
    if (o < a.owners && p0 + COLS > o) {
        const int i = a.perm[o];
        const uint4* list = reinterpret_cast<const uint4*>(a.L.entries + (int64_t)i * a.L.pitch);
        const int count = a.L.count[i];
        const float bound = a.L.bound[i];
        const float* col = a.XT + p;
        float acc[4], t0[4], t1[4];
        {
            const bool symmetric = asym && *asym == 0;  // A[x][z] is A[z][x] then: no gather through the order
            const float4 e1 = ldg4(col + (int64_t)i * a.ldt);  // A[z][x]
            const float v1[4] = {e1.x, e1.y, e1.z, e1.w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const bool live = p + c > o && p + c < a.cols;  // z == x goes in any case
                acc[c] = -INFINITY;
                t1[c] = live ? dpi_threshold(v1[c], tm) : -INFINITY;
                t0[c] = !live || symmetric ? t1[c] : dpi_threshold(__ldg(a.O + (int64_t)i * a.ldo + a.perm[p + c]), tm);
            }
        }
        auto any_open = [&](float next) {
            bool open = false;
#pragma unroll
            for (int c = 0; c < 4; ++c) open |= dpi_open(acc[c], next, t0[c], t1[c]);
            return __any_sync(FULL, open);
        };
        bool open = any_open(INFINITY);
        for (int t = 0; t < count && open; t += BATCH) {
            uint4 e[BATCH / 2];
            float4 b[BATCH];
#pragma unroll
            for (int u = 0; u < BATCH / 2; ++u) e[u] = __ldg(list + t / 2 + u);
#pragma unroll
            for (int u = 0; u < BATCH / 2; ++u) {
                b[2 * u] = ldg4(col + (int64_t)e[u].y * a.ldt);
                b[2 * u + 1] = ldg4(col + (int64_t)e[u].w * a.ldt);
            }
            const float next = t + BATCH < count ? __uint_as_float(__ldg(&list[t / 2 + BATCH / 2].x)) : bound;
#pragma unroll
            for (int u = 0; u < BATCH / 2; ++u) {
                const float v0 = __uint_as_float(e[u].x), v1 = __uint_as_float(e[u].z);
                acc[0] = fmax3(acc[0], fmin2(v0, b[2 * u].x), fmin2(v1, b[2 * u + 1].x));
                acc[1] = fmax3(acc[1], fmin2(v0, b[2 * u].y), fmin2(v1, b[2 * u + 1].y));
                acc[2] = fmax3(acc[2], fmin2(v0, b[2 * u].z), fmin2(v1, b[2 * u + 1].z));
                acc[3] = fmax3(acc[3], fmin2(v0, b[2 * u].w), fmin2(v1, b[2 * u + 1].w));
            }
            open = any_open(next);
        }
        if (open) {
            unsigned m[4];
            int total = 0;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                m[c] = __ballot_sync(FULL, dpi_open(acc[c], bound, t0[c], t1[c]));
                total += __popc(m[c]);
            }
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(a.pending_n, (unsigned long long)total);
            base = __shfl_sync(FULL, base, 0);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const unsigned long long at = base + __popc(m[c] & ((1u << lane) - 1u));
                if (((m[c] >> lane) & 1u) && at < (unsigned long long)a.pending_cap)
                    a.pending[at] = RankedPending{o, p + c, acc[c]};
                base += __popc(m[c]);
            }
        }
        float* dst = a.P + (int64_t)o * a.ldp + p;
        if (p > o) *reinterpret_cast<float4*>(dst) = make_float4(acc[0], acc[1], acc[2], acc[3]);
        else
#pragma unroll
            for (int c = 1; c < 4; ++c)
                if (p + c > o) dst[c] = acc[c];
        *reinterpret_cast<float4*>(&tile[w][lane * 4]) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    }
    __syncthreads();
    const int r = threadIdx.x >> 1, h = (threadIdx.x & 1) * 4;
    const int pp = p0 + r;
    if (pp < a.cols) {
        float* dst = a.P + (int64_t)pp * a.ldp + o0 + h;
        if (o0 + h + 3 < a.owners && pp > o0 + h + 3) {
            *reinterpret_cast<float4*>(dst) = make_float4(tile[h][r], tile[h + 1][r], tile[h + 2][r], tile[h + 3][r]);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (o0 + h + q < a.owners && pp > o0 + h + q) dst[q] = tile[h + q][r];
        }
    }
}

// One warp per pending pair: the other row's list, then both whole rows without x and z.
__global__ void __launch_bounds__(256) dpi_ranked_pending_kernel(const RankedArgs a, const DpiMult tm) {
    if (gave_up(a)) return;
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t count = (int64_t)*a.pending_n;
    for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < count; w += nw) {
        const RankedPending d = a.pending[w];
        const int x = a.perm[d.o], z = a.perm[d.p];
        const float* rx = a.O + (int64_t)x * a.ldo;
        const float* rz = a.O + (int64_t)z * a.ldo;
        const float t0 = dpi_threshold(__ldg(rx + z), tm), t1 = dpi_threshold(__ldg(rz + x), tm);
        float acc = d.m;
        const uint2* list = a.L.entries + (int64_t)z * a.L.pitch;
        const int c = a.L.count[z];
        float bound = a.L.bound[x];
        const float bz = a.L.bound[z];
        auto best = [&]() { return okey_value(__reduce_max_sync(FULL, okey(acc))); };
        bool open = true;
        for (int t = 0; t < c && open; t += 32) {
            if (t + lane < c) {
                const uint2 e = __ldg(list + t + lane);
                if ((int)e.y != x) acc = fmax2(acc, fmin2(__uint_as_float(e.x), __ldg(rx + e.y)));
            }
            const float next = t + 32 < c ? __uint_as_float(__ldg(&list[t + 32].x)) : bz;
            acc = best();
            open = dpi_open(acc, next, t0, t1);
        }
        bound = fminf(bound, bz);
        if (open) open = dpi_open(acc, bound, t0, t1);
        for (int y0 = 0; y0 < a.k && open; y0 += 128) {
            const int y = y0 + lane * 4;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (y + q < a.k && y + q != x && y + q != z) acc = fmax2(acc, fmin2(__ldg(rx + y + q), __ldg(rz + y + q)));
            acc = best();
            open = dpi_open(acc, bound, t0, t1);
        }
        if (lane == 0) {
            a.P[(int64_t)d.o * a.ldp + d.p] = acc;
            a.P[(int64_t)d.p * a.ldp + d.o] = acc;
        }
    }
}

// out = the entries that stay, mask, and the number of entries that changed.
__global__ void __launch_bounds__(512) dpi_finish_kernel(const RankedArgs a, const int* __restrict__ rank, const DpiMult tm,
                                                         float* __restrict__ out, int64_t ldo, uint8_t* __restrict__ mask,
                                                         int64_t ldmask, unsigned long long* removed) {
    extern __shared__ float prow[];
    if (__syncthreads_or(threadIdx.x == 0 && gave_up(a))) return;
    unsigned long long cnt = 0;
    const int n = a.owners;
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        const float* src = a.P + (int64_t)rank[i] * a.ldp;
        const float* row = a.O + (int64_t)i * a.ldo;
        __syncthreads();
        for (int j = threadIdx.x * 4; j < n; j += 512 * 4)
            *reinterpret_cast<float4*>(prow + j) = *reinterpret_cast<const float4*>(src + j);
        __syncthreads();
        for (int j0 = threadIdx.x; j0 < n; j0 += 4 * 512) {  // four columns' loads in flight
            int c[4];
            float e[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int j = j0 + u * 512;
                c[u] = j < n ? rank[j] : 0;
                e[u] = j < n ? row[j] : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int j = j0 + u * 512;
                if (j >= n) break;
                const bool del = i == j || prow[c[u]] >= dpi_threshold(e[u], tm);
                const float o = del ? 0.0f : e[u];
                out[i * ldo + j] = o;
                cnt += (o != e[u]);
                if (mask) mask[i * ldmask + j] = del ? 1 : 0;
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(FULL, cnt, o);
    if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(removed, cnt);
}

// The finishing kernels hold a product row of up to RANKED_MAX_COLS columns in shared memory.  The attribute is
// the process's, and always the same value: with each call's own size, another thread's smaller call between the
// setting and the launch made the launch fail.
cudaError_t allow_row_buffer(const void* kernel) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(RANKED_MAX_COLS * sizeof(float)));
}

int isqrt_ceil(int64_t v) { return (int)ceil(sqrt((double)v)); }

}  // namespace

int ranked_list_cap(int64_t k) {
    // four square roots of the candidate count cover 99 % of the outputs of the measured matrices
    int64_t c = (4 * (int64_t)isqrt_ceil(k) + 31) / 32 * 32;
    // one entry per thread of the sort (k up to 25,600): the DPI gains throughout (24,000 genes 17.8 ms, 18.6 with 640
    // entries), products up to about 21,000 (22.2 and 22.0 ms; at 24,000 32.4 and 29.9)
    if (c > LIST_TPB && c <= LIST_TPB + 128) c = LIST_TPB;
    return (int)(c > LIST_MAX ? LIST_MAX : c);
}

cudaError_t launch_ranked_lists(const float* O, int64_t ldo, int64_t rows, int64_t k, int skip_diag, const RankedLists& L,
                                unsigned long long* nan, cudaStream_t st, int64_t* launches,
                                const unsigned long long* only_above, unsigned long long above, const RankedOther& alt) {
    const int cap = ranked_list_cap(k), want = cap * 3 / 4, at = 2 * isqrt_ceil(k);
    if (k > (int64_t)LIST_TPB * 64 || L.pitch < cap) return cudaErrorInvalidValue;
    if (launches) ++*launches;
    // a launch that may have nothing to do: few CTAs (8,192 that return at once take 10 us)
    const int64_t most = std::max<int64_t>(rows, alt.flip ? alt.rows : 0);
    const unsigned g = (unsigned)(only_above ? std::min<int64_t>(most, 152 * 4) : most);
    auto launch = [&](auto* kernel) {
        kernel<<<g, LIST_TPB, 0, st>>>(O, ldo, (int)rows, (int)k, want, cap, at, skip_diag, L, nan, only_above, above, alt);
        return cudaGetLastError();
    };
    if (k <= LIST_TPB * 4) return launch(only_above ? lists_kernel<4, true> : lists_kernel<4, false>);
    if (k <= LIST_TPB * 16) return launch(only_above ? lists_kernel<16, true> : lists_kernel<16, false>);
    if (k <= LIST_TPB * 40) return launch(only_above ? lists_kernel<40, true> : lists_kernel<40, false>);
    return launch(only_above ? lists_kernel<64, true> : lists_kernel<64, false>);
}

cudaError_t launch_ranked_order(const RankedLists& L, int64_t n, int* rank, int* perm, cudaStream_t st,
                                int64_t* launches) {
    if (launches) ++*launches;
    order_kernel<<<(unsigned)ceil_div(n, 8), 256, 0, st>>>(L.strength, (int)n, rank, perm);
    return cudaGetLastError();
}

cudaError_t launch_ranked_transpose(const float* X, int64_t ldx, int64_t rows, int64_t k, int skip_diag,
                                    const int* perm, float* XT,
                                    int64_t ldt, unsigned long long* nan, cudaStream_t st, int64_t* launches) {
    if (launches) ++*launches;
    dim3 grid((unsigned)(ldt / 32), (unsigned)ceil_div(k, 32));
    transpose_kernel<<<grid, 256, 0, st>>>(X, ldx, (int)rows, (int)k, skip_diag, perm, XT, ldt, nan);
    return cudaGetLastError();
}

cudaError_t launch_ranked_choose(const RankedArgs& a, int* flip, unsigned long long* sum, float* XT,
                                 cudaStream_t st, int64_t* launches) {
    if (launches) *launches += 3;
    const int most = (int)(SAMPLES * a.pending_cap * 5 / ((int64_t)a.owners * a.cols * 8));
    choose_kernel<<<SAMPLES, CHOOSE_TPB, 0, st>>>(a, ranked_list_cap(a.k), most, flip, sum);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const RankedOther alt{a.X, a.ldx, a.cols, a.flip};
    if (launches) --*launches;  // counted below
    e = launch_ranked_lists(a.O, a.ldo, a.owners, a.k, 0, a.L, const_cast<unsigned long long*>(a.nan), st, launches, nullptr, 0,
                            alt);
    if (e != cudaSuccess) return e;
    const int64_t tiles = ceil_div(std::max(a.owners, a.cols), COLS) * (COLS / 32) * ceil_div(a.k, 32);
    transpose_chosen_kernel<<<(unsigned)std::min<int64_t>(tiles, 152 * 64), 256, 0, st>>>(
        a, XT, const_cast<unsigned long long*>(a.nan));
    return cudaGetLastError();
}

cudaError_t launch_ranked_walk(const RankedArgs& a, int symmetric, cudaStream_t st, int64_t* launches) {
    if (launches) *launches += 2;
    const dim3 grid = tile_grid(a);
    if (symmetric) walk_kernel<true><<<grid, OWN * 32, 0, st>>>(a);
    else if (a.flip) walk_kernel<false, true><<<grid, OWN * 32, 0, st>>>(a);
    else walk_kernel<false><<<grid, OWN * 32, 0, st>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (!symmetric && a.LX.entries) {
        // An owner with many large entries against a row without: only the other row's list settles
        // that early.  Its lists are built when such pairs are many.
        e = launch_ranked_lists(a.X, a.ldx, a.cols, a.k, 0, a.LX, const_cast<unsigned long long*>(a.nan), st, launches,
                                a.pending_n, a.lx_above, RankedOther{a.O, a.ldo, a.owners, a.flip});
        if (e != cudaSuccess) return e;
    }
    const unsigned g = 152 * 8;
    if (symmetric) pending_kernel<true><<<g, 256, 0, st>>>(a);
    else if (a.flip) pending_kernel<false, true><<<g, 256, 0, st>>>(a);
    else pending_kernel<false><<<g, 256, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_ranked_finish(const RankedArgs& a, const int* rrank, const int* crank, int64_t rows, int64_t cols,
                                 float* C, int64_t ldc, const float* E, int64_t lde, float* R, int64_t ldr,
                                 cudaStream_t st, int64_t* launches) {
    if (launches) ++*launches;
    const unsigned g = (unsigned)(rows < 152 * 16 ? rows : 152 * 16);
    if (crank) {
        const size_t smem = (size_t)((cols + 3) / 4 * 4) * sizeof(float);
        cudaError_t e = allow_row_buffer((const void*)finish_kernel<true>);
        if (e != cudaSuccess) return e;
        finish_kernel<true><<<g, 512, smem, st>>>(a, rrank, crank, (int)rows, (int)cols, C, ldc, E, lde, R, ldr);
    } else {
        finish_kernel<false><<<g, 512, 0, st>>>(a, rrank, crank, (int)rows, (int)cols, C, ldc, E, lde, R, ldr);
    }
    return cudaGetLastError();
}

cudaError_t launch_ranked_dpi(const RankedArgs& a, const int* rank, double tol_mult, float* out, int64_t ldo,
                              uint8_t* mask, int64_t ldmask, unsigned long long* removed, unsigned long long* asym,
                              cudaStream_t st, int64_t* launches) {
    if (launches) *launches += 4;
    dim3 grid((unsigned)ceil_div(a.owners, OWN), (unsigned)ceil_div(a.cols, COLS));
    const DpiMult tm = dpi_mult(tol_mult);
    // (a matrix that fits L2 gathers its thresholds cheaply: no check there)
    if (a.owners < 4096) asym = nullptr;
    const unsigned tiles = (unsigned)ceil_div(a.owners, 64);
    if (asym) symmetry_kernel<<<dim3(tiles, tiles), 256, 0, st>>>(a.O, a.ldo, a.owners, asym);
    dpi_walk_kernel<<<grid, OWN * 32, 0, st>>>(a, tm, asym);
    dpi_ranked_pending_kernel<<<152 * 8, 256, 0, st>>>(a, tm);
    const size_t smem = (size_t)((a.cols + 3) / 4 * 4) * sizeof(float);
    cudaError_t e = allow_row_buffer((const void*)dpi_finish_kernel);
    if (e != cudaSuccess) return e;
    dpi_finish_kernel<<<(unsigned)(a.owners < 152 * 16 ? a.owners : 152 * 16), 512, smem, st>>>(
        a, rank, tm, out, ldo, mask, ldmask, removed);
    return cudaGetLastError();
}

// After launch_ranked_walk (owner = rows of C).
cudaError_t launch_ranked_witness(const RankedArgs& a, int symmetric, const int* rank, int* PK,
                                  unsigned long long* open_n, int64_t rows, int64_t cols, float* C, int64_t ldc,
                                  int32_t* K, int64_t ldk, cudaStream_t st, int64_t* launches) {
    if (launches) *launches += 3;
    const dim3 grid = tile_grid(a);
    const unsigned g = (unsigned)(rows < 152 * 16 ? rows : 152 * 16);
    if (symmetric) {
        witness_walk_kernel<true><<<grid, OWN * 32, 0, st>>>(a, PK, open_n);
        witness_pending_kernel<true><<<152 * 8, 256, 0, st>>>(a, PK, open_n);
        witness_finish_kernel<true><<<g, 256, 0, st>>>(a, PK, open_n, rank, (int)rows, (int)cols, C, ldc, K, ldk);
    } else {
        if (a.flip) {
            witness_walk_kernel<false, true><<<grid, OWN * 32, 0, st>>>(a, PK, open_n);
            witness_pending_kernel<false, true><<<152 * 8, 256, 0, st>>>(a, PK, open_n);
        } else {
            witness_walk_kernel<false><<<grid, OWN * 32, 0, st>>>(a, PK, open_n);
            witness_pending_kernel<false><<<152 * 8, 256, 0, st>>>(a, PK, open_n);
        }
        witness_finish_kernel<false><<<g, 256, 0, st>>>(a, PK, open_n, nullptr, (int)rows, (int)cols, C, ldc, K, ldk);
    }
    return cudaGetLastError();
}

}  // namespace mcpg
