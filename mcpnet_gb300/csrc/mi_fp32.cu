// Plain-FP32 B-spline MI on CUDA cores (K2').  First the dense kernel, for any bins and order,
// then the one that skips zero weight rows (10 bins, order 3).  Both contract
//   P_ij[a][b] = (1/m) sum_s w_i[a](s) w_j[b](s)
// with the joint entropy and Hx + Hy - Hxy fused into the epilogue, so the
// joint tables never leave registers.  Whole-matrix form of
// BSplineEntropyKernel::entropy2d_simd + BSplineMIKernel::operator()
// (include/mcp/correlation/BSplineMI.hpp:288-315,492-499) under
// InnerProduct<..., SYMM=true> (apps/pipeline/mcpnet_helper.hpp:88-98).
//
// Shape: CTA = 16 x 16 genes, 256 threads, one gene pair per thread with its
// BINS x BINS joint counts in registers.  Weights are sample-major
// (Wt[s][gene*BINS + a]) so one sample of 16 genes is one contiguous 640-byte
// row: a 4-stage cp.async pipeline stages 16 samples per step.  Per sample a
// thread loads 2*BINS floats (LDS.64, broadcast across the warp's 4 x 8 pair
// layout) and issues BINS^2 FFMA.  Only tiles with j-block >= i-block run.
// Epilogue: p = count * (1/m) (float, as the reference's norm_factor),
// row sums of p*log2(p) in float, the BINS row sums and the combine
// H_i + H_j - H_ij in double.
#include <math.h>

#include "common.cuh"
#include "internal.h"

namespace mcpg {
namespace {

constexpr int G = 16;          // genes per tile side
constexpr int BKS = 16;        // samples per stage
constexpr int STAGES = 4;
constexpr int THREADS = 256;

template <int BINS>
struct MiCfg {
    static constexpr int ROW = G * BINS;                  // floats per sample per operand tile
    static constexpr int STAGE_FLOATS = 2 * BKS * ROW;    // A and B
    static constexpr size_t SMEM = (size_t)STAGES * STAGE_FLOATS * sizeof(float);
};

// Upper-triangular tile index -> (ti, tj) with tj >= ti, row-major.
__device__ __forceinline__ void tri_tile(int64_t b, int64_t T, int64_t& ti, int64_t& tj) {
    // rows r have (T - r) tiles; start(r) = r*T - r(r-1)/2
    double tt = (double)(2 * T + 1);
    int64_t r = (int64_t)floor((tt - sqrt(tt * tt - 8.0 * (double)b)) * 0.5);
    if (r < 0) r = 0;
    if (r >= T) r = T - 1;
    while (r > 0 && r * T - r * (r - 1) / 2 > b) --r;
    while (r + 1 < T && (r + 1) * T - (r + 1) * r / 2 <= b) ++r;
    ti = r;
    tj = r + (b - (r * T - r * (r - 1) / 2));
}

// Adjoint epilogue arguments (EPI >= 1): Q[i * BINS + a][(j - j0) * BINS + b]
// = Gs_ij (log2 P_ab + 1/ln 2) for P_ab > 0 (else 0), Gs_ij = G[i][j] + G[j][i]
// for i != j and 0 on the diagonal, for all genes i and the genes j in [j0, j1).  Q over all
// genes is symmetric bit for bit (the sums' products commute).
struct QArgs {
    const float* G; int64_t ldg;
    float* Q; int64_t ldq;
    int64_t j0, j1;
};

template <int BINS, int EPI>
__global__ void __launch_bounds__(THREADS, 1)
    mi_fp32_kernel(const float* __restrict__ Wt, int64_t ldwt, const double* __restrict__ H, int64_t n,
                   int64_t m_pad, float inv_m, float* __restrict__ MI, int64_t ldmi, int64_t T, const QArgs qa,
                   int64_t tile_base) {
    using C = MiCfg<BINS>;
    extern __shared__ float4 smem_f4[];
    float* smem = reinterpret_cast<float*>(smem_f4);

    int64_t ti, tj;
    if (EPI == 0) {
        tri_tile(tile_base + blockIdx.x, T, ti, tj);
    } else {
        const int64_t slab = (qa.j1 - qa.j0 + G - 1) / G;
        ti = blockIdx.x / slab;
        tj = qa.j0 / G + blockIdx.x % slab;
    }
    const int64_t gi0 = ti * G, gj0 = tj * G;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int il = ((warp >> 1) << 2) + (lane >> 3);  // 0..15
    const int jl = ((warp & 1) << 3) + (lane & 7);    // 0..15

    // staging: per sample and operand, ROW floats = ROW/4 chunks of 16 bytes
    constexpr int CHUNKS_PER_ROW = C::ROW / 4;              // 40 for BINS = 10
    constexpr int CHUNKS = 2 * BKS * CHUNKS_PER_ROW;         // per stage
    const float* srcA = Wt + gi0 * BINS;
    const float* srcB = Wt + gj0 * BINS;
    auto load = [&](int stage, int64_t s0) {
        float* dst = smem + stage * C::STAGE_FLOATS;
        for (int c = tid; c < CHUNKS; c += THREADS) {
            const int op = c / (BKS * CHUNKS_PER_ROW);
            const int rem = c - op * (BKS * CHUNKS_PER_ROW);
            const int srow = rem / CHUNKS_PER_ROW, ch = rem - srow * CHUNKS_PER_ROW;
            const float* src = (op ? srcB : srcA) + (s0 + srow) * ldwt + ch * 4;
            cp_async16(dst + op * BKS * C::ROW + srow * C::ROW + ch * 4, src, 16);
        }
    };

    float acc[BINS][BINS];
#pragma unroll
    for (int a = 0; a < BINS; ++a)
#pragma unroll
        for (int b = 0; b < BINS; ++b) acc[a][b] = 0.0f;

    const int64_t ksteps = m_pad / BKS;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < ksteps) load(s, (int64_t)s * BKS);
        cp_async_commit();
    }
    for (int64_t t = 0; t < ksteps; ++t) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();
        {
            const int64_t tn = t + STAGES - 1;
            if (tn < ksteps) load((int)(tn % STAGES), tn * BKS);
            cp_async_commit();
        }
        const float* As = smem + (t % STAGES) * C::STAGE_FLOATS + il * BINS;
        const float* Bs = smem + (t % STAGES) * C::STAGE_FLOATS + BKS * C::ROW + jl * BINS;
#pragma unroll 2
        for (int s = 0; s < BKS; ++s) {
            float a[BINS], b[BINS];
            if (BINS % 2 == 0) {
#pragma unroll
                for (int q = 0; q < BINS / 2; ++q) {
                    const float2 va = *reinterpret_cast<const float2*>(As + s * C::ROW + 2 * q);
                    const float2 vb = *reinterpret_cast<const float2*>(Bs + s * C::ROW + 2 * q);
                    a[2 * q] = va.x; a[2 * q + 1] = va.y;
                    b[2 * q] = vb.x; b[2 * q + 1] = vb.y;
                }
            } else {
#pragma unroll
                for (int q = 0; q < BINS; ++q) { a[q] = As[s * C::ROW + q]; b[q] = Bs[s * C::ROW + q]; }
            }
#pragma unroll
            for (int x = 0; x < BINS; ++x)
#pragma unroll
                for (int y = 0; y < BINS; ++y) acc[x][y] = fmaf(a[x], b[y], acc[x][y]);
        }
    }
    cp_async_wait<0>();

    const int64_t i = gi0 + il, j = gj0 + jl;
    if (EPI == 1) {
        if (i >= n || j >= n) return;
        const float gs = (i == j) ? 0.0f : qa.G[i * qa.ldg + j] + qa.G[j * qa.ldg + i];
        const float c = 1.4426950408889634f;  // 1 / ln 2
        float* Qr = qa.Q + i * BINS * qa.ldq + (j - qa.j0) * BINS;
#pragma unroll
        for (int x = 0; x < BINS; ++x)
#pragma unroll
            for (int y = 0; y < BINS; ++y) {
                const float pv = acc[x][y] * inv_m;
                Qr[x * qa.ldq + y] = (gs != 0.0f && pv > 0.0f) ? gs * (__log2f(pv) + c) : 0.0f;
            }
        return;
    }
    if (i >= n || j >= n || j < i) return;
    double hxy = 0.0;
#pragma unroll
    for (int x = 0; x < BINS; ++x) {
        float row = 0.0f;
#pragma unroll
        for (int y = 0; y < BINS; ++y) {
            const float pv = acc[x][y] * inv_m;
            if (pv > 0.0f) row += pv * __log2f(pv);
        }
        hxy += (double)row;
    }
    const float v = (float)(H[i] + H[j] + hxy);  // hxy = -H_ij
    MI[i * ldmi + j] = v;
    MI[j * ldmi + i] = v;
}

// ---------------- 10 bins, order 3: only the rows a sample touches ----------------
// A sample has three nonzero weights per gene, so its outer product touches three of the ten
// rows of a pair's table.  A warp takes one gene i and 32 genes j (a lane each, its 10 x 10
// counts in registers): the three rows are the same for every lane, so a uniform branch
// on i's first nonzero bin runs 3 x 10 of the 10 x 10 multiply-adds (as 15 packed
// fma.f32x2).  The products left out are exact zeros and each count still sums its
// samples in ascending order: the bits are those of the dense kernel above.  Where some
// sample has a nonzero weight outside three neighbouring bins (NaN or infinite input),
// *irregular is set and every row is multiplied.
// Per 32 pairs and sample: 1,280 B of j weights and a broadcast entry of i from shared
// memory (12 clocks with the staging writes), 7.5 clocks of packed multiply-adds.  Measured
// (weights excluded): 2,000 x 2,000 16.7 -> 7.0 ms, 4,000 x 2,000 66.2 -> 27.0 ms, 500 x 500
// 346 -> 151 us; the shared-memory pipe is 82 % busy (ncu, 2,000 x 1,000), the rest are branch and
// table latencies.  16 warps of 128 registers hide those better than 12 of 152 with the j weights double
// buffered (7.4 ms).  Small matrices run a few warps per CTA, so that their tiles reach all SMs.
constexpr int SB = 10, SJ = 32, SCH = 64, SSTG = 2, SWARPS_MAX = 16;
constexpr int SROW = SJ * SB;  // floats of a sample's j weights
// floats of a stage: j weights, entries and their end row
__host__ __device__ constexpr int rows_stage(int warps) { return SCH * SROW + (SCH + 1) * warps * 4; }

__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pack2(float v) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

// One chunk of samples: acc[r .. r + 2][:] += (w0, w1, w2) (x) b for each, with r = the entry's first
// row, the same for the whole warp.  Threaded code in one asm statement: an arm per first row
// fetches the next entry, runs its 15 packed multiply-adds, fetches the next j weights and
// branches through a table straight to the next sample's arm; an entry with row 8 behind the
// chunk ends it.  Left to a C++ switch, the compiler merges the arms and moves the counts around one
// shared copy, or branches through a tree of compares (11.6 ms at 2,000 x 2,000).
// pj: this lane's j weights of sample 0 (rows SROW floats apart); pe: the warp's entry of sample 0
// (WARPS entries apart); shared-memory addresses.
#define MCPG_FMA2(d, w, b) "fma.rn.f32x2 %" #d ", " #w ", " #b ", %" #d ";\n\t"
#define MCPG_ROW(w, d0, d1, d2, d3, d4) \
    MCPG_FMA2(d0, w, b0) MCPG_FMA2(d1, w, b1) MCPG_FMA2(d2, w, b2) MCPG_FMA2(d3, w, b3) MCPG_FMA2(d4, w, b4)
#define MCPG_ENTRY "ld.shared.v4.b32 {x0, x1, x2, xr}, [pe];\n\t"
#define MCPG_WEIGHTS                                                                                  \
    "ld.shared.b64 b0, [pj];\n\tld.shared.b64 b1, [pj + 8];\n\tld.shared.b64 b2, [pj + 16];\n\t"      \
    "ld.shared.b64 b3, [pj + 24];\n\tld.shared.b64 b4, [pj + 32];\n\t"
#define MCPG_NEXT                                                                                     \
    "mov.b64 w0, {x0, x0};\n\tmov.b64 w1, {x1, x1};\n\tmov.b64 w2, {x2, x2};\n\t"                     \
    "add.u32 pe, pe, %52;\n\tadd.u32 pj, pj, %53;\n\t" MCPG_ENTRY
template <int WARPS>
__device__ __forceinline__ void add_chunk(unsigned long long (&acc)[SB][SB / 2], uint32_t pj, uint32_t pe) {
    asm volatile(
        "{\n\t.reg .b64 b<5>, w0, w1, w2;\n\t.reg .b32 pj, pe, x0, x1, x2, xr;\n\t"
        "mov.b32 pj, %50;\n\tmov.b32 pe, %51;\n\t"
        "ROWS: .branchtargets R0, R1, R2, R3, R4, R5, R6, R7, DONE;\n\t"
        MCPG_ENTRY MCPG_WEIGHTS "brx.idx.uni xr, ROWS;\n\t"
        "R0: " MCPG_NEXT MCPG_ROW(w0, 0, 1, 2, 3, 4) MCPG_ROW(w1, 5, 6, 7, 8, 9)
        MCPG_ROW(w2, 10, 11, 12, 13, 14) MCPG_WEIGHTS "brx.idx.uni xr, ROWS;\n\t"
        "R1: " MCPG_NEXT MCPG_ROW(w0, 5, 6, 7, 8, 9) MCPG_ROW(w1, 10, 11, 12, 13, 14)
        MCPG_ROW(w2, 15, 16, 17, 18, 19) MCPG_WEIGHTS "brx.idx.uni xr, ROWS;\n\t"
        "R2: " MCPG_NEXT MCPG_ROW(w0, 10, 11, 12, 13, 14) MCPG_ROW(w1, 15, 16, 17, 18, 19)
        MCPG_ROW(w2, 20, 21, 22, 23, 24) MCPG_WEIGHTS "brx.idx.uni xr, ROWS;\n\t"
        "R3: " MCPG_NEXT MCPG_ROW(w0, 15, 16, 17, 18, 19) MCPG_ROW(w1, 20, 21, 22, 23, 24)
        MCPG_ROW(w2, 25, 26, 27, 28, 29) MCPG_WEIGHTS "brx.idx.uni xr, ROWS;\n\t"
        "R4: " MCPG_NEXT MCPG_ROW(w0, 20, 21, 22, 23, 24) MCPG_ROW(w1, 25, 26, 27, 28, 29)
        MCPG_ROW(w2, 30, 31, 32, 33, 34) MCPG_WEIGHTS "brx.idx.uni xr, ROWS;\n\t"
        "R5: " MCPG_NEXT MCPG_ROW(w0, 25, 26, 27, 28, 29) MCPG_ROW(w1, 30, 31, 32, 33, 34)
        MCPG_ROW(w2, 35, 36, 37, 38, 39) MCPG_WEIGHTS "brx.idx.uni xr, ROWS;\n\t"
        "R6: " MCPG_NEXT MCPG_ROW(w0, 30, 31, 32, 33, 34) MCPG_ROW(w1, 35, 36, 37, 38, 39)
        MCPG_ROW(w2, 40, 41, 42, 43, 44) MCPG_WEIGHTS "brx.idx.uni xr, ROWS;\n\t"
        "R7: " MCPG_NEXT MCPG_ROW(w0, 35, 36, 37, 38, 39) MCPG_ROW(w1, 40, 41, 42, 43, 44)
        MCPG_ROW(w2, 45, 46, 47, 48, 49) MCPG_WEIGHTS "brx.idx.uni xr, ROWS;\n\t"
        "DONE:\n\t}"
        : "+l"(acc[0][0]), "+l"(acc[0][1]), "+l"(acc[0][2]), "+l"(acc[0][3]), "+l"(acc[0][4]), "+l"(acc[1][0]),
          "+l"(acc[1][1]), "+l"(acc[1][2]), "+l"(acc[1][3]), "+l"(acc[1][4]), "+l"(acc[2][0]), "+l"(acc[2][1]),
          "+l"(acc[2][2]), "+l"(acc[2][3]), "+l"(acc[2][4]), "+l"(acc[3][0]), "+l"(acc[3][1]), "+l"(acc[3][2]),
          "+l"(acc[3][3]), "+l"(acc[3][4]), "+l"(acc[4][0]), "+l"(acc[4][1]), "+l"(acc[4][2]), "+l"(acc[4][3]),
          "+l"(acc[4][4]), "+l"(acc[5][0]), "+l"(acc[5][1]), "+l"(acc[5][2]), "+l"(acc[5][3]), "+l"(acc[5][4]),
          "+l"(acc[6][0]), "+l"(acc[6][1]), "+l"(acc[6][2]), "+l"(acc[6][3]), "+l"(acc[6][4]), "+l"(acc[7][0]),
          "+l"(acc[7][1]), "+l"(acc[7][2]), "+l"(acc[7][3]), "+l"(acc[7][4]), "+l"(acc[8][0]), "+l"(acc[8][1]),
          "+l"(acc[8][2]), "+l"(acc[8][3]), "+l"(acc[8][4]), "+l"(acc[9][0]), "+l"(acc[9][1]), "+l"(acc[9][2]),
          "+l"(acc[9][3]), "+l"(acc[9][4])
        : "r"(pj), "r"(pe), "n"(WARPS * 16), "n"(SROW * 4)
        : "memory");
}
#undef MCPG_NEXT
#undef MCPG_WEIGHTS
#undef MCPG_ENTRY
#undef MCPG_ROW
#undef MCPG_FMA2

// Genes i in [i0, i1).  Wt as for the dense kernel, ent[s][gene] = {w0, w1, w2, first row}, both
// zero-padded to ldg genes (whole tiles on either side) and whole chunks of SCH samples.
template <int WARPS, int EPI>
__global__ void __launch_bounds__(WARPS * 32, 1)
    mi_rows_kernel(const float* __restrict__ Wt, int64_t ldwt, const float4* __restrict__ ent, int64_t ldg,
                   const int* __restrict__ irregular, const double* __restrict__ H, int64_t n, int64_t m_pad,
                   float inv_m, float* __restrict__ MI, int64_t ldmi, int64_t i0, int64_t i1, const QArgs qa) {
    constexpr int SSTAGE = rows_stage(WARPS);
    extern __shared__ float4 smem_f4[];
    float* smem = reinterpret_cast<float*>(smem_f4);
    // grid: 4 j tiles (fastest), i tiles, groups of 4 j tiles
    const int64_t gi0 = i0 + (int64_t)blockIdx.y * WARPS, gj0 = ((int64_t)blockIdx.z * 4 + blockIdx.x) * SJ + (EPI == 1 ? qa.j0 : 0);
    if (gj0 >= (EPI == 1 ? qa.j1 : n) || (EPI != 1 && gj0 + SJ <= gi0)) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // a warp copies whole samples: 80 chunks of j weights, then the entries
    const float* srcj = Wt + gj0 * SB + lane * 4;
    const float4* srci = ent + gi0 + (lane - 16);
    auto load = [&](int stage, int64_t s0) {
        float* dj = smem + stage * SSTAGE + lane * 4;
        float* di = smem + stage * SSTAGE + SCH * SROW + (lane - 16) * 4;
        for (int r = warp; r < SCH; r += WARPS) {
            const float* sj = srcj + (s0 + r) * ldwt;
            cp_async16(dj + r * SROW, sj, 16);
            cp_async16(dj + r * SROW + 128, sj + 128, 16);
            if (lane < 16) cp_async16(dj + r * SROW + 256, sj + 256, 16);
            else if (lane < 16 + WARPS) cp_async16(di + r * WARPS * 4, srci + (s0 + r) * ldg, 16);
        }
    };

    unsigned long long acc[SB][SB / 2];
#pragma unroll
    for (int a = 0; a < SB; ++a)
#pragma unroll
        for (int q = 0; q < SB / 2; ++q) acc[a][q] = 0ull;

    const bool dense = *irregular != 0;
    const int64_t steps = m_pad / SCH;
    if (lane < SSTG)  // the end rows: no copy writes them
        *reinterpret_cast<float4*>(smem + lane * SSTAGE + SCH * SROW + (SCH * WARPS + warp) * 4) =
            make_float4(0.0f, 0.0f, 0.0f, __int_as_float(8));
    load(0, 0);
    cp_async_commit();
    for (int64_t t = 0; t < steps; ++t) {
        cp_async_wait<0>();
        __syncthreads();
        if (t + 1 < steps) load((int)((t + 1) & 1), (t + 1) * SCH);
        cp_async_commit();
        const float* st = smem + (t & 1) * SSTAGE;
        const float* bj = st + lane * SB;
        if (dense) {
            for (int s = 0; s < SCH; ++s) {
#pragma unroll
                for (int a = 0; a < SB; ++a) {
                    const unsigned long long w = pack2(Wt[(t * SCH + s) * ldwt + (gi0 + warp) * SB + a]);
#pragma unroll
                    for (int q = 0; q < SB / 2; ++q)
                        fma2(acc[a][q], w, *reinterpret_cast<const unsigned long long*>(bj + s * SROW + 2 * q));
                }
            }
            continue;
        }
        add_chunk<WARPS>(acc, (uint32_t)__cvta_generic_to_shared(bj),
                  (uint32_t)__cvta_generic_to_shared(st + SCH * SROW + warp * 4));
    }
    cp_async_wait<0>();

    const int64_t i = gi0 + warp, j = gj0 + lane;
    if (EPI >= 1) {
        if (i >= i1 || j >= (EPI == 1 ? qa.j1 : n) || (EPI == 2 && j < i)) return;
        const float gs = (i == j) ? 0.0f : qa.G[i * qa.ldg + j] + qa.G[j * qa.ldg + i];
        const float c = 1.4426950408889634f;  // 1 / ln 2
        float* Qr = qa.Q + i * SB * qa.ldq + (j - qa.j0) * SB;
        float2 v[SB][SB / 2];
#pragma unroll
        for (int x = 0; x < SB; ++x)
#pragma unroll
            for (int y = 0; y < SB / 2; ++y) {
                const float2 u = unpack2(acc[x][y]);
                const float p0 = u.x * inv_m, p1 = u.y * inv_m;
                v[x][y] = make_float2((gs != 0.0f && p0 > 0.0f) ? gs * (__log2f(p0) + c) : 0.0f,
                                      (gs != 0.0f && p1 > 0.0f) ? gs * (__log2f(p1) + c) : 0.0f);
                *reinterpret_cast<float2*>(Qr + x * qa.ldq + 2 * y) = v[x][y];
            }
        if (EPI == 2 && i != j) {
            float* Qm = qa.Q + j * SB * qa.ldq + i * SB;
#pragma unroll
            for (int y = 0; y < SB / 2; ++y)
#pragma unroll
                for (int x = 0; x < SB; x += 2) {
                    *reinterpret_cast<float2*>(Qm + (2 * y) * qa.ldq + x) = make_float2(v[x][y].x, v[x + 1][y].x);
                    *reinterpret_cast<float2*>(Qm + (2 * y + 1) * qa.ldq + x) = make_float2(v[x][y].y, v[x + 1][y].y);
                }
        }
        return;
    }
    if (i >= i1 || j >= n || j < i) return;
    double hxy = 0.0;
#pragma unroll
    for (int x = 0; x < SB; ++x) {
        float row = 0.0f;
#pragma unroll
        for (int y = 0; y < SB / 2; ++y) {
            const float2 u = unpack2(acc[x][y]);
            const float p0 = u.x * inv_m, p1 = u.y * inv_m;
            if (p0 > 0.0f) row += p0 * __log2f(p0);
            if (p1 > 0.0f) row += p1 * __log2f(p1);
        }
        hxy += (double)row;
    }
    const float v = (float)(H[i] + H[j] + hxy);  // hxy = -H_ij
    MI[i * ldmi + j] = v;
    MI[j * ldmi + i] = v;
}

// ent[s][g] from the dense weights of (s, g): the three weights from the first nonzero bin on.
__global__ void __launch_bounds__(256) mi_entries_kernel(const float* __restrict__ Wt, int64_t ldwt, int64_t ldg,
                                                         int64_t m_pad, float4* __restrict__ ent,
                                                         int* __restrict__ irregular) {
    const int64_t g = (int64_t)blockIdx.x * 32 + (threadIdx.x & 31);
    for (int64_t s = (int64_t)blockIdx.y * 8 + (threadIdx.x >> 5); s < m_pad; s += (int64_t)gridDim.y * 8) {
        const float2* w = reinterpret_cast<const float2*>(Wt + s * ldwt + g * SB);
        float v[SB];
#pragma unroll
        for (int q = 0; q < SB / 2; ++q) {
            const float2 u = w[q];
            v[2 * q] = u.x;
            v[2 * q + 1] = u.y;
        }
        int r = SB - 3;
#pragma unroll
        for (int a = SB - 4; a >= 0; --a)
            if (v[a] != 0.0f) r = a;
        float4 e = make_float4(v[SB - 3], v[SB - 2], v[SB - 1], __int_as_float(r));
#pragma unroll
        for (int a = 0; a < SB - 3; ++a)
            if (r == a) {
                e.x = v[a];
                e.y = v[a + 1];
                e.z = v[a + 2];
            }
        ent[s * ldg + g] = e;
        // every nonzero weight is in the window, or the sample is irregular (a NaN counts as nonzero)
        int nonzero = 0;
#pragma unroll
        for (int a = 0; a < SB; ++a) nonzero += v[a] != 0.0f;
        if (nonzero != (e.x != 0.0f) + (e.y != 0.0f) + (e.z != 0.0f)) *irregular = 1;
    }
}

template <int WARPS, int EPI>
cudaError_t launch_rows_warps(const float* Wt, int64_t ldwt, const float4* ent, int64_t ldg, const int* irregular,
                              const double* H, int64_t n, int64_t m, float* MI, int64_t ldmi, int64_t i0, int64_t i1,
                              const QArgs& qa, cudaStream_t stream) {
    constexpr size_t smem = (size_t)SSTG * rows_stage(WARPS) * sizeof(float);
    auto kern = mi_rows_kernel<WARPS, EPI>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    dim3 grid(4, (unsigned)ceil_div(i1 - i0, WARPS), (unsigned)ceil_div(EPI == 1 ? qa.j1 - qa.j0 : n, 4 * SJ));
    kern<<<grid, WARPS * 32, smem, stream>>>(Wt, ldwt, ent, ldg, irregular, H, n, ceil_div(m, SCH) * SCH,
                                             1.0f / (float)m, MI, ldmi, i0, i1, qa);
    return cudaGetLastError();
}

// The widest CTA (16 warps) once its tiles fill the SMs (one CTA each); below that 4 or 8 warps: with 16,
// 64 x 500 and 200 x 500 took 74 and 78 us, with 4 and 8 they take 49 and 54 us.
template <int EPI>
cudaError_t launch_rows(const float* Wt, int64_t ldwt, const float4* ent, int64_t ldg, const int* irregular,
                        const double* H, int64_t n, int64_t m, float* MI, int64_t ldmi, int64_t i0, int64_t i1,
                        const QArgs& qa, cudaStream_t stream) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t jt = ceil_div(EPI == 1 ? qa.j1 - qa.j0 : n, SJ);
    // EPI 0, 2: about half of the tiles hold some j >= i
    auto tiles = [&](int64_t w) { return ceil_div(i1 - i0, w) * jt / (EPI == 1 ? 1 : 2); };
    if (tiles(4) <= sms)
        return launch_rows_warps<4, EPI>(Wt, ldwt, ent, ldg, irregular, H, n, m, MI, ldmi, i0, i1, qa, stream);
    if (tiles(8) <= sms)
        return launch_rows_warps<8, EPI>(Wt, ldwt, ent, ldg, irregular, H, n, m, MI, ldmi, i0, i1, qa, stream);
    return launch_rows_warps<16, EPI>(Wt, ldwt, ent, ldg, irregular, H, n, m, MI, ldmi, i0, i1, qa, stream);
}

template <int BINS>
cudaError_t launch_bins(const float* Wt, int64_t ldwt, const double* H, int64_t n, int64_t m, float* MI, int64_t ldmi,
                        cudaStream_t stream, int64_t t0, int64_t t1) {
    using C = MiCfg<BINS>;
    auto kern = mi_fp32_kernel<BINS, 0>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    if (e != cudaSuccess) return e;
    const int64_t T = ceil_div(n, G);
    if (t1 > T) t1 = T;
    if (t0 >= t1) return cudaSuccess;
    // triangle rows [t0, t1): tiles start(t) = t*T - t(t-1)/2
    const int64_t start0 = t0 * T - t0 * (t0 - 1) / 2, start1 = t1 * T - t1 * (t1 - 1) / 2;
    const int64_t tiles = start1 - start0;
    const int64_t m_pad = ceil_div(m, BKS) * BKS;
    const float inv_m = 1.0f / (float)m;  // norm_factor = FT(1) / FT(m), BSplineMI.hpp:321
    kern<<<(unsigned)tiles, THREADS, C::SMEM, stream>>>(Wt, ldwt, H, n, m_pad, inv_m, MI, ldmi, T, QArgs{}, start0);
    return cudaGetLastError();
}

template <int BINS>
cudaError_t launch_q_bins(const float* Wt, int64_t ldwt, int64_t n, int64_t m, const QArgs& qa, cudaStream_t stream) {
    using C = MiCfg<BINS>;
    auto kern = mi_fp32_kernel<BINS, 1>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    if (e != cudaSuccess) return e;
    const int64_t T = ceil_div(n, G);
    const int64_t m_pad = ceil_div(m, BKS) * BKS;
    const float inv_m = 1.0f / (float)m;
    kern<<<(unsigned)(T * ceil_div(qa.j1 - qa.j0, G)), THREADS, C::SMEM, stream>>>(Wt, ldwt, nullptr, n, m_pad, inv_m,
                                                                                   nullptr, 0, T, qa, 0);
    return cudaGetLastError();
}

}  // namespace

// n genes and the overhang of a tile on either side
int64_t mi_rows_genes(int64_t n) { return ceil_div(n + SWARPS_MAX, SJ) * SJ; }
int64_t mi_rows_samples(int64_t m) { return ceil_div(m, SCH) * SCH; }

cudaError_t launch_mi_entries(const float* Wt, int64_t ldwt, int64_t ldg, int64_t m, float4* ent, int* irregular,
                              cudaStream_t stream, int64_t* launches) {
    const int64_t m_pad = mi_rows_samples(m);
    if (launches) ++*launches;
    dim3 grid((unsigned)(ldg / 32), (unsigned)(m_pad / 8 < 1024 ? m_pad / 8 : 1024));
    mi_entries_kernel<<<grid, 256, 0, stream>>>(Wt, ldwt, ldg, m_pad, ent, irregular);
    return cudaGetLastError();
}

cudaError_t launch_mi_rows(const float* Wt, int64_t ldwt, const float4* ent, int64_t ldg, const int* irregular,
                           const double* H, int64_t n, int64_t m, float* MI, int64_t ldmi, int64_t gene0,
                           int64_t gene1, cudaStream_t stream, int64_t* launches) {
    if (gene1 < 0 || gene1 > n) gene1 = n;
    if (n <= 0 || gene0 >= gene1) return cudaSuccess;
    if (ldg != mi_rows_genes(n) || ldwt < ldg * SB) return cudaErrorInvalidValue;
    if (launches) ++*launches;
    return launch_rows<0>(Wt, ldwt, ent, ldg, irregular, H, n, m, MI, ldmi, gene0, gene1, QArgs{}, stream);
}

cudaError_t launch_mi_q_rows(const float* Wt, int64_t ldwt, const float4* ent, int64_t ldge, const int* irregular,
                             const float* G, int64_t ldg, int64_t n, int64_t m, int64_t j0, int64_t j1, float* Q,
                             int64_t ldq, cudaStream_t stream, int64_t* launches) {
    if (n <= 0 || j0 >= j1) return cudaSuccess;
    if (ldge != mi_rows_genes(n) || ldwt < ldge * SB || j0 % SJ || j1 > n || ldq % 2) return cudaErrorInvalidValue;
    if (launches) ++*launches;
    const QArgs qa{G, ldg, Q, ldq, j0, j1};
    if (j0 == 0 && j1 == n)
        return launch_rows<2>(Wt, ldwt, ent, ldge, irregular, nullptr, n, m, nullptr, 0, 0, n, qa, stream);
    return launch_rows<1>(Wt, ldwt, ent, ldge, irregular, nullptr, n, m, nullptr, 0, 0, n, qa, stream);
}

// Adjoint slab: Q for all genes i and the genes j in [j0, j1), j0 a multiple of 16.
cudaError_t launch_mi_q(const float* Wt, int64_t ldwt, const float* G, int64_t ldg, int64_t n, int64_t m, int bins,
                        int64_t j0, int64_t j1, float* Q, int64_t ldq, cudaStream_t stream, int64_t* launches) {
    if (n <= 0 || j0 >= j1) return cudaSuccess;
    if (j0 % 16 || j1 > n) return cudaErrorInvalidValue;
    if (launches) ++*launches;
    QArgs qa{G, ldg, Q, ldq, j0, j1};
    switch (bins) {
        case 2: return launch_q_bins<2>(Wt, ldwt, n, m, qa, stream);
        case 3: return launch_q_bins<3>(Wt, ldwt, n, m, qa, stream);
        case 4: return launch_q_bins<4>(Wt, ldwt, n, m, qa, stream);
        case 5: return launch_q_bins<5>(Wt, ldwt, n, m, qa, stream);
        case 6: return launch_q_bins<6>(Wt, ldwt, n, m, qa, stream);
        case 7: return launch_q_bins<7>(Wt, ldwt, n, m, qa, stream);
        case 8: return launch_q_bins<8>(Wt, ldwt, n, m, qa, stream);
        case 9: return launch_q_bins<9>(Wt, ldwt, n, m, qa, stream);
        case 10: return launch_q_bins<10>(Wt, ldwt, n, m, qa, stream);
        case 11: return launch_q_bins<11>(Wt, ldwt, n, m, qa, stream);
        case 12: return launch_q_bins<12>(Wt, ldwt, n, m, qa, stream);
        default: return cudaErrorNotSupported;
    }
}

// Wt must be zero-padded: ldwt >= ceil(n/16)*16*bins (multiple of 4), rows
// s in [m, ceil(m/16)*16) zero.
cudaError_t launch_mi_fp32(const float* Wt, int64_t ldwt, const double* H, int64_t n, int64_t m, int bins, float* MI,
                           int64_t ldmi, cudaStream_t stream, int64_t* launches, int64_t gene0, int64_t gene1) {
    if (gene1 < 0 || gene1 > n) gene1 = n;
    if (n <= 0 || gene0 >= gene1) return cudaSuccess;
    if (gene0 % G) return cudaErrorInvalidValue;
    const int64_t t0 = gene0 / G, t1 = ceil_div(gene1, G);
    if (launches) ++*launches;
    switch (bins) {
        case 2: return launch_bins<2>(Wt, ldwt, H, n, m, MI, ldmi, stream, t0, t1);
        case 3: return launch_bins<3>(Wt, ldwt, H, n, m, MI, ldmi, stream, t0, t1);
        case 4: return launch_bins<4>(Wt, ldwt, H, n, m, MI, ldmi, stream, t0, t1);
        case 5: return launch_bins<5>(Wt, ldwt, H, n, m, MI, ldmi, stream, t0, t1);
        case 6: return launch_bins<6>(Wt, ldwt, H, n, m, MI, ldmi, stream, t0, t1);
        case 7: return launch_bins<7>(Wt, ldwt, H, n, m, MI, ldmi, stream, t0, t1);
        case 8: return launch_bins<8>(Wt, ldwt, H, n, m, MI, ldmi, stream, t0, t1);
        case 9: return launch_bins<9>(Wt, ldwt, H, n, m, MI, ldmi, stream, t0, t1);
        case 10: return launch_bins<10>(Wt, ldwt, H, n, m, MI, ldmi, stream, t0, t1);
        case 11: return launch_bins<11>(Wt, ldwt, H, n, m, MI, ldmi, stream, t0, t1);
        case 12: return launch_bins<12>(Wt, ldwt, H, n, m, MI, ldmi, stream, t0, t1);
        default: return cudaErrorNotSupported;
    }
}

}  // namespace mcpg
