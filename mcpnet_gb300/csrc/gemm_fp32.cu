// FP32 product of two k-major operands for the MI adjoint,
//   C[r][s] = sum_k A[k][r] B[k][s],
// each element one multiply-add chain over ascending k.
//
// Bound by the FP32 multiply-add pipe (128 lanes per clock and SM).  CTA tile 128 x 128, 256
// threads, 8 x 8 elements each, as packed fma.f32x2 over pairs of rows r: half the instructions to
// issue, so that loads and the duplication of B's values fit beside them.  Both operands are k-major,
// a 16-deep slice is two 8 KB blocks of whole 512-byte rows: four cp.async stages (64 KB), two CTAs per SM.
// The s tiles are the fast grid axis: the CTAs in flight share B's rows in L2.
//
// Measured: 40,960 x 1,024 x 40,960 in 53.9 ms (3.2e13 multiply-adds/s, 79 % of the pipe; nine waves of
// tiles, the last 42 % full), 20,480 x 1,000 x 20,480 in 14.3 ms (73 %; the last of five waves is
// 21 % full).  The form before took both operands row-major through the max-min kernel's loop with
// unpacked multiply-adds.
#include "common.cuh"
#include "internal.h"

namespace mcpg {
namespace {

constexpr int T = 128, BK = 16, STG = 4, TPB = 256;
constexpr size_t SMEM = (size_t)STG * 2 * BK * T * sizeof(float);

__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long twice(float v) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}

__global__ void __launch_bounds__(TPB, 2) gemm_fp32_kernel(const float* __restrict__ A, int64_t lda,
                                                           const float* __restrict__ B, int64_t ldb, int64_t R,
                                                           int64_t S, int64_t K, float* __restrict__ C, int64_t ldc) {
    extern __shared__ float4 gemm_smem[];
    float* smem = reinterpret_cast<float*>(gemm_smem);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t s0 = (int64_t)blockIdx.x * T, r0 = (int64_t)blockIdx.y * T;
    // a warp is 4 x 8 threads; a thread takes rows ty * 4 + {0..3, 64..67}, columns likewise
    const int ty = ((warp >> 1) << 2) + (lane >> 3), tx = ((warp & 1) << 3) + (lane & 7);
    const int lk = tid >> 5, lc = (tid & 31) * 4;  // loader: k rows lk and lk + 8, 16 bytes each
    const float* pa = A + r0 + lc;
    const float* pb = B + s0 + lc;
    auto load = [&](int stage, int64_t k0) {
        float* as = smem + stage * 2 * BK * T;
        float* bs = as + BK * T;
#pragma unroll
        for (int h = 0; h < BK; h += 8) {
            const int64_t k = k0 + lk + h;
            const bool ok = k < K;  // rows beyond K: zeros, which leave every sum as it is
            cp_async16(as + (lk + h) * T + lc, pa + (ok ? k : 0) * lda, ok ? 16 : 0);
            cp_async16(bs + (lk + h) * T + lc, pb + (ok ? k : 0) * ldb, ok ? 16 : 0);
        }
    };
    unsigned long long acc[4][8];  // pairs of rows x columns
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
    const int64_t steps = ceil_div(K, BK);
#pragma unroll
    for (int s = 0; s < STG - 1; ++s) {
        if (s < steps) load(s, (int64_t)s * BK);
        cp_async_commit();
    }
    for (int64_t t = 0; t < steps; ++t) {
        cp_async_wait<STG - 2>();
        __syncthreads();
        {
            const int64_t tn = t + STG - 1;
            if (tn < steps) load((int)(tn % STG), tn * BK);
            cp_async_commit();
        }
        const float* as = smem + (t % STG) * 2 * BK * T + ty * 4;
        const float* bs = smem + (t % STG) * 2 * BK * T + BK * T + tx * 4;
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(as + k * T);
            const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(as + k * T + 64);
            const float4 b0 = *reinterpret_cast<const float4*>(bs + k * T);
            const float4 b1 = *reinterpret_cast<const float4*>(bs + k * T + 64);
            const unsigned long long a[4] = {a0.x, a0.y, a1.x, a1.y};
            const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const unsigned long long bb = twice(b[j]);
#pragma unroll
                for (int i = 0; i < 4; ++i) fma2(acc[i][j], a[i], bb);
            }
        }
    }
    cp_async_wait<0>();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float2 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) asm("mov.b64 {%0, %1}, %2;" : "=f"(v[j].x), "=f"(v[j].y) : "l"(acc[i][j]));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int64_t r = r0 + ty * 4 + (i >> 1) * 64 + (i & 1) * 2 + h;
            if (r >= R) continue;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int64_t s = s0 + tx * 4 + (j >> 2) * 64 + (j & 3);
                if (s < S) C[r * ldc + s] = h ? v[j].y : v[j].x;
            }
        }
    }
}

}  // namespace

cudaError_t launch_gemm_fp32(const float* A, int64_t lda, const float* B, int64_t ldb, int64_t R, int64_t S, int64_t K,
                             float* C, int64_t ldc, cudaStream_t stream, int64_t* launches) {
    if (R <= 0 || S <= 0) return cudaSuccess;
    if (lda % T || ldb % T || lda < R || ldb < S || ((uintptr_t)A & 15u) || ((uintptr_t)B & 15u))
        return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(gemm_fp32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    if (e != cudaSuccess) return e;
    if (launches) ++*launches;
    dim3 grid((unsigned)ceil_div(S, T), (unsigned)ceil_div(R, T));
    gemm_fp32_kernel<<<grid, TPB, SMEM, stream>>>(A, lda, B, ldb, R, S, K, C, ldc);
    return cudaGetLastError();
}

}  // namespace mcpg
