// Matrix product of the true 32-bit path, out[t, n] = sum_k x[t, k] * w[n, k], for operands that 16-byte copies can fetch: FMA on the
// CUDA cores in ascending k for every output, the same bits as gemm_plain_kernel whatever T and the tile are.
//
// Both operands keep their rows in shared memory as they lie in memory (k runs along a row; rows of BK + 4 floats, so that the four-float
// reads of eight neighbouring rows fall on all 32 banks) and come by cp.async, STAGES - 1 steps of BK ahead.  A thread owns TM x TN
// outputs, its rows BM / TM and its columns BN / TN apart; for four k it reads TM + TN vectors for 4 TM TN multiply-adds.  A warp's read of
// a vector takes four cycles of the SM's shared memory and a warp's multiply-add a cycle of its quarter of the SM: a tile of 8 x 4 a
// thread is bound by the reads (1.5 of the multiply-adds' time; 0.64 of the multiply-adds' rate at 2,048 tokens, N = 12,288), yet 8 x 8 and 16 x 8,
// which are not, were no faster anywhere (2,193 and 2,466 us against 2,266): fewer warps, with 168 and 255 registers.
#pragma once
#include "common.cuh"

__device__ __forceinline__ void gf_copy16(uint32_t dst, const float *src, bool valid) {
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

template <int BM, int BN, int TM, int TN, int BK, int STAGES>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_kernel(const float *__restrict__ x, const float *__restrict__ w, float *__restrict__ out, int Tn, int N, int K, long long ldx,
                long long ldw, long long ldo) {
    constexpr int THREADS = (BM / TM) * (BN / TN), LD = BK + 4, CHUNKS = BK / 4, ROWS = BM + BN, TX = BN / TN;
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float gf_sm[];            // [STAGES][x rows, then w rows][LD]
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    const int t0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const uint32_t sm = (uint32_t)__cvta_generic_to_shared(gf_sm);
    auto fetch = [&](int step) {
        const int k0 = step * BK;
        const uint32_t to = sm + (uint32_t)(step % STAGES) * ROWS * LD * 4;
#pragma unroll
        for (int i = 0; i < (ROWS * CHUNKS + THREADS - 1) / THREADS; ++i) {
            const int idx = tid + i * THREADS;
            if (ROWS * CHUNKS % THREADS != 0 && idx >= ROWS * CHUNKS) break;
            const int r = idx / CHUNKS, k = k0 + (idx % CHUNKS) * 4;
            const bool is_x = r < BM;
            const int row = is_x ? t0 + r : n0 + r - BM;
            const bool valid = row < (is_x ? Tn : N) && k < K;
            const float *from = is_x ? x : w;
            if (valid) from += (size_t)row * (is_x ? ldx : ldw) + k;
            gf_copy16(to + (uint32_t)(r * LD + (idx % CHUNKS) * 4) * 4, from, valid);
        }
    };
    const int steps = (K + BK - 1) / BK;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) fetch(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
    for (int s = 0; s < steps; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                        // step s is there for all, and all are done with the stage that is filled next
        if (s + STAGES - 1 < steps) fetch(s + STAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float *xs = gf_sm + (size_t)(s % STAGES) * ROWS * LD + ty * LD, *ws = gf_sm + (size_t)(s % STAGES) * ROWS * LD + (BM + tx) * LD;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            float4 b[TN];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4 *>(ws + j * TX * LD + k);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float4 a = *reinterpret_cast<const float4 *>(xs + i * (BM / TM) * LD + k);
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    acc[i][j] = fmaf(a.x, b[j].x, acc[i][j]);
                    acc[i][j] = fmaf(a.y, b[j].y, acc[i][j]);
                    acc[i][j] = fmaf(a.z, b[j].z, acc[i][j]);
                    acc[i][j] = fmaf(a.w, b[j].w, acc[i][j]);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int t = t0 + ty + i * (BM / TM);
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx + j * TX;
            if (t < Tn && n < N) out[(size_t)t * ldo + n] = acc[i][j];
        }
    }
}

template <int BM, int BN, int TM, int TN, int BK, int STAGES>
static int gf_launch(const float *x, const float *w, float *out, int T, int N, int K, long long ldx, long long ldw, long long ldo, cudaStream_t stream) {
    constexpr size_t smem = (size_t)STAGES * (BM + BN) * (BK + 4) * sizeof(float);
    static bool attr_set = false;
    if (!attr_set) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_f32_kernel<BM, BN, TM, TN, BK, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return kestrel_fail(-3, "gemm_plain: cannot raise the shared-memory limit: %s", cudaGetErrorString(e));
        attr_set = true;
    }
    const dim3 grid((N + BN - 1) / BN, (T + BM - 1) / BM);
    KESTREL_REQUIRE(grid.y <= 65535, "gemm_plain: T=%d needs more than 65535 row tiles", T);
    kestrel_launch(gemm_f32_kernel<BM, BN, TM, TN, BK, STAGES>, grid, dim3((BM / TM) * (BN / TN)), smem, stream, x, w, out, T, N, K, ldx, ldw, ldo);
    return kestrel_check_launch("gemm_plain");
}
