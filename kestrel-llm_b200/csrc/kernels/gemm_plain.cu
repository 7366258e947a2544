// Plain matrix product on the CUDA cores: out[t, n] = sum_k x[t, k] * w[n, k], float32
// accumulation by FMA in ascending k for every output, whatever T is (the reference's
// float32 product, st.c:8880-8892, is the same sum row by row).  It is the whole product of
// the true 32-bit path, the fallback of the bfloat16 path for sizes the tensor-core kernel
// refuses, and the twin that the tensor-core kernel is tested against.  Any T, N, K.
//
// float32 operands whose rows 16-byte copies can fetch go to the kernel of gemm_f32.cuh, the same bits; this one
// takes the others: tile 64x64, 256 threads, 4x4 outputs per thread, K in steps of 16 through shared memory.
#include "common.cuh"
#include "gemm_f32.cuh"

#define PG_BM 64
#define PG_BN 64
#define PG_BK 16

template <typename T>
__global__ void __launch_bounds__(256)
gemm_plain_kernel(const T *__restrict__ x, const T *__restrict__ w, float *__restrict__ out,
                  int Tn, int N, int K, long long ldx, long long ldw, long long ldo) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float xs[PG_BK][PG_BM + 4];
    __shared__ float ws[PG_BK][PG_BN + 4];
    int tid = threadIdx.x;
    int t0 = blockIdx.y * PG_BM, n0 = blockIdx.x * PG_BN;
    int ty = tid / 16, tx = tid % 16;          // 16 x 16 threads, each 4 rows x 4 cols
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += PG_BK) {
        // 64 rows x 16 k = 1024 elements per operand, 4 per thread
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            int idx = tid + 256 * e;
            int r = idx / PG_BK, kk = idx % PG_BK;
            int gk = k0 + kk;
            float xv = 0.f, wv = 0.f;
            if (gk < K) {
                if (t0 + r < Tn) xv = to_f32<T>(x[(size_t)(t0 + r) * ldx + gk]);
                if (n0 + r < N) wv = to_f32<T>(w[(size_t)(n0 + r) * ldw + gk]);
            }
            xs[kk][r] = xv;
            ws[kk][r] = wv;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < PG_BK; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = xs[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int t = t0 + ty * 4 + i;
        if (t >= Tn) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            int n = n0 + tx * 4 + j;
            if (n < N) out[(size_t)t * ldo + n] = acc[i][j];
        }
    }
}

KESTREL_API int kestrel_gemm_plain(const void *x, const void *w, float *out, int dtype, int T, int N,
                                   int K, long long ldx, long long ldw, long long ldo,
                                   cudaStream_t stream) {
    if (T == 0) return 0;
    KESTREL_REQUIRE(T > 0 && N > 0 && K > 0, "gemm_plain: bad sizes T=%d N=%d K=%d", T, N, K);
    if (dtype == KESTREL_F32 && K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0) {
        // The largest tile of which there are two a SM; beyond that what few tokens waste of a tile counts (a tile of 64 rows for 16 tokens
        // of N = 32,000 takes 225 us, one of 16 rows 113).  Measured, N = 2,048, K = 6,144 | N = 12,288, K = 2,048 in us, beside the one tile
        // of 64 x 64 in steps of 16 this replaces: T = 1 30 | 28 (619 | 407), T = 8 40 | 31 (618 | 411), T = 100 167 | 171 (593 | 472),
        // T = 411 306 | 545 (1,188 | 1,195), T = 2,048 1,158 | 2,266 (2,477 | 4,578).
        const float *xf = (const float *)x, *wf = (const float *)w;
        const long long want = 2ll * kestrel_sms();
        auto tiles = [&](int bm, int bn) { return (long long)((T + bm - 1) / bm) * ((N + bn - 1) / bn); };
        if (T > 32 && tiles(64, 64) >= want) return gf_launch<64, 64, 8, 4, 32, 3>(xf, wf, out, T, N, K, ldx, ldw, ldo, stream);
        if (T > 16 && tiles(32, 32) >= want) return gf_launch<32, 32, 4, 4, 32, 4>(xf, wf, out, T, N, K, ldx, ldw, ldo, stream);
        if (T > 8) return gf_launch<16, 32, 4, 2, 64, 6>(xf, wf, out, T, N, K, ldx, ldw, ldo, stream);
        if (T > 4 && tiles(8, 32) >= want) return gf_launch<8, 32, 2, 2, 64, 6>(xf, wf, out, T, N, K, ldx, ldw, ldo, stream);
        return gf_launch<4, 16, 1, 1, 128, 6>(xf, wf, out, T, N, K, ldx, ldw, ldo, stream);
    }
    dim3 grid((N + PG_BN - 1) / PG_BN, (T + PG_BM - 1) / PG_BM);
    KESTREL_REQUIRE(grid.y <= 65535, "gemm_plain: T=%d needs more than 65535 row tiles", T);
    if (dtype == KESTREL_F32)
        kestrel_launch(gemm_plain_kernel<float>, dim3(grid), dim3(256), 0, stream, (const float *)x, (const float *)w, out, T, N, K, ldx, ldw, ldo);
    else if (dtype == KESTREL_BF16)
        kestrel_launch(gemm_plain_kernel<__nv_bfloat16>, dim3(grid), dim3(256), 0, stream, (const __nv_bfloat16 *)x, (const __nv_bfloat16 *)w, out, T, N, K, ldx, ldw, ldo);
    else
        return kestrel_fail(-2, "gemm_plain: unknown dtype %d", dtype);
    return kestrel_check_launch("gemm_plain");
}
