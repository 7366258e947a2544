// Causal softmax attention of prompt portions over cache rows that are key AND value, on the 5th-generation tensor cores: a key is
// a whole row of `hd` numbers (up to 256), a value the row's first `vd`; all query heads of a kv head share the rows.  It is the
// form in which attention over cached latents runs.
//
// A CTA owns 128 rows - (token, query head of one kv group) pairs, token-major - and walks the cache rows they may see in tiles of
// 64, anchored at multiples of 64 of the absolute position.  A tile is fetched once and read twice: as the K-major operand of
// S = Q K^T and as the MN-major operand of O += P V, so the two products cost one load.  Six warps in three roles, coupled by mbarriers:
//   softmax  (warps 0-3)  a thread owns a row (TMEM lane): its 64 scores come out of TMEM once, maximum, exp2 and sum in float32, P goes
//            back as packed bfloat16 over the first 32 columns of its score buffer;
//   loader   (warp 4)     pages by TMA (boxes of a page, or of 64 rows of a larger page, by 64 columns; 128-byte swizzle) into a ring of
//            six stages: a stage is freed by the tile's second product, five tiles before its next content is needed;
//   issuer   (warp 5)     S(0) | S(t + 1), O += P(t) V(t): the scores of the next tile are made while this tile is softmaxed, for which
//            there are two score buffers of 64 columns.
// TMEM: S 2 x 64, Q 128 (two numbers to a column), O up to 256 columns.  Q is operand A of S from TMEM: from shared memory each product of
// 128 x 64 x 16 read 4 KB of Q beside 2 KB of keys.  What bounds the kernel is the chain of a tile: scores out, softmax, P in, hand-overs.
// 1,024 tokens of 16 heads behind 2,000, rows of 256, values of 192: 72.0 us (78.6 with Q in shared memory and a ring of four), where the
// mma.sync kernel (attention_window.cu) took 389.
// As in attention_tc.cu the output is rescaled only when a row's maximum has outgrown its reference by more than 2^8, keys a row may
// not see are masked in S, rows outside the CTA's key range are zeroed in shared memory before they are read as values (a page may hold
// another request's stale numbers), key ranges may be cut into slices that attention_merge combines, tiles with most keys go first, and
// every wait is bounded (kestrel_attention_rows_tc_error).
#include "attention_params.cuh"
#include "tcgen05.cuh"
#include <math.h>

#define AR_THREADS 192
#define AR_BM 128
#define AR_BN 64
#define AR_STAGES 6
#define AR_MAX_HD 256
#define AR_K_PANEL (AR_BN * 128)            // bytes of a panel of 64 columns: 64 cache rows
#define AR_RESCALE_STEP 8.0f

__device__ int g_ar_error = 0;

__device__ __forceinline__ float ar_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// 32 consecutive TMEM columns of this thread's lane
__device__ __forceinline__ void ar_ld32(uint32_t taddr, uint32_t *r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void ar_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void ar_st16(uint32_t taddr, const uint32_t *r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void ar_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D (TMEM) = or += A (TMEM, 128 x 16 bfloat16 packed two to a column) x B (shared memory)
__device__ __forceinline__ void ar_mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}

enum { R_Q_FULL = 0, R_K_FULL = 1, R_K_EMPTY = R_K_FULL + AR_STAGES, R_S_FULL = R_K_EMPTY + AR_STAGES, R_P_FULL = R_S_FULL + 2, R_PV_DONE = R_P_FULL + 2,
       R_COUNT = R_PV_DONE + 2 };

struct ArParams {
    AttnParams a;               // v_cache unused; window, gate, slices as there
    int vd;
};

__global__ void __launch_bounds__(AR_THREADS, 1)
attention_rows_tc_kernel(const __grid_constant__ CUtensorMap map_k, const ArParams ap, int cache_pages, int rows_per_tile) {
    const AttnParams &p = ap.a;
    const int hd = p.hd, vd = ap.vd;
    const int panels = (hd + 63) / 64, k_steps = (hd + 15) / 16, vd16 = (vd + 15) / 16 * 16;
    // M = 128, bf16 x bf16 -> f32; S: N = 64, both K-major; PV: N = vd rounded up to 16, B MN-major
    const uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(AR_BM >> 4) << 24);
    const uint32_t idesc_s = IDESC | ((uint32_t)(AR_BN >> 3) << 17), idesc_pv = IDESC | (1u << 16) | ((uint32_t)(vd16 >> 3) << 17);
    const uint32_t stage_bytes = (uint32_t)panels * AR_K_PANEL;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *aligned = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t k_s = base;
    const uint32_t bar_off = (uint32_t)panels * AR_STAGES * AR_K_PANEL;
    const uint32_t bars = base + bar_off, tmem_slot = bars + 8 * R_COUNT;
    volatile uint32_t *tmem_slot_ptr = (volatile uint32_t *)(aligned + bar_off + 8 * R_COUNT);
    uint8_t *k_ptr = aligned;
    auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        mbar_init(bar(R_Q_FULL), 4);
        for (int b = 0; b < AR_STAGES; ++b) { mbar_init(bar(R_K_FULL + b), 1); mbar_init(bar(R_K_EMPTY + b), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(bar(R_S_FULL + b), 1); mbar_init(bar(R_P_FULL + b), 4); mbar_init(bar(R_PV_DONE + b), 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot_ptr, tmem_q = tmem + 2 * AR_BN, tmem_o = tmem + 256;
    pdl_launch_dependents();            // after the allocation: a dependent's CTA that holds TMEM waits for this grid
    pdl_wait();

    const int kvh = blockIdx.x % p.nkv, tile = (int)(gridDim.x / p.nkv) - 1 - (int)(blockIdx.x / p.nkv), slice = blockIdx.z;
    const int G = p.nq / p.nkv;
    int seq, row0;
    if (p.tile_seq) seq = p.tile_seq[tile], row0 = p.tile_row0[tile];
    else attn_find_tile(p.cu_seqlens, p.nseq, G, rows_per_tile, tile, seq, row0);
    const int tok_begin = p.cu_seqlens[seq], n_tok = p.cu_seqlens[seq + 1] - tok_begin;
    const int pos_begin = p.kv_lens[seq] - n_tok;
    const int rows_here = min(rows_per_tile, n_tok * G - row0);
    const int *table = p.block_table + (size_t)seq * p.table_stride;
    const int first_tok = row0 / G, last_tok = (row0 + rows_here - 1) / G;
    // keys these rows may see, cut to the slice of the key range (slices are multiples of 128)
    const int k_hi = min(pos_begin + last_tok + 1, (slice + 1) * p.slice_len);
    const int k_first = max(p.window > 0 ? max(0, pos_begin + first_tok - p.window + 1) : 0, slice * p.slice_len);
    const int k_lo = (k_first / AR_BN) * AR_BN;
    const int n_tiles = k_hi > k_lo ? (k_hi - k_lo + AR_BN - 1) / AR_BN : 0;

    if (warp == 4) {
        // ------------------------------------------------------------------ loader: lane l fetches the l-th page of a tile
        const int box_rows = min(p.page_size, AR_BN), boxes = AR_BN / box_rows;
        for (int t = 0; t < n_tiles; ++t) {
            const int b = t % AR_STAGES;
            int row = 0;
            if (lane < boxes) {
                const int s0 = k_lo + t * AR_BN + lane * box_rows, idx = s0 / p.page_size;
                int page = idx < p.table_width ? table[idx] : 0;
                if (page < 0 || page >= cache_pages) page = 0;      // a released or absent page: masked, and zeroed as values
                row = (page * p.nkv + kvh) * p.page_size + s0 % p.page_size;
            }
            if (!mbar_wait(bar(R_K_EMPTY + b), ((uint32_t)(t / AR_STAGES) & 1u) ^ 1u)) { atomicExch(&g_ar_error, 1); break; }
            if (lane == 0) mbar_expect_tx(bar(R_K_FULL + b), stage_bytes);
            __syncwarp();
            if (lane < boxes) {
                const uint32_t dst = k_s + b * stage_bytes + lane * box_rows * 128;
                for (int c = 0; c < panels; ++c) tma_load_2d(dst + c * AR_K_PANEL, &map_k, bar(R_K_FULL + b), c * 64, row);
            }
        }
    } else if (warp == 5) {
        // ------------------------------------------------------------------ issuer
        if (lane == 0 && n_tiles > 0) {
            bool ok = mbar_wait(bar(R_Q_FULL), 0);
            if (!ok) atomicExch(&g_ar_error, 2);
            tc_fence_after();
            auto issue_s = [&](int t) {
                const int b = t % AR_STAGES;
                if (!mbar_wait(bar(R_K_FULL + b), (uint32_t)(t / AR_STAGES) & 1u)) { atomicExch(&g_ar_error, 3); return false; }
                tc_fence_after();
                for (int ks = 0; ks < k_steps; ++ks)
                    ar_mma_ts(tmem + (t & 1) * AR_BN, tmem_q + ks * 8, smem_desc(k_s + b * stage_bytes + (ks >> 2) * AR_K_PANEL + (ks & 3) * 32), idesc_s,
                              ks > 0 ? 1u : 0u);
                tc_commit(bar(R_S_FULL + (t & 1)));
                return true;
            };
            if (ok) ok = issue_s(0);
            for (int t = 0; t < n_tiles && ok; ++t) {
                // the other score buffer held P(t - 1), which the product before this one in the queue reads
                if (t + 1 < n_tiles && !(ok = issue_s(t + 1))) break;
                if (!mbar_wait(bar(R_P_FULL + (t & 1)), (uint32_t)(t >> 1) & 1u)) { atomicExch(&g_ar_error, 4); break; }
                tc_fence_after();
                const int b = t % AR_STAGES;
#pragma unroll
                for (int ks = 0; ks < AR_BN / 16; ++ks)      // P: 16 keys are 8 columns; V: 16 rows are two groups of 8
                    ar_mma_ts(tmem_o, tmem + (t & 1) * AR_BN + ks * 8, smem_desc_mn_major(k_s + b * stage_bytes + ks * 2048, AR_K_PANEL), idesc_pv,
                              (t > 0 || ks > 0) ? 1u : 0u);
                tc_commit(bar(R_K_EMPTY + b));
                tc_commit(bar(R_PV_DONE + (t & 1)));
            }
        }
    } else {
        // ------------------------------------------------------------------ softmax: thread r owns row r (TMEM lane r)
        const int r = tid;
        const int chunks = panels * 8;                       // 16-byte chunks of a cache row in shared memory
        // the row's query, two numbers to a column as P's, zeros beyond hd and for rows that are not there
        const uint32_t q_addr = tmem_q + (((uint32_t)(32 * warp)) << 16);
        const int q_row = row0 + min(r, rows_here - 1);
        const uint4 *q = reinterpret_cast<const uint4 *>(p.q + ((size_t)(tok_begin + q_row / G) * p.nq + kvh * G + q_row % G) * hd);
        for (int c = 0; c < k_steps * 8; c += 16) {
            uint32_t w[16];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const bool in = r < rows_here && (c / 4 + k) * 8 < hd;
                const uint4 x = in ? q[c / 4 + k] : make_uint4(0, 0, 0, 0);
                w[4 * k] = x.x, w[4 * k + 1] = x.y, w[4 * k + 2] = x.z, w[4 * k + 3] = x.w;
            }
            ar_st16(q_addr + c, w);
        }
        ar_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(R_Q_FULL));

        const bool row_ok = r < rows_here;
        const int my_pos = row_ok ? pos_begin + (row0 + r) / G : -1;
        const int my_lo = p.window > 0 ? max(0, my_pos - p.window + 1) : 0;
        const bool warp_has_rows = 32 * warp < rows_here;
        const uint32_t lane_base = ((uint32_t)(32 * warp)) << 16;
        float m_ref = -INFINITY, l_run = 0.f;
        bool ok = true;             // after a wait gave up the loop runs on without waiting, so that the warps still meet
        for (int t = 0; t < n_tiles; ++t) {
            const int kbase = k_lo + t * AR_BN, b = t % AR_STAGES;
            const uint32_t s_addr = tmem + lane_base + (t & 1) * AR_BN;
            if (ok && !mbar_wait(bar(R_S_FULL + (t & 1)), (uint32_t)(t >> 1) & 1u)) { atomicExch(&g_ar_error, 5); ok = false; }
            tc_fence_after();
            if (warp_has_rows) {
                uint32_t sr[AR_BN];
                ar_ld32(s_addr, sr);
                ar_ld32(s_addr + 32, sr + 32);
                ar_ld_wait();
                const bool whole = kbase >= k_first && kbase + AR_BN <= k_hi && kbase + AR_BN - 1 <= my_pos && kbase >= my_lo;
                if (!__all_sync(0xffffffffu, whole)) {
#pragma unroll
                    for (int j = 0; j < AR_BN; ++j) {
                        const int key = kbase + j;
                        if (!(key <= my_pos && key >= my_lo && key < k_hi && key >= k_first)) sr[j] = 0xff800000u;
                    }
                }
                float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int j = 0; j < AR_BN; ++j) m4[j & 3] = fmaxf(m4[j & 3], __uint_as_float(sr[j]));
                const float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * p.scale_log2;      // the scale is positive
                const bool grow = mx > m_ref + AR_RESCALE_STEP || (m_ref == -INFINITY && mx > -INFINITY);
                float alpha = 1.f;
                if (grow) {
                    if (m_ref != -INFINITY) alpha = ar_exp2(m_ref - mx);
                    m_ref = mx;
                }
                l_run *= alpha;
                const float shift = m_ref == -INFINITY ? 0.f : -m_ref;
                float l4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int c = 0; c < AR_BN / 2; c += 16) {
                    uint32_t w[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float e0 = ar_exp2(fmaf(__uint_as_float(sr[2 * (c + j)]), p.scale_log2, shift));
                        const float e1 = ar_exp2(fmaf(__uint_as_float(sr[2 * (c + j) + 1]), p.scale_log2, shift));
                        l4[j & 3] += e0 + e1;
                        __nv_bfloat162 b2 = __floats2bfloat162_rn(e0, e1);
                        w[j] = *reinterpret_cast<uint32_t *>(&b2);
                    }
                    ar_st16(s_addr + c, w);
                }
                l_run += (l4[0] + l4[1]) + (l4[2] + l4[3]);
                if (__any_sync(0xffffffffu, alpha != 1.f)) {
                    // the whole warp walks its rows' outputs; the product of the tile before must be done (S(t) is done, so the one
                    // before that is: each of the two barriers is at the phase waited for or just past it)
                    if (ok && !mbar_wait(bar(R_PV_DONE + ((t - 1) & 1)), (uint32_t)((t - 1) >> 1) & 1u)) { atomicExch(&g_ar_error, 6); ok = false; }
                    tc_fence_after();
                    for (int c = 0; c < vd16; c += 32) {
                        uint32_t o[32];
                        ar_ld32(tmem_o + lane_base + c, o);
                        ar_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
                        ar_st16(tmem_o + lane_base + c, o);
                        ar_st16(tmem_o + lane_base + c + 16, o + 16);
                    }
                }
                ar_st_wait();
            }
            if (kbase < k_first || kbase + AR_BN > k_hi) {
                // rows of keys outside the CTA's range become zero before they are read as values; the scores have read them already
                const int lo_rows = max(0, k_first - kbase), hi_row = min(AR_BN, k_hi - kbase);
                for (int idx = r; idx < AR_BN * chunks; idx += 128) {
                    const int row = idx / chunks, c = idx % chunks;
                    if (row < lo_rows || row >= hi_row)
                        *reinterpret_cast<uint4 *>(k_ptr + b * stage_bytes + (c >> 3) * AR_K_PANEL + row * 128 + (c & 7) * 16) = make_uint4(0, 0, 0, 0);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // zeroed rows -> tensor-core reads
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(R_P_FULL + (t & 1)));
        }
        if (n_tiles > 0 && ok && !mbar_wait(bar(R_PV_DONE + ((n_tiles - 1) & 1)), (uint32_t)((n_tiles - 1) >> 1) & 1u)) { atomicExch(&g_ar_error, 7); ok = false; }
        tc_fence_after();
        if (warp_has_rows) {
            const bool write = row_ok && ok;
            const int row = row0 + r;
            const size_t qrow = write ? (size_t)(tok_begin + row / G) * p.nq + kvh * G + row % G : 0;
            float inv = p.slices > 1 ? 1.f : 1.0f / l_run;
            if (write && p.gate) inv *= p.gate[qrow];
            for (int c = 0; c < vd16; c += 32) {
                uint32_t o[32];
                if (n_tiles > 0) {
                    ar_ld32(tmem_o + lane_base + c, o);             // warp-wide, whatever rows exist
                    ar_ld_wait();
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) o[j] = 0u;
                }
                if (!write) continue;
                if (p.slices > 1) {
                    float *po = p.part_o + (qrow * p.slices + slice) * vd + c;
#pragma unroll
                    for (int j = 0; j < 32; j += 8) {
                        if (c + j >= vd) break;
                        *reinterpret_cast<uint4 *>(po + j) = make_uint4(o[j], o[j + 1], o[j + 2], o[j + 3]);
                        *reinterpret_cast<uint4 *>(po + j + 4) = make_uint4(o[j + 4], o[j + 5], o[j + 6], o[j + 7]);
                    }
                } else {
                    __nv_bfloat16 *po = p.out + qrow * vd + c;
#pragma unroll
                    for (int j = 0; j < 32; j += 8) {
                        if (c + j >= vd) break;
                        uint32_t w[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            __nv_bfloat162 b2 = __floats2bfloat162_rn(__uint_as_float(o[j + 2 * k]) * inv, __uint_as_float(o[j + 2 * k + 1]) * inv);
                            w[k] = *reinterpret_cast<uint32_t *>(&b2);
                        }
                        *reinterpret_cast<uint4 *>(po + j) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
            }
            if (write && p.slices > 1) {
                p.part_ml[(qrow * p.slices + slice) * 2] = m_ref;
                p.part_ml[(qrow * p.slices + slice) * 2 + 1] = l_run;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 5) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// Whether the kernel takes rows of hd numbers with values of vd in pages of page_size.
KESTREL_API int kestrel_attention_rows_tc_supported(int hd, int vd, int page_size) {
    return hd > 0 && hd <= AR_MAX_HD && hd % 8 == 0 && vd > 0 && vd <= hd && vd % 8 == 0 && page_size > 0 && page_size % 8 == 0 &&
           (AR_BN % page_size == 0 || page_size % AR_BN == 0);
}

// q [T, nq * hd], cache [pages, nkv, page_size, hd], out [T, nq * vd] = gate[token, head] (float32 [T, nq], or null) * softmax(q . row * scale) row[:vd]
// over causal keys (the last `window` of them, 0: all).  Tiles of up to 128 rows, listed by tile_seq / tile_row0, or
// with null for both all of the nseq requests' tiles.  With slices > 1 every CTA takes
// slice_len keys (a multiple of 128); scratch part_o [T * nq, slices, vd], part_ml [T * nq, slices, 2]; the gate is then the merge's.
KESTREL_API int kestrel_attention_rows_tc(const void *q, const void *cache, void *out, float *part_o, float *part_ml, const int *tile_seq,
                                          const int *tile_row0, int tiles, int rows_per_tile, const int *cu_seqlens, int nseq, const int *kv_lens,
                                          const int *block_table, int table_width, int table_stride, int page_size, int cache_pages, int T, int nq,
                                          int nkv, int hd, int vd, int window, int slices, int slice_len, const float *gate, float scale,
                                          cudaStream_t stream) {
    if (T == 0 || tiles == 0) return 0;
    KESTREL_REQUIRE(kestrel_attention_rows_tc_supported(hd, vd, page_size), "attention_rows_tc: rows of %d, values of %d, pages of %d", hd, vd, page_size);
    KESTREL_REQUIRE(rows_per_tile >= 1 && rows_per_tile <= AR_BM, "attention_rows_tc: tiles of %d rows; a CTA takes up to %d", rows_per_tile, AR_BM);
    KESTREL_REQUIRE((tile_seq == nullptr) == (tile_row0 == nullptr) && (tile_seq || nseq > 0), "attention_rows_tc: no tiles, and %d requests to cut into some", nseq);
    KESTREL_REQUIRE(nq > 0 && nkv > 0 && nq % nkv == 0, "attention_rows_tc: %d query heads over %d kv heads", nq, nkv);
    KESTREL_REQUIRE(window >= 0 && scale > 0.f, "attention_rows_tc: window %d, scale %g", window, (double)scale);
    KESTREL_REQUIRE(slices >= 1 && slices <= 1024 && slice_len > 0 && slice_len % 128 == 0, "attention_rows_tc: %d slices of %d keys", slices, slice_len);
    KESTREL_REQUIRE(slices == 1 || (part_o && part_ml), "attention_rows_tc: %d slices without scratch", slices);
    KESTREL_REQUIRE((long long)tiles * nkv < (1ll << 31), "attention_rows_tc: grid too large");
    KESTREL_REQUIRE(cache_pages > 0 && (long long)cache_pages * nkv * page_size < (1ll << 31), "attention_rows_tc: a cache of %d pages is beyond the 32-bit row coordinate", cache_pages);
    KESTREL_REQUIRE((((uintptr_t)q | (uintptr_t)cache | (uintptr_t)out | (uintptr_t)part_o) & 15) == 0, "attention_rows_tc: tensors must start on 16-byte boundaries");
    CUtensorMap map_k;
    int rc = kestrel_tensor_map_bf16(&map_k, cache, (long long)cache_pages * nkv * page_size, hd, hd, page_size < AR_BN ? page_size : AR_BN);
    if (rc) return rc;
    ArParams ap = {};
    AttnParams &p = ap.a;
    p.q = (const __nv_bfloat16 *)q; p.out = (__nv_bfloat16 *)out; p.part_o = part_o; p.part_ml = part_ml; p.tile_seq = tile_seq; p.tile_row0 = tile_row0;
    p.cu_seqlens = cu_seqlens; p.kv_lens = kv_lens; p.block_table = block_table; p.table_width = table_width; p.table_stride = table_stride;
    p.page_size = page_size; p.nq = nq; p.nkv = nkv; p.hd = hd; p.window = window; p.slices = slices; p.slice_len = slice_len;
    p.scale_log2 = scale * 1.4426950408889634f;
    p.nseq = nseq;
    p.gate = slices > 1 ? nullptr : gate;
    ap.vd = vd;
    // as much for every size: a CTA has all of an SM's TMEM and shares the SM with no other kernel that takes some
    const size_t smem = (size_t)(AR_MAX_HD / 64) * AR_STAGES * AR_K_PANEL + 8 * R_COUNT + 16 + 1024;
    static bool attr_set = false;
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(attention_rows_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return kestrel_fail(-3, "attention_rows_tc: cannot raise the shared-memory limit: %s", cudaGetErrorString(e));
        attr_set = true;
    }
    kestrel_launch(attention_rows_tc_kernel, dim3((unsigned)((long long)tiles * nkv), 1, slices), dim3(AR_THREADS), smem, stream, map_k, ap, cache_pages, rows_per_tile);
    rc = kestrel_check_launch("attention_rows_tc");
    if (rc || slices == 1) return rc;
    return attention_merge_gated(part_o, part_ml, out, tile_seq, tile_row0, tiles, rows_per_tile, cu_seqlens, nseq, slices, vd, nq, nkv, nullptr, gate, stream);
}

// Error word of the bounded waits (0: none; 1 loader, 2-4 issuer, 5-7 softmax).  Synchronises the device and clears the word.
KESTREL_API int kestrel_attention_rows_tc_error(void) {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_ar_error, sizeof(int)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_ar_error, &zero, sizeof(int));
    return v;
}
