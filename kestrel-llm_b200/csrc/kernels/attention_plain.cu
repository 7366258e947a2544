// Plain causal attention over the paged cache, one block per (token, query head).
//
// For the token at position p of its request the keys are positions lo..p of the same
// request, lo = 0 or p - window + 1 for a windowed layer; the mask is this loop bound, as in
// the reference (st.c:1974, st.c:10833-10849).  kv head = (h * nkv) / nq (st.c:10782);
// score = dot * scale (st.c:10846); softmax in float32 with a running maximum (the
// reference's tiled online form, st.c:9762-9859); out = sum_s w_s V_s.
//
// The four warps of a block take keys lo+w, lo+w+4, ... in groups of four; their running
// (max, sum, out) states are merged in warp order.  The order of every sum depends on
// (lo, p) alone: a token's result is bit-identical however the step was cut or batched.
// Works for any head size up to 576 and any numbers of heads.  It is the attention of the
// true 32-bit path and the twin that the fast kernels are tested against.
//
// Three options beyond the reference's attention, each off by default: `keep_first` tokens at
// the start of a request stay visible to a windowed layer after they have left the window (the
// keys are then positions 0..min(keep_first, lo)-1 followed by lo..p, walked in this order);
// values may have a size `vd` of their own (the V planes are [page][kv_head][slot][vd]); and
// `gate`, float32 [T, nq], multiplies each head's output.
//
// A layer may also change the scores and the way keys are weighed (`ScoreOpts`, attention_score.cuh):
// a cap, a logarithmic distance term, a softmax with a valueless extra term exp(sink) in its
// denominator (sink a number per head, or 0) - it enters the merge as one more state (max sink, sum 1, out 0) in front of the warps'
// - or sigmoid weights that are not normalised, where the states are plain sums.
#include "common.cuh"
#include "attention_score.cuh"
#include <math.h>

#define PA_WARPS 4
#define PA_MAX_PER_LANE 18    // head size up to 576 (a cached latent of 512 numbers beside a shared key part of 64)
#define PA_KEYS 4

template <typename T, typename TO>
__global__ void __launch_bounds__(PA_WARPS * 32)
attention_plain_kernel(const T *__restrict__ q, const T *__restrict__ k_cache, const T *__restrict__ v_cache,
                       const int *__restrict__ positions, const int *__restrict__ seq_of_token,
                       const int *__restrict__ block_table, int table_stride, int page_size,
                       TO *__restrict__ out, int nq, int nkv, int hd, int vd, int v_ld, int window, int keep_first,
                       const float *__restrict__ gate, float scale, const ScoreOpts opts) {
    pdl_launch_dependents();
    pdl_wait();
    int t = blockIdx.x, h = blockIdx.y;
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int kvh = (h * nkv) / nq;
    int pos = positions[t];
    int lo = window > 0 ? max(0, pos - window + 1) : 0;
    const int *table = block_table + (size_t)seq_of_token[t] * table_stride;
    int per_lane = (hd + 31) / 32, per_lane_v = (vd + 31) / 32;
    int n_kept = window > 0 ? min(keep_first, lo) : 0;      // visible keys before the window
    int n_keys = n_kept + (pos - lo + 1);

    float qv[PA_MAX_PER_LANE], acc[PA_MAX_PER_LANE];
    const T *qrow = q + ((size_t)t * nq + h) * hd;
#pragma unroll
    for (int c = 0; c < PA_MAX_PER_LANE; ++c) {
        int i = lane + 32 * c;
        qv[c] = (c < per_lane && i < hd) ? to_f32<T>(qrow[i]) : 0.f;
        acc[c] = 0.f;
    }
    float m = -INFINITY, l = 0.f;
    const HeadScore score(opts, h);
    const bool sigmoid = opts.weighting == KESTREL_WEIGH_SIGMOID;

    for (int base = warp * PA_KEYS; base < n_keys; base += PA_WARPS * PA_KEYS) {
        float sc[PA_KEYS];
        const T *vrow[PA_KEYS];
#pragma unroll
        for (int u = 0; u < PA_KEYS; ++u) {
            int j = base + u;
            int s = j < n_kept ? j : lo + (j - n_kept);
            float dot = 0.f;
            vrow[u] = nullptr;
            if (j < n_keys) {
                int page = table[s / page_size];
                size_t row = ((size_t)page * nkv + kvh) * page_size + (s % page_size);
                const T *krow = k_cache + row * hd;
                vrow[u] = v_cache + row * v_ld;
#pragma unroll
                for (int c = 0; c < PA_MAX_PER_LANE; ++c) {
                    int i = lane + 32 * c;
                    if (c < per_lane && i < hd) dot = fmaf(qv[c], to_f32<T>(krow[i]), dot);
                }
            }
            dot = warp_sum(dot);
            sc[u] = (j < n_keys) ? score(dot * scale, pos - s) : -INFINITY;
        }
        if (sigmoid) {                      // no running maximum: the weights are sums as they are
#pragma unroll
            for (int u = 0; u < PA_KEYS; ++u) {
                if (vrow[u]) {
                    const float p = sigmoid_f32(sc[u]);
#pragma unroll
                    for (int c = 0; c < PA_MAX_PER_LANE; ++c) {
                        int i = lane + 32 * c;
                        if (c < per_lane_v && i < vd) acc[c] = fmaf(p, to_f32<T>(vrow[u][i]), acc[c]);
                    }
                }
            }
            continue;
        }
        float mn = m;
#pragma unroll
        for (int u = 0; u < PA_KEYS; ++u) mn = fmaxf(mn, sc[u]);
        float corr = expf(m - mn);          // m = -inf on the first group: exp(-inf) = 0
        l *= corr;
#pragma unroll
        for (int c = 0; c < PA_MAX_PER_LANE; ++c) acc[c] *= corr;
#pragma unroll
        for (int u = 0; u < PA_KEYS; ++u) {
            if (vrow[u]) {
                float p = expf(sc[u] - mn);
                l += p;
#pragma unroll
                for (int c = 0; c < PA_MAX_PER_LANE; ++c) {
                    int i = lane + 32 * c;
                    if (c < per_lane_v && i < vd) acc[c] = fmaf(p, to_f32<T>(vrow[u][i]), acc[c]);
                }
            }
        }
        m = mn;
    }

    // merge the warps' states in warp order
    __shared__ float sm_m[PA_WARPS], sm_l[PA_WARPS];
    __shared__ float sm_acc[PA_WARPS][PA_MAX_PER_LANE * 32];
    if (lane == 0) { sm_m[warp] = m; sm_l[warp] = l; }
#pragma unroll
    for (int c = 0; c < PA_MAX_PER_LANE; ++c) sm_acc[warp][lane + 32 * c] = acc[c];
    __syncthreads();
    if (warp == 0) {
        const bool sink = opts.weighting == KESTREL_WEIGH_SOFTMAX_SINK;
        float M = sink ? score.sink : -INFINITY;
#pragma unroll
        for (int w = 0; w < PA_WARPS; ++w) M = fmaxf(M, sm_m[w]);
        float L = sink ? expf(score.sink - M) : 0.f;
        float o[PA_MAX_PER_LANE];
#pragma unroll
        for (int c = 0; c < PA_MAX_PER_LANE; ++c) o[c] = 0.f;
#pragma unroll
        for (int w = 0; w < PA_WARPS; ++w) {
            if (sigmoid) {
#pragma unroll
                for (int c = 0; c < PA_MAX_PER_LANE; ++c) o[c] += sm_acc[w][lane + 32 * c];
                continue;
            }
            if (sm_m[w] == -INFINITY) continue;     // a warp that saw no key
            float f = expf(sm_m[w] - M);
            L += sm_l[w] * f;
#pragma unroll
            for (int c = 0; c < PA_MAX_PER_LANE; ++c) o[c] += sm_acc[w][lane + 32 * c] * f;
        }
        float inv = sigmoid ? 1.0f : 1.0f / L;
        if (gate) inv *= gate[(size_t)t * nq + h];
        TO *orow = out + ((size_t)t * nq + h) * vd;
#pragma unroll
        for (int c = 0; c < PA_MAX_PER_LANE; ++c) {
            int i = lane + 32 * c;
            if (c < per_lane_v && i < vd) orow[i] = from_f32<TO>(o[c] * inv);
        }
    }
}

// The same attention for float32 layers that see every earlier token and have no options: up to eight rows - (token, head) pairs of one kv
// head and request - a block, the warps' streams of keys and every sum of a row as above, so that a row's bits still depend on its position
// alone, whatever rows share its block.  One row a block read every key again for each row and spent five shuffles, ten
// additions and five exponentials in all lanes on a key of a row; here a warp reads four keys for all rows, the 32 dot products of four
// keys and eight rows take 31 exchanges together (the same tree over the lanes), a lane makes the exponential of one of them, and
// the weights go through shared memory: 411 tokens of 16 / 4 heads 604 -> 72 us, bound by the issue of what is left.
#define PR_ROWS 8

template <int N, int MASK> __device__ __forceinline__ void pr_exchange(float *x, int lane) {
    const bool up = (lane & MASK) != 0;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
        const float keep = up ? x[i + N / 2] : x[i], give = up ? x[i] : x[i + N / 2];
        x[i] = keep + __shfl_xor_sync(0xffffffffu, give, MASK);
    }
}

// C: channels of a lane; chunk: heads of a kv head's group that a block takes, tokens: tokens of its rows
template <int C>
__global__ void __launch_bounds__(PA_WARPS * 32)
attention_plain_rows_kernel(const float *__restrict__ q, const float *__restrict__ k_cache, const float *__restrict__ v_cache,
                            const int *__restrict__ positions, const int *__restrict__ seq_of_token, const int *__restrict__ block_table,
                            int table_stride, int page_size, float *__restrict__ out, int T, int nq, int nkv, int hd, int vd, int v_ld,
                            const float *__restrict__ gate, float scale, int chunk, int tokens) {
    __shared__ float sm_m[PA_WARPS][PR_ROWS], sm_l[PA_WARPS][PR_ROWS], sm_acc[PA_WARPS][PR_ROWS][C * 32];
    __shared__ __align__(16) float sm_p[PA_WARPS][PR_ROWS][4], sm_c[PA_WARPS][PR_ROWS];
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = nq / nkv, chunks = (G + chunk - 1) / chunk;
    const int kvh = blockIdx.y / chunks, h0 = kvh * G + (blockIdx.y % chunks) * chunk;
    const int heads = min(chunk, (kvh + 1) * G - h0);
    const int tile = (int)gridDim.x - 1 - (int)blockIdx.x;                  // late tokens see the most keys: they go first
    const int t_end = min(T, (tile + 1) * tokens);
    for (int ta = tile * tokens; ta < t_end;) {
        // the tile's tokens of one request
        const int seq = seq_of_token[ta];
        int tb = ta + 1;
        while (tb < t_end && seq_of_token[tb] == seq) ++tb;
        const int rows = (tb - ta) * heads;
        const int *table = block_table + (size_t)seq * table_stride;
        float qv[PR_ROWS][C], acc[PR_ROWS][C];
#pragma unroll
        for (int r = 0; r < PR_ROWS; ++r)
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int i = lane + 32 * c;
                qv[r][c] = r < rows && i < hd ? q[((size_t)(ta + r / heads) * nq + h0 + r % heads) * hd + i] : 0.f;
                acc[r][c] = 0.f;
            }
        // this lane's row among the softmax lanes (row lane / 4, key lane % 4 of a group), and the keys it sees
        const int my_row = lane >> 2, my_key = lane & 3;
        const int my_keys = my_row < rows ? positions[ta + my_row / heads] + 1 : 0;
        int n_keys = my_keys;
#pragma unroll
        for (int o = 16; o >= 4; o >>= 1) n_keys = max(n_keys, __shfl_xor_sync(0xffffffffu, n_keys, o));
        float m = -INFINITY, l = 0.f;
        float kk[PA_KEYS][C], vv[PA_KEYS][C];
        auto load = [&](int base) {
#pragma unroll
            for (int u = 0; u < PA_KEYS; ++u) {
                const int s = base + u;
                const bool in = s < n_keys;
                const size_t row = in ? ((size_t)table[s / page_size] * nkv + kvh) * page_size + s % page_size : 0;
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    const int i = lane + 32 * c;
                    kk[u][c] = in && i < hd ? k_cache[row * hd + i] : 0.f;
                    vv[u][c] = in && i < vd ? v_cache[row * v_ld + i] : 0.f;
                }
            }
        };
        for (int base = warp * PA_KEYS; base < n_keys; base += PA_WARPS * PA_KEYS) {
            load(base);
            float x[4 * PR_ROWS];
#pragma unroll
            for (int r = 0; r < PR_ROWS; ++r)
#pragma unroll
                for (int u = 0; u < PA_KEYS; ++u) {
                    float dot = 0.f;
#pragma unroll
                    for (int c = 0; c < C; ++c) dot = fmaf(qv[r][c], kk[u][c], dot);
                    x[r * 4 + u] = dot;
                }
            pr_exchange<32, 16>(x, lane);
            pr_exchange<16, 8>(x, lane);
            pr_exchange<8, 4>(x, lane);
            pr_exchange<4, 2>(x, lane);
            pr_exchange<2, 1>(x, lane);
            const bool seen = base + my_key < my_keys;
            const uint32_t visible = __ballot_sync(0xffffffffu, seen);        // bit 4 r + u: row r sees key u of the group
            const float sc = seen ? x[0] * scale : -INFINITY;
            float mn = fmaxf(sc, __shfl_xor_sync(0xffffffffu, sc, 1));
            mn = fmaxf(m, fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 2)));
            const bool any = base < my_keys;              // a row that sees none of the group's keys stays as it is
            const float corr = any ? expf(m - mn) : 1.f;
            const float p = seen ? expf(sc - mn) : 0.f;
            if (any) m = mn;
            __syncwarp();
            sm_p[warp][my_row][my_key] = p;
            if (my_key == 0) sm_c[warp][my_row] = corr;
            __syncwarp();
            const float4 mine = *reinterpret_cast<const float4 *>(sm_p[warp][my_row]);
            l = __fmul_rn(l, corr);
            l = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(l, mine.x), mine.y), mine.z), mine.w);
#pragma unroll
            for (int r = 0; r < PR_ROWS; ++r) {
                const float4 pr = *reinterpret_cast<const float4 *>(sm_p[warp][r]);
                const float cr = sm_c[warp][r];
                const float w[4] = {pr.x, pr.y, pr.z, pr.w};
#pragma unroll
                for (int c = 0; c < C; ++c) acc[r][c] = __fmul_rn(acc[r][c], cr);
                // a key that the row does not see adds nothing, whatever its value (0 x inf would not be 0)
#pragma unroll
                for (int u = 0; u < PA_KEYS; ++u)
#pragma unroll
                    for (int c = 0; c < C; ++c) acc[r][c] = (visible >> (4 * r + u)) & 1u ? fmaf(w[u], vv[u][c], acc[r][c]) : acc[r][c];
            }
        }
        // merge the warps' states in warp order: a warp closes two rows
        if (my_key == 0) {
            sm_m[warp][my_row] = m;
            sm_l[warp][my_row] = l;
        }
#pragma unroll
        for (int r = 0; r < PR_ROWS; ++r)
#pragma unroll
            for (int c = 0; c < C; ++c) sm_acc[warp][r][lane + 32 * c] = acc[r][c];
        __syncthreads();
#pragma unroll
        for (int e = 0; e < PR_ROWS / PA_WARPS; ++e) {
            const int r = warp * (PR_ROWS / PA_WARPS) + e;
            if (r >= rows) continue;
            float M = -INFINITY, L = 0.f, o[C];
#pragma unroll
            for (int w = 0; w < PA_WARPS; ++w) M = fmaxf(M, sm_m[w][r]);
#pragma unroll
            for (int c = 0; c < C; ++c) o[c] = 0.f;
#pragma unroll
            for (int w = 0; w < PA_WARPS; ++w) {
                if (sm_m[w][r] == -INFINITY) continue;              // a warp that saw no key
                const float f = expf(sm_m[w][r] - M);
                L = fmaf(sm_l[w][r], f, L);
#pragma unroll
                for (int c = 0; c < C; ++c) o[c] = fmaf(sm_acc[w][r][lane + 32 * c], f, o[c]);
            }
            const size_t at = (size_t)(ta + r / heads) * nq + h0 + r % heads;
            float inv = 1.0f / L;
            if (gate) inv *= gate[at];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const int i = lane + 32 * c;
                if (i < vd) out[at * vd + i] = o[c] * inv;
            }
        }
        ta = tb;
        if (ta < t_end) __syncthreads();
    }
}

KESTREL_API int kestrel_attention_plain_scored(const void *q, const void *k_cache, const void *v_cache,
                                               const int *positions, const int *seq_of_token,
                                               const int *block_table, int table_stride, int page_size,
                                               void *out, int dtype, int T, int nq, int nkv, int hd, int vd, int window,
                                               int keep_first, const float *gate, float scale, float softcap, const float *r1,
                                               const float *r2, const float *head_bias, int weighting, const float *sink,
                                               cudaStream_t stream) {
    return kestrel_attention_plain_biased(q, k_cache, v_cache, positions, seq_of_token, block_table, table_stride, page_size, out, dtype, T, nq, nkv,
                                          hd, vd, window, keep_first, gate, scale, softcap, r1, r2, head_bias, weighting, sink, nullptr, nullptr, 0, 0,
                                          stream);
}

KESTREL_API int kestrel_attention_plain_biased(const void *q, const void *k_cache, const void *v_cache,
                                               const int *positions, const int *seq_of_token,
                                               const int *block_table, int table_stride, int page_size,
                                               void *out, int dtype, int T, int nq, int nkv, int hd, int vd, int window,
                                               int keep_first, const float *gate, float scale, float softcap, const float *r1,
                                               const float *r2, const float *head_bias, int weighting, const float *sink,
                                               const float *rel, const int *rel_bucket, int rel_far, int v_ld, cudaStream_t stream) {
    return kestrel_attention_plain_to(q, k_cache, v_cache, positions, seq_of_token, block_table, table_stride, page_size, out, dtype, 0, T, nq, nkv,
                                      hd, vd, window, keep_first, gate, scale, softcap, r1, r2, head_bias, weighting, sink, rel, rel_bucket, rel_far,
                                      v_ld, stream);
}

// the same with a learned number per head and bucket of distances added to the scores: rel [buckets, nq], the bucket of
// a distance from rel_bucket [rel_far + 1] (distances beyond rel_far share its bucket); `v_ld` > 0: the V plane's rows hold v_ld
// numbers of which the first vd are the value (a V plane that is the K plane of longer rows); `out_f32`: the output is float32 whatever the storage type (heads
// that are combined further before they are rounded)
KESTREL_API int kestrel_attention_plain_to(const void *q, const void *k_cache, const void *v_cache,
                                               const int *positions, const int *seq_of_token,
                                               const int *block_table, int table_stride, int page_size,
                                               void *out, int dtype, int out_f32, int T, int nq, int nkv, int hd, int vd, int window,
                                               int keep_first, const float *gate, float scale, float softcap, const float *r1,
                                               const float *r2, const float *head_bias, int weighting, const float *sink,
                                               const float *rel, const int *rel_bucket, int rel_far, int v_ld, cudaStream_t stream) {
    if (T == 0) return 0;
    KESTREL_REQUIRE(v_ld == 0 || v_ld >= vd, "attention_plain: value rows of %d numbers for values of %d", v_ld, vd);
    KESTREL_REQUIRE(weighting >= 0 && weighting <= 2 && softcap >= 0.f && (r1 == nullptr) == (r2 == nullptr), "attention_plain: bad score options");
    KESTREL_REQUIRE(!rel || (rel_bucket && rel_far >= 0), "attention_plain: a distance table without its buckets");
    const ScoreOpts opts = {softcap, r1, r2, head_bias, weighting, sink, rel, rel_bucket, rel_far, nq};
    KESTREL_REQUIRE(T > 0 && nq > 0 && nkv > 0 && hd > 0 && vd > 0 && keep_first >= 0, "attention_plain: bad sizes");
    KESTREL_REQUIRE(hd <= 32 * PA_MAX_PER_LANE && vd <= 32 * PA_MAX_PER_LANE, "attention_plain: head size %d / %d exceeds %d", hd, vd, 32 * PA_MAX_PER_LANE);
    KESTREL_REQUIRE(nq <= 65535, "attention_plain: %d query heads exceed the grid", nq);
    dim3 grid(T, nq);
    // Whether a layer takes the kernel of eight rows depends on the layer alone, not on the step: a row has the same bits in every step.
    if (dtype == KESTREL_F32 && window == 0 && softcap == 0.f && !r1 && !rel && weighting == KESTREL_WEIGH_SOFTMAX && hd <= 128 && vd <= 128 && nq % nkv == 0) {
        const int G = nq / nkv, chunk = G < PR_ROWS ? G : PR_ROWS, chunks = (G + chunk - 1) / chunk;
        // several tokens a block where there are blocks enough, tokens of one request mostly then
        int tokens = PR_ROWS / chunk;
        while (tokens > 1 && (long long)((T + tokens - 1) / tokens) * nkv * chunks < 2 * kestrel_sms()) --tokens;
        const dim3 rows_grid((T + tokens - 1) / tokens, nkv * chunks);
        KESTREL_REQUIRE(rows_grid.y <= 65535, "attention_plain: %d query heads exceed the grid", nq);
        if (hd <= 64 && vd <= 64)
            kestrel_launch(attention_plain_rows_kernel<2>, rows_grid, dim3(PA_WARPS * 32), 0, stream, (const float *)q, (const float *)k_cache, (const float *)v_cache, positions,
                           seq_of_token, block_table, table_stride, page_size, (float *)out, T, nq, nkv, hd, vd, v_ld > 0 ? v_ld : vd, gate, scale, chunk, tokens);
        else
            kestrel_launch(attention_plain_rows_kernel<4>, rows_grid, dim3(PA_WARPS * 32), 0, stream, (const float *)q, (const float *)k_cache, (const float *)v_cache, positions,
                           seq_of_token, block_table, table_stride, page_size, (float *)out, T, nq, nkv, hd, vd, v_ld > 0 ? v_ld : vd, gate, scale, chunk, tokens);
        return kestrel_check_launch("attention_plain");
    }
    if (dtype == KESTREL_F32)
        kestrel_launch(attention_plain_kernel<float, float>, dim3(grid), dim3(PA_WARPS * 32), 0, stream, (const float *)q, (const float *)k_cache, (const float *)v_cache, positions, seq_of_token,
            block_table, table_stride, page_size, (float *)out, nq, nkv, hd, vd, v_ld > 0 ? v_ld : vd, window, keep_first, gate, scale, opts);
    else if (dtype == KESTREL_BF16 && out_f32)
        kestrel_launch(attention_plain_kernel<__nv_bfloat16, float>, dim3(grid), dim3(PA_WARPS * 32), 0, stream, (const __nv_bfloat16 *)q, (const __nv_bfloat16 *)k_cache, (const __nv_bfloat16 *)v_cache, positions,
            seq_of_token, block_table, table_stride, page_size, (float *)out, nq, nkv, hd, vd, v_ld > 0 ? v_ld : vd, window, keep_first, gate, scale, opts);
    else if (dtype == KESTREL_BF16)
        kestrel_launch(attention_plain_kernel<__nv_bfloat16, __nv_bfloat16>, dim3(grid), dim3(PA_WARPS * 32), 0, stream, (const __nv_bfloat16 *)q, (const __nv_bfloat16 *)k_cache, (const __nv_bfloat16 *)v_cache, positions,
            seq_of_token, block_table, table_stride, page_size, (__nv_bfloat16 *)out, nq, nkv, hd, vd, v_ld > 0 ? v_ld : vd, window, keep_first, gate, scale, opts);
    else
        return kestrel_fail(-2, "attention_plain: unknown dtype %d", dtype);
    return kestrel_check_launch("attention_plain");
}

KESTREL_API int kestrel_attention_plain_ex(const void *q, const void *k_cache, const void *v_cache,
                                           const int *positions, const int *seq_of_token,
                                           const int *block_table, int table_stride, int page_size,
                                           void *out, int dtype, int T, int nq, int nkv, int hd, int vd, int window,
                                           int keep_first, const float *gate, float scale, cudaStream_t stream) {
    return kestrel_attention_plain_scored(q, k_cache, v_cache, positions, seq_of_token, block_table, table_stride, page_size, out, dtype, T,
                                          nq, nkv, hd, vd, window, keep_first, gate, scale, 0.f, nullptr, nullptr, nullptr, KESTREL_WEIGH_SOFTMAX,
                                          nullptr, stream);
}

KESTREL_API int kestrel_attention_plain(const void *q, const void *k_cache, const void *v_cache,
                                        const int *positions, const int *seq_of_token,
                                        const int *block_table, int table_stride, int page_size,
                                        void *out, int dtype, int T, int nq, int nkv, int hd, int window,
                                        float scale, cudaStream_t stream) {
    return kestrel_attention_plain_ex(q, k_cache, v_cache, positions, seq_of_token, block_table, table_stride, page_size, out, dtype, T,
                                      nq, nkv, hd, hd, window, 0, nullptr, scale, stream);
}
