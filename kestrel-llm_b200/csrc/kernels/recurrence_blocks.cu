// The sequential recurrences of linear_recurrence.cu and delta_rule.cu for portions of many tokens, in blocks of 16: the same sums in
// another order, the products and the sums of pairs in float64, what lies between them in float32.
//
// A token's step, S <- diag(w_t) S + a_t (b_t^T S) + k_t v_t^T, is a chain of two reductions over the key channels, some 600 cycles
// however many threads share it.  Over a block of 16 tokens the state S_0 at its start is all that has to be read in order:
// with P(s, t) the product of the decays of tokens s + 1 .. t (per channel, at most 1, so nothing overflows whatever the decays),
//
//     h_t = b_t^T S_(t-1) = (b_t P(0, t - 1))^T S_0 + sum_(s<t) [b_t P(s, t - 1) a_s] h_s + [b_t P(s, t - 1) k_s] v_s
//     o_t = r_t^T S_t     = (r_t P(0, t))^T S_0     + sum_(s<=t) [r_t P(s, t) a_s] h_s    + [r_t P(s, t) k_s] v_s
//     S_16                = P(0, 16) S_0            + sum_s (P(s, 16) a_s) h_s            + (P(s, 16) k_s) v_s
//
// The brackets are numbers per pair of tokens and head.  `blocks_prepare` makes them for all blocks at once, with the decayed vectors, and
// solves the triangular system, so that all that depends on S_0 is one product with rows made beforehand (X = (I - A)^-1):
//
//     h = F1^T S_0 + M1 v,   F1 = X b,        M1 = X K          S_16 = P(0, 16) S_0 + (a to the end)^T h + (k to the end)^T v
//     o = F2^T S_0 + M2 v,   F2 = r + Qa F1,  M2 = Qa M1 + Qk
//
// `blocks_scan` walks a request's blocks: a CTA takes 16 value columns of a head, transposed, its warps a share of the channels each, S^T in the
// accumulators of m16n8k8 products: the accumulators are the next product's operand A as they stand (the sum over channels may run in any
// order, so the unit's k index takes the channels in the order in which the accumulators hold them).  Per block: S^T times F1 and F2, to which a
// warp adds a share of M1 v and M2 v; one exchange of the warps' sums through shared memory; the writes.  GATE's writes need no sum: a block
// has one barrier, off the state's path; the others have two.  A prepared block (29 KB for DELTA at 128 channels) comes by two bulk copies into a
// ring, what meets the state and what is written to it, the first free again as soon as the products are done; values by cp.async three blocks ahead.
//
// The products are the float64 ones of the tensor cores; a portion's state and what the warps exchange are float64 from its first block to its
// last.  Distance of read-outs and states from a float64 evaluation, at memories of 5 to 300 tokens: 0.44 to 0.9 of the sequential scan's.
// Operands as two terms of 11 bits on the tf32 products were further off than the scan (those accumulators cut off instead of rounding);
// float32 sums exchanged by the warps took read-outs at a memory of 5 from 0.44 to 0.6, states from 0.64 to 0.93.
//
// What bounds it.  An SM makes 64 multiply-adds of float64 a cycle, 64 cycles a product and quarter SM: 640 (GATE, 64 channels), 1,700 (DELTA) and
// 2,200 (REMOVAL) cycles a block and CTA.  Conversions from float32 (8 cycles a warp) run beside them.  A lone CTA takes 1,600 (GATE) to 3,600
// cycles a block, the chain of products, exchange and writes; two share an SM at 58 to 65 % of the products' rate.  GATE gains from eight warps
// (118 us against 142 for the launches below), the others lose more by eight sums to add than they gain (DELTA 216 against 210).  With plain float32 multiply-adds the
// blocks are bound by the shared-memory reads of operands that 16 columns cannot reuse: 322 us for DELTA's scan.
// The preparation reads and converts a token's vectors once for four pairs, and exchanges each sum over the lanes (a third of its instructions).
//
// What is not finite stays so, and reaches the tokens and channels that it reaches in the scan: where a value or a prepared row is not
// finite, its sums are made again from the tokens that count (an infinity may come out as NaN, where terms of both signs meet).
//
// Three forms: GATE (no correction), REMOVAL (a, b given) and DELTA (a gated delta rule: with u = beta (v - (diag(w) S)^T k),
// S <- diag(w) S + k u^T, so that b = w k, the writes u take the place of v, F1 = - X b with X = (I + beta K)^-1 beta, F2 = r + Qk F1,
// M1 = X and M2 = Qk X).
//
// Measured, 16 heads, prepared + scanned in us, beside the blocks that exchanged h and o in turn (four pairs' sums by a warp each) and the
// sequential scan: DELTA (128 channels, requests of 592 and 1,185 tokens) 202 (244; 517); GATE (64 channels, 2,048 tokens) 113 (165; 287);
// REMOVAL (128 channels, 700 tokens in three requests, 350 the longest) 100 (124; 213).
#include "common.cuh"
#include "tcgen05.cuh"
#include <initializer_list>
#include <math.h>

#define RB_B 16                 // tokens of a block
#define RB_LD 24                // floats of a row of a 16 x 16 matrix: pairs of four rows fall on all 32 banks
#define RB_MAT (RB_B * RB_LD)
#define RB_COLS 16              // value columns of a CTA
#define RB_VLD 20               // floats of a token's row of them
#define RB_STAGES 8             // most stages of the ring of prepared blocks

enum { RB_GATE = 0, RB_REMOVAL = 1, RB_DELTA = 2 };

__device__ int g_rb_error = 0;


// A prepared block of a head: what meets the state, [rows that give h | rows that give o | what values add to h | to o], then what is
// written to it, [k to the block's end | a to the block's end | P(0, 16)]; each comes by one bulk copy.
template <int D, int FORM> struct RbLayout {
    static constexpr int ROW_LD = D + 8, END_LD = D + 4;        // rows read as pairs along the channels, and as pairs of rows
    static constexpr bool H = FORM != RB_GATE;
    static constexpr int F1 = 0;
    static constexpr int F2 = H ? RB_B * ROW_LD : 0;
    static constexpr int M1 = F2 + RB_B * ROW_LD;
    static constexpr int M2 = H ? M1 + RB_MAT : M1;
    static constexpr int KW = M2 + RB_MAT;
    static constexpr int AW = KW + RB_B * END_LD;
    static constexpr int DT = FORM == RB_REMOVAL ? AW + RB_B * END_LD : AW;
    static constexpr int FLOATS = DT + D;
    static constexpr int MATS = FORM == RB_GATE ? 1 : FORM == RB_DELTA ? 3 : 6;     // matrices of the preparation
};

// What a CTA of the scan holds beside its ring (a GATE block waits for none of its sums: two buffers of them in turn)
template <int D, int FORM> struct RbScan {
    static constexpr int WARPS = FORM == RB_GATE && D >= 64 ? 8 : 4;   // a share of the channels each
    static constexpr int NT = FORM == RB_GATE ? 2 : 4;                  // tiles of eight rows that meet the state
    static constexpr int LD = RB_B + 8;                                 // (pairs of doubles of two neighbouring columns on all 32 banks)
    unsigned long long bars[RB_STAGES][2];
    double red_h[FORM == RB_GATE ? 1 : WARPS][FORM == RB_GATE ? 1 : RB_COLS][LD];             // the warps' sums by column and token
    double red_o[FORM == RB_GATE ? 2 : 1][WARPS][RB_COLS][LD];
    double corr[FORM == RB_GATE ? 1 : RB_COLS][LD];                     // h (DELTA: the writes), summed
    float vals[4][RB_B][RB_VLD];                // values [token][column] of four blocks in flight: loaded for the next block alone they set the pace (2,400 cycles a block)
};

struct RbParams {
    const float *r, *w, *k, *a, *b, *beta;      // r, k [T, G d] (DELTA) or [T, H d]; w, a, b [T, H d]; beta [T, H]
    const float *v;                             // [T, ldv], head h's columns at h * dv
    size_t ldv;
    float *state;
    size_t state_stride;
    const int *cu_seqlens, *slots;
    float *out;                                 // [T, H dv]
    float *blocks;                              // scratch: block (cu_seqlens[seq] / 16 + seq + i) of a request, head by head
    int H, G, d, dv;
};

// Where the vectors come from when `blocks_prepare` makes them itself, as the gates kernels do, instead of reading what those left:
// GATE and REMOVAL from the columns of a product x (r or q, k, v, f or rate logits), DELTA from x = the convolved q | k | v and, for beta,
// the product y; z: the decay's product (REMOVAL, DELTA).  Sums over slices in ascending order; all rows and columns in whole vectors of four.
struct RbSource {
    const float *x, *y, *z;
    int Sx, Sy, Sz, ldx, ldy, ldz, col_r, col_k, col_v, col_a;      // col_a: rate logits (REMOVAL), f (GATE), beta logits in y (DELTA)
    size_t x_stride, y_stride, z_stride;
    const float *bias, *bias2;                  // GATE: f_bias, lower; REMOVAL: a_bias, w_bias; DELTA: dt_bias, A_log
    float rate;
    float *v_out;                               // [T, H dv]: the values' slices summed, or null where they are one slice and read from there
};
__device__ __forceinline__ float4 rb_sum4(const float *p, int S, size_t stride) {
    float4 v = *reinterpret_cast<const float4 *>(p);
    for (int s = 1; s < S; ++s) {
        const float4 x = *reinterpret_cast<const float4 *>(p + (size_t)s * stride);
        v.x += x.x, v.y += x.y, v.z += x.z, v.w += x.w;
    }
    return v;
}
__device__ __forceinline__ float rb_sigmoid(float z) { return 1.0f / (1.0f + expf(-z)); }

// One exchange of a sum of N values over the lanes: a lane keeps the half of the values that its bit of MASK names and adds the other
// lane's share of them.  Five of them, from 32 values, leave lane l with the sum of value l.
template <int N, int MASK> __device__ __forceinline__ void rb_exchange(double *x, int lane) {
    const bool up = (lane & MASK) != 0;
#pragma unroll
    for (int i = 0; i < N / 2; ++i) {
        const double keep = up ? x[i + N / 2] : x[i], give = up ? x[i] : x[i + N / 2];
        x[i] = keep + __shfl_xor_sync(0xffffffffu, give, MASK);
    }
}

// c += a * b, one step of 8 along the sum, m16n8k8 in float64
__device__ __forceinline__ void rb_mma(double *c, const double *a, double b0, double b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
                 : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}
// Operand A from a row-major pair of numbers per row: (row l / 4: x0 at 2 (l % 4), x1 behind it; row l / 4 + 8: x2, x3).  The unit's k index
// l % 4 is taken for the even, l % 4 + 4 for the odd of the two; operand B pairs its numbers the same way.
struct RbA { double x[4]; };
__device__ __forceinline__ RbA rb_a(double x0, double x1, double x2, double x3) { return {{x0, x2, x1, x3}}; }

__device__ __forceinline__ void rb_put2(double *to, double x, double y) { *reinterpret_cast<double2 *>(to) = make_double2(x, y); }
template <int N> struct RbCount { static constexpr int value = N; };
// V neighbouring numbers in one load
template <int V> __device__ __forceinline__ void rb_load(float *x, const float *p) {
    if constexpr (V == 4) {
        const float4 v = *reinterpret_cast<const float4 *>(p);
        x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
    } else if constexpr (V == 2) {
        const float2 v = *reinterpret_cast<const float2 *>(p);
        x[0] = v.x, x[1] = v.y;
    } else {
        x[0] = p[0];
    }
}

template <int D, int FORM, bool MADE>
__global__ void __launch_bounds__(128)
blocks_prepare_kernel(const RbParams p, const RbSource src) {
    using L = RbLayout<D, FORM>;
    constexpr int V = D / 32;                   // channels of a lane
    pdl_wait();
    const int blk = blockIdx.x, h = blockIdx.y, seq = blockIdx.z;
    const int t0 = p.cu_seqlens[seq] + blk * RB_B, t1 = p.cu_seqlens[seq + 1];
    if (t0 >= t1) return;
    extern __shared__ __align__(16) float rb_sm[];
    // [w | r | k | b | a] of the block's tokens, zero (w: one) beyond the head's channels and the request's tokens
    constexpr int LD = L::END_LD;               // of a token's row
    float *sw = rb_sm, *sr = sw + RB_B * LD, *sk = sr + RB_B * LD, *sb = sk + RB_B * LD, *sa = sb + (FORM == RB_GATE ? 0 : RB_B * LD);
    // per pair of tokens, rows of RB_LD: GATE Qk; DELTA K, Qk, X; REMOVAL K, Qk, A, Qa, X, X K
    constexpr int MATS = L::MATS;
    double *mat = reinterpret_cast<double *>(sa + (FORM == RB_REMOVAL ? RB_B * LD : 0));
    double *mK = mat, *mQk = mat + (MATS > 1 ? RB_MAT : 0), *mA = mat + 2 * RB_MAT, *mQa = mat + 3 * RB_MAT, *mX = mat + (MATS - 2 + (FORM == RB_DELTA)) * RB_MAT,
           *mY = mat + 5 * RB_MAT;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kh = FORM == RB_DELTA ? h / (p.H / p.G) : h, KH = FORM == RB_DELTA ? p.G : p.H;
    __shared__ float sbeta[RB_B], sinv[2][RB_B];
    if (FORM == RB_DELTA && !MADE && tid < RB_B) sbeta[tid] = t0 + tid < t1 ? p.beta[(size_t)(t0 + tid) * p.H + h] : 0.f;
    const bool vec = MADE || (p.d % 4 == 0 && (((uintptr_t)p.r | (uintptr_t)p.w | (uintptr_t)p.k | (uintptr_t)p.a | (uintptr_t)p.b) & 15) == 0);
    if (MADE) {
        constexpr int N = RB_B * D / 512;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        float4 rs[N], ks[N], as[N], zs[N];       // all of a thread's loads in flight together, then the gates
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int idx = (tid + 128 * i) * 4, t = idx / D, c = idx % D;
            rs[i] = ks[i] = as[i] = zs[i] = zero;
            if (t0 + t < t1 && c < p.d) {
                const float *row = src.x + (size_t)(t0 + t) * src.ldx;
                rs[i] = rb_sum4(row + src.col_r + kh * p.d + c, src.Sx, src.x_stride);
                if (FORM != RB_GATE) ks[i] = rb_sum4(row + src.col_k + kh * p.d + c, src.Sx, src.x_stride);
                if (FORM != RB_DELTA) as[i] = rb_sum4(row + src.col_a + h * p.d + c, src.Sx, src.x_stride);
                if (FORM != RB_GATE) zs[i] = rb_sum4(src.z + (size_t)(t0 + t) * src.ldz + h * p.d + c, src.Sz, src.z_stride);
            }
        }
        const float A = FORM == RB_DELTA ? expf(src.bias2[h]) : 0.f;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int idx = (tid + 128 * i) * 4, t = idx / D, c = idx % D;
            float4 r4 = rs[i], k4 = ks[i], a4 = as[i], w4 = make_float4(1.f, 1.f, 1.f, 1.f);
            if (t0 + t < t1 && c < p.d) {
                float *r = &r4.x, *k = &k4.x, *a = &a4.x, *w = &w4.x;
                const float *z = &zs[i].x;
                const int hc = h * p.d + c;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    if (FORM == RB_GATE) {
                        const float lo = src.bias2 ? src.bias2[hc + e] : 0.f;
                        w[e] = lo + (1.0f - lo) * rb_sigmoid(a[e] + (src.bias ? src.bias[hc + e] : 0.f));
                        r[e] *= rb_sigmoid(r[e]);
                        k[e] = 1.0f - w[e];
                    } else if (FORM == RB_REMOVAL) {
                        a[e] = rb_sigmoid(a[e] + (src.bias ? src.bias[hc + e] : 0.f));
                        w[e] = expf(-src.rate * rb_sigmoid(z[e] + (src.bias2 ? src.bias2[hc + e] : 0.f)));
                    } else {
                        const float x = z[e] + src.bias[hc + e];
                        w[e] = expf(-A * (x > 20.f ? x : log1pf(expf(x))));
                    }
                }
            }
            const int at = t * LD + c;
            *reinterpret_cast<float4 *>(sw + at) = w4;
            *reinterpret_cast<float4 *>(sr + at) = r4;
            *reinterpret_cast<float4 *>(sk + at) = k4;
            if (FORM == RB_REMOVAL) *reinterpret_cast<float4 *>(sa + at) = a4;
        }
        if (FORM == RB_DELTA && tid < RB_B) {
            float z = 0.f;
            if (t0 + tid < t1) z = sum_slices(src.y, src.Sy, src.y_stride, (size_t)(t0 + tid) * src.ldy + src.col_a + h);
            sbeta[tid] = t0 + tid < t1 ? rb_sigmoid(z) : 0.f;
        }
        if (FORM != RB_DELTA && src.v_out)
            for (int idx = tid; idx < RB_B * p.dv; idx += 128) {
                const int t = t0 + idx / p.dv, c = h * p.dv + idx % p.dv;
                if (t < t1) src.v_out[(size_t)t * p.H * p.dv + c] = sum_slices(src.x, src.Sx, src.x_stride, (size_t)t * src.ldx + src.col_v + c);
            }
        if (FORM != RB_GATE) {                  // unit keys (DELTA: and queries): a warp a token's head, four tokens a warp
            __syncthreads();
#pragma unroll
            for (int i = 0; i < RB_B / 4; ++i) {
                const int t = warp * (RB_B / 4) + i;
                float sk2 = 0.f, sr2 = 0.f;
#pragma unroll
                for (int j = 0; j < V; ++j) {
                    const float k = sk[t * LD + lane * V + j], r = sr[t * LD + lane * V + j];
                    sk2 = fmaf(k, k, sk2);
                    sr2 = fmaf(r, r, sr2);
                }
                sk2 = warp_sum(sk2);
                if (FORM == RB_DELTA) sr2 = warp_sum(sr2);
                if (lane == 0) {
                    sinv[0][t] = 1.0f / sqrtf(sk2 + 1e-6f);
                    sinv[1][t] = (1.0f / sqrtf(sr2 + 1e-6f)) * (1.0f / sqrtf((float)p.d));
                }
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < RB_B * D / 128; ++i) {
                const int t = (tid + 128 * i) / D, at = t * LD + (tid + 128 * i) % D;
                const float u = sk[at] * sinv[0][t];
                if (FORM == RB_REMOVAL) {
                    sb[at] = u;
                    sa[at] = -(sa[at] * u);
                } else {
                    sk[at] = u;
                    sr[at] *= sinv[1][t];
                    sb[at] = sw[at] * u;
                }
            }
        }
    } else
    if (vec) {                                  // all of a thread's loads in flight together
        constexpr int N = RB_B * D / 512;
        float4 w4[N], r4[N], k4[N], a4[FORM == RB_REMOVAL ? N : 1], b4[FORM == RB_REMOVAL ? N : 1];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int idx = (tid + 128 * i) * 4, t = idx / D, c = idx % D;
            const bool in = t0 + t < t1 && c < p.d;
            const size_t oh = in ? ((size_t)(t0 + t) * p.H + h) * p.d + c : 0, ok = in ? ((size_t)(t0 + t) * KH + kh) * p.d + c : 0;
            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
            w4[i] = in ? *reinterpret_cast<const float4 *>(p.w + oh) : make_float4(1.f, 1.f, 1.f, 1.f);
            r4[i] = in ? *reinterpret_cast<const float4 *>(p.r + ok) : zero;
            k4[i] = in ? *reinterpret_cast<const float4 *>(p.k + ok) : zero;
            if (FORM == RB_REMOVAL) {
                a4[i] = in ? *reinterpret_cast<const float4 *>(p.a + oh) : zero;
                b4[i] = in ? *reinterpret_cast<const float4 *>(p.b + oh) : zero;
            }
        }
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int at = (tid + 128 * i) * 4 / D * LD + (tid + 128 * i) * 4 % D;
            *reinterpret_cast<float4 *>(sw + at) = w4[i];
            *reinterpret_cast<float4 *>(sr + at) = r4[i];
            *reinterpret_cast<float4 *>(sk + at) = k4[i];
            if (FORM == RB_REMOVAL) {
                *reinterpret_cast<float4 *>(sb + at) = b4[i];
                *reinterpret_cast<float4 *>(sa + at) = a4[i];
            }
            if (FORM == RB_DELTA)
                *reinterpret_cast<float4 *>(sb + at) = make_float4(w4[i].x * k4[i].x, w4[i].y * k4[i].y, w4[i].z * k4[i].z, w4[i].w * k4[i].w);
        }
    } else {
#pragma unroll 4
        for (int idx = tid; idx < RB_B * D; idx += 128) {
            const int t = idx / D, c = idx % D;
            const bool in = t0 + t < t1 && c < p.d;
            const size_t oh = ((size_t)(t0 + t) * p.H + h) * p.d + c, ok = ((size_t)(t0 + t) * KH + kh) * p.d + c;
            const float w = in ? p.w[oh] : 1.f, k = in ? p.k[ok] : 0.f;
            const int at = t * LD + c;
            sw[at] = w;
            sr[at] = in ? p.r[ok] : 0.f;
            sk[at] = k;
            if (FORM == RB_REMOVAL) {
                sb[at] = in ? p.b[oh] : 0.f;
                sa[at] = in ? p.a[oh] : 0.f;
            }
            if (FORM == RB_DELTA) sb[at] = w * k;
        }
    }
    for (int idx = tid; idx < MATS * RB_MAT; idx += 128) mat[idx] = 0.0;
    __syncthreads();

    float *blkp = p.blocks + ((size_t)(p.cu_seqlens[seq] / RB_B + seq + blk) * p.H + h) * L::FLOATS;
    // The pairs: a warp takes four neighbouring tokens s and walks t = s .. 15, so that a token's b, r and w are read and converted once
    // for four pairs (16 a cycle and SM, a quarter of the multiply-adds' rate); blocks give the longest walk to another quarter of the SM each.
    // The sums of TG tokens t go through the lanes together.
    constexpr int SUMS = FORM == RB_GATE ? 1 : FORM == RB_DELTA ? 2 : 4, TG = FORM == RB_REMOVAL ? 2 : 4, VALUES = 4 * TG * SUMS;
    {
        const int s0 = ((warp + blk + h) & 3) * 4;
        double xk[4][V], xa[FORM == RB_REMOVAL ? 4 : 1][V];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < V; ++j) {       // neighbouring channels: they come in one load
                xk[i][j] = sk[(s0 + i) * LD + lane * V + j];
                if (FORM == RB_REMOVAL) xa[i][j] = sa[(s0 + i) * LD + lane * V + j];
            }
        // tokens t .. t + TG - 1, OFF or (4) more behind s0
        auto walk = [&](auto off, int t0_) {
            constexpr int OFF = decltype(off)::value;
            double x[VALUES];                   // [t][s][sum]
#pragma unroll
            for (int u = 0; u < TG; ++u) {
                const int o = (t0_ + u) * LD + lane * V;
                float b[V], w[V], r[V];
                if (FORM != RB_GATE) rb_load<V>(b, sb + o);
                rb_load<V>(w, sw + o);
                rb_load<V>(r, sr + o);
                double f[4][SUMS];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int m = 0; m < SUMS; ++m) f[i][m] = 0.0;
#pragma unroll
                for (int j = 0; j < V; ++j) {
                    const double bb = FORM == RB_GATE ? 0.0 : (double)b[j], ww = w[j], rr = r[j];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (OFF + u > i) {
                            if (FORM != RB_GATE) f[i][0] = fma(bb, xk[i][j], f[i][0]);
                            if (FORM == RB_REMOVAL) f[i][2] = fma(bb, xa[i][j], f[i][2]);
                            xk[i][j] *= ww;
                            if (FORM == RB_REMOVAL) xa[i][j] *= ww;
                        }
                        if (OFF + u >= i) {
                            f[i][SUMS > 1 ? 1 : 0] = fma(rr, xk[i][j], f[i][SUMS > 1 ? 1 : 0]);
                            if (FORM == RB_REMOVAL) f[i][3] = fma(rr, xa[i][j], f[i][3]);
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int m = 0; m < SUMS; ++m) x[(u * 4 + i) * SUMS + m] = f[i][m];
            }
            // lane l ends with value l (GATE: l / 2)
            if constexpr (VALUES == 16) {
                rb_exchange<16, 16>(x, lane);
                rb_exchange<8, 8>(x, lane);
                rb_exchange<4, 4>(x, lane);
                rb_exchange<2, 2>(x, lane);
                x[0] += __shfl_xor_sync(0xffffffffu, x[0], 1);
                mQk[(t0_ + (lane >> 3)) * RB_LD + s0 + ((lane >> 1) & 3)] = x[0];
            } else {
                rb_exchange<32, 16>(x, lane);
                rb_exchange<16, 8>(x, lane);
                rb_exchange<8, 4>(x, lane);
                rb_exchange<4, 2>(x, lane);
                rb_exchange<2, 1>(x, lane);
                mat[(lane % SUMS) * RB_MAT + (t0_ + lane / (4 * SUMS)) * RB_LD + s0 + (lane / SUMS) % 4] = x[0];
            }
        };
        walk(RbCount<0>(), s0);
        if (TG == 2) walk(RbCount<2>(), s0 + 2);
#pragma unroll 1
        for (int t = s0 + 4; t < RB_B; t += TG) walk(RbCount<4>(), t);
    }
    __syncthreads();
    // vectors decayed from the block's start (here, where b and r were, for what follows; GATE: done) and to its end, a channel a thread
    for (int idx = tid; idx < 2 * D; idx += 128) {
        const int c = idx % D;
        float run = 1.f;
        if (idx < D) {
#pragma unroll
            for (int t = 0; t < RB_B; ++t) {
                const float w = sw[t * LD + c];
                if (FORM != RB_GATE) sb[t * LD + c] *= run;
                run *= w;
                if (FORM != RB_GATE) sr[t * LD + c] *= run;
                else blkp[L::F2 + t * L::ROW_LD + c] = sr[t * LD + c] * run;
            }
            blkp[L::DT + c] = run;
        } else {
#pragma unroll
            for (int t = RB_B - 1; t >= 0; --t) {
                blkp[L::KW + t * L::END_LD + c] = sk[t * LD + c] * run;
                if (FORM == RB_REMOVAL) blkp[L::AW + t * L::END_LD + c] = sa[t * LD + c] * run;
                run *= sw[t * LD + c];
            }
        }
    }
    if (FORM == RB_GATE) {
        pdl_launch_dependents();
        for (int idx = tid; idx < RB_B * RB_B; idx += 128) blkp[L::M2 + idx / RB_B * RB_LD + idx % RB_B] = (float)mQk[idx / RB_B * RB_LD + idx % RB_B];
        return;
    }
    // X, a column a thread, by substitution: REMOVAL (I - A)^-1; DELTA (I + beta A)^-1 beta with A in mK.  (Zero above the diagonal whatever A holds.)
    if (warp == ((blk + h) & 3) && lane < RB_B) {
        const double *A = FORM == RB_DELTA ? mK : mA;
        double x[RB_B];
#pragma unroll
        for (int t = 0; t < RB_B; ++t) x[t] = 0.0;
#pragma unroll
        for (int t = 0; t < RB_B; ++t) {
            const double one = t == lane ? 1.0 : 0.0, beta = FORM == RB_DELTA ? (double)sbeta[t] : 0.0;
            const double y = FORM == RB_DELTA ? beta * (one - x[t]) : one + x[t];      // x[t]: the sum over the tokens before
            mX[t * RB_LD + lane] = t >= lane ? y : 0.0;
#pragma unroll
            for (int s = t + 1; s < RB_B; ++s) x[s] = fma(A[s * RB_LD + t], y, x[s]);
        }
    }
    __syncthreads();
    // What values add: to h, and through h and directly to o.  (Sums over the tokens up to t alone: a later token's numbers may not be
    // finite, and 0 x inf would not be 0.)
    for (int idx = tid; idx < RB_B * RB_B; idx += 128) {
        const int t = idx / RB_B, j = idx % RB_B;
        double m = 0.0;
#pragma unroll
        for (int s = 0; s < RB_B; ++s)
            if (s <= t) m = FORM == RB_DELTA ? fma(mQk[t * RB_LD + s], mX[s * RB_LD + j], m) : fma(mX[t * RB_LD + s], mK[s * RB_LD + j], m);
        if (FORM == RB_DELTA) {
            blkp[L::M1 + t * RB_LD + j] = (float)mX[t * RB_LD + j];
            blkp[L::M2 + t * RB_LD + j] = (float)m;
        } else {
            blkp[L::M1 + t * RB_LD + j] = (float)m;
            mY[t * RB_LD + j] = m;
        }
    }
    pdl_launch_dependents();                    // (late: the scan's CTAs are then spread over SMs that are free, longest first)
    // What meets the state: F1 = X b (DELTA: - X b) gives h, F2 = r + Q F1 (Q = Qa; DELTA: Qk) gives o.  Transposed, 16 channels a tile of a
    // warp, so that F1's accumulators are the operand of the product with Q.
    const double *mQ = FORM == RB_DELTA ? mQk : mQa;
    const int lr = lane >> 2, lc = (lane & 3) * 2;
    for (int c0 = 16 * warp; c0 < D; c0 += 64) {
        double f1[2][4], f2[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                f1[n][e] = 0.0;
                f2[n][e] = sr[(n * 8 + lc + (e & 1)) * LD + c0 + lr + (e >> 1) * 8];
            }
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            const float *b0 = sb + (ks * 8 + lc) * LD + c0 + lr, *b1 = b0 + LD;
            const RbA a = rb_a(b0[0], b1[0], b0[8], b1[8]);
#pragma unroll
            for (int n = ks; n < 2; ++n) {
                const double2 x = *reinterpret_cast<const double2 *>(mX + (n * 8 + lr) * RB_LD + ks * 8 + lc);
                rb_mma(f1[n], a.x, x.x, x.y);
            }
        }
        if (FORM == RB_DELTA)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) f1[n][e] = -f1[n][e];
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            const RbA a = rb_a(f1[ks][0], f1[ks][1], f1[ks][2], f1[ks][3]);
#pragma unroll
            for (int n = ks; n < 2; ++n) {
                const double2 q = *reinterpret_cast<const double2 *>(mQ + (n * 8 + lr) * RB_LD + ks * 8 + lc);
                rb_mma(f2[n], a.x, q.x, q.y);
            }
        }
        bool number = true;
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) number = number && fabs(f1[n][e]) < INFINITY && fabs(f2[n][e]) < INFINITY;
        if (!__all_sync(0xffffffffu, number)) {     // from the tokens up to t alone, as above
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int t = n * 8 + lc + (e & 1), c = c0 + lr + (e >> 1) * 8;
                    double y = 0.0, z = sr[t * LD + c];
#pragma unroll 1
                    for (int s = 0; s <= t; ++s) {
                        y = 0.0;
#pragma unroll 1
                        for (int q = 0; q <= s; ++q) y = fma(mX[s * RB_LD + q], (double)sb[q * LD + c], y);
                        if (FORM == RB_DELTA) y = -y;
                        z = fma(mQ[t * RB_LD + s], y, z);
                    }
                    f1[n][e] = y;
                    f2[n][e] = z;
                }
        }
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int at = (n * 8 + lc + (e & 1)) * L::ROW_LD + c0 + lr + (e >> 1) * 8;
                blkp[L::F1 + at] = (float)f1[n][e];
                blkp[L::F2 + at] = (float)f2[n][e];
            }
    }
    if (FORM == RB_REMOVAL) {
        __syncthreads();
        for (int idx = tid; idx < RB_B * RB_B; idx += 128) {
            const int t = idx / RB_B, j = idx % RB_B;
            double m = mQk[t * RB_LD + j];
#pragma unroll
            for (int s = 0; s < RB_B; ++s)
                if (s <= t) m = fma(mQa[t * RB_LD + s], mY[s * RB_LD + j], m);
            blkp[L::M2 + t * RB_LD + j] = (float)m;
        }
    }
}

// The request whose portion is the k-th longest, of equal ones the first.  CTAs are placed in the order of their index, so the longest get
// SMs of their own and the shorter ones share: prepared + scanned in us, in the requests' order and by length, DELTA's 592 and 1,185
// tokens 218 and 202, REMOVAL's 117, 233 and 350 122 and 100.
__device__ __forceinline__ int rb_longest(const int *cu, int n, int k) {
    int found = 0;
    for (int i = threadIdx.x & 31; i < n; i += 32) {
        const int mine = cu[i + 1] - cu[i];
        int longer = 0;
        for (int j = 0; j < n; ++j) {
            const int other = cu[j + 1] - cu[j];
            longer += other > mine || (other == mine && j < i);
        }
        if (longer == k) found = i;
    }
    return __reduce_add_sync(0xffffffffu, found);
}

template <int D, int FORM>
__global__ void __launch_bounds__(32 * RbScan<D, FORM>::WARPS)
blocks_scan_kernel(const RbParams p, int stages, bool by_length) {
    using L = RbLayout<D, FORM>;
    constexpr int WARPS = RbScan<D, FORM>::WARPS;
    constexpr int NT = RbScan<D, FORM>::NT;
    constexpr int CT = D / 8 / WARPS;                            // tiles of eight channels of a warp
    constexpr int STAGE = L::FLOATS;
    constexpr bool EARLY = FORM == RB_GATE;                      // a block's writes need none of its sums: its last operands are free a block earlier
    pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char rb_dyn[];
    RbScan<D, FORM> &sm = *reinterpret_cast<RbScan<D, FORM> *>(rb_dyn);
    float *ring = reinterpret_cast<float *>(rb_dyn + (sizeof(sm) + 127) / 128 * 128);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int lr = lane >> 2, lc = (lane & 3) * 2;               // a fragment's row (and row + 8) and its pair of columns
    const int h = blockIdx.y, col0 = blockIdx.x * RB_COLS;
    const int ch0 = warp * (D / WARPS);
    const uint32_t bar0 = smem_u32(&sm.bars[0][0]);
    if (tid == 0) {
        for (int b = 0; b < 2 * stages; ++b) mbar_init(bar0 + 8 * b, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_wait();
    const int seq = by_length ? rb_longest(p.cu_seqlens, gridDim.z, blockIdx.z) : (int)blockIdx.z;
    const int t0 = p.cu_seqlens[seq], T = p.cu_seqlens[seq + 1] - t0;
    const int n_blocks = (T + RB_B - 1) / RB_B;
    const size_t src_step = (size_t)p.H * STAGE;
    const float *src = p.blocks + ((size_t)(t0 / RB_B + seq) * p.H + h) * STAGE;
    // one thread: of the block at `from`, what meets the state, or (part 1) what is written to it, into a stage; each has a barrier
    auto fetch = [&](int stage, const float *from, int part) {
        const uint32_t bar = bar0 + 16u * (uint32_t)stage + 8u * part;
        const int off = part ? L::KW : 0, bytes = (part ? STAGE - L::KW : L::KW) * 4;
        mbar_expect_tx(bar, bytes);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(smem_u32(ring + stage * STAGE + off)), "l"(from + off), "r"(bytes), "r"(bar)
                     : "memory");
    };
    if (tid == 0)
        for (int i = 0; i < min(stages, n_blocks); ++i) fetch(i, src + i * src_step, 0), fetch(i, src + i * src_step, 1);
    const float *ahead = src + stages * src_step;                // block i + stages
    float *Sg = p.state + (size_t)p.slots[seq] * p.state_stride + (size_t)h * p.d * p.dv;     // [d][dv]
    // S^T of the warp's channels: S[ct] = columns lr, lr + 8 of the CTA by channels lc, lc + 1 of the tile
    double S[CT][4];
#pragma unroll
    for (int ct = 0; ct < CT; ++ct)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int c = ch0 + ct * 8 + lc + (e & 1), j = col0 + lr + (e >> 1) * 8;
            S[ct][e] = (c < p.d && j < p.dv) ? Sg[(size_t)c * p.dv + j] : 0.f;
        }
    // a thread moves VN columns of a token's values; zeros beyond the request and the head
    constexpr int VN = 8 / WARPS;
    const int vt = tid / (RB_COLS / VN), vj = tid % (RB_COLS / VN) * VN;
    const uint32_t v_to = smem_u32(&sm.vals[0][vt][vj]);
    const float *v_from = p.v + (size_t)(t0 + vt) * p.ldv + (size_t)h * p.dv + col0 + vj;     // of block i + 3
    int v_left = T - vt;                                         // its tokens from this one on
    auto load_v = [&](int slot) {
#pragma unroll
        for (int e = 0; e < VN; ++e) {
            const bool in = v_left > 0 && col0 + vj + e < p.dv;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(v_to + (uint32_t)(slot * RB_B * RB_VLD + e) * 4), "l"(in ? v_from + e : p.v), "r"(in ? 4 : 0)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        v_from += RB_B * p.ldv;
        v_left -= RB_B;
    };
    load_v(0);
    load_v(1);
    load_v(2);
    asm volatile("cp.async.wait_group 2;" ::: "memory");
    __syncthreads();
    bool ok = true;
    int stage = 0, before = 0, left = T;                         // tokens from the block's first on
    uint32_t phase = 0;
    auto await = [&](int part) {
        if (ok && !mbar_wait(bar0 + 16u * (uint32_t)stage + 8u * part, phase)) { atomicExch(&g_rb_error, 1); ok = false; }
    };
    // the sums and read-outs of a quarter of a block: tokens 8 n + lc, + 1 of columns lr + 8 e
    const int qn = warp & 1, qe = (warp >> 1) & 1, out_j = col0 + lr + 8 * qe;
    float *out = p.out + ((size_t)(t0 + qn * 8 + lc) * p.H + h) * p.dv + out_j;
    const size_t out_row = (size_t)p.H * p.dv;
    for (int i = 0; i < n_blocks; ++i, left -= RB_B, ahead += src_step, out += RB_B * out_row) {
        const float *st = ring + stage * STAGE;
        auto &red_o = sm.red_o[FORM == RB_GATE ? i & 1 : 0];
        const float(*vr)[RB_VLD] = sm.vals[i & 3];
        // operand A of tokens 8 ks .. of the values
        auto values = [&](int ks, float *x) {
            const float *u0 = &vr[ks * 8 + lc][lr], *u1 = &vr[ks * 8 + lc + 1][lr];
            x[0] = u0[0], x[1] = u1[0], x[2] = u0[8], x[3] = u1[8];
        };
        auto decay = [&] {
#pragma unroll
            for (int ct = 0; ct < CT; ++ct) {
                const float2 d2 = *reinterpret_cast<const float2 *>(st + L::DT + ch0 + ct * 8 + lc);
                S[ct][0] *= d2.x;
                S[ct][1] *= d2.y;
                S[ct][2] *= d2.x;
                S[ct][3] *= d2.y;
            }
        };
        auto write = [&](int ks, const RbA &a, int rows) {
#pragma unroll
            for (int ct = 0; ct < CT; ++ct) {
                const float *b = st + rows + (ks * 8 + lc) * L::END_LD + ch0 + ct * 8 + lr;
                rb_mma(S[ct], a.x, b[0], b[L::END_LD]);
            }
        };
        await(0);
        {   // what the warp's channels of the state, and its share of the values, give to the block's h and o
            double acc[NT][4];
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[n][e] = 0.0;
            // The share: the values of tokens 8 ks .. in the sums of tokens 8 half .. of h (eight warps: of h or o)
            const int ks = (warp >> 1) & 1, half = warp & 1;
            constexpr int SHARES = NT / 2;
            if (ks <= half && (WARPS == 4 || SHARES == 2 || warp < 4)) {
                float x[4];
                values(ks, x);
                const bool number = fabsf(x[0]) < INFINITY && fabsf(x[1]) < INFINITY && fabsf(x[2]) < INFINITY && fabsf(x[3]) < INFINITY;
                const bool numbers = __all_sync(0xffffffffu, number);
                const RbA a = rb_a(x[0], x[1], x[2], x[3]);
                auto share = [&](bool of_h, double *y) {
                    const float *mat = st + (of_h ? L::M1 : L::M2);
                    if (numbers) {
                        const float2 b = *reinterpret_cast<const float2 *>(mat + (half * 8 + lr) * RB_LD + ks * 8 + lc);
                        rb_mma(y, a.x, b.x, b.y);
                        return;
                    }
                    // The product meets the zeros of the matrix with the numbers of later tokens, and 0 x inf is not 0: from the tokens that count alone, as
                    // the scan has it
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int t = half * 8 + lc + (e & 1), j = lr + (e >> 1) * 8;
#pragma unroll 1
                        for (int s = ks * 8; s < ks * 8 + 8 && s <= t; ++s)
                            if (!(FORM == RB_REMOVAL && of_h && s == t)) y[e] = fma((double)mat[t * RB_LD + s], (double)vr[s][j], y[e]);
                    }
                };
                double y[4] = {0.0, 0.0, 0.0, 0.0}, z[4] = {0.0, 0.0, 0.0, 0.0};
                constexpr bool BOTH = WARPS == 4 && SHARES == 2;
                const bool of_h = SHARES == 2 && (BOTH || warp < 4);
                share(of_h, y);
                if (BOTH) share(false, z);
#pragma unroll
                for (int n = 0; n < NT; ++n)                     // (neither the share nor its half is a constant)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const bool h_row = SHARES == 2 && n < 2;
                        const double mine = BOTH && !h_row ? z[e] : y[e];
                        acc[n][e] = (n & 1) == half && (BOTH || h_row == of_h) ? mine : 0.0;
                    }
            }
#pragma unroll
            for (int ct = 0; ct < CT; ++ct) {
                const RbA a = rb_a(S[ct][0], S[ct][1], S[ct][2], S[ct][3]);
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    const float2 b = *reinterpret_cast<const float2 *>(st + L::F1 + (n * 8 + lr) * L::ROW_LD + ch0 + ct * 8 + lc);
                    rb_mma(acc[n], a.x, b.x, b.y);
                }
            }
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (FORM != RB_GATE) rb_put2(&sm.red_h[FORM == RB_GATE ? 0 : warp][FORM == RB_GATE ? 0 : lr + 8 * e][n * 8 + lc], acc[n][2 * e], acc[n][2 * e + 1]);
                    rb_put2(&red_o[warp][lr + 8 * e][n * 8 + lc], acc[NT - 2 + n][2 * e], acc[NT - 2 + n][2 * e + 1]);
                }
        }
        if (FORM != RB_DELTA) {                 // what needs none of the sums
            await(1);
            decay();
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
                float x[4];
                values(ks, x);
                write(ks, rb_a(x[0], x[1], x[2], x[3]), L::KW);
            }
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");       // the next block's values; the barrier shows them to all
        __syncthreads();                        // and every warp is done with what the block before needed, and with this block's rows
        if (tid == 32 * (WARPS - 1)) {
            if (i + stages < n_blocks) {
                fetch(stage, ahead, 0);
                if (EARLY) fetch(stage, ahead, 1);
            }
            if (!EARLY && i > 0 && i - 1 + stages < n_blocks) fetch(before, ahead - src_step, 1);
        }
        load_v((i + 3) & 3);
        // the sums over the warps' channels, in their order
        if (FORM != RB_GATE && warp < 4) {      // (none of the tokens beyond the request's end: what is not finite before them reaches their rows too)
            double2 y = make_double2(0.0, 0.0);
#pragma unroll
            for (int w = 0; w < WARPS; ++w) {
                const double2 z = *reinterpret_cast<const double2 *>(&sm.red_h[FORM == RB_GATE ? 0 : w][FORM == RB_GATE ? 0 : lr + 8 * qe][qn * 8 + lc]);
                y.x += z.x;
                y.y += z.y;
            }
            rb_put2(&sm.corr[FORM == RB_GATE ? 0 : lr + 8 * qe][qn * 8 + lc], left > qn * 8 + lc ? y.x : 0.0, left > qn * 8 + lc + 1 ? y.y : 0.0);
        }
        if (WARPS == 4 || warp >= 4) {
            double2 y = make_double2(0.0, 0.0);
#pragma unroll
            for (int w = 0; w < WARPS; ++w) {
                const double2 z = *reinterpret_cast<const double2 *>(&red_o[w][lr + 8 * qe][qn * 8 + lc]);
                y.x += z.x;
                y.y += z.y;
            }
            if (out_j < p.dv) {
                if (left > qn * 8 + lc) out[0] = (float)y.x;
                if (left > qn * 8 + lc + 1) out[out_row] = (float)y.y;
            }
        }
        if (FORM != RB_GATE) {
            if (FORM == RB_DELTA) {
                await(1);
                decay();
            }
            __syncthreads();
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
                const double *y0 = &sm.corr[FORM == RB_GATE ? 0 : lr][ks * 8 + lc], *y1 = &sm.corr[FORM == RB_GATE ? 0 : lr + 8][ks * 8 + lc];
                write(ks, rb_a(y0[0], y0[1], y1[0], y1[1]), FORM == RB_DELTA ? L::KW : L::AW);
            }
        }
        before = stage;
        if (++stage == stages) stage = 0, phase ^= 1u;
    }
#pragma unroll
    for (int ct = 0; ct < CT; ++ct)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int c = ch0 + ct * 8 + lc + (e & 1), j = col0 + lr + (e >> 1) * 8;
            if (c < p.d && j < p.dv) Sg[(size_t)c * p.dv + j] = (float)S[ct][e];
        }
}

static int rb_padded(int d) { return d <= 32 ? 32 : d <= 64 ? 64 : 128; }
static long long rb_floats(int D, int form) {
    const int rows = form == RB_GATE ? 1 : 2, ends = form == RB_REMOVAL ? 2 : 1;
    return (long long)RB_B * (rows * (D + 8) + ends * (D + 4)) + D + (long long)rows * RB_MAT;
}

// Whether the scan takes the requests by length: up to 64 of them, and not equal ones, which stay in their order and would
// pay for the look (eight of 256 tokens, us: DELTA 203.4 with it, 202.5 without, GATE 74.4 and 73.5).
KESTREL_API int kestrel_recurrence_blocks_by_length(int T, int nseq, int max_count) {
    return nseq > 1 && nseq <= 64 && (long long)T < (long long)nseq * max_count ? 1 : 0;
}

template <int D, int FORM>
static int rb_launch(const RbParams &p, const RbSource *src, int T, int nseq, int max_count, cudaStream_t stream) {
    static_assert(RbLayout<D, FORM>::FLOATS % 4 == 0 && RbLayout<D, FORM>::KW % 4 == 0, "bulk copies move 16 bytes");
    const size_t prep = (size_t)(FORM == RB_GATE ? 3 : FORM == RB_DELTA ? 4 : 5) * RB_B * RbLayout<D, FORM>::END_LD * sizeof(float) + RbLayout<D, FORM>::MATS * RB_MAT * sizeof(double);
    constexpr size_t stage = (size_t)RbLayout<D, FORM>::FLOATS * sizeof(float), fixed = (sizeof(RbScan<D, FORM>) + 127) / 128 * 128;
    static bool attr_set = false;
    if (!attr_set) {
        if (cudaFuncSetAttribute(blocks_prepare_kernel<D, FORM, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prep) != cudaSuccess ||
            cudaFuncSetAttribute(blocks_prepare_kernel<D, FORM, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prep) != cudaSuccess ||
            cudaFuncSetAttribute(blocks_scan_kernel<D, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, KESTREL_SMEM_MAX_DYNAMIC) != cudaSuccess)
            return kestrel_fail(-3, "recurrence_blocks: cannot set the shared memory size");
        attr_set = true;
    }
    const dim3 blocks((max_count + RB_B - 1) / RB_B, p.H, nseq);
    if (src) kestrel_launch(blocks_prepare_kernel<D, FORM, true>, blocks, dim3(128), prep, stream, p, *src);
    else kestrel_launch(blocks_prepare_kernel<D, FORM, false>, blocks, dim3(128), prep, stream, p, RbSource());
    static_assert(2 * stage + fixed <= KESTREL_SMEM_MAX_DYNAMIC, "two stages fit an SM");
    const dim3 grid((p.dv + RB_COLS - 1) / RB_COLS, p.H, nseq);
    // as many stages as the CTAs that share an SM leave room for, two at least
    const size_t smem = kestrel_spread_smem((long)grid.x * grid.y * grid.z, 2 * stage + fixed), room = smem - fixed;
    const int stages = (int)(room / stage) < RB_STAGES ? (int)(room / stage) : RB_STAGES;
    kestrel_launch(blocks_scan_kernel<D, FORM>, grid, dim3(32 * RbScan<D, FORM>::WARPS), smem, stream, p, stages,
                   kestrel_recurrence_blocks_by_length(T, nseq, max_count) != 0);
    return kestrel_check_launch("recurrence_blocks");
}

template <int FORM>
static int rb_run(const RbParams &p, int T, int nseq, int max_count, cudaStream_t stream, const RbSource *src = nullptr) {
    switch (rb_padded(p.d)) {
        case 32: return rb_launch<32, FORM>(p, src, T, nseq, max_count, stream);
        case 64: return rb_launch<64, FORM>(p, src, T, nseq, max_count, stream);
        default: return rb_launch<128, FORM>(p, src, T, nseq, max_count, stream);
    }
}

static int rb_check(const RbParams &p, int T, int nseq, int max_count, long long floats, int form) {
    KESTREL_REQUIRE(T > 0 && nseq > 0 && max_count > 0 && p.H > 0 && p.G > 0 && p.H % p.G == 0 && p.d > 0 && p.dv > 0, "recurrence_blocks: bad sizes");
    KESTREL_REQUIRE(p.d <= 128, "recurrence_blocks: %d key channels; the kernel holds up to 128", p.d);
    KESTREL_REQUIRE(p.H <= 65535 && nseq <= 65535, "recurrence_blocks: grid too large");
    KESTREL_REQUIRE(floats >= ((long long)T / RB_B + nseq) * p.H * rb_floats(rb_padded(p.d), form), "recurrence_blocks: scratch of %lld floats is too small", floats);
    KESTREL_REQUIRE(((uintptr_t)p.blocks & 15) == 0, "recurrence_blocks: the scratch must start on a 16-byte boundary");
    return 0;
}

// floats of scratch for a step of T tokens of nseq requests; form 0: no correction, 1: with a and b, 2: the gated delta rule
KESTREL_API long long kestrel_recurrence_blocks_floats(int T, int nseq, int H, int d, int form) {
    if (T <= 0 || nseq <= 0 || H <= 0 || d <= 0 || d > 128 || form < 0 || form > 2) return -1;
    return ((long long)T / RB_B + nseq) * H * rb_floats(rb_padded(d), form);
}

// kestrel_recurrence_scan for portions of many tokens (max_count: the most tokens of one request); a and b null: no correction
KESTREL_API int kestrel_recurrence_blocks(const float *r, const float *w, const float *k, const float *v, const float *a, const float *b,
                                          float *state, long long state_stride, long long state_off, const int *cu_seqlens, const int *slots,
                                          float *out, float *scratch, long long scratch_floats, int T, int nseq, int max_count, int H, int d, int dv,
                                          cudaStream_t stream) {
    if (T == 0 || nseq == 0) return 0;
    KESTREL_REQUIRE((a == nullptr) == (b == nullptr), "recurrence_blocks: a and b come together");
    const RbParams p = {r, w, k, a, b, nullptr, v, (size_t)H * dv, state + state_off, (size_t)state_stride, cu_seqlens, slots, out, scratch, H, H, d, dv};
    const int rc = rb_check(p, T, nseq, max_count, scratch_floats, a ? RB_REMOVAL : RB_GATE);
    if (rc) return rc;
    return a ? rb_run<RB_REMOVAL>(p, T, nseq, max_count, stream) : rb_run<RB_GATE>(p, T, nseq, max_count, stream);
}

// kestrel_delta_scan for portions of many tokens
KESTREL_API int kestrel_delta_blocks(const float *qn, const float *kn, const float *decay, const float *v, long long ldv, const float *beta,
                                     float *state, long long state_stride, const int *cu_seqlens, const int *slots, float *out, float *scratch,
                                     long long scratch_floats, int T, int nseq, int max_count, int H, int G, int d, int dv, cudaStream_t stream) {
    if (T == 0 || nseq == 0) return 0;
    const RbParams p = {qn, decay, kn, nullptr, nullptr, beta, v, (size_t)ldv, state, (size_t)state_stride, cu_seqlens, slots, out, scratch, H, G, d, dv};
    const int rc = rb_check(p, T, nseq, max_count, scratch_floats, RB_DELTA);
    if (rc) return rc;
    return rb_run<RB_DELTA>(p, T, nseq, max_count, stream);
}

// Whether vectors of four fetch everything that a kernel with gates reads
static bool rb_whole(int d, std::initializer_list<long long> sizes, std::initializer_list<const void *> ptrs) {
    bool ok = d % 4 == 0;
    for (const long long x : sizes) ok = ok && x % 4 == 0;
    for (const void *p : ptrs) ok = ok && ((uintptr_t)p & 15) == 0;
    return ok;
}

// The whole recurrence of a mixer in blocks, its gates included: forget_gates / removal_gates (wz not null) and recurrence_scan.  x: the product,
// S slices; vsum: scratch [T, H dv] for the values of a product of several slices (may be null for one).  Returns 1 if vectors of four do not fit.
KESTREL_API int kestrel_gated_blocks(const float *x, int S, long long slice_stride, int ld, int col_r, int col_k, int col_v, int col_a,
                                     const float *bias, const float *bias2, const float *wz, int Sw, long long w_stride, float rate, float *vsum,
                                     float *state, long long state_stride, const int *cu_seqlens, const int *slots, float *out, float *scratch,
                                     long long scratch_floats, int T, int nseq, int max_count, int H, int d, int dv, cudaStream_t stream) {
    if (T == 0 || nseq == 0) return 0;
    KESTREL_REQUIRE(S > 0 && (!wz || Sw > 0) && (S == 1 || vsum), "gated_blocks: bad slices");
    if (!rb_whole(d, {slice_stride, ld, col_r, col_k, col_a, w_stride}, {x, wz})) return 1;
    RbSource src = {};
    src.x = x; src.Sx = S; src.x_stride = (size_t)slice_stride; src.ldx = ld;
    src.z = wz; src.Sz = Sw; src.z_stride = (size_t)w_stride; src.ldz = H * d;
    src.col_r = col_r; src.col_k = col_k; src.col_v = col_v; src.col_a = col_a;
    src.bias = bias; src.bias2 = bias2; src.rate = rate;
    src.v_out = S > 1 ? vsum : nullptr;
    RbParams p = {};
    p.v = S > 1 ? vsum : x + col_v;
    p.ldv = S > 1 ? (size_t)H * dv : (size_t)ld;
    p.state = state; p.state_stride = (size_t)state_stride; p.cu_seqlens = cu_seqlens; p.slots = slots; p.out = out; p.blocks = scratch;
    p.H = H; p.G = H; p.d = d; p.dv = dv;
    const int rc = rb_check(p, T, nseq, max_count, scratch_floats, wz ? RB_REMOVAL : RB_GATE);
    if (rc) return rc;
    return wz ? rb_run<RB_REMOVAL>(p, T, nseq, max_count, stream, &src) : rb_run<RB_GATE>(p, T, nseq, max_count, stream, &src);
}

// delta_gates (a decay per head and channel) and delta_scan in blocks.  act [T, C] = q | k | v after the convolution; beta logits at col_beta of
// the product y, decay logits the product a [T, H d].  Returns 1 if vectors of four do not fit.
KESTREL_API int kestrel_gated_delta_blocks(const float *act, int C, int col_v, const float *y, int Sy, long long y_stride, int ldy, int col_beta,
                                           const float *a, int Sa, long long a_stride, const float *A_log, const float *dt_bias, float *state,
                                           long long state_stride, const int *cu_seqlens, const int *slots, float *out, float *scratch,
                                           long long scratch_floats, int T, int nseq, int max_count, int H, int G, int d, int dv, cudaStream_t stream) {
    if (T == 0 || nseq == 0) return 0;
    KESTREL_REQUIRE(Sy > 0 && Sa > 0, "gated_delta_blocks: bad slices");
    if (!rb_whole(d, {C, a_stride}, {act, a})) return 1;
    RbSource src = {};
    src.x = act; src.Sx = 1; src.ldx = C; src.col_r = 0; src.col_k = G * d;
    src.y = y; src.Sy = Sy; src.y_stride = (size_t)y_stride; src.ldy = ldy; src.col_a = col_beta;
    src.z = a; src.Sz = Sa; src.z_stride = (size_t)a_stride; src.ldz = H * d;
    src.bias = dt_bias; src.bias2 = A_log;
    RbParams p = {};
    p.v = act + col_v;
    p.ldv = (size_t)C;
    p.state = state; p.state_stride = (size_t)state_stride; p.cu_seqlens = cu_seqlens; p.slots = slots; p.out = out; p.blocks = scratch;
    p.H = H; p.G = G; p.d = d; p.dv = dv;
    const int rc = rb_check(p, T, nseq, max_count, scratch_floats, RB_DELTA);
    if (rc) return rc;
    return rb_run<RB_DELTA>(p, T, nseq, max_count, stream, &src);
}

// Error word of the bounded waits (0: none, 1: a block's copy).  Synchronises the device and clears the word.
KESTREL_API int kestrel_recurrence_blocks_error(void) {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_rb_error, sizeof(int)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_rb_error, &zero, sizeof(int));
    return v;
}
