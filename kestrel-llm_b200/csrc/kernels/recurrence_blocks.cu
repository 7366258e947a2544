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
// The brackets are numbers per pair of tokens and head.  `blocks_prepare` makes them for all blocks at once, with the decayed vectors,
// and solves the triangular system: h = X (b^T S_0) + XK v with X = (I - A)^-1, and what o takes from b^T S_0 and v.  `blocks_scan` then
// walks a request's blocks: a CTA takes 16 value columns of a head, transposed, its four warps a quarter of the channels each, S^T in the
// accumulators of m16n8k8 products: the accumulators are the next product's operand A as they stand (the sum over channels may run in any
// order, so the unit's k index takes the channels in the order in which the accumulators hold them).  Per block: S^T times the decayed b and r
// (the warps' parts meet in shared memory), the 16 x 16 matrices, S^T update; two barriers.  A prepared block (38 KB at 128 channels) comes
// by one bulk copy into a ring, values by cp.async four blocks ahead.
//
// The products are the float64 ones of the tensor cores, and a portion's state is float64 from its first block to its last.  Read-outs and states
// are then closer to a float64 evaluation than the sequential scan's: 0.7 to 0.97 of its distance in a model of the roundings, at memories of 5
// to 300 tokens.  Operands as two terms of 11 bits on the tf32 products were not: those accumulators cut off instead of rounding, and with the
// state among them the read-outs were 1.8 (memory 20) to 4.3 times (300) as far as the scan's; summed afresh each block still 1.3 times.
// An SM makes 64 multiply-adds of float64 a cycle, 64 cycles a product and warp: 1,150 (GATE), 1,660 (DELTA) and 2,300 (REMOVAL) cycles a
// block and CTA, beside which come the conversions and the barriers: 2,250 cycles a block with one CTA an SM (GATE), 4,960 with two (DELTA).
// Prepared and scanned without their gates, tf32 -> float64: DELTA 213 -> 245 us, GATE 137 -> 165, REMOVAL 106 -> 123 (sizes below).  With plain
// float32 multiply-adds the same blocks are bound by the shared-memory reads of operands that 16 columns cannot reuse: 322 us for DELTA's scan.
//
// What is not finite stays so, and reaches the tokens and channels that it reaches in the scan: a block whose read-outs or corrections are
// not finite sums them again token by token (an infinity may come out as NaN, where terms of both signs meet).
//
// Three forms: GATE (no correction), REMOVAL (a, b given) and DELTA (a gated delta rule: with u = beta (v - (diag(w) S)^T k),
// S <- diag(w) S + k u^T, so that b = w k and the writes u = X beta (v - b^T S_0) take the place of v).
//
// Measured, 16 heads, prepared + scanned against the sequential scan, the gates in either case made before: DELTA (128 channels, requests of 592
// and 1,185 tokens) 245 us against 517; GATE (64 channels, 2,048 tokens) 165 against 287; REMOVAL (128 channels, 700 tokens in three
// requests, 350 the longest) 123 against 213.  The layers, which make their gates in the preparation, take 81 + 190, 26 + 147 and
// 55 + 93 us for the two launches, where gates kernel and scan took 37 + 523, 27 + 291 and 55 + 205.
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


// a prepared block of a head: [b decayed | r decayed | k to the block's end | a to the block's end | P(0, 16) | matrices]
template <int D, int FORM> struct RbLayout {
    static constexpr int ROW_LD = D + 8, END_LD = D + 4;        // rows read as pairs along the channels, and as pairs of rows
    static constexpr int BD = 0;
    static constexpr int RD = FORM == RB_GATE ? 0 : RB_B * ROW_LD;
    static constexpr int KW = RD + RB_B * ROW_LD;
    static constexpr int AW = KW + RB_B * END_LD;
    static constexpr int DT = FORM == RB_REMOVAL ? AW + RB_B * END_LD : AW;
    static constexpr int M = DT + D;            // GATE: Qk; DELTA: X beta, Qk X beta; REMOVAL: X, X K, Qa X, Qa X K + Qk
    static constexpr int FLOATS = M + (FORM == RB_GATE ? 1 : FORM == RB_DELTA ? 2 : 4) * RB_MAT;
};

// What a CTA of the scan holds beside its ring (a GATE block corrects nothing, and alternates between two buffers of sums)
template <int FORM> struct RbScan {
    static constexpr int ROWS = FORM == RB_GATE ? RB_B : 2 * RB_B;      // rows that meet the state: b and r
    static constexpr int RED_LD = ROWS + 8;
    unsigned long long bars[RB_STAGES];
    float red[FORM == RB_GATE ? 2 : 1][4][RB_COLS][RED_LD];
    float vals[4][RB_B][RB_VLD];                // values [token][column] of four blocks in flight: loaded for the next block alone they set the pace (2,400 cycles a block)
    float corr[FORM == RB_GATE ? 1 : RB_COLS][RB_LD];
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

template <int D, int FORM, bool MADE>
__global__ void __launch_bounds__(128)
blocks_prepare_kernel(const RbParams p, const RbSource src) {
    using L = RbLayout<D, FORM>;
    constexpr int V = D / 32;                   // channels of a lane
    pdl_launch_dependents();
    pdl_wait();
    const int blk = blockIdx.x, h = blockIdx.y, seq = blockIdx.z;
    const int t0 = p.cu_seqlens[seq] + blk * RB_B, t1 = p.cu_seqlens[seq + 1];
    if (t0 >= t1) return;
    extern __shared__ __align__(16) float rb_sm[];
    // [w | r | k | b | a] of the block's tokens, zero (w: one) beyond the head's channels and the request's tokens
    float *sw = rb_sm, *sr = sw + RB_B * D, *sk = sr + RB_B * D, *sb = sk + RB_B * D, *sa = sb + (FORM == RB_GATE ? 0 : RB_B * D);
    float *mat = sa + (FORM == RB_REMOVAL ? RB_B * D : 0);                     // A, K, Qa, Qk and two more, rows of RB_LD
    float *mA = mat, *mK = mA + RB_MAT, *mQa = mK + RB_MAT, *mQk = mQa + RB_MAT, *mX = mQk + RB_MAT, *mY = mX + RB_MAT;
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
            *reinterpret_cast<float4 *>(sw + idx) = w4;
            *reinterpret_cast<float4 *>(sr + idx) = r4;
            *reinterpret_cast<float4 *>(sk + idx) = k4;
            if (FORM == RB_REMOVAL) *reinterpret_cast<float4 *>(sa + idx) = a4;
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
                    const float k = sk[t * D + lane * V + j], r = sr[t * D + lane * V + j];
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
                const int idx = tid + 128 * i, t = idx / D;
                const float u = sk[idx] * sinv[0][t];
                if (FORM == RB_REMOVAL) {
                    sb[idx] = u;
                    sa[idx] = -(sa[idx] * u);
                } else {
                    sk[idx] = u;
                    sr[idx] *= sinv[1][t];
                    sb[idx] = sw[idx] * u;
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
            const int idx = (tid + 128 * i) * 4;
            *reinterpret_cast<float4 *>(sw + idx) = w4[i];
            *reinterpret_cast<float4 *>(sr + idx) = r4[i];
            *reinterpret_cast<float4 *>(sk + idx) = k4[i];
            if (FORM == RB_REMOVAL) {
                *reinterpret_cast<float4 *>(sb + idx) = b4[i];
                *reinterpret_cast<float4 *>(sa + idx) = a4[i];
            }
            if (FORM == RB_DELTA)
                *reinterpret_cast<float4 *>(sb + idx) = make_float4(w4[i].x * k4[i].x, w4[i].y * k4[i].y, w4[i].z * k4[i].z, w4[i].w * k4[i].w);
        }
    } else {
#pragma unroll 4
        for (int idx = tid; idx < RB_B * D; idx += 128) {
            const int t = idx / D, c = idx % D;
            const bool in = t0 + t < t1 && c < p.d;
            const size_t oh = ((size_t)(t0 + t) * p.H + h) * p.d + c, ok = ((size_t)(t0 + t) * KH + kh) * p.d + c;
            const float w = in ? p.w[oh] : 1.f, k = in ? p.k[ok] : 0.f;
            sw[idx] = w;
            sr[idx] = in ? p.r[ok] : 0.f;
            sk[idx] = k;
            if (FORM == RB_REMOVAL) {
                sb[idx] = in ? p.b[oh] : 0.f;
                sa[idx] = in ? p.a[oh] : 0.f;
            }
            if (FORM == RB_DELTA) sb[idx] = w * k;
        }
    }
    for (int idx = tid; idx < 6 * RB_MAT; idx += 128) mat[idx] = 0.f;
    __syncthreads();

    float *blkp = p.blocks + ((size_t)(p.cu_seqlens[seq] / RB_B + seq + blk) * p.H + h) * L::FLOATS;
    // vectors decayed from the block's start and to its end, a channel a thread
    for (int c = tid; c < D; c += 128) {
        float run = 1.f;
#pragma unroll
        for (int t = 0; t < RB_B; ++t) {
            if (FORM != RB_GATE) blkp[L::BD + t * L::ROW_LD + c] = sb[t * D + c] * run;
            run *= sw[t * D + c];
            blkp[L::RD + t * L::ROW_LD + c] = sr[t * D + c] * run;
        }
        blkp[L::DT + c] = run;
        run = 1.f;
#pragma unroll
        for (int t = RB_B - 1; t >= 0; --t) {
            blkp[L::KW + t * L::END_LD + c] = sk[t * D + c] * run;
            if (FORM == RB_REMOVAL) blkp[L::AW + t * L::END_LD + c] = sa[t * D + c] * run;
            run *= sw[t * D + c];
        }
    }
    // the pairs: a warp takes four tokens s, evenly long walks t = s .. 15 among them; the sums of TG t's go through the lanes together
    constexpr int TG = FORM == RB_REMOVAL ? 8 : RB_B;
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
        const int s = i == 0 ? warp : i == 1 ? 7 - warp : i == 2 ? 8 + warp : 15 - warp;
        double xk[V], xa[V];
#pragma unroll
        for (int j = 0; j < V; ++j) {           // neighbouring channels: they come in one load
            xk[j] = sk[s * D + lane * V + j];
            xa[j] = FORM == RB_REMOVAL ? sa[s * D + lane * V + j] : 0.f;
        }
#pragma unroll 1
        for (int part = s / TG; part < RB_B / TG; ++part) {
            double x[32];                       // [t][the form's matrices]
#pragma unroll
            for (int u = 0; u < TG; ++u) {
                const int t = part * TG + u;
                double fA = 0.0, fK = 0.0, fQa = 0.0, fQk = 0.0;
                if (t >= s) {
#pragma unroll
                    for (int j = 0; j < V; ++j) {
                        const int o = t * D + lane * V + j;
                        if (t > s) {
                            if (FORM != RB_GATE) {
                                const double bb = sb[o];
                                fK = fma(bb, xk[j], fK);
                                if (FORM == RB_REMOVAL) fA = fma(bb, xa[j], fA);
                            }
                            const double ww = sw[o];
                            xk[j] *= ww;
                            if (FORM == RB_REMOVAL) xa[j] *= ww;
                        }
                        const double rr = sr[o];
                        fQk = fma(rr, xk[j], fQk);
                        if (FORM == RB_REMOVAL) fQa = fma(rr, xa[j], fQa);
                    }
                }
                if (FORM == RB_REMOVAL) x[4 * u] = fA, x[4 * u + 1] = fK, x[4 * u + 2] = fQa, x[4 * u + 3] = fQk;
                else if (FORM == RB_DELTA) x[2 * u] = fK, x[2 * u + 1] = fQk;
                else x[u] = fQk;
            }
            // lane l ends with value l (GATE: l / 2)
            if (FORM == RB_GATE) {
                rb_exchange<16, 16>(x, lane);
                rb_exchange<8, 8>(x, lane);
                rb_exchange<4, 4>(x, lane);
                rb_exchange<2, 2>(x, lane);
                x[0] += __shfl_xor_sync(0xffffffffu, x[0], 1);
                mQk[(lane >> 1) * RB_LD + s] = (float)x[0];
            } else {
                rb_exchange<32, 16>(x, lane);
                rb_exchange<16, 8>(x, lane);
                rb_exchange<8, 4>(x, lane);
                rb_exchange<4, 2>(x, lane);
                rb_exchange<2, 1>(x, lane);
                if (FORM == RB_REMOVAL) mat[(lane & 3) * RB_MAT + (part * TG + (lane >> 2)) * RB_LD + s] = (float)x[0];
                else (lane & 1 ? mQk : mK)[(lane >> 1) * RB_LD + s] = (float)x[0];
            }
        }
    }
    __syncthreads();
    if (FORM == RB_GATE) {
        for (int idx = tid; idx < RB_MAT; idx += 128) blkp[L::M + idx] = mQk[idx];
        return;
    }
    // X, a column a thread, by substitution: REMOVAL (I - A)^-1; DELTA (I + beta A)^-1 beta with A in mK
    if (tid < RB_B) {
        double x[RB_B];
#pragma unroll
        for (int t = 0; t < RB_B; ++t) {
            const float beta = FORM == RB_DELTA ? sbeta[t] : 0.f;
            double sum = 0;
#pragma unroll
            for (int s = 0; s < t; ++s) sum = fma((double)(FORM == RB_DELTA ? mK : mA)[t * RB_LD + s], x[s], sum);
            const float one = t == tid ? 1.f : 0.f;
            x[t] = FORM == RB_DELTA ? beta * (one - sum) : one + sum;
            mX[t * RB_LD + tid] = (float)x[t];
        }
    }
    __syncthreads();
    // (sums over the tokens up to t alone: a later token's numbers may not be finite, and 0 x inf would not be 0)
    for (int idx = tid; idx < RB_B * RB_B; idx += 128) {
        const int t = idx / RB_B, j = idx % RB_B;
        if (FORM == RB_DELTA) {
            float m = 0.f;
#pragma unroll
            for (int s = 0; s < RB_B; ++s)
                if (s <= t) m = fmaf(mQk[t * RB_LD + s], mX[s * RB_LD + j], m);
            blkp[L::M + t * RB_LD + j] = mX[t * RB_LD + j];
            blkp[L::M + RB_MAT + t * RB_LD + j] = m;
        } else {
            float xk = 0.f, m1 = 0.f;
#pragma unroll
            for (int s = 0; s < RB_B; ++s)
                if (s <= t) {
                    xk = fmaf(mX[t * RB_LD + s], mK[s * RB_LD + j], xk);
                    m1 = fmaf(mQa[t * RB_LD + s], mX[s * RB_LD + j], m1);
                }
            mY[t * RB_LD + j] = xk;
            blkp[L::M + t * RB_LD + j] = mX[t * RB_LD + j];
            blkp[L::M + RB_MAT + t * RB_LD + j] = xk;
            blkp[L::M + 2 * RB_MAT + t * RB_LD + j] = m1;
        }
    }
    if (FORM == RB_REMOVAL) {
        __syncthreads();
        for (int idx = tid; idx < RB_B * RB_B; idx += 128) {
            const int t = idx / RB_B, j = idx % RB_B;
            float m2 = mQk[t * RB_LD + j];
#pragma unroll
            for (int s = 0; s < RB_B; ++s)
                if (s <= t) m2 = fmaf(mQa[t * RB_LD + s], mY[s * RB_LD + j], m2);
            blkp[L::M + 3 * RB_MAT + t * RB_LD + j] = m2;
        }
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

template <int D, int FORM>
__global__ void __launch_bounds__(128)
blocks_scan_kernel(const RbParams p, int stages) {
    using L = RbLayout<D, FORM>;
    constexpr int NT = RbScan<FORM>::ROWS / 8;                   // tiles of eight rows that meet the state
    constexpr int CT = D / 32;                                   // tiles of eight channels of a warp
    constexpr int STAGE = L::FLOATS, RED_LD = RbScan<FORM>::RED_LD;
    pdl_launch_dependents();
    extern __shared__ float4 rb_smem4[];
    float *ring = reinterpret_cast<float *>(rb_smem4);
    __shared__ __align__(16) RbScan<FORM> sm;
    auto &vals = sm.vals;
    auto &corr = sm.corr;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int lr = lane >> 2, lc = (lane & 3) * 2;               // a fragment's row (and row + 8) and its pair of columns
    const int h = blockIdx.y, seq = blockIdx.z, col0 = blockIdx.x * RB_COLS;
    const int ch0 = warp * (D / 4);
    const uint32_t bar0 = smem_u32(&sm.bars[0]);
    if (tid == 0) {
        for (int b = 0; b < stages; ++b) mbar_init(bar0 + 8 * b, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_wait();
    const int t0 = p.cu_seqlens[seq], t1 = p.cu_seqlens[seq + 1];
    const int n_blocks = (t1 - t0 + RB_B - 1) / RB_B;
    const float *src = p.blocks + ((size_t)(t0 / RB_B + seq) * p.H + h) * STAGE;
    auto fetch = [&](int i) {           // one thread: block i into stage i % stages
        const uint32_t bar = bar0 + 8u * (uint32_t)(i % stages);
        mbar_expect_tx(bar, STAGE * 4);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(smem_u32(ring + (i % stages) * STAGE)), "l"(src + (size_t)i * p.H * STAGE), "r"(STAGE * 4), "r"(bar)
                     : "memory");
    };
    if (tid == 0)
        for (int i = 0; i < min(stages, n_blocks); ++i) fetch(i);
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
    // thread moves columns vj, vj + 1 of token vt; zeros beyond the request and the head
    const int vt = tid >> 3, vj = (tid & 7) * 2;
    auto load_v = [&](int i) {
        const int t = t0 + i * RB_B + vt;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const bool in = i < n_blocks && t < t1 && col0 + vj + e < p.dv;
            const float *from = in ? p.v + (size_t)t * p.ldv + (size_t)h * p.dv + col0 + vj + e : p.v;
            const int bytes = in ? 4 : 0;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(&vals[i & 3][vt][vj + e])), "l"(from), "r"(bytes) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load_v(0);
    load_v(1);
    load_v(2);
    bool ok = true;
    for (int i = 0; i < n_blocks; ++i) {
        const int stage = i % stages;
        const float *st = ring + stage * STAGE;
        float(*red)[RB_COLS][RED_LD] = sm.red[FORM == RB_GATE ? i & 1 : 0];       // GATE has one barrier a block: two buffers in turn
        asm volatile("cp.async.wait_group 2;" ::: "memory");       // this block's values; the barrier below shows them to all
        if (ok && !mbar_wait(bar0 + 8u * stage, (uint32_t)(i / stages) & 1u)) { atomicExch(&g_rb_error, 1); ok = false; }
        {   // what the warp's channels of the state give to the block's rows
            double acc[NT][4];
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[n][e] = 0.0;
#pragma unroll
            for (int ct = 0; ct < CT; ++ct) {
                const RbA a = rb_a(S[ct][0], S[ct][1], S[ct][2], S[ct][3]);
#pragma unroll
                for (int n = 0; n < NT; ++n) {                   // rows: BD, then RD (GATE: RD)
                    const float2 b = *reinterpret_cast<const float2 *>(st + (n * 8 + lr) * L::ROW_LD + ch0 + ct * 8 + lc);
                    rb_mma(acc[n], a.x, b.x, b.y);
                }
            }
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    *reinterpret_cast<float2 *>(&red[warp][lr + 8 * e][n * 8 + lc]) = make_float2((float)acc[n][2 * e], (float)acc[n][2 * e + 1]);
        }
        __syncthreads();                        // and every warp is done with the block before
        if (tid == 0 && i > 0 && i - 1 + stages < n_blocks) fetch(i - 1 + stages);
        load_v(i + 3);
        const float(*vr)[RB_VLD] = vals[i & 3];
        // sum over the warps' channels of rows 8 n + lc, + 1 for columns lr, lr + 8
        auto total = [&](int n, float *x) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float2 s = make_float2(0.f, 0.f);
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    const float2 y = *reinterpret_cast<const float2 *>(&red[w][lr + 8 * e][n * 8 + lc]);
                    s.x += y.x;
                    s.y += y.y;
                }
                x[2 * e] = s.x;
                x[2 * e + 1] = s.y;
            }
        };
        // columns by tokens: warps 0, 1 the corrections (DELTA: the writes) of tokens 0-7, 8-15, warps 2, 3 the read-outs
        const bool reads = warp >= 2;
        const int half = warp & 1;
        if (reads || FORM != RB_GATE) {
            double sum[4] = {0.0, 0.0, 0.0, 0.0};
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            const float *m0 = st + L::M, *m1 = m0 + RB_MAT;
            const int row = (half * 8 + lr) * RB_LD + lc;
            if (reads) total((FORM == RB_GATE ? 0 : 2) + half, acc);
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
                const float *u0 = &vr[ks * 8 + lc][lr], *u1 = &vr[ks * 8 + lc + 1][lr];
                RbA av;
                if (FORM == RB_DELTA) {         // v - b^T S_0 takes the values' place
                    float x[4];
                    total(ks, x);
                    av = rb_a((double)u0[0] - x[0], (double)u1[0] - x[1], (double)u0[8] - x[2], (double)u1[8] - x[3]);
                } else {
                    av = rb_a(u0[0], u1[0], u0[8], u1[8]);
                }
                const float *mv = FORM == RB_GATE ? m0 : FORM == RB_DELTA ? (reads ? m1 : m0) : (reads ? m0 + 3 * RB_MAT : m1);
                float2 b = *reinterpret_cast<const float2 *>(mv + row + ks * 8);
                rb_mma(sum, av.x, b.x, b.y);
                if (FORM == RB_REMOVAL) {
                    float x[4];
                    total(ks, x);
                    const RbA ah = rb_a(x[0], x[1], x[2], x[3]);
                    b = *reinterpret_cast<const float2 *>((reads ? m0 + 2 * RB_MAT : m0) + row + ks * 8);
                    rb_mma(sum, ah.x, b.x, b.y);
                }
            }
            bool number = true;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                acc[e] = (float)(sum[e] + acc[e]);
                number = number && fabsf(acc[e]) < INFINITY;
            }
            if (!__all_sync(0xffffffffu, number)) {
                // The products above meet the zeros of the matrices with the numbers of later tokens, and 0 x inf is not 0: a token's
                // result from itself and the tokens before it alone, as the scan has it.
                auto total_of = [&](int n, int j) { return red[0][j][n] + red[1][j][n] + red[2][j][n] + red[3][j][n]; };
#pragma unroll 1
                for (int e = 0; e < 4; ++e) {
                    const int t = half * 8 + lc + (e & 1), j = lr + (e >> 1) * 8;
                    float x = reads ? total_of((FORM == RB_GATE ? 0 : RB_B) + t, j) : 0.f;
#pragma unroll 1
                    for (int s = 0; s <= t; ++s) {
                        const float *m = m0 + t * RB_LD + s;        // matrix i at i * RB_MAT
                        const float v = vr[s][j], h = FORM == RB_GATE ? 0.f : total_of(s, j);
                        if (FORM == RB_GATE) x = fmaf(m[0], v, x);
                        if (FORM == RB_DELTA) x = fmaf(m[reads ? RB_MAT : 0], v - h, x);
                        if (FORM == RB_REMOVAL) {
                            x = fmaf(m[reads ? 2 * RB_MAT : 0], h, x);
                            if (reads || s < t) x = fmaf(m[(reads ? 3 : 1) * RB_MAT], v, x);
                        }
                    }
                    acc[0] = e == 0 ? x : acc[0], acc[1] = e == 1 ? x : acc[1], acc[2] = e == 2 ? x : acc[2], acc[3] = e == 3 ? x : acc[3];
                }
            }
            if (reads) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int t = t0 + i * RB_B + half * 8 + lc + (e & 1), j = col0 + lr + (e >> 1) * 8;
                    if (t < t1 && j < p.dv) p.out[((size_t)t * p.H + h) * p.dv + j] = acc[e];
                }
            } else {
                // (none of the tokens beyond the request's end: what is not finite before them reaches their rows too)
                const int left = t1 - t0 - i * RB_B - half * 8 - lc;
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    *reinterpret_cast<float2 *>(&corr[lr + 8 * e][half * 8 + lc]) = make_float2(left > 0 ? acc[2 * e] : 0.f, left > 1 ? acc[2 * e + 1] : 0.f);
            }
        }
        if (FORM != RB_GATE) __syncthreads();
        // the state at the block's end
#pragma unroll
        for (int ct = 0; ct < CT; ++ct) {
            const float2 d2 = *reinterpret_cast<const float2 *>(st + L::DT + ch0 + ct * 8 + lc);
            S[ct][0] *= d2.x;
            S[ct][1] *= d2.y;
            S[ct][2] *= d2.x;
            S[ct][3] *= d2.y;
        }
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            auto write = [&](const RbA &a, const float *rows) {
#pragma unroll
                for (int ct = 0; ct < CT; ++ct) {
                    const float *b = rows + (ks * 8 + lc) * L::END_LD + ch0 + ct * 8 + lr;
                    rb_mma(S[ct], a.x, b[0], b[L::END_LD]);
                }
            };
            if (FORM != RB_DELTA) {
                const float *u0 = &vr[ks * 8 + lc][lr], *u1 = &vr[ks * 8 + lc + 1][lr];
                write(rb_a(u0[0], u1[0], u0[8], u1[8]), st + L::KW);
            }
            if (FORM != RB_GATE) {
                const float2 x0 = *reinterpret_cast<const float2 *>(&corr[lr][ks * 8 + lc]), x1 = *reinterpret_cast<const float2 *>(&corr[lr + 8][ks * 8 + lc]);
                write(rb_a(x0.x, x0.y, x1.x, x1.y), st + (FORM == RB_DELTA ? L::KW : L::AW));
            }
        }
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
    const int rows = form == RB_GATE ? 1 : 2, ends = form == RB_REMOVAL ? 2 : 1, mats = form == RB_GATE ? 1 : form == RB_DELTA ? 2 : 4;
    return (long long)RB_B * (rows * (D + 8) + ends * (D + 4)) + D + (long long)mats * RB_MAT;
}

template <int D, int FORM>
static int rb_launch(const RbParams &p, const RbSource *src, int nseq, int max_count, cudaStream_t stream) {
    static_assert(RbLayout<D, FORM>::FLOATS % 4 == 0, "bulk copies move 16 bytes");
    const size_t prep = (size_t)((FORM == RB_GATE ? 3 : FORM == RB_DELTA ? 4 : 5) * RB_B * D + 6 * RB_MAT) * sizeof(float);
    constexpr size_t stage = (size_t)RbLayout<D, FORM>::FLOATS * sizeof(float), fixed = (sizeof(RbScan<FORM>) + 1023) / 1024 * 1024;
    static bool attr_set = false;
    if (!attr_set) {
        if (cudaFuncSetAttribute(blocks_prepare_kernel<D, FORM, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prep) != cudaSuccess ||
            cudaFuncSetAttribute(blocks_prepare_kernel<D, FORM, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prep) != cudaSuccess ||
            cudaFuncSetAttribute(blocks_scan_kernel<D, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(KESTREL_SMEM_MAX_DYNAMIC - fixed)) != cudaSuccess)
            return kestrel_fail(-3, "recurrence_blocks: cannot set the shared memory size");
        attr_set = true;
    }
    const dim3 blocks((max_count + RB_B - 1) / RB_B, p.H, nseq);
    if (src) kestrel_launch(blocks_prepare_kernel<D, FORM, true>, blocks, dim3(128), prep, stream, p, *src);
    else kestrel_launch(blocks_prepare_kernel<D, FORM, false>, blocks, dim3(128), prep, stream, p, RbSource());
    static_assert(2 * stage + fixed <= KESTREL_SMEM_MAX_DYNAMIC, "two stages fit an SM");
    const dim3 grid((p.dv + RB_COLS - 1) / RB_COLS, p.H, nseq);
    // as many stages as the CTAs that share an SM leave room for, two at least
    const size_t room = kestrel_spread_smem((long)grid.x * grid.y * grid.z, 2 * stage + fixed) - fixed;
    const int stages = (int)(room / stage) < RB_STAGES ? (int)(room / stage) : RB_STAGES;
    kestrel_launch(blocks_scan_kernel<D, FORM>, grid, dim3(128), room, stream, p, stages);
    return kestrel_check_launch("recurrence_blocks");
}

template <int FORM>
static int rb_run(const RbParams &p, int nseq, int max_count, cudaStream_t stream, const RbSource *src = nullptr) {
    switch (rb_padded(p.d)) {
        case 32: return rb_launch<32, FORM>(p, src, nseq, max_count, stream);
        case 64: return rb_launch<64, FORM>(p, src, nseq, max_count, stream);
        default: return rb_launch<128, FORM>(p, src, nseq, max_count, stream);
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
    return a ? rb_run<RB_REMOVAL>(p, nseq, max_count, stream) : rb_run<RB_GATE>(p, nseq, max_count, stream);
}

// kestrel_delta_scan for portions of many tokens
KESTREL_API int kestrel_delta_blocks(const float *qn, const float *kn, const float *decay, const float *v, long long ldv, const float *beta,
                                     float *state, long long state_stride, const int *cu_seqlens, const int *slots, float *out, float *scratch,
                                     long long scratch_floats, int T, int nseq, int max_count, int H, int G, int d, int dv, cudaStream_t stream) {
    if (T == 0 || nseq == 0) return 0;
    const RbParams p = {qn, decay, kn, nullptr, nullptr, beta, v, (size_t)ldv, state, (size_t)state_stride, cu_seqlens, slots, out, scratch, H, G, d, dv};
    const int rc = rb_check(p, T, nseq, max_count, scratch_floats, RB_DELTA);
    if (rc) return rc;
    return rb_run<RB_DELTA>(p, nseq, max_count, stream);
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
    return wz ? rb_run<RB_REMOVAL>(p, nseq, max_count, stream, &src) : rb_run<RB_GATE>(p, nseq, max_count, stream, &src);
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
    return rb_run<RB_DELTA>(p, nseq, max_count, stream, &src);
}

// Error word of the bounded waits (0: none, 1: a block's copy).  Synchronises the device and clears the word.
KESTREL_API int kestrel_recurrence_blocks_error(void) {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_rb_error, sizeof(int)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_rb_error, &zero, sizeof(int));
    return v;
}
