// Token selection on the device: argmax, and sampling with temperature, top-k, min-p and
// top-p over rows of float32 logits.  Only token ids leave the GPU.  A row is sampled by the
// CTAs of a cluster that keep it in shared memory (sample_cluster_kernel, further down), or,
// where it does not fit, by one block over global memory (sample_kernel).
//
// Meaning of the options follows the reference's host sampler
// (src/core/vllm_transformer.c:357-479): temperature <= 0 or top_p <= 0 selects the first
// maximum (:362-367); else p = exp((l - max)/T) / sum (:393-404); top-k keeps the k most
// probable (:413); min-p drops p < min_p * max p (:418-423); top-p keeps the shortest
// descending prefix whose mass reaches top_p, without renormalising in between (:426-458);
// the draw is the first index whose running sum of kept p reaches u * total (:464-471).  The
// reference's zeroing of ids 0, 1 and 3 (:406-409) belongs to its toy tokenizer and is not
// taken over.  The uniform number u in (0, 1] comes from the caller, one per row, so a
// request's draws do not depend on what else is in the batch.
//
// No sort: the k-th largest logit and the top-p cut are found by building the threshold's
// bit pattern from the top bits down, one counting (or mass) pass per bit (sample_kernel), or in
// the bin of values that holds it (sample_cluster_kernel).  Entries equal to a
// threshold are all kept, where the reference's heap keeps the lower indices; the two differ
// only on exact ties at a cut.
#include "common.cuh"
#include <math.h>

#define SP_THREADS 1024

__device__ __forceinline__ unsigned ordered_key(float f) {
    unsigned b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__device__ float block_sum(float v, float *red) {
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float tot = 0.f;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) tot += red[k];
    return tot;
}

__device__ float block_max(float v, float *red) {
    v = warp_max(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float tot = -INFINITY;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) tot = fmaxf(tot, red[k]);
    return tot;
}

// first maximum of a row; ties go to the lower index
__device__ int block_argmax(const float *__restrict__ row, int V, float *red, int *redi) {
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int i = threadIdx.x; i < V; i += blockDim.x) {
        float v = row[i];
        if (v > best || (v == best && i < bi)) { best = v; bi = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        float ov = __shfl_xor_sync(0xffffffffu, best, o);
        int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) { red[threadIdx.x >> 5] = best; redi[threadIdx.x >> 5] = bi; }
    __syncthreads();
    float b = red[0];
    int idx = redi[0];
    for (int k = 1; k < (int)(blockDim.x >> 5); ++k)
        if (red[k] > b || (red[k] == b && redi[k] < idx)) { b = red[k]; idx = redi[k]; }
    return idx == 0x7fffffff ? 0 : idx;   // a row of NaN or -inf: index 0, as a strict > scan gives
}

__global__ void __launch_bounds__(SP_THREADS)
argmax_kernel(const float *__restrict__ logits, long long ld, int V, int *__restrict__ out) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float red[SP_THREADS / 32];
    __shared__ int redi[SP_THREADS / 32];
    int idx = block_argmax(logits + (size_t)blockIdx.x * ld, V, red, redi);
    if (threadIdx.x == 0) out[blockIdx.x] = idx;
}

// A large vocabulary in two passes, so that a row is read by many SMs: each block finds the
// first maximum of a chunk of ARGMAX_CHUNK entries and writes (value, index) to scratch; then
// one thread per row takes the first maximum over the chunks in ascending order.
#define ARGMAX_CHUNK 8192

__global__ void __launch_bounds__(256)
argmax_chunks_kernel(const float *__restrict__ logits, long long ld, int V, float *__restrict__ cand_v,
                     int *__restrict__ cand_i) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float red[8];
    __shared__ int redi[8];
    int row = blockIdx.x, chunk = blockIdx.y, chunks = gridDim.y;
    int b = chunk * ARGMAX_CHUNK, n = min(ARGMAX_CHUNK, V - b);
    int idx = block_argmax(logits + (size_t)row * ld + b, n, red, redi);
    if (threadIdx.x == 0) {
        cand_v[(size_t)row * chunks + chunk] = logits[(size_t)row * ld + b + idx];
        cand_i[(size_t)row * chunks + chunk] = b + idx;
    }
}

__global__ void argmax_final_kernel(const float *__restrict__ cand_v, const int *__restrict__ cand_i, int chunks,
                                    int R, int *__restrict__ out) {
    pdl_launch_dependents();
    pdl_wait();
    int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= R) return;
    const float *v = cand_v + (size_t)row * chunks;
    int best = 0;
    for (int c = 1; c < chunks; ++c)
        if (v[c] > v[best]) best = c;
    out[row] = cand_i[(size_t)row * chunks + best];
}

// scratch (used for V > ARGMAX_CHUNK): float [R * chunks] and int [R * chunks], chunks = ceil(V / 8192)
KESTREL_API int kestrel_argmax(const float *logits, long long ld, int R, int V, int *out, float *cand_v, int *cand_i,
                               cudaStream_t stream) {
    if (R == 0) return 0;
    KESTREL_REQUIRE(R > 0 && V > 0, "argmax: bad sizes R=%d V=%d", R, V);
    int chunks = (V + ARGMAX_CHUNK - 1) / ARGMAX_CHUNK;
    if (chunks == 1 || !cand_v || !cand_i) {
        kestrel_launch(argmax_kernel, dim3(R), dim3(SP_THREADS), 0, stream, logits, ld, V, out);
        return kestrel_check_launch("argmax");
    }
    KESTREL_REQUIRE(chunks <= 65535, "argmax: vocabulary %d too large", V);
    kestrel_launch(argmax_chunks_kernel, dim3(dim3(R, chunks)), dim3(256), 0, stream, logits, ld, V, cand_v, cand_i);
    kestrel_launch(argmax_final_kernel, dim3((R + 63) / 64), dim3(64), 0, stream, cand_v, cand_i, chunks, R, out);
    return kestrel_check_launch("argmax");
}

KESTREL_API int kestrel_argmax_chunks(int V) { return (V + ARGMAX_CHUNK - 1) / ARGMAX_CHUNK; }

__global__ void __launch_bounds__(SP_THREADS)
sample_kernel(const float *__restrict__ logits, long long ld, int V, const float *__restrict__ temperature,
              const int *__restrict__ top_k, const float *__restrict__ top_p, const float *__restrict__ min_p,
              const float *__restrict__ uniform, int *__restrict__ out) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float red[SP_THREADS / 32];
    __shared__ int redi[SP_THREADS / 32];
    __shared__ float scan[SP_THREADS];
    __shared__ int pick;
    const float *row = logits + (size_t)blockIdx.x * ld;
    float temp = temperature[blockIdx.x], tp = top_p[blockIdx.x], mp = min_p[blockIdx.x];
    int tk = top_k[blockIdx.x];
    if (temp <= 0.f || tp <= 0.f) {
        int idx = block_argmax(row, V, red, redi);
        if (threadIdx.x == 0) out[blockIdx.x] = idx;
        return;
    }
    float mx = -INFINITY;
    for (int i = threadIdx.x; i < V; i += SP_THREADS) mx = fmaxf(mx, row[i]);
    mx = block_max(mx, red);
    float z = 0.f;
    for (int i = threadIdx.x; i < V; i += SP_THREADS) z += expf((row[i] - mx) / temp);
    z = block_sum(z, red);
    float inv_z = 1.0f / z;

    // top-k: largest key x with count(key >= x) >= k
    unsigned key_k = 0u;
    if (tk > 0 && tk < V) {
        for (int bit = 31; bit >= 0; --bit) {
            unsigned cand = key_k | (1u << bit);
            float cnt = 0.f;
            for (int i = threadIdx.x; i < V; i += SP_THREADS) cnt += ordered_key(row[i]) >= cand ? 1.f : 0.f;
            cnt = block_sum(cnt, red);
            if (cnt >= (float)tk) key_k = cand;
        }
    }
    // min-p against the largest probability, which is exp(0)/z
    float floor_p = mp > 0.f ? mp * inv_z : 0.f;
    // top-p: largest key x whose mass(key >= x) reaches top_p among the entries still kept
    unsigned key_p = 0u;
    if (tp < 1.0f) {
        for (int bit = 31; bit >= 0; --bit) {
            unsigned cand = key_p | (1u << bit);
            float mass = 0.f;
            for (int i = threadIdx.x; i < V; i += SP_THREADS) {
                unsigned key = ordered_key(row[i]);
                float p = expf((row[i] - mx) / temp) * inv_z;
                if (key >= key_k && !(p < floor_p) && key >= cand) mass += p;
            }
            mass = block_sum(mass, red);
            if (mass >= tp) key_p = cand;
        }
    }
    unsigned cut = key_k > key_p ? key_k : key_p;

    // draw: contiguous chunk per thread, scan of the chunk sums, then a walk inside one chunk
    int chunk = (V + SP_THREADS - 1) / SP_THREADS;
    int b = threadIdx.x * chunk, e = min(V, b + chunk);
    float s = 0.f;
    for (int i = b; i < e; ++i) {
        float p = expf((row[i] - mx) / temp) * inv_z;
        if (ordered_key(row[i]) >= cut && !(p < floor_p)) s += p;
    }
    scan[threadIdx.x] = s;
    if (threadIdx.x == 0) pick = SP_THREADS;
    __syncthreads();
    for (int off = 1; off < SP_THREADS; off <<= 1) {
        float add = threadIdx.x >= off ? scan[threadIdx.x - off] : 0.f;
        __syncthreads();
        scan[threadIdx.x] += add;
        __syncthreads();
    }
    float total = scan[SP_THREADS - 1];
    float r = uniform[blockIdx.x] * total;
    float incl = scan[threadIdx.x];
    if (s > 0.f && incl >= r) atomicMin(&pick, (int)threadIdx.x);
    __syncthreads();
    if ((int)threadIdx.x == pick) {
        float c = threadIdx.x ? scan[threadIdx.x - 1] : 0.f;
        int chosen = -1, last = -1;
        for (int i = b; i < e && chosen < 0; ++i) {
            float p = expf((row[i] - mx) / temp) * inv_z;
            if (ordered_key(row[i]) >= cut && !(p < floor_p)) {
                c += p;
                last = i;
                if (c >= r) chosen = i;
            }
        }
        out[blockIdx.x] = chosen >= 0 ? chosen : last;
    }
    if (pick == SP_THREADS) {            // nothing kept (a row of NaN): first maximum
        int idx = block_argmax(row, V, red, redi);
        if (threadIdx.x == 0) out[blockIdx.x] = idx;
    }
}

// ------------------------------------------------------------------------------------------
// The same selection for vocabularies that fit the shared memory of a cluster: the row is cut
// over the CTAs of a cluster (up to 8), each CTA keeps its slice - logits and, where they fit
// too, probabilities - in shared memory, reads global memory once, and every further pass runs
// from there.  A threshold takes one pass that counts (top-k) or weighs (top-p) the entries by
// bins of values, a scan of the cluster's bins, and a look at the entries of the bin in which
// the threshold lies: few (SC_LIST; after a top-k all that are left of the row) are gathered and
// compared pair by pair, more go into bins of their keys until few are left or one key is.
//
// Counts and masses of bins are whole numbers (a probability relative to the largest, in units
// of a power of two that keeps all of its 24 bits), and the drawn sums of a gathered row too, so
// atomics in any order leave the same bits and a row's token does not depend on what else is in
// the batch; float32 sums are taken in a fixed order (thread, warp, block, rank).
//
// Bound by latency: a row's slices come in some 3 us, the rest are passes of 37 entries a thread
// and cluster barriers (five with a top-k whose list is short, seven with top-p alone).  Rows of
// 151,936, 16 | 1 of them, us: top-k 50, top-p and min-p 25 | 20, top-p alone 47 | 33, no filter
// 21 | 11; passes of four bits over the whole row, sixteen with an exchange each, took 165 | 79,
// 130 | 61 and 34 | 14.  Nearly flat rows, whose bins hold thousands: 60 | 40 (130 | 62).
// ------------------------------------------------------------------------------------------
#define SC_THREADS 512
#define SC_WARPS (SC_THREADS / 32)
#define SC_MAX_CLUSTER 8
#define SC_SMEM_LIMIT (200 * 1024)
#define SC_BINS 2048
#define SC_LIST SC_THREADS          // entries that are compared pair by pair, one a thread

__device__ __forceinline__ uint32_t sc_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t sc_ranks() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void sc_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// what lies at the same shared-memory address in CTA `rank` of this cluster
__device__ __forceinline__ uint32_t sc_at(const void *local, uint32_t rank) {
    uint32_t addr = (uint32_t)__cvta_generic_to_shared(local), remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
    return remote;
}
__device__ __forceinline__ float sc_remote(const float *local, uint32_t rank) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(sc_at(local, rank)) : "memory");
    return v;
}
__device__ __forceinline__ unsigned sc_remote(const unsigned *local, uint32_t rank) {
    unsigned v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(sc_at(local, rank)) : "memory");
    return v;
}
__device__ __forceinline__ uint2 sc_remote(const uint2 *local, uint32_t rank) {
    uint2 v;
    asm volatile("ld.shared::cluster.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(sc_at(local, rank)) : "memory");
    return v;
}
__device__ __forceinline__ double sc_remote(const double *local, uint32_t rank) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(sc_at(local, rank)) : "memory");
    return v;
}

struct ScEntries {                      // [SC_LIST] entries of a row
    unsigned key[SC_LIST], index[SC_LIST], what[SC_LIST];      // what: the entry's weight, or its probability
};
struct ScShared {
    float wred[SC_WARPS][4];            // per-warp partial results
    double wscan[SC_WARPS];
    float xch[2][4];                    // this CTA's results, read by the other ranks; two turns
    float res[4];                       // the cluster's
    ScEntries list;                     // this CTA's entries of a bin, read by the other ranks
    unsigned listed;                    // how many
    unsigned cut;                       // a bin or a key that the block's threads agree on
    unsigned low, high;                 // the least and the largest key of a bin
    int pick, last;
};
// A bin's weight: x in units of 2^13, y in units of one, each summed by 32-bit atomics; then, in the segment of bins that this
// CTA has added up over the cluster, their running sum in its place (nobody else reads a CTA's bins of its own segment).
union ScBin {
    uint2 w;
    double run;
};

// v[0..n) summed over the block (lane tree, then warps in ascending order) and over the
// cluster (ranks in ascending order); every thread of every CTA gets the same totals in sh.res.
// One cluster barrier a call; `turn` alternates so that a slot is not overwritten while a
// slower CTA still reads it.
template <int N>
__device__ __forceinline__ void sc_reduce(float (&v)[N], ScShared &sh, int &turn) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int b = 0; b < N; ++b) v[b] = warp_sum(v[b]);
    if (lane == 0) {
#pragma unroll
        for (int b = 0; b < N; ++b) sh.wred[warp][b] = v[b];
    }
    __syncthreads();
    if (threadIdx.x < N) {
        float t = 0.f;
        for (int w = 0; w < SC_WARPS; ++w) t += sh.wred[w][threadIdx.x];
        sh.xch[turn][threadIdx.x] = t;
    }
    sc_cluster_sync();
    if (threadIdx.x < N) {
        float t = 0.f;
        const uint32_t n = sc_ranks();
        for (uint32_t r = 0; r < n; ++r) t += sc_remote(&sh.xch[turn][threadIdx.x], r);
        sh.res[threadIdx.x] = t;
    }
    __syncthreads();
    turn ^= 1;
}

// Bins for counting, by the distance d >= 0 from the row's maximum: 128 to an octave from 2^-8 to 2^8, so that the entries
// around the k-th are told apart whether they lie close under the maximum or far below it.
__device__ __forceinline__ int sc_distance_bin(float d) {
    return min(max((int)(__float_as_uint(d) >> 16) - ((127 - 8) << 7), 0), SC_BINS - 1);
}
// Bins for weighing, by x = (l - max) / T <= 0: 128 to a factor e, down to e^-16
__device__ __forceinline__ int sc_mass_bin(float x) { return (int)fminf(-128.f * x, (float)(SC_BINS - 1)); }
// e = exp(x) of a bin lies in (2^-(s + 2), 2^-s]: in units of 2^-(26 + s) it is whole and below 2^27 (the last bin is cut off there)
__device__ __forceinline__ int sc_mass_shift(int bin) { return (int)((float)bin * (1.4426950f / 128.f)); }
__device__ __forceinline__ unsigned sc_mass_units(float e, int bin) {
    return __float2uint_rz(e * __uint_as_float((unsigned)(127 + 26 + sc_mass_shift(bin)) << 23));
}
__device__ __forceinline__ double sc_power(int exponent) { return __hiloint2double((1023 + exponent) << 20, 0); }

// The first bin with which the running weight, in which a bin's weight counts unit(bin) times, reaches what `reached` asks for; the
// running weight with it and before it.  False if none does.  Two cluster barriers, behind the first of which every CTA's bins are complete.
template <class Unit, class Reached>
__device__ __forceinline__ bool sc_find_bin(ScBin *bins, ScShared &sh, Unit unit, Reached reached, int &bin, double &before, double &with) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t nr = sc_ranks(), rank = sc_rank();
    const int per = SC_BINS / (int)nr, first = (int)rank * per;         // this CTA's segment
    const int own = max(1, per / SC_THREADS);                           // bins of a thread, one behind the other
    constexpr int MOST = SC_BINS / SC_THREADS;
    if (tid == 0) sh.cut = SC_BINS;
    sc_cluster_sync();
    double run[MOST], sum = 0.0;
#pragma unroll
    for (int i = 0; i < MOST; ++i) {
        run[i] = 0.0;
        const int b = first + tid * own + i;
        if (i < own && tid * own < per) {
            unsigned long long x = 0, y = 0;
#pragma unroll
            for (uint32_t r = 0; r < SC_MAX_CLUSTER; ++r)
                if (r < nr) {
                    const uint2 w = sc_remote(&bins[b].w, r);
                    x += w.x;
                    y += w.y;
                }
            sum += (double)((x << 13) + y) * unit(b);
            run[i] = sum;
        }
    }
    double incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double add = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += add;
    }
    if (lane == 31) sh.wscan[warp] = incl;
    __syncthreads();
    double offset = incl - sum;
    for (int w = 0; w < warp; ++w) offset += sh.wscan[w];
#pragma unroll
    for (int i = 0; i < MOST; ++i)
        if (i < own && tid * own < per) bins[first + tid * own + i].run = offset + run[i];
    sc_cluster_sync();
    double base = 0.0;
    int owner = -1;
    for (uint32_t r = 0; r < nr && owner < 0; ++r) {
        const double total = sc_remote(&bins[(r + 1) * per - 1].run, r);
        if (reached(base + total)) owner = (int)r;
        else base += total;
    }
    if (owner < 0) return false;                                        // (the same sums, the same answer, in every CTA)
    for (int b = tid; b < per; b += SC_THREADS)
        if (reached(base + sc_remote(&bins[owner * per + b].run, owner))) atomicMin(&sh.cut, (unsigned)(owner * per + b));
    __syncthreads();
    bin = (int)sh.cut;
    with = base + sc_remote(&bins[bin].run, owner);
    before = base + (bin > owner * per ? sc_remote(&bins[bin - 1].run, owner) : 0.0);
    return true;
}

// The lists of all CTAs, SC_LIST entries at most, into `all` (over the bins: every CTA is done with them behind the barrier)
__device__ __forceinline__ int sc_gather(ScEntries *all, ScShared &sh) {
    sc_cluster_sync();
    int before = 0;
    const uint32_t nr = sc_ranks();
    for (uint32_t r = 0; r < nr; ++r) {
        const int m = (int)sc_remote(&sh.listed, r), j = (int)threadIdx.x - before;
        if (j >= 0 && j < m) {
            all->key[threadIdx.x] = sc_remote(&sh.list.key[j], r);
            all->index[threadIdx.x] = sc_remote(&sh.list.index[j], r);
            all->what[threadIdx.x] = sc_remote(&sh.list.what[j], r);
        }
        before += m;
    }
    __syncthreads();
    return before;
}

// The smallest key that is kept among a bin's entries: one is kept unless the weight of the larger ones reaches the limit
template <class Reached>
__device__ __forceinline__ unsigned sc_list_cut(const ScEntries *all, int n, ScShared &sh, Reached reached) {
    if (threadIdx.x == 0) sh.cut = 0xffffffffu;
    __syncthreads();
    if ((int)threadIdx.x < n) {
        const unsigned key = all->key[threadIdx.x];
        unsigned long long larger = 0;
        for (int j = 0; j < n; ++j)
            if (all->key[j] > key) larger += all->what[j];
        if (!reached((double)larger)) atomicMin(&sh.cut, key);
    }
    __syncthreads();
    return sh.cut;
}

__device__ __forceinline__ void sc_clear_bins(ScBin *bins) {
    for (int i = threadIdx.x; i < SC_BINS / 2; i += SC_THREADS) reinterpret_cast<uint4 *>(bins)[i] = make_uint4(0, 0, 0, 0);
}
__device__ __forceinline__ void sc_add_units(ScBin &bin, unsigned units) {
    atomicAdd(&bin.w.x, units >> 13);
    if (units & 8191u) atomicAdd(&bin.w.y, units & 8191u);
}

// The largest key x for which the weight of the entries with key >= x reaches the limit, where `before` is the weight above the entries
// for which in(i, key) holds and with theirs it is reached.  units(i) is an entry's weight in whole units of `unit`.  The entries' keys
// are one range, and no other entry's lies in it.
template <class In, class Units, class Reached>
__device__ __forceinline__ unsigned sc_refine(ScBin *bins, ScEntries *all, const float *vals, int n, ScShared &sh, double before, double unit, In in, Units units,
                                              Reached reached) {
    const int tid = threadIdx.x;
    unsigned low = 0u, high = 0xffffffffu;          // of the entries' keys, from the first level on
    for (bool first = true;; first = false) {
        auto member = [&](int i, unsigned key) { return key >= low && key <= high && (!first || in(i, key)); };
        if (tid == 0) sh.listed = 0, sh.low = 0xffffffffu, sh.high = 0u;        // (the other CTAs have read earlier ones: a barrier lies between)
        __syncthreads();
        unsigned least = 0xffffffffu, most = 0u;
        for (int i = tid; i < n; i += SC_THREADS) {
            const unsigned key = ordered_key(vals[i]);
            if (!member(i, key)) continue;
            least = min(least, key), most = max(most, key);
            const unsigned at = atomicAdd(&sh.listed, 1u);
            if (at < SC_LIST) {
                sh.list.key[at] = key;
                sh.list.what[at] = units(i);
            }
        }
        if (most) atomicMin(&sh.low, least), atomicMax(&sh.high, most);
        sc_cluster_sync();
        unsigned listed = 0;
        low = 0xffffffffu, high = 0u;
        const uint32_t nr = sc_ranks();
        for (uint32_t r = 0; r < nr; ++r) {
            listed += sc_remote(&sh.listed, r);
            low = min(low, sc_remote(&sh.low, r)), high = max(high, sc_remote(&sh.high, r));
        }
        if (low >= high) return high;
        if (listed <= SC_LIST) {
            sc_gather(all, sh);
            return sc_list_cut(all, (int)listed, sh, [&](double w) { return reached(before + w * unit); });
        }
        // bins of keys from the largest down, a key a bin where they are few
        const int shift = max(0, 32 - __clz(high - low) - 11);
        sc_clear_bins(bins);
        __syncthreads();
        for (int i = tid; i < n; i += SC_THREADS) {
            const unsigned key = ordered_key(vals[i]);
            if (key >= low && key <= high) sc_add_units(bins[(high - key) >> shift], units(i));
        }
        int bin = 0;
        double above = 0.0, with = 0.0;
        if (sc_find_bin(bins, sh, [&](int) { return unit; }, [&](double w) { return reached(before + w); }, bin, above, with)) {
            before += above;
            high -= (unsigned)bin << shift;
            low = max(low, high - ((1u << shift) - 1u));
        } else {
            high = low;                             // (but for rounding it is reached with the last of them)
        }
    }
}

template <bool STORE_P>
__global__ void __launch_bounds__(SC_THREADS, 2)
sample_cluster_kernel(const float *__restrict__ logits, long long ld, int V, int S, const float *__restrict__ temperature,
                      const int *__restrict__ top_k, const float *__restrict__ top_p, const float *__restrict__ min_p,
                      const float *__restrict__ uniform, int *__restrict__ out) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) float sc_dyn[];
    __shared__ ScShared sh;
    ScBin *bins = reinterpret_cast<ScBin *>(sc_dyn);                    // [SC_BINS]
    ScEntries *all = reinterpret_cast<ScEntries *>(sc_dyn);             // in their place
    static_assert(sizeof(ScEntries) % 8 == 0 && sizeof(ScEntries) + SC_LIST * 8 <= SC_BINS * sizeof(ScBin), "gathered entries and their masses take the bins' place");
    float *vals = sc_dyn + SC_BINS * 2;             // [S] this CTA's logits
    float *probs = vals + (STORE_P ? S : 0);        // [S] their probabilities (relative to the largest), if kept
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t rank = sc_rank(), nr = sc_ranks();
    const int rowi = blockIdx.y;
    const int base = (int)rank * S, n = max(0, min(S, V - base));
    sc_clear_bins(bins);
    pdl_wait();
    const float temp = temperature[rowi], tp = top_p[rowi], mp = min_p[rowi], u = uniform[rowi];
    const int tk = top_k[rowi];
    const float *row = logits + (size_t)rowi * ld + base;
    int turn = 0;

    // the slice into shared memory; its first maximum on the way
    float best = -INFINITY;
    int bi = 0x7fffffff;
    const int whole = ((uintptr_t)row & 15) == 0 ? n & ~3 : 0;          // in vectors of four, eight of a thread in flight
    for (int i0 = 4 * tid; i0 < whole; i0 += 32 * SC_THREADS) {
        float4 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (i0 + 4 * SC_THREADS * j < whole) v[j] = __ldcs(reinterpret_cast<const float4 *>(row + i0 + 4 * SC_THREADS * j));
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int i = i0 + 4 * SC_THREADS * j;
            if (i >= whole) break;
            *reinterpret_cast<float4 *>(vals + i) = v[j];
            if (v[j].x > best) { best = v[j].x; bi = base + i; }        // ascending i per thread: the first of equals stays
            if (v[j].y > best) { best = v[j].y; bi = base + i + 1; }
            if (v[j].z > best) { best = v[j].z; bi = base + i + 2; }
            if (v[j].w > best) { best = v[j].w; bi = base + i + 3; }
        }
    }
#pragma unroll 8
    for (int i = whole + tid; i < n; i += SC_THREADS) {
        const float v = row[i];
        vals[i] = v;
        if (v > best) { best = v; bi = base + i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        float ov = __shfl_xor_sync(0xffffffffu, best, o);
        int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    if (lane == 0) { sh.wred[warp][0] = best; sh.wred[warp][1] = __int_as_float(bi); }
    __syncthreads();
    if (tid == 0) {
        float b = sh.wred[0][0], low = b;
        int idx = __float_as_int(sh.wred[0][1]);
        for (int w = 1; w < SC_WARPS; ++w) {
            float wv = sh.wred[w][0];
            int wi = __float_as_int(sh.wred[w][1]);
            low = fminf(low, wv);
            if (wv > b || (wv == b && wi < idx)) { b = wv; idx = wi; }
        }
        sh.xch[turn][0] = b;
        sh.xch[turn][1] = __int_as_float(idx);
        sh.xch[turn][2] = low;
        sh.listed = 0;
    }
    sc_cluster_sync();
    float mx = -INFINITY, low = INFINITY;
    int arg = 0x7fffffff;
    for (uint32_t r = 0; r < nr; ++r) {             // ranks in ascending order hold ascending indices
        float rv = sc_remote(&sh.xch[turn][0], r);
        int ri = __float_as_int(sc_remote(&sh.xch[turn][1], r));
        low = fminf(low, sc_remote(&sh.xch[turn][2], r));
        if (rv > mx || (rv == mx && ri < arg)) { mx = rv; arg = ri; }
    }
    turn ^= 1;
    if (arg == 0x7fffffff) arg = 0;                     // a row of NaN or -inf
    const bool greedy = temp <= 0.f || tp <= 0.f;
    bool done = greedy;
    if (!greedy) {
        // probabilities relative to the largest, and their sum
        auto relative = [&](float v) { return expf((v - mx) / temp); };
        auto rel = [&](int i) { return STORE_P ? probs[i] : relative(vals[i]); };
        float z[1] = {0.f};
#pragma unroll 2
        for (int i = 4 * tid; i < (n & ~3); i += 4 * SC_THREADS) {
            const float4 v = *reinterpret_cast<const float4 *>(vals + i);
            const float4 e = make_float4(relative(v.x), relative(v.y), relative(v.z), relative(v.w));
            if (STORE_P) *reinterpret_cast<float4 *>(probs + i) = e;
            z[0] += e.x, z[0] += e.y, z[0] += e.z, z[0] += e.w;
        }
        for (int i = (n & ~3) + tid; i < n; i += SC_THREADS) {
            const float e = relative(vals[i]);
            if (STORE_P) probs[i] = e;
            z[0] += e;
        }
        sc_reduce<1>(z, sh, turn);
        const float total_e = sh.res[0], inv_z = 1.0f / total_e;
        const float floor_p = mp > 0.f ? mp * inv_z : 0.f;
        unsigned key_k = 0u, key_p = 0u;
        bool drawn = !(total_e < INFINITY);             // NaN or an infinity in the row: the first maximum
        if (tk > 0 && tk < V && !drawn) {               // top-k: the largest key x with count(key >= x) >= k
            // every warp of the cluster has an entry that is not below the least of their maxima: no fewer than the warps
            const float least = tk <= (int)nr * SC_WARPS ? low : -INFINITY;
            unsigned far = 0;
            auto count = [&](float v) {
                if (!(v >= least)) return;
                const int b = sc_distance_bin(mx - v);
                if (b == SC_BINS - 1) ++far;
                else atomicAdd(&bins[b].w.x, 1u);
            };
            for (int i = 4 * tid; i < (n & ~3); i += 4 * SC_THREADS) {
                const float4 v = *reinterpret_cast<const float4 *>(vals + i);
                if (fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)) >= least) count(v.x), count(v.y), count(v.z), count(v.w);
            }
            for (int i = (n & ~3) + tid; i < n; i += SC_THREADS) count(vals[i]);
            if (far) atomicAdd(&bins[SC_BINS - 1].w.x, far);
            int bin = 0;
            double before = 0.0, with = 0.0;
            sc_find_bin(bins, sh, [](int) { return sc_power(-13); }, [&](double c) { return c >= (double)tk; }, bin, before, with);
            if (with > SC_LIST) {
                key_k = sc_refine(bins, all, vals, n, sh, before, 1.0, [&](int i, unsigned) { return vals[i] >= least && sc_distance_bin(mx - vals[i]) == bin; },
                                  [](int) { return 1u; }, [&](double c) { return c >= (double)tk; });
            } else {
                // all that top-k can keep, one entry a thread of the first CTA
                for (int i = tid; i < n; i += SC_THREADS) {
                    const float v = vals[i];
                    if (!(v >= least) || sc_distance_bin(mx - v) > bin) continue;
                    const unsigned at = atomicAdd(&sh.listed, 1u);
                    sh.list.key[at] = ordered_key(v);
                    sh.list.index[at] = (unsigned)(base + i);
                    sh.list.what[at] = __float_as_uint(rel(i));
                }
                const int m = sc_gather(all, sh);
                drawn = done = true;
                if (rank == 0) {
                    unsigned long long *masses = reinterpret_cast<unsigned long long *>(all + 1);       // in units of 2^-44 of the largest probability
                    const bool mine = tid < m;
                    const unsigned key = mine ? all->key[tid] : 0u, index = mine ? all->index[tid] : 0u;
                    const float e = mine ? __uint_as_float(all->what[tid]) : 0.f;
                    const unsigned long long q = __float2ull_rz(e * 17592186044416.f);
                    int larger = 0;
                    if (mine)
                        for (int j = 0; j < m; ++j) larger += all->key[j] > key ? 1 : 0;
                    const bool kept = mine && larger < tk && !(e * inv_z < floor_p);
                    if (mine) masses[tid] = kept ? q : 0ull;
                    __syncthreads();
                    unsigned long long sum = 0;
                    if (kept && tp < 1.0f)
                        for (int j = 0; j < m; ++j) sum += all->key[j] > key ? masses[j] : 0ull;
                    const bool stays = kept && !(tp < 1.0f && (double)sum * sc_power(-44) * inv_z >= (double)tp);
                    __syncthreads();
                    if (mine) masses[tid] = stays ? q : 0ull;
                    if (tid == 0) sh.pick = 0x7fffffff;
                    __syncthreads();
                    if (stays) {
                        unsigned long long all_mass = 0, upto = 0;
                        for (int j = 0; j < m; ++j) {
                            all_mass += masses[j];
                            upto += all->index[j] <= index ? masses[j] : 0ull;
                        }
                        if (q > 0 && (double)upto >= (double)u * (double)all_mass) atomicMin(&sh.pick, (int)index);
                    }
                    __syncthreads();
                    if (tid == 0) out[rowi] = sh.pick != 0x7fffffff ? sh.pick : arg;    // nothing kept (a floor above every probability): the first maximum
                }
            }
        }
        if (tp < 1.0f && !drawn) {                      // top-p: the largest key x whose mass(key >= x) reaches top_p among the entries still kept
            if (tk > 0 && tk < V) sc_clear_bins(bins);
            __syncthreads();
            unsigned long long beyond = 0;
            for (int i = tid; i < n; i += SC_THREADS) {
                const float v = vals[i], e = rel(i);
                if (ordered_key(v) < key_k || e * inv_z < floor_p) continue;
                const int b = sc_mass_bin((v - mx) / temp);
                const unsigned q = sc_mass_units(e, b);
                if (b == SC_BINS - 1) beyond += q;
                else sc_add_units(bins[b], q);
            }
            if (beyond) {
                atomicAdd(&bins[SC_BINS - 1].w.x, (unsigned)(beyond >> 13));
                atomicAdd(&bins[SC_BINS - 1].w.y, (unsigned)beyond & 8191u);
            }
            auto reached = [&](double mass) { return mass * inv_z >= (double)tp; };
            int bin = 0;
            double before = 0.0, with = 0.0;
            if (sc_find_bin(bins, sh, [](int b) { return sc_power(-26 - sc_mass_shift(b)); }, reached, bin, before, with))      // else all is kept
                key_p = sc_refine(bins, all, vals, n, sh, before, sc_power(-26 - sc_mass_shift(bin)),
                                  [&](int i, unsigned key) {
                                      return key >= key_k && sc_mass_bin((vals[i] - mx) / temp) == bin && !(rel(i) * inv_z < floor_p);
                                  },
                                  [&](int i) { return sc_mass_units(rel(i), bin); }, reached);
        }
        if (!drawn) {
            // draw: a contiguous chunk per thread, scan of the chunk sums over the block, the CTAs'
            // totals over the cluster, then a walk inside one chunk
            const unsigned cut = key_k > key_p ? key_k : key_p;
            auto kept = [&](int i) {                    // the probability of an entry that is kept, or none
                const float p = rel(i) * inv_z;
                return ordered_key(vals[i]) >= cut && !(p < floor_p) ? p : 0.f;
            };
            const int chunk = ((S + SC_THREADS - 1) / SC_THREADS) | 1;  // odd: a warp's threads read from 32 banks
            const int b0 = min(n, tid * chunk), e0 = min(n, b0 + chunk);
            float s = 0.f;
#pragma unroll 4
            for (int i = b0; i < e0; ++i) s += kept(i);
            float incl = s;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float add = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += add;
            }
            if (lane == 31) sh.wred[warp][0] = incl;
            if (tid == 0) sh.pick = SC_THREADS, sh.last = -1;
            __syncthreads();
            float lower = 0.f, cta_total = 0.f;
            for (int w = 0; w < SC_WARPS; ++w) {
                if (w == warp) lower = cta_total;
                cta_total += sh.wred[w][0];
            }
            float below = __shfl_up_sync(0xffffffffu, incl, 1);
            below = lower + (lane ? below : 0.f);
            incl += lower;
            if (tid == 0) sh.xch[turn][0] = cta_total;
            sc_cluster_sync();
            // the CTA in which the running sum of kept probability first reaches u * total: every CTA
            // finds the same one from the same sums
            float total = 0.f;
            for (uint32_t r = 0; r < nr; ++r) total += sc_remote(&sh.xch[turn][0], r);
            const float target = u * total;
            float before = 0.f, run = 0.f;
            int owner_rank = -1;
            for (uint32_t r = 0; r < nr; ++r) {
                float t = sc_remote(&sh.xch[turn][0], r);
                float end = run + t;
                if (owner_rank < 0 && t > 0.f && end >= target) { owner_rank = (int)r; before = run; }
                run = end;
            }
            turn ^= 1;
            if (total > 0.f && owner_rank >= 0) {
                done = true;
                if (owner_rank == (int)rank) {
                    const float rl = fminf(target - before, cta_total);
                    if (s > 0.f) {
                        if (incl >= rl) atomicMin(&sh.pick, tid);
                        atomicMax(&sh.last, tid);
                    }
                    __syncthreads();
                    const int pick = sh.pick < SC_THREADS ? sh.pick : sh.last;          // (rounding may leave the last sum short)
                    if (warp == pick >> 5) {            // the warp walks its thread's chunk, 32 entries a time
                        const int from = __shfl_sync(0xffffffffu, b0, pick & 31), to = __shfl_sync(0xffffffffu, e0, pick & 31);
                        float c = __shfl_sync(0xffffffffu, below, pick & 31);
                        int chosen = -1;
                        for (int i0 = from; i0 < to; i0 += 32) {
                            const float p = i0 + lane < to ? kept(i0 + lane) : 0.f;
                            float upto = p;
#pragma unroll
                            for (int o = 1; o < 32; o <<= 1) {
                                const float add = __shfl_up_sync(0xffffffffu, upto, o);
                                if (lane >= o) upto += add;
                            }
                            const unsigned some = __ballot_sync(0xffffffffu, p > 0.f), there = __ballot_sync(0xffffffffu, p > 0.f && c + upto >= rl);
                            if (some) chosen = i0 + (there ? __ffs(there) - 1 : 31 - __clz(some));
                            if (there) break;
                            c += __shfl_sync(0xffffffffu, upto, 31);
                        }
                        if (lane == 0) out[rowi] = base + chosen;
                    }
                }
            }
        }
    }
    if ((greedy || !done) && rank == 0 && tid == 0) out[rowi] = arg;    // greedy, or nothing kept (a row of NaN): first maximum
    sc_cluster_sync();                  // nobody leaves while its shared memory may still be read
}

// CTAs of a cluster for a vocabulary of V and whether the probabilities fit beside the logits;
// 0 if the row does not fit a cluster's shared memory (the one-block kernel takes it then)
static int sample_cluster_shape(int V, int R, int *slice, int *store_p) {
    static_assert(SC_SMEM_LIMIT + SC_BINS * sizeof(ScBin) + sizeof(ScShared) <= KESTREL_SMEM_MAX_DYNAMIC, "a CTA's slice, bins and lists");
    constexpr size_t half = KESTREL_SMEM_MAX_DYNAMIC / 2 - SC_BINS * sizeof(ScBin) - sizeof(ScShared) - 2048;
    for (int cl = 1; cl <= SC_MAX_CLUSTER; cl *= 2) {
        int S = (((V + cl - 1) / cl) + 3) & ~3;
        bool last = cl == SC_MAX_CLUSTER;
        if (!last && S > 8192) continue;               // more CTAs while a slice is long
        // Many rows: two CTAs on an SM, if leaving the probabilities out lets them fit.  From three quarters of the SMs on: clusters of
        // eight CTAs of an SM each do not fill every part of the chip (16 rows of 151,936 unfiltered took
        // 37 us, twice the time of 8; two CTAs an SM 21).
        bool crowded = 4ll * R * cl > 3ll * kestrel_sms() && (size_t)S * 8 > half && (size_t)S * 4 <= half;
        if (!crowded && (size_t)S * 8 <= SC_SMEM_LIMIT) { *slice = S; *store_p = 1; return cl; }
        if ((size_t)S * 4 <= SC_SMEM_LIMIT) { *slice = S; *store_p = 0; return cl; }
    }
    return 0;
}

// ------------------------------------------------------------------------------------------
// Repetition penalty of the reference's streaming harness (src/main.c:3741-3782): for each of
// the last `window` tokens a request generated, most recent first, the token's logit l becomes
// l / p if l >= 0, else l * p - once per occurrence, so a token that appears twice in the window
// is penalised twice.  history int32 [R, width]: row r holds that request's last tokens (entries
// beyond counts[r], or outside the vocabulary, are skipped); penalty float [R], <= 1 = off.
// One thread a row: the steps on one token follow each other, and there are 64 at most.
// ------------------------------------------------------------------------------------------
__global__ void repetition_penalty_kernel(float *__restrict__ logits, long long ld, int V, const int *__restrict__ history,
                                          int width, const int *__restrict__ counts, const float *__restrict__ penalty, int R) {
    pdl_launch_dependents();
    pdl_wait();
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= R) return;
    float p = penalty[r];
    if (!(p > 1.0f)) return;
    float *row = logits + (size_t)r * ld;
    int n = min(counts[r], width);
    for (int h = 0; h < n; ++h) {
        int tok = history[(size_t)r * width + h];
        if (tok < 0 || tok >= V) continue;
        float l = row[tok];
        row[tok] = l >= 0.0f ? l / p : l * p;
    }
}

KESTREL_API int kestrel_repetition_penalty(float *logits, long long ld, int R, int V, const int *history, int width,
                                           const int *counts, const float *penalty, cudaStream_t stream) {
    if (R == 0) return 0;
    KESTREL_REQUIRE(R > 0 && V > 0 && width > 0, "repetition_penalty: bad sizes R=%d V=%d width=%d", R, V, width);
    kestrel_launch(repetition_penalty_kernel, dim3((R + 63) / 64), dim3(64), 0, stream, logits, ld, V, history, width, counts, penalty, R);
    return kestrel_check_launch("repetition_penalty");
}

static int g_sample_cluster = 1;    // 0: always the one-block kernel (for tests of it)
KESTREL_API void kestrel_sample_set_cluster(int on) { g_sample_cluster = on ? 1 : 0; }

KESTREL_API int kestrel_sample(const float *logits, long long ld, int R, int V, const float *temperature,
                               const int *top_k, const float *top_p, const float *min_p,
                               const float *uniform, int *out, cudaStream_t stream) {
    if (R == 0) return 0;
    KESTREL_REQUIRE(R > 0 && V > 0, "sample: bad sizes R=%d V=%d", R, V);
    int S = 0, store_p = 0;
    int cl = g_sample_cluster && R <= 65535 && V < (1 << 24) ? sample_cluster_shape(V, R, &S, &store_p) : 0;
    if (cl > 0) {
        size_t smem = SC_BINS * sizeof(ScBin) + (size_t)S * 4 * (store_p ? 2 : 1);
        static bool attr_set = false;
        if (!attr_set) {
            const int most = SC_SMEM_LIMIT + SC_BINS * (int)sizeof(ScBin);
            cudaError_t e = cudaFuncSetAttribute(sample_cluster_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(sample_cluster_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
            if (e != cudaSuccess) return kestrel_fail(-3, "sample: cannot raise the shared-memory limit: %s", cudaGetErrorString(e));
            attr_set = true;
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(cl, R);
        cfg.blockDim = dim3(SC_THREADS);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = cl;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = g_kestrel_pdl ? 2 : 1;
        if (store_p) cudaLaunchKernelEx(&cfg, sample_cluster_kernel<true>, logits, ld, V, S, temperature, top_k, top_p, min_p, uniform, out);
        else cudaLaunchKernelEx(&cfg, sample_cluster_kernel<false>, logits, ld, V, S, temperature, top_k, top_p, min_p, uniform, out);
        return kestrel_check_launch("sample");
    }
    kestrel_launch(sample_kernel, dim3(R), dim3(SP_THREADS), 0, stream, logits, ld, V, temperature, top_k, top_p, min_p, uniform, out);
    return kestrel_check_launch("sample");
}
