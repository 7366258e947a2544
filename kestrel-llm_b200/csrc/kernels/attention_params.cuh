// Arguments shared by the tensor-core attention kernels (attention_mma.cu, attention_tc.cu).
#pragma once
#include <cuda_bf16.h>
#include "common.cuh"
#include "attention_score.cuh"
#include "differential.cuh"

struct AttnParams {
    const __nv_bfloat16 *q;         // [T, nq * hd]
    const __nv_bfloat16 *k_cache;   // [pages, nkv, page_size, hd]
    const __nv_bfloat16 *v_cache;
    __nv_bfloat16 *out;             // [T, nq * hd]
    float *part_o;                  // [T * nq, slices, hd]   (slices > 1)
    float *part_ml;                 // [T * nq, slices, 2]
    const int *tile_seq;            // [tiles] request index of the tile
    const int *tile_row0;           // [tiles] first row (token-major, head-minor) among the request's rows
    const int *cu_seqlens;          // [nseq + 1] first token of each request in this step
    const int *kv_lens;             // [nseq] request length after this step
    const int *block_table;         // [nseq, table_stride]
    const int *max_kv_ptr;          // if not null: the longest request's length on the device, from which the slice length follows (a captured step)
    int table_width;                // entries of a request's row that may be read (attention_tc.cu)
    int table_stride, page_size, nq, nkv, hd, window, slices, slice_len;
    float scale_log2;
    // options on the scores and on the weighing of keys; read by attention_tc.cu only, and only if `scored`
    float scale;
    ScoreOpts opts;
    int scored;
    int partial_only;               // attention_decode.cu: the unnormalised outputs go to part_o / part_ml even from one slice
    float cap_in, cap_out;          // attention_decode.cu: a bound on the scores, in base-2 units (cap_out 0: none)
    int slices_from_window;         // attention_decode.cu: slices count from the first key tile the window touches
    // a window that keeps a request's first tokens, and a factor per (token, head) on the outputs (or null); attention_tc.cu's kept form only
    int keep_first;
    const float *gate;
    int nseq;                       // where tile_seq is null: the requests of cu_seqlens, in whose rows a CTA looks for its tile (attn_find_tile)
    // two maps a head over the same values (differential attention); read by attention_tc.cu only
    DifferentialOpts maps;
};

// Keys per slice.  A launch recorded for replay fixes the number of slices; their length then
// follows the step's longest request, read on the device: its share of the keys rounded up to
// a multiple of 128 (a multiple of every kernel's key tile).
__device__ __forceinline__ int attn_slice_len(const AttnParams &p) {
    if (!p.max_kv_ptr) return p.slice_len;
    const int per = (*p.max_kv_ptr + p.slices - 1) / p.slices;
    const int len = (per + 127) / 128 * 128;
    return len < 128 ? 128 : len;
}

// (request, its first row) of a tile where no list was made for the step: every request's rows - `group` a token - cut into tiles of
// rows_per_tile, request by request.  A list costs its making and a copy on the host, once a step and size: 20 us of a step that the host
// paces, which a layer of few tokens does not win back; this is a scan over a warp per 32 requests.  All lanes of a warp take part.
__device__ __forceinline__ void attn_find_tile(const int *cu_seqlens, int nseq, int group, int rows_per_tile, int tile, int &seq, int &row0) {
    const int lane = threadIdx.x & 31;
    int left = tile;
    for (int base = 0; base < nseq; base += 32) {
        const int i = base + lane;
        const int n = i < nseq ? ((cu_seqlens[i + 1] - cu_seqlens[i]) * group + rows_per_tile - 1) / rows_per_tile : 0;
        int end = n;                // tiles of the requests up to this lane's
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += x;
        }
        const uint32_t behind = __ballot_sync(0xffffffffu, left < end);
        if (behind) {
            const int at = __ffs(behind) - 1;
            seq = base + at;
            row0 = (left - __shfl_sync(0xffffffffu, end - n, at)) * rows_per_tile;
            return;
        }
        left -= __shfl_sync(0xffffffffu, end, 31);
    }
    seq = nseq - 1;                 // no such tile: a tile that is there, whose rows another CTA writes too, with the same numbers
    row0 = 0;
}

// attention_mma.cu: merges the key-range slices of the listed tiles into out (kestrel_attention_merge, declared in kestrel.h), or with
// a factor per (token, head) on the outputs; tile_seq null: the tiles of nseq requests, found from cu_seqlens
int attention_merge_gated(const float *part_o, const float *part_ml, void *out, const int *tile_seq, const int *tile_row0, int tiles,
                          int rows_per_tile, const int *cu_seqlens, int nseq, int slices, int hd, int nq, int nkv, const float *sink, const float *gate,
                          cudaStream_t stream, bool contracted = false);
