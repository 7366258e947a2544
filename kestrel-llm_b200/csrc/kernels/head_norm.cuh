// Norm and gate of recurrent heads in vectors of four (linear_recurrence.cu).  False, and nothing launched, if the sizes do not fit it.
#pragma once
#include "common.cuh"

bool kestrel_head_norm_vec(const float *o, const float *w, int w_stride, float eps, const float *g_part, int Sg, size_t g_stride, int g_ld, int g_col0,
                           int g_act, __nv_bfloat16 *out, long long ldo, float scale, int T, int H, int dv, cudaStream_t stream);
