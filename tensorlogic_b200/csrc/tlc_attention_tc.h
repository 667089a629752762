// Prefill attention on the tensor cores (tlc_attention_tc.cu), called by tlc_launch_attention.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>

#include "tlc_internal.h"

struct AttnTc {
    const __half *q, *kc, *vc;  // [batch * I, H, D]; this layer's caches [batch][Tmax][Hkv][D]
    __half *out;
    int batch, I, H, Hkv, D, Tmax, pos0;
    float scale;
    CUtensorMap q_map, k_map, v_map;
};
// Fills in the tensor maps; false where the pointers cannot be described (not 16-byte aligned).
bool tlc_attention_tc_maps(AttnTc &a);
int32_t tlc_launch_attention_tc(tlc_ctx *ctx, const AttnTc &a);
