// The prompt path's attention (jq_prompt_attention.cu), as the decoder calls it.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "jq_common.cuh"

namespace jq {

struct PromptAttention {
    const float *q, *k, *v;          // [T][heads | kv_heads][hd], not rotated yet
    float *k_cache, *v_cache;        // [position][kv_heads][hd]; positions below pos0 are filled
    const float *cos_t, *sin_t;      // [position][hd / 2]
    __nv_bfloat16* out;              // [T][heads][hd]
    int T, pos0, heads, kv_heads;
    float scale;
    // workspace (prompt_attention_layout): operands as two halves per value, and a power of two per row
    __half *qh, *ql, *kh, *kl, *vh, *vl;
    float *qs, *ks, *vs;
    int keys_pad;                    // keys rounded up to whole tiles
};

size_t prompt_attention_bytes(int T, int keys, int heads, int kv_heads, int hd);
void prompt_attention_layout(PromptAttention& p, uint8_t* scratch, int hd);
// Head sizes 64 and 128.
int launch_prompt_attention(const PromptAttention& p, int hd, cudaStream_t s);

}  // namespace jq
