// Arguments of causal attention of prompts over the paged cache (dense_attn.cu, prefill_attn.cu); the ctypes mirror is `AttnParams`
// (`ops/dense.py`).
#pragma once

#include "common.cuh"

struct PagedPrefillParams {
    const bf16* q;                   // [T, n_heads, hd]
    const bf16* k_cache;             // [num_slots, n_kv, hd]
    const bf16* v_cache;
    const int* positions;            // [T] absolute position of each query (keys 0..pos are visible)
    const int* batch_idx;            // [T]
    const int* page_table; int pt_stride, page_size;
    const int* qo_indptr;            // [B + 1]
    int n_heads, n_kv, hd;
    float sm_scale;
    bf16* out;                       // [T, n_heads, hd]
    int T, num_slots;
    int max_keys;                    // longest history (0: not known)
    int* err;                        // error word of bounded waits
};

// Pages of 64 tokens, heads of 64 or 128 values, 16-byte aligned rows (prefill_attn.cu).
int paged_prefill_tcgen05(const PagedPrefillParams* p, int B, int max_q, cudaStream_t s);
