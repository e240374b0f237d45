// Interface between the prefill dispatcher (ktk_prefill.cu) and the tcgen05 prefill kernel (ktk_prefill_umma.cu).
#pragma once

#include "ktk_common.cuh"

namespace ktk {

struct PrefillUmmaParams {
    const void* q;
    void* o;
    const void* cache;
    const int32_t* q_indptr;
    const int32_t* kv_indices;
    const int32_t* kv_indptr;
    const int32_t* kv_last_page_len;
    const int32_t* page_count;
    int sink_tokens;
    int batch, Hkv, G;
    int64_t total_new;
    int tiles;                 // of a CTA: 1 or 2 (set by launch_prefill_umma)
    int64_t num_pages;
    float scale_log2;
    int32_t* status;
};

int launch_prefill_umma(PrefillUmmaParams p, int max_new_tokens, cudaStream_t st);

}  // namespace ktk
