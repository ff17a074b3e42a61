// Prompt attention on tcgen05; see attention_prefill_tc.cu.
#pragma once
#include "attention.cuh"
#include "prompt_cost.cuh"

struct M40PrefillTcArgs {
    M40PrefillCall c;  // c.seg null: packed K, V [rows][kv_heads][hd] with the offsets and lengths below
    const uint32_t* q_offsets;
    const uint32_t* kv_offsets;
    const uint32_t* q_lens;
    const uint32_t* kv_lens;
    uint32_t* status;
    uint32_t two_tiles;   // two tiles of 128 rows per CTA (prompt_cost.cuh)
    uint32_t pair_heads;  // filled in by the launch
};
// kv_rows: rows of the K and V arrays (cache: slots * kv_heads * max_seq_len). 0 when launched, 1 for a call it does not take,
// < 0 on failure.
int m40_attention_prefill_tc(M40llmCudaContext* ctx, cudaStream_t s, const M40PrefillTcArgs& a, uint64_t kv_rows);
