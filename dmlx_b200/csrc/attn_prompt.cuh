// Attention of batches that hold prompt portions, on tcgen05 (bf16 pools of one shape).
#pragma once
#include "kv_pool.cuh"

// Whether b200_attn_prompt takes the call: bf16 pages, GQA groups that divide a tile, q rows that TMA can address.
bool b200_attn_prompt_takes(const b200_kv* kv, const void* d_q, int32_t q_stride, const void* d_out);
b200_status b200_attn_prompt(b200_kv* kv, int32_t layer, const void* d_q, int32_t q_stride, const int32_t* d_row_seq, const int32_t* d_row_ctx,
                             int32_t total_rows, void* d_out, void* stream, bool may_split, bool reuse_plan);
// Integers of the work list that a pool keeps for it.
size_t b200_attn_prompt_plan_ints(int32_t max_rows);
