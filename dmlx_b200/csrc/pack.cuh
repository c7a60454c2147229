// Batch packing for the blocks of one kernel (pack.cu holds the kernels for batches of any size).
#pragma once
#include <cuda_runtime.h>

#include "dmlx_b200.h"

struct PackOut {
  int *cu_seqlens, *position_ids, *row_to_req, *row_seq, *row_ctx, *last_row;
  uint32_t* token_ids;
};

// Row `row` of the batch, a row of request r, whose rows start at `first`.
__device__ __forceinline__ void pack_row(const b200_pack_desc& d, int r, int first, int row, const uint32_t* __restrict__ prefill_tokens,
                                         const uint32_t* __restrict__ last_token, const PackOut& o) {
  const int j = row - first, pos = d.base_pos + j;
  o.token_ids[row] = d.src_offset >= 0 ? prefill_tokens[d.src_offset + j] : last_token[d.seq_slot];
  o.position_ids[row] = pos;
  o.row_to_req[row] = r;
  o.row_seq[row] = d.seq_slot;
  o.row_ctx[row] = pos + 1;
}

// One block of THREADS threads packs up to THREADS requests.
template <int THREADS>
__device__ __forceinline__ void pack_by_block(const b200_pack_desc* __restrict__ desc, int n_req, const uint32_t* __restrict__ prefill_tokens,
                                              const uint32_t* __restrict__ last_token, int total_rows, const PackOut& o) {
  __shared__ int s_cu[THREADS], s_warp[THREADS / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int count = tid < n_req ? max(desc[tid].count, 0) : 0;
  int inc = count;
#pragma unroll
  for (int k = 1; k < 32; k <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, k);
    if (lane >= k) inc += t;
  }
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  for (int w = 0; w < warp; ++w) inc += s_warp[w];
  s_cu[tid] = inc - count;
  if (tid == 0) o.cu_seqlens[0] = 0;
  if (tid < n_req) {
    o.cu_seqlens[tid + 1] = inc;
    o.last_row[tid] = inc - 1;  // -1 for an empty request that opens the batch
  }
  __syncthreads();
  for (int row = tid; row < total_rows && n_req > 0; row += THREADS) {
    int lo = 0, hi = n_req - 1;  // the last request that starts at `row` or before
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (s_cu[mid] <= row) lo = mid; else hi = mid - 1;
    }
    pack_row(desc[lo], lo, s_cu[lo], row, prefill_tokens, last_token, o);
  }
}
