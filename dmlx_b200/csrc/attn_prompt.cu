// Attention of batches that hold prompt portions: softmax(Q K^T / sqrt(D)) V over the page pool on tcgen05, causal by a context per row.
//
// A group is up to 256 / G consecutive tokens of one sequence (G query heads per kv head); a work item is (group, range of keys, kv head).
// Its rows, (token, head of the GQA group), are two tiles of 128; keys come in blocks of 128 (four pages).  One CTA per SM:
//   warp 8      takes items off the list and loads: Q of the item, then K and V of block after block into a ring (TMA);
//   warp 9      issues the products: S = Q K^T into tensor memory, O += P V with P read from there, where it replaces S;
//   warps 0-3   softmax of tile 0, a thread per row; warps 4-7 the same for tile 1.
// While one tile's scores go through softmax the tensor cores work for the other, so the products (2 x 1024 cycles per block) and the
// exponentials (32768 per block, 16 a cycle) overlap.
//
// P is bf16, and which of a row's weights are exact depends on its scale.  A block's weights are scaled by the row's largest score in that block
// (or 2^-8 of its largest so far, if that is more), so that the block's largest weight is 1; the rows' threads, whose tensor-memory lanes hold the
// sums, rescale them to it behind the weights.  The groups of paged_attn.cu scale by the largest of every 32 keys, anew every 256.  What the
// coarser step costs is made good in the blocks that some row does not see whole, which are all the keys of a short context: there the MMAs also
// get what the rounding of P leaves.  Error against 64 bits, as a multiple of theirs, scores of standard deviation 1 / 4: 200 tokens 0.85 / 0.97,
// 512 over 256 cached 0.98 / 1.00, 683 over 700 0.98 / 1.00, 300 over 3000 1.00 / 1.00.  A scale that may lag its scores by 2^8, the published
// way round most of the rescaling, is 1.02 to 1.2 there.
//
// A group that fits one tile (the decoding requests of the batch are groups of one token) would leave half of the CTA idle: there the two
// softmax groups take the blocks in turn, with sums of their own, and put them together at the end.  Such items are bound by the stream of
// pages, 64 KB per block.
//
// A key that a row does not see has weight 0 there, and 0 times a value that is no finite number is no number: a group's rows share their blocks
// of values, so one such value would reach up to 256 / G tokens ahead of its own.  The softmax threads therefore look through the values of the
// blocks that some row does not see whole (one or two of an item, the rest of its last page among them), clear what is not finite, and a row
// that does see it gets it back at the end.  The look, 64 packed multiply-adds per thread and such block, did not show in the time.
//
// Two tiles of 128 rows: a CTA reads 64 KB of pages per block for 256 rows; one tile would read them twice.  Items go longest first, from a
// counter, since contexts differ.  A batch too small to fill the chip has its key ranges split, f32 partial sums, and a combine pass.
//
// The plan is the published one of attention on this chip: two tiles of rows, P in place of S, a warp each for loads and MMAs.
//
// Measured on one B200, bf16, 32/8 heads of 128, a call over 3 portions of 683 tokens over 700..8000 cached, plan included: 981 us in groups of
// 16 rows per warp on mma.sync (paged_attn.cu), 167 us here (plan 8, the kernel 154); a step of four 512-token portions and 57 decoding requests
// through four layers 7.27 and 5.00 ms with the other kernels as they were (4.4 now).
#include <cuda_bf16.h>

#include <algorithm>

#include "attn_prompt.cuh"
#include "common.h"
#include "launch.cuh"
#include "ptx.cuh"
#include "tma.cuh"

namespace {

constexpr int kBlockKeys = 128, kBlockPages = 4, kTileRows = 128;
constexpr int kThreads = 320;
constexpr float kBelow = 8.f;            // log2 units that the scale of a block may lie below a row's largest score so far
constexpr float kHidden = -1e30f;       // score of a key that a row does not see
constexpr float kNoScale = -1e28f;      // scale of a row that has seen no key: exp2 of any hidden score against it is 0
constexpr uint32_t kPolls = 1u << 21;   // a wait inside a CTA is microseconds
constexpr int kExtraItems = 2048;       // of the work list, beyond one per row: what splitting may add
constexpr int kHdr = 8;                 // {items per kv head, pages per chunk, next item, CTAs done, some range is split}

template <int D>
struct Shape {
  static constexpr int kBoxes = D / 64, kSlotBytes = kBoxes * kBlockKeys * 128, kQBytes = kBoxes * kTileRows * 128;
  static constexpr int kSlots = D == 128 ? 5 : 8;  // K and V blocks in flight: what fits beside Q
};

struct Item {
  int kind;  // 0: end of the list, 1: one tile, 2: two tiles
  int head, seq, first_row, n_rows, ctx0, page_begin, page_end;
  int slot0;  // first partial slot, -1: the rows are written
};

struct Args {
  KvDev d;
  int layer, total_rows, n_q_heads, group;  // group: query heads per kv head
  const int *row_seq, *row_ctx, *group_first, *part_base, *chunk_start;
  const int2* items;  // {group, chunk}, longest first
  int* hdr;
  float *part_o, *part_ml;
  __nv_bfloat16* out;
  float scale_log2;
  bool may_split;  // such batches give 0 for a row whose sum is no number, as the decode kernels do; the others what comes out
};

template <int D>
struct Shared {
  uint64_t full[Shape<D>::kSlots], free[Shape<D>::kSlots], q_full, q_free, s_full[2], p_ready[2], o_full[2], item_full[2], item_free[2], merged[2], drain;
  Item items[2];
  uint32_t cleared[4];  // item n of this CTA had values cleared: [n % 4] is n + 1 (a softmax group is never three items ahead of the other)
  uint32_t tmem;
  float m[2][kTileRows], l[2][kTileRows];
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Bounded; once a wait has run out nothing is waited for any more, so that every role comes to its end.
__device__ __forceinline__ void wait(uint64_t* bar, uint32_t parity, bool& ok) {
  if (!ok) return;
  for (uint32_t i = 0; i < kPolls; ++i)
    if (ptx::mbar_try_wait(bar, parity)) return;
  ok = false;
}
// Two at a time.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\tfma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tadd.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// ---- the work list ---------------------------------------------------------------------------------------------
template <bool MAX>
__device__ __forceinline__ int scan(int v, int* warp_buf) {  // inclusive, over the block
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v = MAX ? max(v, t) : v + t;
  }
  __syncthreads();
  if (lane == 31) warp_buf[warp] = v;
  __syncthreads();
  if (warp == 0) {
    int w = lane < (int)(blockDim.x >> 5) ? warp_buf[lane] : (MAX ? -1 : 0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w = MAX ? max(w, t) : w + t;
    }
    warp_buf[lane] = w;
  }
  __syncthreads();
  if (warp > 0) v = MAX ? max(v, warp_buf[warp - 1]) : v + warp_buf[warp - 1];
  return v;
}

constexpr int kLengths = 6;  // blocks per chunk: the whole range, 64, 32, 16, 8, 4
__device__ __forceinline__ int chunk_blocks(int k) { return k == 0 ? 1 << 24 : 128 >> k; }

// Rows that continue one another (same sequence, context one longer) form runs, which are cut into groups of q_tokens.  may_split: the
// key ranges may be cut into chunks; the length is the one with the smallest estimated time among those whose partial sums fit.
// old_limit > 0: batches of this kind are refused (CAPACITY) where groups of old_tokens rows in chunks of 8 pages would need more partial
// slots than that, the documented limit of the pool's scratch.
__global__ void __launch_bounds__(1024) prompt_plan_kernel(const int* row_seq, const int* row_ctx, int total_rows, int page_size,
                                                           int q_tokens, int tile_tokens, int heads, int workers, int may_split, int max_slots,
                                                           int old_tokens, int* __restrict__ chunk_start, int* __restrict__ group_first,
                                                           int* __restrict__ part_base, int* __restrict__ row_group, int2* __restrict__ items,
                                                           int* __restrict__ hdr, int* __restrict__ err) {
  after_previous();
  __shared__ int warp_buf[32], hist[256], carry[4];
  __shared__ int s_max[kLengths], s_items[kLengths], s_total[kLengths], s_slots[kLengths], s_old, s_pick, s_longest;
  __shared__ int2 s_group[1024];  // {rows, blocks} of the first groups
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid < 4) carry[tid] = tid == 0 ? -1 : 0;
  if (tid < kLengths) { s_max[tid] = 0; s_items[tid] = 0; s_total[tid] = 0; s_slots[tid] = 0; }
  if (tid == 0) { s_old = 0; s_longest = 0; s_pick = 0; }
  if (tid < 256) hist[tid] = 0;
  __syncthreads();
  // four neighbouring rows a thread, so that one round of scans is enough for 1024 rows in 256 threads and 4096 in 1024
  constexpr int kRows = 4;
  for (int base = 0; base < total_rows; base += kRows * blockDim.x) {
    const int i0 = base + kRows * tid;
    int seq[kRows + 1], ctx[kRows + 1], run[kRows];
#pragma unroll
    for (int k = 0; k <= kRows; ++k) {
      const int i = i0 + k - 1;
      const bool there = i >= 0 && i < total_rows;
      seq[k] = there ? row_seq[i] : -1;
      ctx[k] = there ? row_ctx[i] : 0;
    }
    int last_start = -1;
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
      const int i = i0 + k;
      const bool joins = i > 0 && seq[k + 1] == seq[k] && ctx[k + 1] == ctx[k] + 1;
      if (i < total_rows && !joins) last_start = i;
      run[k] = last_start;
    }
    const int starts = scan<true>(last_start, warp_buf);  // of this thread's rows and those before
    int before = __shfl_up_sync(0xffffffffu, starts, 1);
    if (lane == 0) before = tid > 0 ? warp_buf[(tid >> 5) - 1] : -1;
    before = max(before, carry[0]);
    int heads = 0;
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
      run[k] = max(run[k], before);
      heads += i0 + k < total_rows && (i0 + k - run[k]) % q_tokens == 0 ? 1 : 0;
    }
    __syncthreads();  // (the scans share a buffer)
    const int heads_incl = scan<false>(heads, warp_buf);
    int gid = carry[1] + heads_incl - heads - 1, old = 0;
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
      const int i = i0 + k;
      if (i >= total_rows) break;
      const bool head = (i - run[k]) % q_tokens == 0;
      gid += head ? 1 : 0;
      row_group[i] = gid;
      if (head) group_first[gid] = i;
      if (old_tokens > 0) {  // slots of this row as the limit counts them: by the context of its group's last row
        const int last = (i - run[k]) / old_tokens * old_tokens + old_tokens - 1 + run[k];
        int end = i;
        while (end < last && end + 1 < total_rows && row_seq[end + 1] == row_seq[end] && row_ctx[end + 1] == row_ctx[end] + 1) ++end;
        old += ((max(row_ctx[end], 0) + page_size - 1) / page_size + 7) / 8;
      }
    }
    if (old_tokens > 0) {
      old = __reduce_add_sync(0xffffffffu, old);
      if (lane == 0) atomicAdd(&s_old, old);
    }
    __syncthreads();
    if (tid == blockDim.x - 1) { carry[0] = max(starts, carry[0]); carry[1] += heads_incl; }
    __syncthreads();
  }
  const int n_groups = carry[1];
  if (tid == 0) group_first[n_groups] = total_rows;
  __syncthreads();
  auto look = [&](int g) {
    const int first = group_first[g], next = group_first[g + 1], pages = (max(row_ctx[next - 1], 0) + page_size - 1) / page_size;
    return make_int2(next - first, (pages + kBlockPages - 1) / kBlockPages);
  };
  for (int base = 0; base < n_groups; base += blockDim.x) {
    const int g = base + tid;
    const bool valid = g < n_groups;
    const int2 rb = valid ? look(g) : make_int2(0, 0);
    if (base == 0) s_group[tid] = rb;
    const int longest = __reduce_max_sync(0xffffffffu, rb.y);
    if (lane == 0) atomicMax(&s_longest, longest);
    if (may_split) {
      // eighths of a block: a two-tile block counts 8, a one-tile block 5; an item's fill, drain and epilogue 10
      const int unit = rb.x > tile_tokens ? 8 : 5;
#pragma unroll
      for (int k = 0; k < kLengths; ++k) {
        const int len = chunk_blocks(k), chunks = valid ? max((rb.y + len - 1) / len, 1) : 0;
        const int top = __reduce_max_sync(0xffffffffu, valid ? unit * min(rb.y, len) + 10 : 0), items_k = __reduce_add_sync(0xffffffffu, chunks);
        const int total = __reduce_add_sync(0xffffffffu, valid ? unit * rb.y + 10 * chunks : 0), slots = __reduce_add_sync(0xffffffffu, chunks > 1 ? chunks * rb.x : 0);
        if (lane == 0) {
          atomicMax(&s_max[k], top);
          atomicAdd(&s_items[k], items_k);
          atomicAdd(&s_total[k], total);
          atomicAdd(&s_slots[k], slots);
        }
      }
    }
  }
  __syncthreads();
  if (tid == 0 && may_split) {
    int pick = 0;
    long long best = 0;
    for (int k = 0; k < kLengths; ++k) {
      if (k > 0 && (s_slots[k] > max_slots || s_items[k] > total_rows + kExtraItems)) continue;
      const long long share = (long long)s_total[k] * heads / workers;
      // a combine pass, and the partial sums' way to memory and back
      const long long extra = k > 0 && s_slots[k] > 0 ? 24 + (long long)(s_slots[k] / 64) : 0;
      const long long cost = max((long long)s_max[k], share + s_max[k] / 2) + extra;
      if (k == 0 || cost < best) { best = cost; pick = k; }
    }
    s_pick = pick;
  }
  __syncthreads();
  const int len = chunk_blocks(s_pick), longest = max(s_longest, 1);
  auto bucket = [&](int blocks) { return 255 - min(255, (int)((long long)blocks * 255 / longest)); };
  for (int base = 0; base < n_groups; base += blockDim.x) {
    const int g = base + tid;
    int chunks = 0, slots = 0;
    if (g < n_groups) {
      const int2 rb = base == 0 ? s_group[g] : look(g);
      chunks = max((rb.y + len - 1) / len, 1);
      slots = chunks > 1 ? chunks * rb.x : 0;
      for (int c = 0; c < chunks; ++c) atomicAdd(&hist[bucket(min(len, rb.y - c * len))], 1);
    }
    const int c_incl = scan<false>(chunks, warp_buf), s_incl = scan<false>(slots, warp_buf);
    if (g < n_groups) {
      chunk_start[g] = carry[2] + c_incl - chunks;
      part_base[g] = carry[3] + s_incl - slots;
    }
    __syncthreads();
    if (tid == blockDim.x - 1) { carry[2] += c_incl; carry[3] += s_incl; }
    __syncthreads();
  }
  // longest first: a counting sort by length
  const int h = tid < 256 ? hist[tid] : 0, h_incl = scan<false>(h, warp_buf);
  __syncthreads();
  if (tid < 256) hist[tid] = h_incl - h;
  __syncthreads();
  for (int g = tid; g < n_groups; g += blockDim.x) {
    const int blocks = g < (int)blockDim.x ? s_group[g].y : look(g).y, chunks = max((blocks + len - 1) / len, 1);
    for (int c = 0; c < chunks; ++c) items[atomicAdd(&hist[bucket(min(len, blocks - c * len))], 1)] = make_int2(g, c);
  }
  if (tid == 0) {
    const bool refused = old_tokens > 0 && s_old > max_slots;
    if (refused) *err = B200_ERR_CAPACITY;
    chunk_start[n_groups] = carry[2];
    hdr[0] = refused ? 0 : carry[2];
    hdr[1] = len >= 1 << 24 ? 1 << 24 : len * kBlockPages;
    hdr[4] = refused ? 0 : (carry[3] > 0 ? 1 : 0);
  }
}

// ---- values that are not finite ------------------------------------------------------------------------------------
// Pieces of 16 bytes from `first` on, one for each thread of a tile in turn, in every box of a block of values: what is not finite becomes 0.
template <int D>
__device__ __noinline__ void clear_pieces(uint4* v, int first, int pieces, uint32_t* mark, uint32_t value) {
  auto clear = [](uint32_t w) { return ((w & 0x7F80u) == 0x7F80u ? 0u : w & 0xFFFFu) | ((w & 0x7F800000u) == 0x7F800000u ? 0u : w & 0xFFFF0000u); };
  for (int i = first; i < pieces; i += kTileRows)
    for (int x = 0; x < Shape<D>::kBoxes; ++x) {
      const uint4 q = v[x * (kBlockKeys * 8) + i], z = make_uint4(clear(q.x), clear(q.y), clear(q.z), clear(q.w));
      if (q.x == z.x && q.y == z.y && q.z == z.z && q.w == z.w) continue;
      *reinterpret_cast<volatile uint32_t*>(mark) = value;
      __threadfence_block();  // (who finds the values cleared finds the mark)
      v[x * (kBlockKeys * 8) + i] = z;
    }
}
// (Written out where it is used, in loops that stay loops: as a function it cost the whole kernel 9 %, for the registers that a call takes.)
// The cleared values that a row sees, onto its columns c_begin..c_end as they were written.
template <int D>
__device__ __forceinline__ void add_cleared(const Args& a, const Item& it, int ctx, int c_begin, int c_end, __nv_bfloat16* row, float* partial) {
  const int begin = it.page_begin * 32, first = max(begin, begin + (it.ctx0 - begin) / kBlockKeys * kBlockKeys);
#pragma unroll 1
  for (int key = first; key < min(ctx, it.page_end * 32); ++key) {
    const size_t page = (size_t)a.layer * a.d.n_pages + a.d.block_table[(size_t)it.seq * a.d.max_pages_per_seq + key / 32];
    const __nv_bfloat16* v = reinterpret_cast<const __nv_bfloat16*>(a.d.v_pool) + ((page * a.d.n_kv_heads + it.head) * 32 + key % 32) * D;
#pragma unroll 1
    for (int c = c_begin; c < c_end; ++c) {
      const float value = __bfloat162float(v[c]);
      if (isfinite(value)) continue;
      if (row) row[c] = __float2bfloat16(__bfloat162float(row[c]) + value);
      else partial[c] += value;
    }
  }
}

// A tile's sums, rescaled by its rows' threads.
template <int D>
__device__ __forceinline__ void rescale(uint32_t t_o, float corr) {
#pragma unroll
  for (int c = 0; c < D; c += 32) {
    uint32_t u[32];
    ptx::tmem_ld32(t_o + c, u);
    ptx::tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 32; ++i) u[i] = __float_as_uint(__uint_as_float(u[i]) * corr);
    ptx::tmem_st32(t_o + c, u);
  }
}
// A row's sums: their scale, the largest score so far (both log2), the sum of its weights.
struct Row {
  float m = kNoScale, most = kNoScale, l = 0.f;
  // Takes the scale of a block whose largest score is `top`; returns the factor of what was summed before.
  __device__ __forceinline__ float next(float top) {
    most = fmaxf(most, top);
    const float scale = fmaxf(top, most - kBelow), corr = ex2(m - scale);
    m = scale;
    return corr;
  }
};
// One block of keys, some of which some rows of the tile do not see: the scores from tensor memory, P into place of the scores, and what its rounding leaves behind it, 64 columns further on.  The blocks that all rows see take the same steps in the kernel itself.
template <int D>
__device__ __noinline__ Row partly_seen_block(uint32_t t_s, uint32_t t_o, int seen, bool first, float scale_log2, Row r) {
  float s[kBlockKeys];
  {
    uint32_t u[4][32];
#pragma unroll
    for (int c = 0; c < 4; ++c) ptx::tmem_ld32(t_s + c * 32, u[c]);
    ptx::tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < kBlockKeys; ++i) s[i] = i < seen ? fmaxf(__uint_as_float(u[i >> 5][i & 31]), kHidden) : kHidden;
  }
  float mx[4] = {kHidden, kHidden, kHidden, kHidden};
#pragma unroll
  for (int i = 0; i < kBlockKeys; ++i) mx[i & 3] = fmaxf(mx[i & 3], s[i]);
  const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * scale_log2;
  const float corr = r.next(top);
  const float2 k2 = make_float2(scale_log2, scale_log2), m2 = make_float2(-r.m, -r.m);
  float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t p[16], left[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float2 x = fma2(make_float2(s[c * 32 + 2 * i], s[c * 32 + 2 * i + 1]), k2, m2), e = make_float2(ex2(x.x), ex2(x.y));
      sum[i & 1] = add2(sum[i & 1], e);
      p[i] = pack2(e.x, e.y);
      const float2 rest = add2(e, make_float2(-__uint_as_float(p[i] << 16), -__uint_as_float(p[i] & 0xFFFF0000u)));
      left[i] = pack2(rest.x, rest.y);
    }
    ptx::tmem_st16(t_s + c * 16, p);
    ptx::tmem_st16(t_s + 64 + c * 16, left);
  }
  const float2 both = add2(sum[0], sum[1]);
  if (!first) rescale<D>(t_o, corr);
  r.l = fmaf(r.l, corr, both.x + both.y);
  return r;
}

// ---- the kernel ---------------------------------------------------------------------------------------------------
template <int D>
__global__ void __launch_bounds__(kThreads, 1)
    prompt_attn_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap, const __grid_constant__ CUtensorMap qmap, const __grid_constant__ Args a) {
  wait_previous();
  using Z = Shape<D>;
  extern __shared__ __align__(1024) unsigned char smem[];  // (there is no room for a base that has to be rounded up)
  unsigned char* qbuf = smem;                        // [tile][box][128 rows][128 B]
  unsigned char* ring = smem + 2 * Z::kQBytes;       // [slot][box][128 keys][128 B], K and V in turn
  Shared<D>& sh = *reinterpret_cast<Shared<D>*>(ring + Z::kSlots * Z::kSlotBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < Z::kSlots; ++s) { ptx::mbar_init(&sh.full[s], 1); ptx::mbar_init(&sh.free[s], 1); }
    ptx::mbar_init(&sh.q_full, 1);
    ptx::mbar_init(&sh.q_free, 1);
    for (int t = 0; t < 2; ++t) {
      ptx::mbar_init(&sh.s_full[t], 1);
      ptx::mbar_init(&sh.p_ready[t], kTileRows);
      ptx::mbar_init(&sh.o_full[t], 1);
      ptx::mbar_init(&sh.item_full[t], 1);
      ptx::mbar_init(&sh.item_free[t], 9);
      ptx::mbar_init(&sh.merged[t], 2 * kTileRows);
    }
    ptx::mbar_init(&sh.drain, 1);
    for (int i = 0; i < 4; ++i) sh.cleared[i] = 0;
    ptx::mbar_fence_init();
  }
  if (warp == 9) {
    ptx::tmem_alloc(&sh.tmem, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem = sh.tmem;
  auto tmem_s = [&](int t) { return tmem + (uint32_t)(t * 128); };
  auto tmem_o = [&](int t) { return tmem + (uint32_t)(256 + t * D); };
  bool ok = (ptx::smem_u32(smem) & 1023) == 0;

  if (warp == 8) {
    // ---- loads; the warp stays together, lane 0 issues ----
    const int n_items = a.hdr[0], chunk_pages = a.hdr[1];
    int slot = 0, loaded = 0;
    uint32_t phase = 0, used = 0;  // bits per slot: parity of its next load; whether it ever had one
    auto wait_all = [&](uint64_t* bar, uint32_t parity) {
      wait(bar, parity, ok);
      ok = __all_sync(0xffffffffu, ok);
    };
    for (uint32_t n = 0;; ++n) {
      int idx = 0;
      if (lane == 0) idx = atomicAdd(&a.hdr[2], 1);
      idx = __shfl_sync(0xffffffffu, idx, 0);
      const int b = n & 1u;
      wait_all(&sh.item_free[b], ((n >> 1) & 1u) ^ 1u);
      Item it{};
      if (ok && idx < n_items * a.d.n_kv_heads) {
        const int2 gc = a.items[idx / a.d.n_kv_heads];
        it.head = idx % a.d.n_kv_heads;
        it.first_row = a.group_first[gc.x];
        it.n_rows = a.group_first[gc.x + 1] - it.first_row;
        it.seq = a.row_seq[it.first_row];
        it.ctx0 = a.row_ctx[it.first_row];
        const int pages = (max(it.ctx0 + it.n_rows - 1, 0) + a.d.page_size - 1) / a.d.page_size;
        it.page_begin = gc.y * chunk_pages;
        it.page_end = min((long long)it.page_begin + chunk_pages, (long long)pages);
        it.slot0 = a.chunk_start[gc.x + 1] - a.chunk_start[gc.x] > 1 ? a.part_base[gc.x] + gc.y * it.n_rows : -1;
        it.kind = it.n_rows * a.group > kTileRows ? 2 : 1;
      }
      if (lane == 0) {
        sh.items[b] = it;
        ptx::mbar_arrive(&sh.item_full[b]);
      }
      __syncwarp();
      if (it.kind == 0) break;
      if (it.page_end <= it.page_begin) continue;  // (rows without a context: written as zeros)
      wait_all(&sh.q_free, (loaded & 1u) ^ 1u);
      if (!ok) continue;  // (the next round ends the list)
      ++loaded;
      if (lane == 0) {
        ptx::mbar_expect_tx(&sh.q_full, it.kind * Z::kQBytes);
        for (int t = 0; t < it.kind; ++t)
          for (int x = 0; x < Z::kBoxes; ++x)
            ptx::tma_load_3d(qbuf + t * Z::kQBytes + x * kTileRows * 128, &qmap, x * 64, it.head * a.group, it.first_row + t * (kTileRows / a.group), &sh.q_full);
      }
      // lanes hold the ids of 32 pages, and of the 32 behind them
      const int* table = a.d.block_table + (size_t)it.seq * a.d.max_pages_per_seq;
      int ids = it.page_begin + lane < it.page_end ? table[it.page_begin + lane] : 0, more = 0;
      for (int pg = it.page_begin; pg < it.page_end && ok; pg += kBlockPages) {
        const int rel = pg - it.page_begin;
        if ((rel & 31) == 0) {
          if (rel > 0) ids = more;
          more = pg + 32 + lane < it.page_end ? table[pg + 32 + lane] : 0;
        }
        const int pages = min(kBlockPages, it.page_end - pg);
        int row0[kBlockPages];
#pragma unroll
        for (int p = 0; p < kBlockPages; ++p) row0[p] = (__shfl_sync(0xffffffffu, ids, (rel & 31) + p) * a.d.n_kv_heads + it.head) * 32;
#pragma unroll
        for (int kv = 0; kv < 2; ++kv) {
          wait_all(&sh.free[slot], ((phase >> slot) & 1u) ^ 1u);
          if (!ok) break;
          if (lane == 0) {
            ptx::mbar_expect_tx(&sh.full[slot], pages * Z::kBoxes * 4096);
            unsigned char* dst = ring + slot * Z::kSlotBytes;
            for (int x = 0; x < Z::kBoxes; ++x)
              for (int p = 0; p < pages; ++p)
                ptx::tma_load_3d(dst + x * kBlockKeys * 128 + p * 4096, kv ? &vmap : &kmap, x * 64, row0[p], a.layer, &sh.full[slot]);
          }
          __syncwarp();
          phase ^= 1u << slot;
          used |= 1u << slot;
          if (++slot == Z::kSlots) slot = 0;
        }
      }
    }
    if (!ok) {  // leave no copy in flight behind
      bool drained = true;
      if (loaded > 0) wait(&sh.q_full, (loaded - 1) & 1u, drained);
      for (int s = 0; s < Z::kSlots; ++s)
        if (used >> s & 1u) wait(&sh.full[s], ((phase >> s) & 1u) ^ 1u, drained);
    }
    if (lane == 0) {  // the last CTA leaves the counters as it found them
      if (atomicAdd(&a.hdr[3], 1) == (int)gridDim.x - 1) { a.hdr[2] = 0; a.hdr[3] = 0; }
    }
  } else if (warp == 9) {
    if (ptx::elect_one()) {
      // ---- products ----
      const uint32_t id_s = ptx::umma_idesc_bf16(kTileRows, kBlockKeys), id_o = ptx::umma_idesc_bf16(kTileRows, D) | ptx::kUmmaBMn;
      const uint64_t q_desc = ptx::umma_desc_k_sw128(ptx::smem_u32(qbuf)), k_desc = ptx::umma_desc_k_sw128(ptx::smem_u32(ring));
      const uint64_t v_desc = ptx::umma_desc_mn_sw128(ptx::smem_u32(ring), kBlockKeys * 128);
      uint32_t phase = 0, n_p[2] = {0, 0}, n_q = 0;  // ring parities by slot; softmaxes waited for; items with keys
      int slot0 = 0;                                 // ring slot of the item's first block
      auto slot_of = [&](int k) { return (slot0 + k) % Z::kSlots; };  // k-th load of the item: K of block j is 2 j, V is 2 j + 1
      auto arrived = [&](int k) {
        const int s = slot_of(k);
        wait(&sh.full[s], (phase >> s) & 1u, ok);
        phase ^= 1u << s;
        ptx::tc_fence_after_sync();
      };
      for (uint32_t n = 0;; ++n) {
        const int b = n & 1u;
        wait(&sh.item_full[b], (n >> 1) & 1u, ok);
        if (!ok) break;
        const int kind = sh.items[b].kind, n_pages = sh.items[b].page_end - sh.items[b].page_begin;
        const int first_partly = (sh.items[b].ctx0 - sh.items[b].page_begin * 32) / kBlockKeys;  // the first block that some row does not see whole
        ptx::mbar_arrive(&sh.item_free[b]);
        if (kind == 0) break;
        if (n_pages <= 0) continue;
        const int nb = (n_pages + kBlockPages - 1) / kBlockPages;
        wait(&sh.q_full, n_q & 1u, ok);
        ++n_q;
        ptx::tc_fence_after_sync();
        auto qk = [&](int t, int j, int q_tile) {  // S of softmax group t from block j
          const uint64_t k0 = k_desc + (uint64_t)(slot_of(2 * j) * (Z::kSlotBytes >> 4)), q0 = q_desc + (uint64_t)(q_tile * (Z::kQBytes >> 4));
#pragma unroll
          for (int k = 0; k < D / 16; ++k) {
            const uint32_t at = (uint32_t)((k >> 2) * (kBlockKeys * 128 >> 4) + (k & 3) * 2);
            ptx::umma_bf16(tmem_s(t), q0 + at, k0 + at, id_s, k > 0 ? 1u : 0u);
          }
          ptx::umma_commit(&sh.s_full[t]);
        };
        auto pv = [&](int t, int j, bool first) {
          const uint64_t v0 = v_desc + (uint64_t)(slot_of(2 * j + 1) * (Z::kSlotBytes >> 4));
          const int steps = min(kBlockPages, n_pages - j * kBlockPages) * 2;  // (what lies behind the last page is not read)
          wait(&sh.p_ready[t], n_p[t] & 1u, ok);
          ++n_p[t];
          ptx::tc_fence_after_sync();
          if (steps == 2 * kBlockPages) {
#pragma unroll
            for (int k = 0; k < 2 * kBlockPages; ++k)
              ptx::umma_bf16_tmem_a(tmem_o(t), tmem_s(t) + k * 8, v0 + k * (2048 >> 4), id_o, first && k == 0 ? 0u : 1u);
          } else {
            for (int k = 0; k < steps; ++k)
              ptx::umma_bf16_tmem_a(tmem_o(t), tmem_s(t) + k * 8, v0 + k * (2048 >> 4), id_o, first && k == 0 ? 0u : 1u);
          }
          if (j >= first_partly)
            for (int k = 0; k < steps; ++k) ptx::umma_bf16_tmem_a(tmem_o(t), tmem_s(t) + 64 + k * 8, v0 + k * (2048 >> 4), id_o, 1u);
        };
        if (kind == 2) {
          arrived(0);
          qk(0, 0, 0);
          qk(1, 0, 1);
          ptx::umma_commit(&sh.free[slot_of(0)]);
          if (nb == 1) ptx::umma_commit(&sh.q_free);
          for (int j = 0; j < nb && ok; ++j) {
            const bool last = j + 1 == nb;
            arrived(2 * j + 1);
            pv(0, j, j == 0);
            if (last) {
              ptx::umma_commit(&sh.o_full[0]);
            } else {
              arrived(2 * j + 2);
              qk(0, j + 1, 0);
            }
            pv(1, j, j == 0);
            ptx::umma_commit(&sh.free[slot_of(2 * j + 1)]);
            if (last) {
              ptx::umma_commit(&sh.o_full[1]);
            } else {
              qk(1, j + 1, 1);
              ptx::umma_commit(&sh.free[slot_of(2 * j + 2)]);
              if (j + 2 == nb) ptx::umma_commit(&sh.q_free);
            }
          }
        } else {
          for (int j = 0; j < min(nb, 2); ++j) {
            arrived(2 * j);
            qk(j, j, 0);
            ptx::umma_commit(&sh.free[slot_of(2 * j)]);
          }
          if (nb <= 2) ptx::umma_commit(&sh.q_free);
          for (int j = 0; j < nb && ok; ++j) {
            const int t = j & 1;
            arrived(2 * j + 1);
            pv(t, j, j < 2);
            ptx::umma_commit(&sh.free[slot_of(2 * j + 1)]);
            if (j + 2 < nb) {
              arrived(2 * j + 4);
              qk(t, j + 2, 0);
              ptx::umma_commit(&sh.free[slot_of(2 * j + 4)]);
              if (j + 3 == nb) ptx::umma_commit(&sh.q_free);
            } else {
              ptx::umma_commit(&sh.o_full[t]);
            }
          }
        }
        slot0 = (slot0 + 2 * nb) % Z::kSlots;
      }
      const bool fine = ok;
      ok = true;
      ptx::umma_commit(&sh.drain);
      wait(&sh.drain, 0, ok);
      ok = ok && fine;
    }
    __syncwarp();
  } else if (warp < 8) {
    // ---- softmax: a thread per row ----
    const int g = warp >> 2, row = (warp & 3) * 32 + lane;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    uint32_t n_s = 0, n_o[2] = {0, 0}, n_m = 0, loads = 0;  // loads: of the items before
    // Clears what is not finite among the values of a block (the group's threads a 16-byte piece each, in turn).
    auto clear_values = [&](uint32_t load, int pages, uint32_t n) {
      wait(&sh.full[load % Z::kSlots], (load / Z::kSlots) & 1u, ok);
      uint4* v = reinterpret_cast<uint4*>(ring + (load % Z::kSlots) * Z::kSlotBytes);
      const __nv_bfloat162 zero = __floats2bfloat162_rn(0.f, 0.f);
      __nv_bfloat162 seen = zero;  // 0 as long as every factor is finite
      for (int i = row; i < pages * 256; i += kTileRows)
#pragma unroll
        for (int x = 0; x < Z::kBoxes; ++x) {
          uint4 q = v[x * (kBlockKeys * 8) + i];
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
          for (int e = 0; e < 4; ++e) seen = __hfma2(h[e], zero, seen);
        }
      if (__any_sync(0xffffffffu, __low2float(seen) != 0.f || __high2float(seen) != 0.f)) {
        clear_pieces<D>(v, row, pages * 256, &sh.cleared[n & 3u], n + 1);
        ptx::fence_proxy_async_smem();
        __syncwarp();
      }
    };
    for (uint32_t n = 0;; ++n) {
      const int b = n & 1u;
      wait(&sh.item_full[b], (n >> 1) & 1u, ok);
      __syncwarp();
      if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      const Item it = sh.items[b];
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&sh.item_free[b]);
      if (it.kind == 0) break;
      const bool shared_tile = it.kind == 1;  // both groups work on tile 0, blocks in turn
      const int at = (shared_tile ? 0 : g * kTileRows) + row, tok = at / a.group, head = at - tok * a.group;
      const bool on = tok < it.n_rows;
      const int ctx = on ? it.ctx0 + tok : 0;
      const int n_pages = it.page_end - it.page_begin, nb = n_pages > 0 ? (n_pages + kBlockPages - 1) / kBlockPages : 0;
      Row r;
      const int j0 = shared_tile ? g : 0, step = shared_tile ? 2 : 1;
      for (int j = j0; j < nb; j += step) {
        wait(&sh.s_full[g], n_s & 1u, ok);
        ++n_s;
        ptx::tc_fence_after_sync();
        __syncwarp();
        const int tok0 = (it.page_begin + j * kBlockPages) * 32;
        const bool partly = tok0 + kBlockKeys > it.ctx0;  // some row does not see all of the block's keys
        if (partly) {
          clear_values(loads + 2 * j + 1, min(kBlockPages, n_pages - j * kBlockPages), n);
          r = partly_seen_block<D>(tmem_s(g) + lanes, tmem_o(g) + lanes, ctx - tok0, j == j0, a.scale_log2, r);
        } else {
          float s[kBlockKeys];
          {
            uint32_t u[4][32];
#pragma unroll
            for (int c = 0; c < 4; ++c) ptx::tmem_ld32(tmem_s(g) + lanes + c * 32, u[c]);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < kBlockKeys; ++i) s[i] = __uint_as_float(u[i >> 5][i & 31]);
          }
          float mx[4] = {kHidden, kHidden, kHidden, kHidden};
#pragma unroll
          for (int i = 0; i < kBlockKeys; ++i) mx[i & 3] = fmaxf(mx[i & 3], s[i]);
          const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * a.scale_log2;
          const float corr = r.next(top);  // (by the row's own scores, whatever its neighbours do)
          const float2 k2 = make_float2(a.scale_log2, a.scale_log2), m2 = make_float2(-r.m, -r.m);
          auto weigh = [&]() {  // P, and its sum
            float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              uint32_t p[32];
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                const float2 x = fma2(make_float2(s[c * 64 + 2 * i], s[c * 64 + 2 * i + 1]), k2, m2);
                const float2 e = make_float2(ex2(x.x), ex2(x.y));
                sum[i & 1] = add2(sum[i & 1], e);
                p[i] = pack2(e.x, e.y);
              }
              ptx::tmem_st32(tmem_s(g) + lanes + c * 32, p);
            }
            const float2 both = add2(sum[0], sum[1]);
            return both.x + both.y;
          };
          float total = weigh();
          // A score that is no number weighs nothing, as a hidden one: it shows in the sum, and the block is done again without it.
          if (__any_sync(0xffffffffu, total != total)) {
#pragma unroll
            for (int i = 0; i < kBlockKeys; ++i) s[i] = fmaxf(s[i], kHidden);
            total = weigh();
          }
          r.l = fmaf(r.l, corr, total);
          if (j != j0) rescale<D>(tmem_o(g) + lanes, corr);  // (the scores' arrival says that the product before them is done)
        }
        ptx::tmem_st_wait();
        ptx::tc_fence_before_sync();
        ptx::mbar_arrive(&sh.p_ready[g]);
      }
      // ---- the rows leave: all columns of this thread's row, or half of them from both groups' sums ----
      const bool both = shared_tile && nb > 1;
      float w0 = 1.f, w1 = 0.f, m = r.m, l = r.l;
      if (nb > 0 && (j0 < nb || both)) wait(&sh.o_full[g], n_o[g] & 1u, ok);
      if (both) {
        wait(&sh.o_full[g ^ 1], n_o[g ^ 1] & 1u, ok);
        sh.m[g][row] = m;
        sh.l[g][row] = l;
        ptx::mbar_arrive(&sh.merged[0]);
        wait(&sh.merged[0], n_m & 1u, ok);
        const float mo = sh.m[g ^ 1][row], lo = sh.l[g ^ 1][row], mm = fmaxf(m, mo), own = ex2(m - mm), other = ex2(mo - mm);
        l = own * l + other * lo;
        m = mm;
        w0 = g == 0 ? own : other;
        w1 = g == 0 ? other : own;
      }
      // phases of the barriers, whether this thread waited or not
      if (shared_tile) {
        if (nb > 0) ++n_o[0];
        if (nb > 1) ++n_o[1];
      } else if (nb > 0) {
        ++n_o[0];
        ++n_o[1];
      }
      ptx::tc_fence_after_sync();
      __syncwarp();
      const bool writes = !shared_tile || both || g == 0;
      if (writes) {
        const int c_begin = both ? g * (D / 2) : 0, c_end = both ? c_begin + D / 2 : D, tile = shared_tile ? 0 : g;
        const bool direct = it.slot0 < 0;
        const float inv = direct ? (l > 0.f ? 1.0f / l : 0.f) : 1.f;
        const bool drop = direct && a.may_split && !(l > 0.f);
        const bool cleared = nb > 0 && l > 0.f && *reinterpret_cast<const volatile uint32_t*>(&sh.cleared[n & 3u]) == n + 1;
        const size_t qh = (size_t)it.head * a.group + head;
        __nv_bfloat16* dst = a.out + ((size_t)(it.first_row + tok) * a.n_q_heads + qh) * D;
        const size_t pidx = (size_t)(max(it.slot0, 0) + tok) * a.n_q_heads + qh;
        float* po = a.part_o + pidx * D;
        if (on && !direct && c_begin == 0) { a.part_ml[pidx * 2] = m; a.part_ml[pidx * 2 + 1] = l; }
#pragma unroll 1
        for (int c = c_begin; c < c_end; c += 32) {
          float x[32];
          if (nb > 0) {
            uint32_t u[32];
            ptx::tmem_ld32(tmem_o(tile) + lanes + c, u);
            if (both) {
              uint32_t v[32];
              ptx::tmem_ld32(tmem_o(1) + lanes + c, v);
              ptx::tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) x[i] = fmaf(w0, __uint_as_float(u[i]), w1 * __uint_as_float(v[i])) * inv;
            } else {
              ptx::tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) x[i] = __uint_as_float(u[i]) * inv;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) x[i] = 0.f;
          }
          if (drop) {
#pragma unroll
            for (int i = 0; i < 32; ++i) x[i] = 0.f;
          }
          if (on) {
            if (direct) {
#pragma unroll
              for (int i = 0; i < 32; i += 8)
                *reinterpret_cast<uint4*>(dst + c + i) = make_uint4(pack2(x[i], x[i + 1]), pack2(x[i + 2], x[i + 3]), pack2(x[i + 4], x[i + 5]), pack2(x[i + 6], x[i + 7]));
            } else {
#pragma unroll
              for (int i = 0; i < 32; i += 4) *reinterpret_cast<float4*>(po + c + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
            }
          }
        }
        if (cleared && on) add_cleared<D>(a, it, ctx, c_begin, c_end, direct ? dst : nullptr, po);
      }
      if (both) {  // neither group's sums are written again before the other has read them
        ptx::tc_fence_before_sync();
        ptx::mbar_arrive(&sh.merged[1]);
        wait(&sh.merged[1], n_m & 1u, ok);
        ptx::tc_fence_after_sync();
        ++n_m;
      }
      loads += 2 * nb;
    }
  }
  if (!ok) atomicExch(a.d.state + ST_ATTN_ERR, B200_ERR_DEVICE_FLAGGED);
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  if (warp == 9) ptx::tmem_dealloc(tmem, 512);
}

// A warp per (row, query head): merges the chunks of rows whose key range was split.
template <int D>
__global__ void __launch_bounds__(256) prompt_combine_kernel(Args a, const int* row_group) {
  after_previous();
  const int u = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (u >= a.total_rows * a.n_q_heads || a.hdr[4] == 0 || a.d.state[ST_ATTN_ERR] != 0) return;
  const int row = u / a.n_q_heads, qh = u - row * a.n_q_heads;
  const int grp = row_group[row], first = a.group_first[grp], size = a.group_first[grp + 1] - first, n = a.chunk_start[grp + 1] - a.chunk_start[grp];
  if (n <= 1) return;
  const size_t slot0 = (size_t)a.part_base[grp] + (row - first);
  constexpr int V = D / 32;
  float mm = kNoScale, ll = 0.f, acc[V] = {};
  for (int c = 0; c < n; ++c) mm = fmaxf(mm, a.part_ml[((slot0 + (size_t)c * size) * a.n_q_heads + qh) * 2]);
#pragma unroll 4
  for (int c = 0; c < n; ++c) {
    const size_t pidx = (slot0 + (size_t)c * size) * a.n_q_heads + qh;
    const float w = ex2(a.part_ml[pidx * 2] - mm);
    ll = fmaf(a.part_ml[pidx * 2 + 1], w, ll);
#pragma unroll
    for (int e = 0; e < V; ++e) acc[e] = fmaf(a.part_o[pidx * D + lane * V + e], w, acc[e]);
  }
  const float inv = ll > 0.f ? 1.0f / ll : 0.f;
  uint32_t* dst = reinterpret_cast<uint32_t*>(a.out + ((size_t)row * a.n_q_heads + qh) * D + lane * V);
#pragma unroll
  for (int e = 0; e < V; e += 2) dst[e / 2] = ll > 0.f ? pack2(acc[e] * inv, acc[e + 1] * inv) : 0u;
}

template <int D>
b200_status launch(b200_kv* kv, const CUtensorMap& qmap, const Args& a, const int* row_group, int sms, bool may_split, cudaStream_t s) {
  using Z = Shape<D>;
  const size_t smem = 2 * Z::kQBytes + Z::kSlots * Z::kSlotBytes + sizeof(Shared<D>);
  static bool configured = false;
  if (!configured) {
    B200_CUDA_TRY(cudaFuncSetAttribute(prompt_attn_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured = true;
  }
  launch_after(prompt_attn_kernel<D>, sms, kThreads, smem, s, kv->kmap, kv->vmap, qmap, a);
  B200_LAUNCH_CHECK();
  if (!may_split) return B200_OK;
  launch_after(prompt_combine_kernel<D>, (a.total_rows * a.n_q_heads + 7) / 8, 256, 0, s, a, row_group);
  B200_LAUNCH_CHECK();
  return B200_OK;
}

int g_prompt_sms = 0;

}  // namespace

size_t b200_attn_prompt_plan_ints(int32_t max_rows) { return kHdr + 2 * ((size_t)max_rows + kExtraItems); }

bool b200_attn_prompt_takes(const b200_kv* kv, const void* d_q, int32_t q_stride, const void* d_out) {
  const b200_kv_config& c = kv->cfg;
  const int g = c.n_kv_heads > 0 ? c.n_q_heads / c.n_kv_heads : 0;
  return !kv->layered && c.kv_dtype == B200_KV_BF16 && (c.head_dim == 64 || c.head_dim == 128) && (g == 1 || g == 2 || g == 4 || g == 8) &&
         ((uintptr_t)d_q & 15) == 0 && ((uintptr_t)d_out & 15) == 0 && q_stride % 8 == 0 && q_stride >= c.n_q_heads * c.head_dim;
}

b200_status b200_attn_prompt(b200_kv* kv, int32_t layer, const void* d_q, int32_t q_stride, const int32_t* d_row_seq, const int32_t* d_row_ctx,
                             int32_t total_rows, void* d_out, void* stream, bool may_split, bool reuse_plan) {
  const b200_kv_config& c = kv->cfg;
  cudaStream_t s = (cudaStream_t)stream;
  if (g_prompt_sms == 0) {
    int dev = 0;
    B200_CUDA_TRY(cudaGetDevice(&dev));
    B200_CUDA_TRY(cudaDeviceGetAttribute(&g_prompt_sms, cudaDevAttrMultiProcessorCount, dev));
  }
  const int g = c.n_q_heads / c.n_kv_heads, stride = c.max_rows + 2;
  Args a;
  a.d = kv->dev; a.layer = layer; a.total_rows = total_rows; a.n_q_heads = c.n_q_heads; a.group = g;
  a.row_seq = d_row_seq; a.row_ctx = d_row_ctx;
  a.group_first = kv->d_groups; a.part_base = kv->d_groups + stride; a.chunk_start = kv->d_chunk_start;
  a.hdr = kv->d_prompt;
  a.items = reinterpret_cast<const int2*>(kv->d_prompt + kHdr);
  a.part_o = kv->d_part_o; a.part_ml = kv->d_part_ml; a.out = (__nv_bfloat16*)d_out;
  a.scale_log2 = 1.4426950408889634f / sqrtf((float)c.head_dim);
  a.may_split = may_split;
  if (!reuse_plan) {
    launch_after(prompt_plan_kernel, 1, total_rows <= 1024 ? 256 : 1024, 0, s, d_row_seq, d_row_ctx, total_rows, c.page_size, 2 * kTileRows / g, kTileRows / g, c.n_kv_heads, g_prompt_sms,
                                          may_split ? 1 : 0, kv->max_chunks, may_split ? 16 / g : 0, kv->d_chunk_start, kv->d_groups, kv->d_groups + stride,
                                          kv->d_groups + 2 * stride, reinterpret_cast<int2*>(kv->d_prompt + kHdr), kv->d_prompt, kv->dev.state + ST_ATTN_ERR);
    B200_LAUNCH_CHECK();
  }
  CUtensorMap qmap;
  const uint64_t dims[3] = {(uint64_t)c.head_dim, (uint64_t)c.n_q_heads, (uint64_t)total_rows};
  const uint64_t strides[2] = {(uint64_t)c.head_dim * 2, (uint64_t)q_stride * 2};
  const uint32_t box[3] = {64, (uint32_t)g, (uint32_t)(kTileRows / g)};
  b200_status st = b200_make_tensor_map(&qmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, d_q, dims, strides, box);
  if (st != B200_OK) return st;
  const int* row_group = kv->d_groups + 2 * stride;
  return c.head_dim == 128 ? launch<128>(kv, qmap, a, row_group, g_prompt_sms, may_split, s) : launch<64>(kv, qmap, a, row_group, g_prompt_sms, may_split, s);
}
