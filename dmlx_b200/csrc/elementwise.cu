// Row-wise pieces of the layer stack: RMSNorm, RoPE, embedding gather, greedy argmax.
// All activations are bf16 with f32 arithmetic; every kernel is a single pass over its rows.
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include "common.h"
#include "launch.cuh"
#include "qmm.cuh"
#include "rows.cuh"

namespace cg = cooperative_groups;

namespace {

// A row by a block; nvec vectors of eight.
__device__ __forceinline__ void rmsnorm_row(const uint4* __restrict__ xr, const uint4* __restrict__ wr, uint4* __restrict__ orow, int nvec, float eps) {
  __shared__ float s_part[32];
  float ss = 0.f;
  for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
    uint4 v = xr[i];
    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 f = __bfloat1622float2(p[j]);
      ss += f.x * f.x + f.y * f.y;
    }
  }
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = ss;
  __syncthreads();
  if (threadIdx.x < 32) {
    float t = threadIdx.x < (blockDim.x >> 5) ? s_part[threadIdx.x] : 0.f;
    t = warp_sum(t);
    if (threadIdx.x == 0) s_part[0] = rsqrtf(t / (float)(8 * nvec) + eps);
  }
  __syncthreads();
  const float r = s_part[0];
  for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
    uint4 v = xr[i], g = wr[i], o;
    const __nv_bfloat162* pv = reinterpret_cast<const __nv_bfloat162*>(&v);
    const __nv_bfloat162* pg = reinterpret_cast<const __nv_bfloat162*>(&g);
    __nv_bfloat162* po = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 f = __bfloat1622float2(pv[j]), gg = __bfloat1622float2(pg[j]);
      po[j] = __floats2bfloat162_rn(f.x * r * gg.x, f.y * r * gg.y);
    }
    orow[i] = o;
  }
}

// One CTA per row; hidden % 8 == 0.
__global__ void rmsnorm_kernel(const __nv_bfloat16* x, const __nv_bfloat16* w, __nv_bfloat16* out, int hidden, float eps) {
  after_previous();
  const size_t at = (size_t)blockIdx.x * hidden;
  rmsnorm_row(reinterpret_cast<const uint4*>(x + at), reinterpret_cast<const uint4*>(w), reinterpret_cast<uint4*>(out + at), hidden / 8, eps);
}

// Non-traditional RoPE: pair (i, i + D/2) of every head rotates by pos * theta^(-2i/D).
// One thread per (row, head, i); q heads first, then k heads.
__global__ void rope_kernel(__nv_bfloat16* q, __nv_bfloat16* k,
                            const int* positions, int rows, int hq, int hkv, int D, int q_stride,
                            int k_stride, float log2_theta) {
  after_previous();
  const int half = D / 2;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long total = (long long)rows * (hq + hkv) * half;
  if (idx >= total) return;
  const int i = idx % half;
  const int head = (idx / half) % (hq + hkv);
  const int row = idx / ((long long)half * (hq + hkv));
  __nv_bfloat16* base = head < hq ? q + (size_t)row * q_stride + (size_t)head * D
                                  : k + (size_t)row * k_stride + (size_t)(head - hq) * D;
  const float inv_freq = exp2f(-log2_theta * (2.0f * i) / (float)D);
  float s, c;
  sincosf((float)positions[row] * inv_freq, &s, &c);
  const float x1 = __bfloat162float(base[i]), x2 = __bfloat162float(base[i + half]);
  base[i] = __float2bfloat16(x1 * c - x2 * s);
  base[i + half] = __float2bfloat16(x1 * s + x2 * c);
}

__global__ void embed_kernel(const __nv_bfloat16* table, const uint32_t* ids,
                             __nv_bfloat16* __restrict__ out, int hidden) {
  after_previous();
  const int row = blockIdx.x;
  const uint4* src = reinterpret_cast<const uint4*>(table + (size_t)ids[row] * hidden);
  uint4* dst = reinterpret_cast<uint4*>(out + (size_t)row * hidden);
  copy_vectors(dst, src, hidden / 8);
}

// First strict maximum of each row (ties keep the smaller index).
// A row belongs to a cluster of CTAs, a contiguous part each (16 rows of 32000 f32 values: 9.9 us by a block each, 6.8 this way).
template <typename T, bool WHOLE>  // WHOLE: a block has a row by itself
__global__ void argmax_kernel(const T* logits, int vocab, uint32_t* __restrict__ out) {
  after_previous();
  __shared__ float s_val[32];
  __shared__ int s_idx[32];
  cg::cluster_group cluster = cg::this_cluster();
  const int parts = WHOLE ? 1 : cluster.num_blocks(), part = WHOLE ? 0 : cluster.block_rank(), row = blockIdx.x / parts;
  const int per = ((vocab + parts - 1) / parts + 7) / 8 * 8, lo = min(part * per, vocab), hi = min(lo + per, vocab);
  const T* lr = logits + (size_t)row * vocab;
  float best = -INFINITY;
  int bi = 0x7fffffff;
  // 16-byte loads where the row allows it (row start and length multiples of 8 elements); a thread
  // meets its elements in increasing index order, so a strict > keeps the first maximum it saw.
  const bool vec = sizeof(T) == 2 && (vocab % 8 == 0) && ((reinterpret_cast<uintptr_t>(lr) & 15) == 0);
  if (vec) {
    const uint4* lv = reinterpret_cast<const uint4*>(lr);
    for (int c = lo / 8 + threadIdx.x; c < hi / 8; c += blockDim.x) {
      const uint4 q = lv[c];
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float lo = __uint_as_float(w[j] << 16), hi = __uint_as_float(w[j] & 0xFFFF0000u);
        if (lo > best) { best = lo; bi = c * 8 + 2 * j; }
        if (hi > best) { best = hi; bi = c * 8 + 2 * j + 1; }
      }
    }
  } else {
    for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
      float v = (float)lr[i];
      if (v > best || (v == best && i < bi)) { best = v; bi = i; }
    }
  }
  auto better = [](float va, int ia, float vb, int ib) { return va > vb || (va == vb && ia < ib); };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    float ov = __shfl_xor_sync(0xffffffffu, best, o);
    int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (better(ov, oi, best, bi)) { best = ov; bi = oi; }
  }
  if ((threadIdx.x & 31) == 0) { s_val[threadIdx.x >> 5] = best; s_idx[threadIdx.x >> 5] = bi; }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int nw = blockDim.x >> 5;
    best = threadIdx.x < nw ? s_val[threadIdx.x] : -INFINITY;
    bi = threadIdx.x < nw ? s_idx[threadIdx.x] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      float ov = __shfl_xor_sync(0xffffffffu, best, o);
      int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (better(ov, oi, best, bi)) { best = ov; bi = oi; }
    }
    if (WHOLE && threadIdx.x == 0) out[row] = bi == 0x7fffffff ? 0u : (uint32_t)bi;
    if (!WHOLE && threadIdx.x == 0) { s_val[0] = best; s_idx[0] = bi; }
  }
  if (WHOLE) return;
  cluster.sync();
  if (part == 0 && threadIdx.x == 0) {
    for (int q = 1; q < parts; ++q) {
      const float ov = *cluster.map_shared_rank(&s_val[0], q);
      const int oi = *cluster.map_shared_rank(&s_idx[0], q);
      if (better(ov, oi, best, bi)) { best = ov; bi = oi; }
    }
    out[row] = bi == 0x7fffffff ? 0u : (uint32_t)bi;
  }
  cluster.sync();  // nobody leaves while its shared memory may be read
}

template <typename T>
b200_status launch_argmax(const T* logits, int rows, int vocab, uint32_t* out, cudaStream_t s) {
  // parts of 4096 values and more, as long as the CTAs run at once, two per SM
  static const int most = ctas_in_clusters(argmax_kernel<T, false>, 8, 2, b200_sm_count(), 512, 0) / 64 * 64;
  int parts = 1;
  while (parts < 8 && vocab >= parts * 8192 && (long long)rows * parts * 2 <= most) parts *= 2;
  if (parts == 1) {  // (as clusters of one 1000 rows of 4097 values took 15.8 us, 9.9 so; 150 rows of 128256 f32 values, scheduled early 45, apart 34)
    if (vocab < 32768) launch_after(argmax_kernel<T, true>, rows, 1024, 0, s, logits, vocab, out);
    else launch_apart(argmax_kernel<T, true>, rows, 1024, 0, s, logits, vocab, out);
    B200_LAUNCH_CHECK();
    return B200_OK;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)rows * parts);
  cfg.blockDim = dim3(512);
  cfg.stream = s;
  cudaLaunchAttribute attr[2]{};
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = parts;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // (as launch_after)
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  B200_CUDA_TRY(cudaLaunchKernelEx(&cfg, argmax_kernel<T, false>, logits, vocab, out));
  B200_LAUNCH_CHECK();
  return B200_OK;
}

__global__ void gather_rows_kernel(const __nv_bfloat16* src, const int* idx,
                                   __nv_bfloat16* __restrict__ dst, int hidden) {
  after_previous();
  const int row = blockIdx.x;
  const int s = max(idx[row], 0);
  const uint4* sp = reinterpret_cast<const uint4*>(src + (size_t)s * hidden);
  uint4* dp = reinterpret_cast<uint4*>(dst + (size_t)row * hidden);
  copy_vectors(dp, sp, hidden / 8);
}

// `flags` points at the pool's eight state words: a step whose page reservation or attention was
// flagged has computed its tokens from stale pages, so the sequences keep the input token they had
// and the step can be run again once the cause (an exhausted pool) is gone.
__global__ void scatter_tokens_kernel(const uint32_t* next, const b200_pack_desc* desc,
                                      uint32_t* __restrict__ last_token, int n_req, const int* flags,
                                      int flag_a, int flag_b, const int* qmm_err, uint32_t* __restrict__ h_next,
                                      int* __restrict__ h_state) {
  after_previous();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  // The host's copies, straight into its pinned buffers: three copies behind the kernel took 6 us each, copy and gap, of an 8-request step.
  if (i < n_req) h_next[i] = next[i];
  if (i < 8) h_state[i] = flags[i];
  if (i == 8) h_state[8] = qmm_err ? *qmm_err : 0;
  if (flags[flag_a] != 0 || flags[flag_b] != 0) return;
  if (i < n_req && desc[i].count > 0) last_token[desc[i].seq_slot] = next[i];
}

}  // namespace

// Rows idx[r] of src -> row r of dst (the last position of every request, src/generation.zig:124-131).
b200_status b200_gather_rows(const void* d_src, const int32_t* d_idx, void* d_dst, int32_t rows, int32_t hidden, void* stream) {
  if (rows <= 0) return B200_OK;
  launch_after(gather_rows_kernel, rows, 128, 0, (cudaStream_t)stream, (const __nv_bfloat16*)d_src, d_idx, (__nv_bfloat16*)d_dst, hidden);
  B200_LAUNCH_CHECK();
  return B200_OK;
}

// The sampled token of request i becomes the next decode input of its sequence slot.  Pinned host buffers: h_next[n_req] gets the tokens,
// h_state[0..7] the pool's state words, h_state[8] the matmuls' error word.
b200_status b200_scatter_tokens(const uint32_t* d_next, const b200_pack_desc* d_desc, uint32_t* d_last_token, int32_t n_req,
                                const int* d_flags, int flag_a, int flag_b, uint32_t* h_next, int32_t* h_state, void* stream) {
  if (n_req <= 0) return B200_OK;
  launch_after(scatter_tokens_kernel, (n_req + 127) / 128, 128, 0, (cudaStream_t)stream, d_next, d_desc, d_last_token, n_req, d_flags,
               flag_a, flag_b, b200_qmm_err_word_device(), h_next, h_state);
  B200_LAUNCH_CHECK();
  return B200_OK;
}

extern "C" {

b200_status b200_rmsnorm(const void* d_x, const void* d_weight, void* d_out, int32_t rows, int32_t hidden, float eps,
                         void* stream) {
  b200_status st = b200_require_device();
  if (st != B200_OK) return st;
  if (hidden % 8 != 0) { b200_set_error("rmsnorm: hidden must be a multiple of 8"); return B200_ERR_INVALID_ARGUMENT; }
  if (rows <= 0) return B200_OK;
  launch_after(rmsnorm_kernel, rows, 256, 0, (cudaStream_t)stream, (const __nv_bfloat16*)d_x, (const __nv_bfloat16*)d_weight,
                                                        (__nv_bfloat16*)d_out, hidden, eps);
  B200_LAUNCH_CHECK();
  return B200_OK;
}

b200_status b200_rope(void* d_q, void* d_k, const int32_t* d_positions, int32_t rows, int32_t n_q_heads,
                      int32_t n_kv_heads, int32_t head_dim, int32_t q_stride, int32_t k_stride, float theta,
                      void* stream) {
  b200_status st = b200_require_device();
  if (st != B200_OK) return st;
  if (rows <= 0) return B200_OK;
  long long total = (long long)rows * (n_q_heads + n_kv_heads) * (head_dim / 2);
  launch_after(rope_kernel, (unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)stream,
      (__nv_bfloat16*)d_q, (__nv_bfloat16*)d_k, d_positions, rows, n_q_heads, n_kv_heads, head_dim, q_stride, k_stride,
      log2f(theta));
  B200_LAUNCH_CHECK();
  return B200_OK;
}

b200_status b200_embed_gather(const void* d_table, const uint32_t* d_ids, void* d_out, int32_t rows, int32_t hidden,
                              void* stream) {
  b200_status st = b200_require_device();
  if (st != B200_OK) return st;
  if (hidden % 8 != 0) { b200_set_error("embed: hidden must be a multiple of 8"); return B200_ERR_INVALID_ARGUMENT; }
  if (rows <= 0) return B200_OK;
  launch_after(embed_kernel, rows, 128, 0, (cudaStream_t)stream, (const __nv_bfloat16*)d_table, d_ids, (__nv_bfloat16*)d_out, hidden);
  B200_LAUNCH_CHECK();
  return B200_OK;
}

b200_status b200_argmax(const void* d_logits, int32_t rows, int32_t vocab, uint32_t* d_out, void* stream) {
  b200_status st = b200_require_device();
  if (st != B200_OK) return st;
  if (rows <= 0) return B200_OK;
  return launch_argmax((const __nv_bfloat16*)d_logits, rows, vocab, d_out, (cudaStream_t)stream);
}

b200_status b200_argmax_f32(const float* d_logits, int32_t rows, int32_t vocab, uint32_t* d_out, void* stream) {
  b200_status st = b200_require_device();
  if (st != B200_OK) return st;
  if (rows <= 0) return B200_OK;
  return launch_argmax(d_logits, rows, vocab, d_out, (cudaStream_t)stream);
}

}  // extern "C"
