// Sampling beyond greedy on the device: temperature, top-k and top-p per row
// (src/sampling.zig:42-72, 175-242, 258-268, 298-322, 328-375), so that only one token id per
// request crosses PCIe for non-greedy requests too.  The uniform variate of each draw is an input.
//
// A row belongs to a cluster of up to eight CTAs, a contiguous part of the vocabulary each; it is read from L2 a few times and what has to be
// known of the whole row goes through distributed shared memory to the cluster's first CTA.  Ordering follows the reference's stable
// descending sort: a candidate is the 64-bit key (descending score bits << 32 | token id), so equal scores keep index order.
//
// Nothing of vocabulary size is sorted.  The scores are counted in 2048 bins by their distance from the maximum (1/64 each, the last one for
// all beyond 32), with the bins' weights; the k-th candidate, the end of the nucleus and the drawn token are each found first by bin, from
// the bins' running sums, and then inside it, among its few keys, sorted in shared memory.  Where all bins up to the one that matters hold
// no more than 2048 keys they are sorted at once and everything is decided on that list; for up to 512 candidates that is tried first on the
// bins that hold as many of the threads' maxima, without counting the row.  A bin with more keys than that is counted again
// in 2048 finer ranges of keys, as often as it takes (keys are unique, so at most five times).
//
// A bin's weight is edge * (count - deficit): 1 - exp(-x), x the distance behind the bin's near edge, is below 2^-6 and is summed in units of
// 2^-22 in an integer, so sums do not depend on the order of the additions.  (Equal scores round alike, so the unit is the same for every
// vocabulary: a CTA of more than 65535 words counts how often a bin's 32 bits are full.)  Running sums over bins and candidates are f64.
//
// Bound by the latency of its passes (loads, cluster barriers), not by bytes.  64 rows of 128256 bf16 words on one B200: greedy 20 us, top-k 50 40,
// the whole distribution 48, a nucleus of 0.9 over all words 75, 3000 candidates 87.  One CTA per row that walked the sorted order 512
// candidates at a time, one thread adding, took 1286 us for a mixture of these rows (800 to 1760 from call to call); this takes 80, upload of
// the rows' parameters included.  More than 148 rows are a CTA each; 256 rows, before and now: greedy 44 and 48 us, top-k 50
// 149 and 59, the whole distribution 202 and 155, a nucleus of 0.9 5943 and 166, 3000 candidates 1716 and 193.
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#include "common.h"
#include "launch.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int kThreads = 512, kWarps = kThreads / 32;
constexpr int kBins = 2048, kPerThread = kBins / kThreads;
constexpr int kCap = 2048;     // keys sorted in shared memory
constexpr int kMaxCluster = 8;
constexpr int kFew = 512;      // candidates that the threads' maxima are asked for
constexpr float kBinsPerUnit = 64.f;
constexpr float kUnits = 4194304.f;  // of a deficit: 2^-22
constexpr int kFullWords = 65535;    // whose deficits, below 2^16 units each, add up in 32 bits

struct Bins {  // running sums over the bins, inclusive
  unsigned n[kBins];
  double m[kBins];
};

struct Shared {
  unsigned hist_n[kBins], hist_d[kBins];  // this CTA's part: keys, deficits
  unsigned hist_c[kBins];                 // multiples of 2^32 of the deficits, where the CTA has more than kFullWords
  Bins row;                               // (first CTA)
  union {
    Bins fine;                            // of the ranges inside one bin
    struct {
      unsigned long long key[kCap];
      float weight[kCap];
    } list;
  };
  double red_d[kWarps];
  float red_f[kWarps];
  int red_i[kWarps];
  unsigned red_u[kWarps];
  unsigned long long red_k[2 * kWarps];
  // what a CTA hands to the others
  float part_max;
  int part_arg;
  double part_sum[2];                     // of exp(logit - max), and of exp((logit - max) / temperature)
  double warp_sum[kWarps];                // the latter by warp, in the order of the vocabulary
  unsigned long long part_lo, part_hi;
  // what the first CTA found
  unsigned found, count;
  double before, mass;
  unsigned n_before;
  unsigned token;
  int owner;
  double target;
};

template <typename T> struct Row {
  const T* p;
  int V;
  bool vec;  // 16-byte loads: the row starts on a 16-byte boundary and V % 8 == 0
};

__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }

// Eight consecutive elements starting at i0 (a multiple of 8); returns how many are inside the row.
__device__ __forceinline__ int load8(const Row<__nv_bfloat16>& r, int i0, float (&v)[8]) {
  const int n = min(max(r.V - i0, 0), 8);
  if (r.vec && n == 8) {
    const uint4 q = *reinterpret_cast<const uint4*>(r.p + i0);
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[2 * j] = __uint_as_float(w[j] << 16);
      v[2 * j + 1] = __uint_as_float(w[j] & 0xFFFF0000u);
    }
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = j < n ? __bfloat162float(r.p[i0 + j]) : 0.f;
  }
  return n;
}
__device__ __forceinline__ int load8(const Row<float>& r, int i0, float (&v)[8]) {
  const int n = min(max(r.V - i0, 0), 8);
  if (r.vec && n == 8) {
    const float4 a = *reinterpret_cast<const float4*>(r.p + i0), b = *reinterpret_cast<const float4*>(r.p + i0 + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = j < n ? r.p[i0 + j] : 0.f;
  }
  return n;
}

// (score descending, token id ascending) as one ascending 64-bit key; -0 is folded into +0 so that
// scores that compare equal share their bits.
__device__ __forceinline__ float score_of(float logit, float temperature) { return logit / temperature + 0.0f; }
__device__ __forceinline__ unsigned long long key_of(float score, int idx) {
  unsigned u = __float_as_uint(score);
  u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
  return ((unsigned long long)(~u) << 32) | (unsigned)idx;
}
__device__ __forceinline__ float key_score(unsigned long long c) {
  const unsigned u = ~(unsigned)(c >> 32);
  return __uint_as_float((u & 0x80000000u) ? (u ^ 0x80000000u) : ~u);
}
__device__ __forceinline__ int bin_of(float distance) { return (int)fminf(fmaxf(distance * kBinsPerUnit, 0.f), (float)(kBins - 1)); }

// One row's work: the CTA's threads, its part of the vocabulary, and the cluster it belongs to.
template <typename T>
struct Sampler {
  cg::cluster_group cluster;
  Shared& s;
  Row<T> r;
  int ranks, rank, tid, lane, warp;
  int warp_part, lo, hi;  // a warp's part of the vocabulary (a multiple of 8), and this warp's
  bool carries;           // deficits of one bin may exceed 32 bits

  __device__ Sampler(Shared& sh, const Row<T>& row) : cluster(cg::this_cluster()), s(sh), r(row) {
    ranks = cluster.num_blocks();
    rank = cluster.block_rank();
    tid = threadIdx.x; lane = tid & 31; warp = tid >> 5;
    warp_part = ((r.V + ranks * kWarps - 1) / (ranks * kWarps) + 7) / 8 * 8;
    lo = min((rank * kWarps + warp) * warp_part, r.V);
    hi = min(lo + warp_part, r.V);
    carries = warp_part * kWarps > kFullWords;
  }
  __device__ Shared& of(int q) { return *cluster.map_shared_rank(&s, q); }

  // f(logits, first token, how many) over the thread's elements, eight neighbours at a time; Q of these loads are in flight
  template <int Q, typename F>
  __device__ __forceinline__ void each8(F f) {
    int base = lo;
    for (; base + Q * 256 <= hi; base += Q * 256) {
      float v[Q][8];
#pragma unroll
      for (int q = 0; q < Q; ++q) load8(r, base + (q * 32 + lane) * 8, v[q]);
#pragma unroll
      for (int q = 0; q < Q; ++q) f(v[q], base + (q * 32 + lane) * 8, 8);
    }
#pragma unroll 1
    for (int i0 = base + lane * 8; i0 < hi; i0 += 256) {
      float v[8];
      load8(r, i0, v);
      f(v, i0, min(hi - i0, 8));
    }
  }
  // f(logit, token) over the thread's elements with a logit from `least` to `most`
  template <typename F>
  __device__ __forceinline__ void each_within(float least, float most, F f) {
    each8<2>([&](const float (&v)[8], int i0, int n) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < n && !(v[j] < least) && !(v[j] > most)) f(v[j], i0 + j);
    });
  }
  // Logits whose scores may fall into bins first..last (a little wider: rounding).
  __device__ __forceinline__ void logits_of(int first, int last, float temperature, float gmax, float* least, float* most) {
    const float slack = 1e-5f * (fabsf(gmax) + 32.f * temperature);
    *most = first == 0 ? INFINITY : gmax - (float)first * (1.f / kBinsPerUnit) * temperature + slack;
    *least = last == kBins - 1 ? -INFINITY : gmax - (float)(last + 1) * (1.f / kBinsPerUnit) * temperature - slack;
  }

  __device__ double block_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) s.red_d[warp] = v;
    __syncthreads();
    double t = 0.0;
    for (int w = 0; w < kWarps; ++w) t += s.red_d[w];
    return t;
  }

  // First strict maximum of the row (src/sampling.zig:22-39).
  __device__ int first_max(float* out_max, float* thread_max) {
    float best = -INFINITY;
    int bi = 0x7fffffff;
    each8<4>([&](const float (&v)[8], int i0, int n) {
      float top = -INFINITY;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < n) top = fmaxf(top, v[j]);
      if (top > best) {
        best = top;
#pragma unroll
        for (int j = 7; j >= 0; --j)
          if (j < n && v[j] == top) bi = i0 + j;
      }
    });
    *thread_max = best;
    auto better = [](float va, int ia, float vb, int ib) { return va > vb || (va == vb && ia < ib); };
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (better(ov, oi, best, bi)) { best = ov; bi = oi; }
    }
    if (lane == 0) { s.red_f[warp] = best; s.red_i[warp] = bi; }
    __syncthreads();
    if (tid == 0) {
      for (int w = 1; w < kWarps; ++w)
        if (better(s.red_f[w], s.red_i[w], best, bi)) { best = s.red_f[w]; bi = s.red_i[w]; }
      s.part_max = best;
      s.part_arg = bi;
    }
    cluster.sync();
    best = of(0).part_max;
    bi = of(0).part_arg;
    for (int q = 1; q < ranks; ++q) {
      const float ov = of(q).part_max;
      const int oi = of(q).part_arg;
      if (better(ov, oi, best, bi)) { best = ov; bi = oi; }
    }
    *out_max = best;
    return bi == 0x7fffffff ? 0 : bi;
  }

  __device__ void clear_hist() {
    for (int b = tid; b < kBins; b += kThreads) { s.hist_n[b] = 0; s.hist_d[b] = 0; s.hist_c[b] = 0; }
    __syncthreads();
  }
  __device__ void count(int bin, float x) {  // x: distance behind the near edge of the score's bin, below 1/64
    const float deficit = x * (1.f - x * (0.5f - x * (1.f / 6.f - x * (1.f / 24.f))));
    atomicAdd(&s.hist_n[bin], 1u);
    const unsigned d = (unsigned)(deficit * kUnits + 0.5f);
    if (!carries) {
      atomicAdd(&s.hist_d[bin], d);
    } else if (const unsigned old = atomicAdd(&s.hist_d[bin], d); old + d < old) {
      atomicAdd(&s.hist_c[bin], 1u);
    }
  }
  // First CTA: running sums of the whole row's bins.  `edge`: weight at the near edge of bin b; `counted` false: the bin weighs nothing.
  template <typename F>
  __device__ void sum_bins(Bins& out, F edge) {
    cluster.sync();
    if (rank == 0) {
      unsigned n[kPerThread];
      double m[kPerThread];
#pragma unroll
      for (int k = 0; k < kPerThread; ++k) n[k] = 0;
      double deficit[kPerThread] = {};
      for (int q = 0; q < ranks; ++q) {
        const Shared& o = of(q);
#pragma unroll
        for (int k = 0; k < kPerThread; ++k) {
          n[k] += o.hist_n[tid * kPerThread + k];
          deficit[k] += (double)o.hist_d[tid * kPerThread + k];
          if (carries) deficit[k] += 4294967296.0 * (double)o.hist_c[tid * kPerThread + k];
        }
      }
      unsigned nt = 0;
      double mt = 0.0;
#pragma unroll
      for (int k = 0; k < kPerThread; ++k) {
        m[k] = edge(tid * kPerThread + k) * ((double)n[k] - deficit[k] * (1.0 / (double)kUnits));
        nt += n[k]; n[k] = nt;
        mt += m[k]; m[k] = mt;
      }
      unsigned ni = nt;
      double mi = mt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned a = __shfl_up_sync(0xffffffffu, ni, o);
        const double b = __shfl_up_sync(0xffffffffu, mi, o);
        if (lane >= o) { ni += a; mi += b; }
      }
      if (lane == 31) { s.red_u[warp] = ni; s.red_d[warp] = mi; }
      __syncthreads();
      unsigned nb = ni - nt;
      double mb = mi - mt;
      for (int w = 0; w < warp; ++w) { nb += s.red_u[w]; mb += s.red_d[w]; }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < kPerThread; ++k) { out.n[tid * kPerThread + k] = nb + n[k]; out.m[tid * kPerThread + k] = mb + m[k]; }
    }
    cluster.sync();
  }

  // A set of keys that follow one another in the order: a range inside a bin, with what lies ahead of it.
  struct Range {
    int bin;
    unsigned long long lo, hi;
    unsigned n_before, n;
    double m_before;
  };
  // The first bin whose running count reaches `rank_wanted` (by_mass false) or whose running weight exceeds `target`.  All CTAs get the answer.
  __device__ unsigned search(const Bins& bins, bool by_mass, unsigned rank_wanted, double target, unsigned last) {
    if (rank == 0) {
      if (tid == 0) s.found = last;
      __syncthreads();
#pragma unroll
      for (int k = 0; k < kPerThread; ++k) {
        const int b = tid * kPerThread + k;
        const bool here = by_mass ? bins.m[b] > target && (b == 0 || !(bins.m[b - 1] > target)) : bins.n[b] >= rank_wanted && (b == 0 || bins.n[b - 1] < rank_wanted);
        if (here) atomicMin(&s.found, (unsigned)b);
      }
      __syncthreads();
      if (tid == 0) {
        // (a bin that adds nothing but rounding is passed over)
        unsigned b = s.found;
        while (b > 0 && bins.n[b] == bins.n[b - 1]) --b;
        s.found = b;
        s.n_before = b ? bins.n[b - 1] : 0;
        s.count = bins.n[b] - s.n_before;
        s.before = b ? bins.m[b - 1] : 0.0;
      }
    }
    cluster.sync();
    return of(0).found;
  }
  // Narrows a search down to at most kCap keys.
  __device__ Range find(float temperature, float gmax, float max_score, bool by_mass, unsigned rank_wanted, double target, unsigned last) {
    Range g;
    g.bin = (int)search(s.row, by_mass, rank_wanted, target, last);
    g.lo = 0;
    g.hi = ~0ull;
    const Shared& f = of(0);
    g.n_before = f.n_before;
    g.n = f.count;
    g.m_before = f.before;
    cluster.sync();
    const double edge = g.bin == kBins - 1 ? 0.0 : exp(-(double)g.bin / (double)kBinsPerUnit);
    while (g.n > kCap) {
      // the range's first and last key, then its keys counted in 2048 parts
      unsigned long long kl = ~0ull, kh = 0ull;
      auto mine = [&](float v, int i, auto f) {
        const float sc = score_of(v, temperature), dist = max_score - sc;
        if (bin_of(dist) != g.bin) return;
        const unsigned long long k = key_of(sc, i);
        if (k >= g.lo && k <= g.hi) f(k, dist);
      };
      float least, most;
      logits_of(g.bin, g.bin, temperature, gmax, &least, &most);
      each_within(least, most, [&](float v, int i) { mine(v, i, [&](unsigned long long k, float) { kl = min(kl, k); kh = max(kh, k); }); });
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        kl = min(kl, __shfl_xor_sync(0xffffffffu, kl, o));
        kh = max(kh, __shfl_xor_sync(0xffffffffu, kh, o));
      }
      __syncthreads();
      if (lane == 0) { s.red_k[warp] = kl; s.red_k[kWarps + warp] = kh; }
      __syncthreads();
      if (tid == 0) {
        for (int w = 0; w < kWarps; ++w) { kl = min(kl, s.red_k[w]); kh = max(kh, s.red_k[kWarps + w]); }
        s.part_lo = kl;
        s.part_hi = kh;
      }
      cluster.sync();
      for (int q = 0; q < ranks; ++q) { kl = min(kl, of(q).part_lo); kh = max(kh, of(q).part_hi); }
      int shift = 0;
      while (((kh - kl) >> shift) >= kBins) ++shift;
      clear_hist();
      each_within(least, most, [&](float v, int i) {
        mine(v, i, [&](unsigned long long k, float dist) { count((int)((k - kl) >> shift), g.bin == kBins - 1 ? 0.f : fmaxf(dist - (float)g.bin * (1.f / kBinsPerUnit), 0.f)); });
      });
      sum_bins(s.fine, [&](int) { return edge; });
      const unsigned part = search(s.fine, by_mass, rank_wanted - g.n_before, target - g.m_before, (unsigned)((kh - kl) >> shift));
      g.lo = kl + ((unsigned long long)part << shift);
      g.hi = g.lo + ((1ull << shift) - 1);
      g.n_before += f.n_before;
      g.n = f.count;
      g.m_before += f.before;
      cluster.sync();
    }
    return g;
  }

  // The keys of bins first..last between klo and khi, sorted, into the first CTA's list; returns how many.
  __device__ int gather(float temperature, float gmax, float max_score, int first, int last, unsigned long long klo, unsigned long long khi) {
    return gather(temperature, gmax, max_score, first, last, klo, khi, [](const float (&)[8], int) {});
  }
  // `also`: done to all the thread's elements on the way.  More keys than fit: the list is not made.
  template <typename F>
  __device__ int gather(float temperature, float gmax, float max_score, int first, int last, unsigned long long klo, unsigned long long khi, F also) {
    Shared& f = of(0);
    if (rank == 0 && tid == 0) s.count = 0;
    cluster.sync();
    float least, most;
    logits_of(first, last, temperature, gmax, &least, &most);
    each8<2>([&](const float (&v)[8], int i0, int n) {
      also(v, n);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (j >= n || v[j] < least || v[j] > most) continue;
        const float sc = score_of(v[j], temperature);
        const int b = bin_of(max_score - sc);
        if (b < first || b > last) continue;
        const unsigned long long k = key_of(sc, i0 + j);
        if (k < klo || k > khi) continue;
        const unsigned at = atomicAdd(&f.count, 1u);
        if (at < kCap) f.list.key[at] = k;
      }
    });
    cluster.sync();
    const int n = (int)f.count;
    if (rank == 0 && n <= kCap) {
      int n2 = 2;
      while (n2 < n) n2 <<= 1;
      for (int i = n + tid; i < n2; i += kThreads) s.list.key[i] = ~0ull;
      __syncthreads();
      for (int k = 2; k <= n2; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
          for (int i = tid; i < n2; i += kThreads) {
            const int x = i ^ j;
            if (x > i) {
              const unsigned long long a = s.list.key[i], c = s.list.key[x];
              if ((a > c) == ((i & k) == 0)) { s.list.key[i] = c; s.list.key[x] = a; }
            }
          }
          __syncthreads();
        }
      }
      for (int i = tid; i < n; i += kThreads) s.list.weight[i] = expf(key_score(s.list.key[i]) - max_score);
      __syncthreads();
    }
    return n;
  }

  // First CTA, all its threads: the first of list[0, n) at which base + running weight exceeds target, n if none does; *upto gets the
  // running sum with it (or all).  A thread takes four neighbours.
  __device__ int walk(int n, double base, double target, double* upto) {
    constexpr int E = kCap / kThreads;
    double w[E], t = 0.0;
#pragma unroll
    for (int k = 0; k < E; ++k) {
      const int i = tid * E + k;
      t += i < n ? (double)s.list.weight[i] : 0.0;
      w[k] = t;
    }
    double incl = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double a = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += a;
    }
    __syncthreads();
    if (lane == 31) s.red_d[warp] = incl;
    if (tid == 0) s.found = (unsigned)n;
    __syncthreads();
    double ahead = base + incl - t;
    for (int q = 0; q < warp; ++q) ahead += s.red_d[q];
    int at = n;
#pragma unroll
    for (int k = E - 1; k >= 0; --k)
      if (tid * E + k < n && ahead + w[k] > target) at = tid * E + k;
    if (at < n) atomicMin(&s.found, (unsigned)at);
    __syncthreads();
    const int found = (int)s.found;
    const int last = min(found, n - 1);  // whose running sum is wanted
#pragma unroll
    for (int k = 0; k < E; ++k)
      if (tid * E + k == last) s.mass = ahead + w[k];
    if (n == 0 && tid == 0) s.mass = base;
    __syncthreads();
    *upto = s.mass;
    __syncthreads();
    return found;
  }

  // First CTA: end of the nucleus and draw on the sorted list, whose first `keep` keys are the candidates; total: their weight.
  __device__ void decide(int keep, double total, bool cut, float top_p, float u) {
    double nucleus, drawn;
    const int end = walk(keep, 0.0, cut ? (double)top_p * total : (double)INFINITY, &nucleus), members = min(end + 1, keep);
    const int at = min(walk(members, 0.0, (double)u * nucleus, &drawn), members - 1);
    if (tid == 0) s.token = (unsigned)s.list.key[at];
    __syncthreads();
  }

  // topKTopPSampler (src/sampling.zig:175-242).  `part` gets the thread's sum of exp(logit - max) where sums is set.
  __device__ unsigned top_k_top_p(float temperature, int k_eff, float top_p, float u, float gmax, float max_score, float thread_max, bool sums, double* part) {
    const Shared& f = of(0);
    const bool all = k_eff >= r.V;
    const bool cut = top_p < 1.0f;
    if (k_eff <= kFew) {
      // The few best: as many threads' maxima as candidates are wanted lie in the bins up to some bin, hence as many words; all words of
      // those bins are a prefix of the order, little longer than wanted.
      clear_hist();
      if (lo < hi) atomicAdd(&s.hist_n[bin_of(max_score - score_of(thread_max, temperature))], 1u);
      sum_bins(s.row, [](int) { return 0.0; });
      const unsigned last = search(s.row, false, (unsigned)k_eff, 0.0, kBins - 1);
      const int n = gather(temperature, gmax, max_score, 0, (int)last, 0ull, ~0ull, [&](const float (&v)[8], int m) {
        if (!sums) return;
        float a = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j < m) a += expf(v[j] - gmax);
        *part += (double)a;
      });
      if (n <= kCap) {
        if (rank == 0) {
          const int keep = min(n, k_eff);
          double total;
          walk(keep, 0.0, INFINITY, &total);
          decide(keep, total, cut, top_p, u);
        }
        cluster.sync();
        return f.token;
      }
      sums = false;
      cluster.sync();
    }
    clear_hist();
    each8<2>([&](const float (&v)[8], int i0, int n) {
      float a = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < n) {
          if (sums) a += expf(v[j] - gmax);
          const float dist = max_score - score_of(v[j], temperature);
          const int b = bin_of(dist);
          count(b, b == kBins - 1 ? 0.f : fmaxf(dist - (float)b * (1.f / kBinsPerUnit), 0.f));
        }
      *part += (double)a;
    });
    sum_bins(s.row, [](int b) { return b == kBins - 1 ? 0.0 : exp(-(double)b / (double)kBinsPerUnit); });
    // the bin that ends the list of candidates: by rank, or by weight where every word is one
    double total = f.row.m[kBins - 1];
    const unsigned last = search(s.row, all && cut, (unsigned)k_eff, (double)top_p * total, kBins - 1);
    const unsigned upto = f.n_before + f.count;
    cluster.sync();
    unsigned token = 0;
    if (upto <= kCap) {
      // they fit: everything is decided on the sorted list
      const int n = gather(temperature, gmax, max_score, 0, (int)last, 0ull, ~0ull);
      if (rank == 0) {
        const int keep = min(n, k_eff);
        if (!all) walk(keep, 0.0, INFINITY, &total);
        decide(keep, total, cut, top_p, u);
      }
    } else {
      // position by position: the last candidate, the end of the nucleus (s.token is the last member so far), the draw
      Range k_end{};
      unsigned n_keep = (unsigned)r.V;
      if (!all) {
        k_end = find(temperature, gmax, max_score, false, (unsigned)k_eff, 0.0, kBins - 1);
        const int n = gather(temperature, gmax, max_score, k_end.bin, k_end.bin, k_end.lo, k_end.hi);
        if (rank == 0) {
          double sum;
          const int here = min(n, k_eff - (int)k_end.n_before);
          walk(here, k_end.m_before, INFINITY, &sum);
          if (tid == 0) { s.target = sum; s.token = (unsigned)s.list.key[here - 1]; }
          __syncthreads();
        }
        cluster.sync();
        total = f.target;
        n_keep = (unsigned)k_eff;
        cluster.sync();
      }
      unsigned members = n_keep;
      double nucleus = total;
      if (cut) {
        const Range g = find(temperature, gmax, max_score, true, 0u, (double)top_p * total, all ? kBins - 1 : (unsigned)k_end.bin);
        const int n = gather(temperature, gmax, max_score, g.bin, g.bin, g.lo, g.hi);
        if (rank == 0) {
          double sum;
          const int here = (int)min((unsigned)n, n_keep - min(n_keep, g.n_before));
          const int at = walk(here, g.m_before, (double)top_p * total, &sum);
          if (tid == 0) {
            s.target = sum;
            s.n_before = min(n_keep, g.n_before + (unsigned)min(at + 1, here));
            if (here > 0) s.token = (unsigned)s.list.key[min(at, here - 1)];
          }
          __syncthreads();
        }
        cluster.sync();
        nucleus = f.target;
        members = f.n_before;
        cluster.sync();
      }
      const Range g = find(temperature, gmax, max_score, true, 0u, (double)u * nucleus, kBins - 1);
      const int n = gather(temperature, gmax, max_score, g.bin, g.bin, g.lo, g.hi);
      if (rank == 0) {
        double sum;
        // (behind the last member, by rounding: s.token is that one already)
        const int here = (int)min((unsigned)n, members - min(members, g.n_before));
        const int at = min(walk(here, g.m_before, (double)u * nucleus, &sum), here - 1);
        if (tid == 0 && here > 0) s.token = (unsigned)s.list.key[at];
        __syncthreads();
      }
    }
    cluster.sync();
    token = f.token;
    return token;
  }

  // temperatureSample (src/sampling.zig:42-72): softmax of (logit - max) / T in index order, first index whose cumulative probability
  // exceeds u.  The warps' sums say which warp's part it falls into; there a lane takes a run of neighbours.
  __device__ unsigned full_softmax(float temperature, float gmax, float u) {
    cluster.sync();
    if (rank == 0 && tid == 0) {
      double sum = 0.0, cum = 0.0;
      for (int q = 0; q < ranks; ++q) sum += of(q).part_sum[1];
      const double target = (double)u * sum;
      s.owner = -1;
      s.token = (unsigned)(r.V - 1);  // sampleFromProbs returns n - 1 when u is never exceeded (:267)
      for (int q = 0; q < ranks && s.owner < 0; ++q)
        for (int w = 0; w < kWarps; ++w) {
          const double next = cum + of(q).warp_sum[w];
          if (next > target) { s.owner = q * kWarps + w; s.target = target - cum; break; }
          cum = next;
        }
    }
    cluster.sync();
    Shared& f = of(0);
    if (f.owner == rank * kWarps + warp) {
      const double target = f.target;
      const int run = (warp_part + 31) / 32, b = min(lo + lane * run, hi), e = min(b + run, hi);
      double mine = 0.0;
      for (int i = b; i < e; ++i) mine += (double)expf((to_f32(r.p[i]) - gmax) / temperature);
      double incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      const unsigned over = __ballot_sync(0xffffffffu, incl > target && e > b);
      if (over == 0) {
        if (lane == 0) f.token = (unsigned)(hi - 1);
      } else if (lane == __ffs(over) - 1) {
        double cum = incl - mine;
        int i = b;
        for (; i < e - 1; ++i) {
          cum += (double)expf((to_f32(r.p[i]) - gmax) / temperature);
          if (cum > target) break;
        }
        f.token = (unsigned)i;
      }
    }
    cluster.sync();
    return f.token;
  }

  __device__ void run(const b200_sample_params& p, uint32_t* out_token, float* out_logprob) {
    float gmax, thread_max;
    unsigned token = (unsigned)first_max(&gmax, &thread_max);
    const bool sums = out_logprob != nullptr, greedy = !(p.temperature > 0.0f), whole = !greedy && p.top_p >= 1.0f && (p.top_k <= 0 || p.top_k >= r.V);
    double part = 0.0, part_t = 0.0;
    if (!greedy && !whole) {
      // the largest score is the largest logit's: division by a positive temperature keeps the order
      token = top_k_top_p(p.temperature, (p.top_k <= 0 || p.top_k > r.V) ? r.V : p.top_k, p.top_p, p.uniform, gmax, score_of(gmax, p.temperature), thread_max, sums, &part);
    } else if (sums || whole) {
      each8<2>([&](const float (&v)[8], int i0, int n) {
        float a = 0.f, b = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (sums && j < n) a += expf(v[j] - gmax);
          if (whole && j < n) b += expf((v[j] - gmax) / p.temperature);
        }
        part += (double)a;
        part_t += (double)b;
      });
    }
    const double sum = block_sum(part);
    if (tid == 0) s.part_sum[0] = sum;
    if (whole) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) part_t += __shfl_xor_sync(0xffffffffu, part_t, o);
      if (lane == 0) s.warp_sum[warp] = part_t;
      __syncthreads();
      if (tid == 0) {
        double t = 0.0;
        for (int w = 0; w < kWarps; ++w) t += s.warp_sum[w];
        s.part_sum[1] = t;
      }
      token = full_softmax(p.temperature, gmax, p.uniform);
    }
    cluster.sync();
    if (rank == 0 && tid == 0) {
      if (out_logprob != nullptr) {
        double all = 0.0;
        for (int q = 0; q < ranks; ++q) all += of(q).part_sum[0];
        *out_logprob = token < (unsigned)r.V ? to_f32(r.p[token]) - (gmax + logf((float)all)) : -INFINITY;
      }
      *out_token = token;
    }
    cluster.sync();  // nobody leaves while its shared memory may be read
  }
};

// The rows' parameters: in device memory, or of up to 1024 rows in the arguments of the launch (24 KB; 128 rows 3 KB), which spares an upload ahead of
// the kernel (64 rows in passes behind one another: pageable upload 105 us, pinned 88, in the arguments 80; the first pass on new buffers 163, 170,
// 148.  256 rows of 128256 bf16 words in passes behind one another 182, 177, 167, waited for one by one 265, 264, 253; 1024 rows 461, 457, 447).
struct InMemory {
  const b200_sample_params* p;
  __device__ __forceinline__ const b200_sample_params& operator[](int row) const { return p[row]; }
};
template <int ROWS>
struct InArguments {
  b200_sample_params p[ROWS];
  __device__ __forceinline__ const b200_sample_params& operator[](int row) const { return p[row]; }
};

template <typename T, typename Params>
__global__ void __launch_bounds__(kThreads, 2) sample_rows_kernel(const T* logits, int V, const __grid_constant__ Params params,
                                                                  const uint32_t* ctx, const int* ctx_off,
                                                                  float* __restrict__ scratch, uint32_t* __restrict__ tokens,
                                                                  float* __restrict__ logprobs) {
  wait_previous();
  extern __shared__ __align__(16) unsigned char sample_dyn[];
  Shared& s = *reinterpret_cast<Shared*>(sample_dyn);
  cg::cluster_group cluster = cg::this_cluster();
  const int ranks = cluster.num_blocks(), rank = cluster.block_rank(), row = blockIdx.x / ranks;
  const b200_sample_params p = params[row];
  const T* x = logits + (size_t)row * V;
  float* lp = logprobs ? logprobs + row : nullptr;
  const int ctx_lo = ctx_off ? ctx_off[row] : 0, ctx_n = ctx_off ? ctx_off[row + 1] - ctx_lo : 0;
  const bool penalised = p.repetition_penalty > 1.0f && ctx_n > 0 && scratch != nullptr;
  float* y = penalised ? scratch + (size_t)row * V : nullptr;
  if (penalised) {
    // applyRepetitionPenalty (src/sampling.zig:328-354): every occurrence of a token divides a positive
    // logit by the penalty or multiplies a non-positive one; occurrences commute, so they may race.
    for (int i = rank * kThreads + threadIdx.x; i < V; i += ranks * kThreads) y[i] = to_f32(x[i]);
    __threadfence();
    cluster.sync();
    for (int c = rank * kThreads + threadIdx.x; c < ctx_n; c += ranks * kThreads) {
      const uint32_t tok = ctx[ctx_lo + c];
      if (tok < (uint32_t)V) {
        unsigned* a = reinterpret_cast<unsigned*>(y + tok);
        unsigned old = *reinterpret_cast<volatile unsigned*>(a), assumed;
        do {
          assumed = old;
          const float f = __uint_as_float(assumed);
          old = atomicCAS(a, assumed, __float_as_uint(f > 0.f ? f / p.repetition_penalty : f * p.repetition_penalty));
        } while (old != assumed);
      }
    }
    __threadfence();
    cluster.sync();
  }
  auto sampled = [&](auto* from) {
    using U = std::remove_const_t<std::remove_pointer_t<decltype(from)>>;
    Sampler<U>(s, Row<U>{from, V, V % 8 == 0 && (reinterpret_cast<uintptr_t>(from) & 15) == 0}).run(p, tokens + row, lp);
  };
  // (One call for f32 rows: with one for each source the compiler kept the sampler as a function, its row's
  // parameters in local memory, where these come in the arguments: 64 rows of 128256 words 101 us, 70 now; from device memory 78 and 70.)
  if constexpr (sizeof(T) == 4) sampled(penalised ? y : x);
  else if (penalised) sampled(y);
  else sampled(x);
}

template <typename T, typename Params>
b200_status launch(const T* logits, int rows, int vocab, const Params& params, const uint32_t* ctx, const int* ctx_off, float* scratch,
                   uint32_t* tokens, float* logprobs, cudaStream_t s) {
  // (asked for at every launch: the attribute belongs to the device that the calling thread uses)
  B200_CUDA_TRY(cudaFuncSetAttribute(sample_rows_kernel<T, Params>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Shared)));
  // CTAs per row: 8192 words each at least (16 a thread), and no more altogether than run at the same time (37 rows, a nucleus of 0.9: 111 us in eight
  // CTAs a row, 88 in four).
  // Of eights less the last few, which find a place late: 33 rows of 128256 words, a nucleus of 0.9, 81 us as eights and 76 as fours; 129 rows take
  // 150 us in a CTA each, 107 in pairs, 65 rows 94 us in pairs and 80 as fours.
  auto at_once = [](int size) { return ctas_in_clusters(sample_rows_kernel<T, Params>, size, 2, b200_sm_count(), kThreads, sizeof(Shared)); };
  static_assert(kMaxCluster == 8);
  static const int most[] = {at_once(2), at_once(4), at_once(8) / 64 * 64};
  int ranks = 1;
  for (int i = 0; i < 3 && vocab > ranks * 8192 && (long long)rows * ranks * 2 <= most[i]; ++i) ranks *= 2;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)rows * ranks);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = sizeof(Shared);
  cfg.stream = s;
  cudaLaunchAttribute attr[2]{};
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ranks;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // (as launch_after)
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  B200_CUDA_TRY(cudaLaunchKernelEx(&cfg, sample_rows_kernel<T, Params>, logits, vocab, params, ctx, ctx_off, scratch, tokens, logprobs));
  B200_LAUNCH_CHECK();
  return B200_OK;
}

template <typename Params>
b200_status sample(const void* d_logits, int32_t logits_f32, int32_t rows, int32_t vocab, const Params& params, bool no_params, const uint32_t* d_ctx_tokens,
                   const int32_t* d_ctx_offsets, float* d_scratch, uint32_t* d_tokens, float* d_logprobs, void* stream) {
  if (vocab < 1 || vocab > (1 << 24) || d_logits == nullptr || no_params || d_tokens == nullptr) {
    b200_set_error("sample_rows: vocab %d outside 1..2^24 or a null argument", vocab);
    return B200_ERR_INVALID_ARGUMENT;
  }
  if ((d_ctx_offsets != nullptr) != (d_ctx_tokens != nullptr) || (d_ctx_offsets != nullptr && d_scratch == nullptr)) {
    b200_set_error("sample_rows: context tokens, their offsets and the f32 scratch go together");
    return B200_ERR_INVALID_ARGUMENT;
  }
  cudaStream_t cs = (cudaStream_t)stream;
  return logits_f32 ? launch((const float*)d_logits, rows, vocab, params, d_ctx_tokens, d_ctx_offsets, d_scratch, d_tokens, d_logprobs, cs)
                    : launch((const __nv_bfloat16*)d_logits, rows, vocab, params, d_ctx_tokens, d_ctx_offsets, d_scratch, d_tokens, d_logprobs, cs);
}

}  // namespace

extern "C" {

b200_status b200_sample_rows(const void* d_logits, int32_t logits_f32, int32_t rows, int32_t vocab,
                             const b200_sample_params* d_params, const uint32_t* d_ctx_tokens, const int32_t* d_ctx_offsets,
                             float* d_scratch, uint32_t* d_tokens, float* d_logprobs, void* stream) {
  b200_status st = b200_require_device();
  if (st != B200_OK) return st;
  if (rows <= 0) return B200_OK;
  return sample(d_logits, logits_f32, rows, vocab, InMemory{d_params}, d_params == nullptr, d_ctx_tokens, d_ctx_offsets, d_scratch, d_tokens, d_logprobs, stream);
}

b200_status b200_sample_rows_host(const void* d_logits, int32_t logits_f32, int32_t rows, int32_t vocab,
                                  const b200_sample_params* h_params, const uint32_t* d_ctx_tokens, const int32_t* d_ctx_offsets,
                                  float* d_scratch, uint32_t* d_tokens, float* d_logprobs, void* stream) {
  b200_status st = b200_require_device();
  if (st != B200_OK) return st;
  if (rows <= 0) return B200_OK;
  if (rows > B200_SAMPLE_HOST_ROWS) {
    b200_set_error("sample_rows_host: %d rows, %d at most", rows, B200_SAMPLE_HOST_ROWS);
    return B200_ERR_INVALID_ARGUMENT;
  }
  auto run = [&](auto params) {
    if (h_params) std::copy_n(h_params, rows, params.p);
    return sample(d_logits, logits_f32, rows, vocab, params, h_params == nullptr, d_ctx_tokens, d_ctx_offsets, d_scratch, d_tokens, d_logprobs, stream);
  };
  return rows <= 128 ? run(InArguments<128>{}) : run(InArguments<B200_SAMPLE_HOST_ROWS>{});
}

}  // extern "C"
