// ThresholdTopK on the device (reference: src/threshold.hxx:127-242).
//
// The reference estimates the magnitude cut from a strided sample of
// (rests + input): position (int)(i * (float)n / samples), samples =
// max(default_subsamples, subsample_factor / topK) (or every element when the
// vector is shorter), and takes the element of rank ceil(samples*topK)-1 in
// descending |x| order; when that rank is <= 0 the threshold is max|x| + 1
// so that nothing is sent.  This kernel reproduces that rule bit for bit: the
// sample keys are the bit patterns of |x| (monotonic for non-negative floats),
// and one CTA finds the element of that rank (select_cached; by radix where that does not apply).
// The result stays in device memory, where the compress kernel reads it, so
// no host round trip sits between the two.
//
// Gathering the sample is the expensive part for small top-k fractions (10 000
// strided elements at 0.1 %: 20 000 separate 32-byte sectors, more than one SM's
// load path moves in the time the rest of the kernel takes).  Above 2048 samples the
// kernel therefore runs as a thread-block cluster of 8 CTAs: every CTA gathers one
// eighth of the sample and stores the keys through distributed shared memory into
// the first CTA, which then selects alone.
//
// Samples of up to 2048 elements have a kernel of their own (threshold_small_kernel).  The selection is a chain
// of dependent block-wide steps, so it takes as few as the rank
// allows (see select_cached).  Sampling rules ask for rank 9 unless the fraction is above 1 %.
//
// Several vectors (the buckets of an optimizer step) share one launch, one cluster each: the
// kernel is all latency, and one after the other they would leave the GPU idle in between.
#include <cooperative_groups.h>
#include <math.h>
#include <string.h>

#include "cx_fold.cuh"

namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kSmemKeys = 11008;  // 43 KB of cached sample keys
constexpr int kVectors = 24;      // vectors per launch: their parameters stay within 4 KB

struct ThreshParams {
  const void* g;
  const float* r;
  int64_t n;
  int32_t samples;   // number of sampled elements
  int32_t use_all;   // sample == the whole vector
  float stepsize;
  int32_t topk_pos;  // rank in descending order; <= 0 selects the sentinel
  float* thr_out;
  CxFold fold;       // FOLD: the vector is folded from gradient tensors instead of read from g
};
template <int NV>
struct ThreshBatch {
  ThreshParams v[NV];
};

// element that sample i looks at (the reference's float arithmetic)
__device__ __forceinline__ int64_t sample_position(int i, int64_t n, int use_all, float stepsize) {
  if (use_all) return i;
  const int64_t pos = (int64_t)(int)__fmul_rn((float)i, stepsize);
  return pos > n - 1 ? n - 1 : pos;
}

// Up to 32 keys, one per lane (the same in every warp), of which warp w looks at key w: true if that is
// the key of rank `rank` in descending order.  Two ballots where one warp that ranks them all takes a
// chain of 32 shuffles (1 us behind the barrier).
__device__ __forceinline__ bool has_rank(uint32_t key, uint32_t valid, int w, uint32_t rank) {
  const uint32_t mine = __shfl_sync(0xffffffffu, key, w);
  const uint32_t gt = __popc(__ballot_sync(0xffffffffu, key > mine) & valid);
  const uint32_t ge = __popc(__ballot_sync(0xffffffffu, key >= mine) & valid);
  return ((valid >> w) & 1u) && gt <= rank && rank < ge;
}

template <typename T, bool FOLD>
__device__ __forceinline__ uint32_t sample_key(const ThreshParams& p, int i) {
  const int64_t pos = sample_position(i, p.n, p.use_all, p.stepsize);
  float x = 0.f;
  if (p.r) x = p.r[pos];
  if (FOLD) x = x + cx::fold_at<T>(p.fold, pos);
  else if (p.g) x = x + cx::Elem<T>::to_f(reinterpret_cast<const T*>(p.g)[pos]);
  return __float_as_uint(fabsf(x));
}

constexpr int kGather = 4;  // loads of one thread that are in flight together

// One warp: the digit of `hist` (256 bins, walked from the top) that holds rank `rank`, and the
// rank inside that bin.  All lanes return the same values.
__device__ __forceinline__ uint32_t pick_digit(const uint32_t* hist, uint32_t& rank, int lane) {
  uint32_t h[8], gsum = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) { h[j] = hist[255 - 8 * lane - j]; gsum += h[j]; }
  uint32_t incl = gsum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += t;
  }
  const uint32_t before = incl - gsum;
  uint32_t digit = 0, left = 0;
  const bool mine = rank >= before && rank < incl;   // exactly one lane (rank < number of keys)
  if (mine) {
    uint32_t cum = before;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (rank >= cum && rank < cum + h[j]) { digit = 255 - 8 * lane - j; left = rank - cum; }
      cum += h[j];
    }
  }
  const uint32_t who = __ffs(__ballot_sync(0xffffffffu, mine)) - 1;
  digit = __shfl_sync(0xffffffffu, digit, who & 31);
  rank = __shfl_sync(0xffffffffu, left, who & 31);
  return digit;
}

// One key per thread (threads from `count` on hold none): the largest t with more than `rank` keys at
// or above it, which is the key of that rank, in every thread.  One block-wide count per bit until the
// keys that agree with t so far are few enough to be ranked together.  s_few: 32 words, s_two: two.
__device__ __forceinline__ uint32_t block_rank(uint32_t key, int count, uint32_t rank, uint32_t* s_few, uint32_t* s_two) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool have = (int)threadIdx.x < count;
  uint32_t t = 0, at_t = count, above = 0;    // keys at or above t; keys at or above the end of its interval
  if (threadIdx.x == 0) s_two[0] = 0;
  int bit = 30;
  do {
    const uint32_t c = t | (1u << bit);
    const uint32_t m = __syncthreads_count(have && key >= c);
    if (m > rank) { t = c; at_t = m; } else above = m;
    --bit;
  } while (bit >= 0 && at_t - above > 32);
  if (bit < 0) return t;
  if (have && key >= t && (key >> (bit + 1)) == (t >> (bit + 1))) s_few[atomicAdd(&s_two[0], 1u)] = key;
  __syncthreads();
  const uint32_t k = s_few[lane];
  if (has_rank(k, 0xffffffffu >> (32 - (at_t - above)), w, rank - above) && lane == w) s_two[1] = k;
  __syncthreads();
  return s_two[1];
}

// The key of rank `rank` among s_keys[0, s), for a sample that fits the block's shared memory, to *out.
// s_max: the largest keys of `maxima` (a multiple of 32) disjoint parts that cover the sample.
//  * A lower bound with at least rank + 1 keys at or above it leaves few keys to rank.  Up to rank 31
//    it is the (rank + 1)-th largest of 32 parts' maxima, and the warps rank what is left together;
//    up to rank 767 it is that of the threads' maxima.
//  * What is left (a large rank, or many ties): four radix passes of 8 bits.
// With one warp that ranks by shuffles 25 M elements (10 000 samples) took 57.7 us instead of 57.2.
// (Samples of up to 2048 come here only beside a larger one in the same launch.)
__device__ __forceinline__ void select_cached(uint32_t* s_keys, int s, uint32_t rank, const uint32_t* s_max, int maxima,
                                              uint32_t* s_hist, uint32_t* s_sel, float* out) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  if (rank < 768) {
    uint32_t bound;
    if (tid == 0) s_sel[0] = 0;
    if (rank < 32) {
      uint32_t m = 0;
      for (int i = lane; i < maxima; i += 32) m = max(m, s_max[i]);
      if (has_rank(m, 0xffffffffu, w, rank) && lane == w) s_sel[1] = m;
      __syncthreads();
      bound = s_sel[1];
    } else {
      uint32_t mymax = 0;
      for (int i = tid; i < s; i += kThreads) mymax = max(mymax, s_keys[i]);
      bound = block_rank(mymax, kThreads, rank, s_hist, s_sel + 2);
    }
    for (int i = tid; i < s; i += kThreads) {
      const uint32_t k = s_keys[i];
      if (k >= bound) {
        const uint32_t at = atomicAdd(&s_sel[0], 1u);
        if (at < kThreads) s_hist[at] = k;
      }
    }
    __syncthreads();
    const uint32_t left = s_sel[0];
    if (left <= 32) {
      const uint32_t key = s_hist[lane];        // (what lies behind `left` is not counted)
      if (has_rank(key, 0xffffffffu >> (32 - left), w, rank) && lane == w) *out = __uint_as_float(key);
      return;
    }
    if (left <= kThreads) {
      const uint32_t key = block_rank(tid < (int)left ? s_hist[tid] : 0u, (int)left, rank, s_hist, s_sel + 2);
      if (tid == 0) *out = __uint_as_float(key);
      return;
    }
  }
  uint32_t prefix = 0, prefmask = 0;
  const int s_round = (s + kThreads - 1) / kThreads * kThreads;
  for (int shift = 24; shift >= 0; shift -= 8) {
    __syncthreads();
    if (tid < 256) s_hist[tid] = 0;
    __syncthreads();
    for (int i = tid; i < s_round; i += kThreads) {
      uint32_t digit = 0xffffffffu;
      if (i < s && (s_keys[i] & prefmask) == prefix) digit = (s_keys[i] >> shift) & 255u;
      const uint32_t peers = __match_any_sync(0xffffffffu, digit);
      if (digit != 0xffffffffu && lane == __ffs(peers) - 1) atomicAdd(&s_hist[digit], __popc(peers));
    }
    __syncthreads();
    if (tid < 32) {
      const uint32_t digit = pick_digit(s_hist, rank, lane);
      if (tid == 0) { s_sel[0] = digit; s_sel[1] = rank; }
    }
    __syncthreads();
    prefix |= s_sel[0] << shift;
    prefmask |= 255u << shift;
    rank = s_sel[1];
  }
  if (tid == 0) *out = __uint_as_float(prefix);
}

template <typename T, bool FOLD, int NV>
__global__ void __launch_bounds__(kThreads) threshold_kernel(const __grid_constant__ ThreshBatch<NV> batch) {
  namespace cg = cooperative_groups;
  __shared__ uint32_t s_keys[kSmemKeys];
  __shared__ uint32_t s_hist[kThreads];
  __shared__ uint32_t s_sel[4];
  uint32_t* s_max = s_hist;  // the warps' maxima (of a cluster launch in the first CTA's copy), until it selects
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned ncta = cluster.num_blocks();      // 1 unless launched as a cluster (only when cached)
  const unsigned crank = cluster.block_rank();
  const ThreshParams& p = batch.v[NV == 1 ? 0 : blockIdx.x / ncta];
  const int s = p.samples;
  const bool cached = s <= kSmemKeys;
  uint32_t* keys0 = ncta > 1 ? cluster.map_shared_rank(s_keys, 0) : s_keys;
  if (ncta > 1) cluster.barrier_arrive();
  cx::pdl_wait();     // resident early: what the kernel in front wrote may be read from here on
  if (ncta > 1) cluster.barrier_wait();   // every CTA runs: its shared memory may be written

  // pass 0: gather the sample (and its maximum, for the sentinel case); CTA c of a cluster
  // takes the samples [c, c+1) * s / ncta
  const int lo = (int)((int64_t)s * crank / ncta), hi = (int)((int64_t)s * (crank + 1) / ncta);
  uint32_t mx = 0;
  for (int i0 = lo + tid; i0 < hi; i0 += kGather * kThreads) {
    uint32_t k[kGather];
#pragma unroll
    for (int u = 0; u < kGather; ++u) {
      const int i = i0 + u * kThreads;
      k[u] = i < hi ? sample_key<T, FOLD>(p, i) : 0u;
    }
#pragma unroll
    for (int u = 0; u < kGather; ++u) {
      const int i = i0 + u * kThreads;
      if (i < hi) {
        if (cached) keys0[i] = k[u];
        mx = max(mx, k[u]);
      }
    }
  }
  // the compress kernel queued behind this one may start now: it loads what both only read, and waits
  // for this grid to finish before it reads the threshold or writes the residual.  (Let in before the
  // gather, its 20 MB of loads were in front of the sample's.)
  cx::pdl_trigger();
  const uint32_t wm = __reduce_max_sync(0xffffffffu, mx);
  if (lane == 0) (ncta > 1 ? cluster.map_shared_rank(s_max, 0) : s_max)[crank * kWarps + (tid >> 5)] = wm;
  if (ncta > 1) {
    cluster.sync();              // keys and maxima of all CTAs are in the first CTA's shared memory
    if (crank != 0) return;      // (no CTA touches another CTA's shared memory after this point)
  } else {
    __syncthreads();
  }
  if (p.topk_pos <= 0) {
    if (tid < 32) {
      uint32_t m = 0;
      for (unsigned i = lane; i < ncta * kWarps; i += 32) m = max(m, s_max[i]);
      m = __reduce_max_sync(0xffffffffu, m);
      if (tid == 0) *p.thr_out = __uint_as_float(m) + 1.0f;
    }
    return;
  }
  if (cached) {
    select_cached(s_keys, s, (uint32_t)p.topk_pos, s_max, (int)(ncta * kWarps), s_hist, s_sel, p.thr_out);
    return;
  }

  // a sample larger than the cache (and no workspace for the grid-wide selection below): the keys
  // are gathered again in every radix pass
  const int64_t s_round = ((int64_t)s + kThreads - 1) / kThreads * kThreads;
  uint32_t prefix = 0, prefmask = 0;
  uint32_t rank = (uint32_t)p.topk_pos;
  for (int shift = 24; shift >= 0; shift -= 8) {
    if (tid < 256) s_hist[tid] = 0;
    __syncthreads();
    for (int64_t i = tid; i < s_round; i += kThreads) {
      uint32_t digit = 0xffffffffu;
      if (i < s) {
        const uint32_t k = sample_key<T, FOLD>(p, (int)i);
        if ((k & prefmask) == prefix) digit = (k >> shift) & 255u;
      }
      const uint32_t peers = __match_any_sync(0xffffffffu, digit);
      if (digit != 0xffffffffu && lane == __ffs(peers) - 1) atomicAdd(&s_hist[digit], __popc(peers));
    }
    __syncthreads();
    if (tid < 32) {
      const uint32_t digit = pick_digit(s_hist, rank, lane);
      if (tid == 0) { s_sel[0] = digit; s_sel[1] = rank; }
    }
    __syncthreads();
    prefix |= s_sel[0] << shift;
    prefmask |= 255u << shift;
    rank = s_sel[1];
    __syncthreads();
  }
  if (tid == 0) *p.thr_out = __uint_as_float(prefix);
}

// ---- samples of up to 2048 elements ------------------------------------------------------------
// All latency: the chain is the gather, then steps of the whole CTA.  256 threads hold the keys in registers,
// up to eight each, with all their loads in flight: a barrier of 8 warps and a handful of them, where 32 warps
// that keep the keys in shared memory spent half of the kernel in barriers (exchange of 2^16 / 2^20 elements
// 11.4 / 14.1 -> 10.7 / 13.1 us, LeNet-5 step 18.7 -> 18.4).  A folded vector's dependent look-ups go side by side.
constexpr int kSmallThreads = 256, kSmallEach = 8, kSmallWarps = kSmallThreads / 32;
constexpr int kSmallSample = kSmallThreads * kSmallEach;
constexpr int kSmallRound = 4;       // samples of a thread whose loads go together

// keys of samples tid, tid + 256, ... (kSmallRound of them from `first` on)
template <typename T, bool FOLD>
__device__ __forceinline__ void gather_small(const ThreshParams& p, int first, uint32_t (&k)[kSmallRound]) {
  int64_t pos[kSmallRound];
  float x[kSmallRound], y[kSmallRound];
  bool in[kSmallRound];
#pragma unroll
  for (int u = 0; u < kSmallRound; ++u) {
    const int i = first + u * kSmallThreads;
    in[u] = i < p.samples;
    pos[u] = in[u] ? sample_position(i, p.n, p.use_all, p.stepsize) : 0;
    x[u] = p.r && in[u] ? p.r[pos[u]] : 0.f;
    y[u] = 0.f;
  }
  if (FOLD) {
    // cx::fold_at for all of them step by step, so that the steps' loads are in flight together
    const CxFold& f = p.fold;
    int seg[kSmallRound];
    int64_t end[kSmallRound], off[kSmallRound];
    float m[kSmallRound], coef[kSmallRound];
    const T* g[kSmallRound];
#pragma unroll
    for (int u = 0; u < kSmallRound; ++u) {
      seg[u] = in[u] ? f.sub_seg[pos[u] / CX_SUBTILE] : f.nseg;
      m[u] = in[u] && f.mu != 0.f ? f.u[pos[u]] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < kSmallRound; ++u) end[u] = seg[u] < f.nseg ? f.seg_end[seg[u]] : INT64_MAX;
    for (bool again = true; again;) {
      again = false;
#pragma unroll
      for (int u = 0; u < kSmallRound; ++u) {
        if (end[u] <= f.base + pos[u]) {
          ++seg[u];
          end[u] = seg[u] < f.nseg ? f.seg_end[seg[u]] : INT64_MAX;
          again = true;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < kSmallRound; ++u) {
      const bool t = seg[u] < f.nseg;
      off[u] = t ? f.seg_off[seg[u]] : INT64_MAX;
      g[u] = t ? reinterpret_cast<const T*>(f.seg_ptr[seg[u]]) : nullptr;
      coef[u] = t ? f.coef[seg[u]] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < kSmallRound; ++u)       // (a gap between tensors: 0)
      if (off[u] <= f.base + pos[u]) y[u] = f.mu * m[u] + coef[u] * cx::Elem<T>::to_f(g[u][f.base + pos[u] - off[u]]);
  } else if (p.g) {
#pragma unroll
    for (int u = 0; u < kSmallRound; ++u) if (in[u]) y[u] = cx::Elem<T>::to_f(reinterpret_cast<const T*>(p.g)[pos[u]]);
  }
#pragma unroll
  for (int u = 0; u < kSmallRound; ++u) k[u] = in[u] ? __float_as_uint(fabsf(FOLD || p.g ? x[u] + y[u] : x[u])) : 0u;
}

template <typename T, bool FOLD, int NV>
__global__ void __launch_bounds__(kSmallThreads) threshold_small_kernel(const __grid_constant__ ThreshBatch<NV> batch) {
  __shared__ __align__(16) uint32_t s_max[kSmallRound * kSmallWarps];     // 32 disjoint parts of the sample
  __shared__ uint32_t s_sum[2][kSmallWarps];
  __shared__ uint32_t s_few[kSmallThreads];
  __shared__ uint32_t s_left;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const ThreshParams& p = batch.v[NV == 1 ? 0 : blockIdx.x];
  const int s = p.samples;
  if (tid == 0) s_left = 0;
  cx::pdl_wait();     // resident early: what the kernel in front wrote may be read from here on
  uint32_t k[kSmallEach];
  {
    uint32_t a[kSmallRound], b[kSmallRound] = {0u, 0u, 0u, 0u};
    gather_small<T, FOLD>(p, tid, a);
    if (s > kSmallRound * kSmallThreads) gather_small<T, FOLD>(p, tid + kSmallRound * kSmallThreads, b);
#pragma unroll
    for (int u = 0; u < kSmallRound; ++u) {
      k[u] = a[u];
      k[kSmallRound + u] = b[u];
      const uint32_t m = __reduce_max_sync(0xffffffffu, max(a[u], b[u]));
      if (lane == 0) s_max[kSmallRound * w + u] = m;
    }
  }
  // the compress kernel queued behind this one may start now: it loads what both only read, and waits
  // for this grid to finish before it reads the threshold or writes the residual.  (Let in before the
  // gather, its 20 MB of loads were in front of the sample's.)
  cx::pdl_trigger();
  __syncthreads();
  const uint32_t mine = s_max[lane];
  if (p.topk_pos <= 0) {
    const uint32_t m = __reduce_max_sync(0xffffffffu, mine);
    if (tid == 0) *p.thr_out = __uint_as_float(m) + 1.0f;
    return;
  }
  const uint32_t rank = (uint32_t)p.topk_pos;
  // keys in [lo, hi] are candidates, `above` keys are larger than those
  uint32_t lo = 0, hi = 0x7fffffffu, above = 0;
  bool few = false;
  if (rank < 32) {
    // the (rank + 1)-th largest of the parts' maxima: at least rank + 1 keys are as large.  Every warp for itself.
    uint32_t gt = 0, ge = 0;
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      const uint4 q = *reinterpret_cast<const uint4*>(s_max + j);
      gt += (q.x > mine) + (q.y > mine) + (q.z > mine) + (q.w > mine);
      ge += (q.x >= mine) + (q.y >= mine) + (q.z >= mine) + (q.w >= mine);
    }
    const uint32_t who = __ballot_sync(0xffffffffu, gt <= rank && rank < ge);
    lo = __shfl_sync(0xffffffffu, mine, __ffs(who) - 1);
    few = lo > 0;            // (0: fewer than rank + 1 parts hold anything)
  }
  for (int attempt = 0;; ++attempt) {
    if (!few) {
      // bisection over the bits: t is the largest value so far with more than `rank` keys at or above it
      uint32_t t = 0, at_t = (uint32_t)s;
      above = 0;
      int bit = 30;
      do {
        const uint32_t c = t | (1u << bit);
        uint32_t n = 0;
#pragma unroll
        for (int u = 0; u < kSmallEach; ++u) n += k[u] >= c ? 1u : 0u;
        n = __reduce_add_sync(0xffffffffu, n);
        uint32_t* sum = s_sum[bit & 1];           // (written again two rounds on, behind the other's barrier)
        if (lane == 0) sum[w] = n;
        __syncthreads();
        n = 0;
#pragma unroll
        for (int j = 0; j < kSmallWarps; ++j) n += sum[j];
        if (n > rank) { t = c; at_t = n; } else above = n;
        --bit;
      } while (bit >= 0 && at_t - above > 64);
      if (bit < 0) {                              // all candidates are equal
        if (tid == 0) *p.thr_out = __uint_as_float(t);
        return;
      }
      lo = t;
      hi = t | ((2u << bit) - 1u);
    }
#pragma unroll
    for (int u = 0; u < kSmallEach; ++u) {
      if (k[u] >= lo && k[u] <= hi && (u * kSmallThreads + tid) < s) {
        const uint32_t at = atomicAdd(&s_left, 1u);
        if (at < (uint32_t)kSmallThreads) s_few[at] = k[u];
      }
    }
    __syncthreads();
    const uint32_t left = s_left;
    if (left <= (uint32_t)kSmallThreads) {
      if (tid < (int)left) {                      // every candidate counts the ones above it; equal ones write the same
        const uint32_t key = s_few[tid];
        uint32_t gt = above, ge = above;
        for (uint32_t j = 0; j < left; ++j) {
          gt += s_few[j] > key ? 1u : 0u;
          ge += s_few[j] >= key ? 1u : 0u;
        }
        if (gt <= rank && rank < ge) *p.thr_out = __uint_as_float(key);
      }
      return;
    }
    __syncthreads();                              // many ties: bisect (at most 64 candidates, or all equal)
    if (tid == 0) s_left = 0;
    few = false;
    __syncthreads();
  }
}

// ---- exact selection over the whole vector, grid-wide ----------------------------------------
// With sampling switched off (every element is a sample) the single CTA above would walk the
// vector four times on its own.  Here every radix pass is a grid-wide histogram instead: each
// CTA replays the digits chosen so far from the global histograms of the earlier passes (256
// counters each), counts the next digit of the keys that still match into shared memory and
// adds its counts to the global histogram of this pass.  Four such launches and a one-warp
// finish read the vector four times at full bandwidth.  The result is the key of rank topk_pos
// in descending order, the same value the single CTA finds.
constexpr int kExactThreads = 256;

struct ExactParams {
  const void* g;
  const float* r;
  int64_t n;
  uint32_t topk_pos;
  int pass;            // 0..3: digit at shift 24 - 8 * pass; 4: finish
  uint32_t* hist;      // [4][256], zero before the first pass; the finish zeroes it again
  float* thr_out;
  uint32_t vec;        // 16-byte accesses are possible
};

template <typename T>
__global__ void __launch_bounds__(kExactThreads) exact_select_kernel(const ExactParams p) {
  __shared__ uint32_t s_hist[256];
  __shared__ uint32_t s_prefix;
  const int tid = threadIdx.x, lane = tid & 31;
  s_hist[tid] = 0;
  if (tid < 32) {      // the decisions of the earlier passes
    uint32_t prefix = 0, rank = p.topk_pos;
    for (int q = 0; q < p.pass && q < 4; ++q) prefix |= pick_digit(p.hist + 256 * q, rank, lane) << (24 - 8 * q);
    if (tid == 0) s_prefix = prefix;
  }
  __syncthreads();
  const uint32_t prefix = s_prefix;
  if (p.pass >= 4) {   // finish: the key of that rank is the threshold; leave the scratch clean
    if (blockIdx.x == 0) {
      if (tid == 0) *p.thr_out = __uint_as_float(prefix);
      for (int i = tid; i < 4 * 256; i += kExactThreads) p.hist[i] = 0;
    }
    return;
  }
  const int shift = 24 - 8 * p.pass;
  const uint32_t prefmask = p.pass == 0 ? 0u : (0xffffffffu << (shift + 8));
  const T* g = reinterpret_cast<const T*>(p.g);
  auto count = [&](float x, bool valid) {
    const uint32_t k = __float_as_uint(fabsf(x));
    const uint32_t digit = (valid && (k & prefmask) == prefix) ? ((k >> shift) & 255u) : 0xffffffffu;
    const uint32_t peers = __match_any_sync(0xffffffffu, digit);
    if (digit != 0xffffffffu && lane == __ffs(peers) - 1) atomicAdd(&s_hist[digit], __popc(peers));
  };
  const int64_t gsz = (int64_t)gridDim.x * kExactThreads;
  const int64_t nv = (p.n + 3) / 4;
  const int64_t rounds = (nv + gsz - 1) / gsz;      // every lane runs every round: the counting is warp-wide
  for (int64_t it = 0; it < rounds; ++it) {
    const int64_t i = (it * gsz + (int64_t)blockIdx.x * kExactThreads + tid) * 4;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (p.vec && i + 3 < p.n) {
      if (p.r) cx::load4(p.r + i, v);
      if (g) {
        float b[4];
        cx::load4(g + i, b);
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = v[e] + b[e];
      }
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (i + e < p.n) {
          if (p.r) v[e] = p.r[i + e];
          if (g) v[e] = v[e] + cx::Elem<T>::to_f(g[i + e]);
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) count(v[e], i + e < p.n);
  }
  __syncthreads();
  if (s_hist[tid]) atomicAdd(&p.hist[256 * p.pass + tid], s_hist[tid]);
}

// ---- exact selection with one pass over the vector -----------------------------------------------
// With scratch for candidates (cx_threshold_exact_bytes) the four passes become one:
//   1. bracket: two keys lo <= hi from a sample of 8192 elements, one per stratum at a hashed position
//      (a fixed stride could meet the same column of every row), between which the wanted key lies
//      unless the sample is off by more than four standard deviations,
//   2. collect: one pass counts the keys above hi, at hi and at lo, and appends the ones between to
//      the candidate list (about 1 % of the vector), counting them by their 11 highest bits,
//   3. finish:  the counts name the bin; a cluster picks the few candidates in it and ranks those
//      (more than fit: it goes on by radix).  If the counts show that the bracket
//      missed, or the candidates did not fit, it selects over the whole vector instead: always exact,
//      only slower.
// 10 M elements, fp32 vector and residual, top-k 1 %: 96 us with four passes.
constexpr int kBracket = 8192;
constexpr int kCluster = 8;
constexpr int kBracketThreads = 512;   // fits next to a receive kernel's CTAs
constexpr int kBins = 2048;          // 11 bits per radix pass of the finish
constexpr int kCollectThreads = 256;
constexpr int kCollectEach = 8;      // elements per thread and round
constexpr int kBuffer = 3072;        // candidates a CTA keeps before it appends them to the list
constexpr int kCollectRounds = 16;   // rounds between two looks at how full that buffer is
constexpr int kCollectPerSm = 5;     // registers

struct ExactState {                  // in the workspace behind the histograms; zero between calls
  uint32_t lo, hi;
  uint32_t above, at_hi, at_lo;      // elements with key > hi, == hi, == lo (lo < hi)
  uint32_t found;                    // candidates with lo < key < hi (not all of them stored when over cap)
  uint32_t pad[58];
  uint32_t hist[kBins];              // candidates by their 11 highest bits between lo and hi
};

// candidates are lo + 1 .. hi - 1; how far their distance from lo + 1 is shifted for its bin
__device__ __forceinline__ uint32_t bracket_base(uint32_t lo) { return lo + 1; }
__device__ __forceinline__ int bracket_bits(uint32_t lo, uint32_t hi) {
  return 32 - __clz((min(hi, 0x80000000u) - 1 - bracket_base(lo)) | 1u);
}

struct OnePassParams {
  const void* g;
  const float* r;
  int64_t n;
  uint32_t rank;         // in descending order
  uint32_t cap;          // candidates that fit the list
  uint32_t hi_rank;      // ranks of the bracket in the sample; hi_rank == ~0u: no upper bound
  uint32_t lo_rank;      // ~0u: no lower bound
  ExactState* st;
  uint32_t* list;
  float* thr_out;
  uint32_t vec;
};

template <typename T>
__device__ __forceinline__ uint32_t key_at(const OnePassParams& p, int64_t i) {
  float x = p.r ? p.r[i] : 0.f;
  if (p.g) x = x + cx::Elem<T>::to_f(reinterpret_cast<const T*>(p.g)[i]);
  return __float_as_uint(fabsf(x));
}

// The digit of a 2048-bin histogram that holds `rank`, walked from the top; all THREADS threads.
template <int THREADS>
__device__ __forceinline__ uint32_t pick_bin(const uint32_t* hist, uint32_t& rank, uint32_t* s_warp, uint32_t* s_out) {
  constexpr int kEach = kBins / THREADS;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  uint32_t h[kEach], sum = 0;
#pragma unroll
  for (int j = 0; j < kEach; ++j) { h[j] = hist[kBins - 1 - kEach * tid - j]; sum += h[j]; }
  uint32_t incl = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += t;
  }
  if (lane == 31) s_warp[w] = incl;
  __syncthreads();
  // lane j holds warp j's sum: the warps before mine
  uint32_t before = __reduce_add_sync(0xffffffffu, lane < w ? s_warp[lane] : 0u) + incl - sum;
#pragma unroll
  for (int j = 0; j < kEach; ++j) {
    if (rank >= before && rank < before + h[j]) { s_out[0] = kBins - 1 - kEach * tid - j; s_out[1] = rank - before; }
    before += h[j];
  }
  __syncthreads();
  rank = s_out[1];
  return s_out[0];
}

// The key of rank `rank` among s_keys[0, count): three radix passes (11, 11, 9 bits).
template <int THREADS>
__device__ __forceinline__ uint32_t radix_rank(const uint32_t* s_keys, int count, uint32_t rank, uint32_t* s_hist,
                                               uint32_t* s_warp, uint32_t* s_out) {
  uint32_t prefix = 0, mask = 0;
#pragma unroll
  for (int pass = 0; pass < 3; ++pass) {
    const int shift = pass == 0 ? 20 : pass == 1 ? 9 : 0;
    const uint32_t low = pass == 2 ? 511u : 2047u;
    for (int i = threadIdx.x; i < kBins; i += THREADS) s_hist[i] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < count; i += THREADS) {
      const uint32_t k = s_keys[i];
      if ((k & mask) == prefix) atomicAdd(&s_hist[(k >> shift) & low], 1u);
    }
    __syncthreads();
    prefix |= pick_bin<THREADS>(s_hist, rank, s_warp, s_out) << shift;
    mask |= low << shift;
  }
  return prefix;
}

template <typename T>
__global__ void __launch_bounds__(kBracketThreads) bracket_kernel(const __grid_constant__ OnePassParams p) {
  namespace cg = cooperative_groups;
  __shared__ uint32_t s_keys[kBracket];
  __shared__ uint32_t s_hist[kBins];
  __shared__ uint32_t s_out[2];
  __shared__ uint32_t s_warp[kBracketThreads / 32];
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned crank = cluster.block_rank();
  const int tid = threadIdx.x;
  uint32_t* k0 = cluster.map_shared_rank(s_keys, 0);
  uint32_t* k1 = cluster.map_shared_rank(s_keys, 1);
  cluster.barrier_arrive();
  cx::pdl_wait();
  cx::pdl_trigger();
  cluster.barrier_wait();             // every CTA runs: the first two's shared memory may be written
  {
    constexpr int kEach = kBracket / kCluster / kBracketThreads;
    uint32_t k[kEach];
#pragma unroll
    for (int u = 0; u < kEach; ++u) {
      const uint32_t i = (crank * kEach + u) * kBracketThreads + tid;
      const int64_t a = (int64_t)(((uint64_t)p.n * i) / kBracket), b = (int64_t)(((uint64_t)p.n * (i + 1)) / kBracket);
      const uint32_t h = (i + 1) * 2654435761u;
      k[u] = key_at<T>(p, a + (int64_t)(((uint64_t)(h ^ (h >> 15)) * (uint64_t)(b - a)) >> 32));
    }
#pragma unroll
    for (int u = 0; u < kEach; ++u) k0[(crank * kEach + u) * kBracketThreads + tid] = k1[(crank * kEach + u) * kBracketThreads + tid] = k[u];
  }
  cluster.sync();                     // CTA 0 selects lo, CTA 1 hi, each in its own shared memory
  if (crank > 1) return;
  const uint32_t rank = crank == 0 ? p.lo_rank : p.hi_rank;
  uint32_t key = crank == 0 ? 0u : 0xffffffffu;
  if (rank != ~0u) key = radix_rank<kBracketThreads>(s_keys, kBracket, rank, s_hist, s_warp, s_out);
  if (tid == 0) {
    if (crank == 0) p.st->lo = key;
    else p.st->hi = key;
  }
}

// Bound by instructions, then by the read of the vector.  A thread compares its eight elements with the bracket
// and keeps two bits of each; only those inside the bracket (1 %) are looked at one by one, and nobody waits for
// the other warps: the CTA's buffer is emptied every 16 rounds, and what finds it full goes to the list at once.
// With a vote for every element and two barriers a round 10 M fp32 elements took 23.5 us by itself, now 19.6; an
// exchange of 1 M elements 30.9 -> 29.4 us (10 M: 63.4 -> 63.0).
template <typename T>
__global__ void __launch_bounds__(kCollectThreads, kCollectPerSm) collect_kernel(const __grid_constant__ OnePassParams p) {
  __shared__ uint32_t s_buf[kBuffer];
  __shared__ uint32_t s_hist[kBins];
  __shared__ uint32_t s_fill, s_kept, s_base;    // s_kept: where the buffer's entries end once it was full
  __shared__ uint32_t s_cnt[3];
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid == 0) { s_fill = 0; s_kept = kBuffer; }
  for (int i = tid; i < kBins; i += kCollectThreads) s_hist[i] = 0;
  if (tid < 3) s_cnt[tid] = 0;
  cx::pdl_wait();
  cx::pdl_trigger();
  const uint32_t lo = p.st->lo, hi = p.st->hi;
  const float lof = __uint_as_float(lo), hif = __uint_as_float(hi);      // (no upper bound: a NaN)
  const int shift = max(bracket_bits(lo, hi) - 11, 0);
  const T* g = reinterpret_cast<const T*>(p.g);
  uint32_t above = 0, at_hi = 0, at_lo = 0;
  __syncthreads();
  const int64_t round = (int64_t)kCollectThreads * kCollectEach;
  auto flush = [&]() {                // all threads
    const uint32_t fill = min(s_fill, s_kept);
    if (tid == 0) s_base = atomicAdd(&p.st->found, fill);
    __syncthreads();
    for (uint32_t i = tid; i < fill; i += kCollectThreads)
      if (s_base + i < p.cap) p.list[s_base + i] = s_buf[i];
    __syncthreads();
    if (tid == 0) { s_fill = 0; s_kept = kBuffer; }
    __syncthreads();
  };
  int rounds = 0;
  for (int64_t b = (int64_t)blockIdx.x * round; b < p.n; b += (int64_t)gridDim.x * round) {
    float v[kCollectEach];
    const bool whole = p.vec && b + round <= p.n;
    uint32_t valid = (1u << kCollectEach) - 1u;
    if (whole) {
      constexpr int kQ = kCollectEach / 4;
      float y[kQ][4];
      typename cx::Raw4<T>::type z[kQ];
#pragma unroll
      for (int k = 0; k < kQ; ++k) {
        const int64_t i = b + (int64_t)k * kCollectThreads * 4 + tid * 4;
        if (p.r) cx::load4(p.r + i, y[k]);
        if (g) z[k] = cx::Raw4<T>::load(g + i);
      }
#pragma unroll
      for (int k = 0; k < kQ; ++k) {
        float t[4] = {0.f, 0.f, 0.f, 0.f};
        if (g) cx::Raw4<T>::to_f(z[k], t);
#pragma unroll
        for (int e = 0; e < 4; ++e) v[4 * k + e] = p.r ? (g ? y[k][e] + t[e] : y[k][e]) : t[e];
      }
    } else {
      valid = 0;
#pragma unroll
      for (int k = 0; k < kCollectEach; ++k) {
        const int64_t i = b + (int64_t)(k / 4) * kCollectThreads * 4 + tid * 4 + (k & 3);
        v[k] = 0.f;
        if (i < p.n) {
          if (p.r) v[k] = p.r[i];
          if (g) v[k] = v[k] + cx::Elem<T>::to_f(g[i]);
          valid |= 1u << k;
        }
      }
    }
    // keys are compared as integers below; as floats, every key that is not plainly below or above the bracket
    // (a NaN never is) counts as inside
    uint32_t from_lo = 0, over = 0;
#pragma unroll
    for (int k = 0; k < kCollectEach; ++k) {
      if (!(fabsf(v[k]) < lof)) from_lo |= 1u << k;
      if (fabsf(v[k]) > hif) over |= 1u << k;
    }
    above += __popc(over & valid);
    uint32_t mid = from_lo & ~over & valid;
    while (__any_sync(0xffffffffu, mid != 0)) {
      const bool have = mid != 0;
      const int k = have ? __ffs(mid) - 1 : 0;
      mid &= mid - 1;
      float x[kCollectEach / 2];
#pragma unroll
      for (int j = 0; j < kCollectEach / 2; ++j) x[j] = k & 1 ? v[2 * j + 1] : v[2 * j];
#pragma unroll
      for (int j = 0; j < kCollectEach / 4; ++j) x[j] = k & 2 ? x[2 * j + 1] : x[2 * j];
      static_assert(kCollectEach == 8, "three levels");
      const uint32_t key = __float_as_uint(fabsf(k & 4 ? x[1] : x[0]));
      const bool near = have && key >= lo;
      above += near && key > hi;
      at_hi += near && key == hi;
      at_lo += near && key == lo && lo != hi;
      const bool cand = near && key > lo && key < hi;
      const uint32_t who = __ballot_sync(0xffffffffu, cand);
      if (who) {
        const uint32_t number = __popc(who);
        const int first = __ffs(who) - 1;
        uint32_t at = 0;
        if (lane == first) at = atomicAdd(&s_fill, number);
        at = __shfl_sync(0xffffffffu, at, first);
        const bool room = at + number <= kBuffer;       // once it is false it stays so until the buffer is emptied
        uint32_t to = at;
        if (!room) {
          if (lane == first) { atomicMin(&s_kept, at); to = atomicAdd(&p.st->found, number); }
          to = __shfl_sync(0xffffffffu, to, first);
        }
        if (cand) {
          to += __popc(who & ((1u << lane) - 1u));
          if (room) s_buf[to] = key;
          else if (to < p.cap) p.list[to] = key;
          atomicAdd(&s_hist[(key - bracket_base(lo)) >> shift], 1u);
        }
      }
    }
    if (++rounds % kCollectRounds == 0) {
      __syncthreads();
      if (s_fill > kBuffer / 2) flush();                // uniform
      else __syncthreads();
    }
  }
  if (above) atomicAdd(&s_cnt[0], above);
  if (at_hi) atomicAdd(&s_cnt[1], at_hi);
  if (at_lo) atomicAdd(&s_cnt[2], at_lo);
  __syncthreads();
  if (tid == 0) {
    if (s_cnt[0]) atomicAdd(&p.st->above, s_cnt[0]);
    if (s_cnt[1]) atomicAdd(&p.st->at_hi, s_cnt[1]);
    if (s_cnt[2]) atomicAdd(&p.st->at_lo, s_cnt[2]);
  }
  for (int i = tid; i < kBins; i += kCollectThreads) if (s_hist[i]) atomicAdd(&p.st->hist[i], s_hist[i]);
  if (s_fill) flush();
}

template <typename T>
__global__ void __launch_bounds__(kThreads) exact_finish_kernel(const __grid_constant__ OnePassParams p) {
  namespace cg = cooperative_groups;
  __shared__ uint32_t s_hists[3][kBins];     // one per radix pass
  __shared__ uint32_t s_warp[kThreads / 32];
  __shared__ uint32_t s_out[2];
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned crank = cluster.block_rank();
  const int tid = threadIdx.x;
  for (int i = tid; i < 3 * kBins; i += kThreads) s_hists[0][i] = 0;
  uint32_t* out0 = cluster.map_shared_rank(s_out, 0);
  cx::pdl_wait();
  cx::pdl_trigger();
  struct { uint32_t lo, hi, above, at_hi, at_lo, found; } st;
  st.lo = p.st->lo; st.hi = p.st->hi; st.above = p.st->above; st.at_hi = p.st->at_hi; st.at_lo = p.st->at_lo; st.found = p.st->found;
  s_hists[2][tid] = p.st->hist[tid];          // (the third radix pass is behind a cluster barrier that clears it again)
  s_hists[2][tid + kThreads] = p.st->hist[tid + kThreads];
  cluster.sync();                     // every CTA has read the state and cleared its histograms
  if (crank == 0 && tid == 0) p.st->above = p.st->at_hi = p.st->at_lo = p.st->found = 0;
  if (crank == 1) p.st->hist[tid] = p.st->hist[tid + kThreads] = 0;
  uint32_t rank = p.rank, base = 0, top = 0x7fffffffu;
  bool list = false;
  if (st.found <= p.cap && rank >= st.above) {
    const uint32_t left = rank - st.above;
    if (left < st.at_hi) { if (crank == 0 && tid == 0) *p.thr_out = __uint_as_float(st.hi); return; }
    if (left - st.at_hi < st.found) {
      list = true;
      rank = left - st.at_hi;
      base = bracket_base(st.lo);
      top = min(st.hi, 0x80000000u) - 1;
    } else if (left - st.at_hi - st.found < st.at_lo) {
      if (crank == 0 && tid == 0) *p.thr_out = __uint_as_float(st.lo);
      return;
    }
  }
  const int bits = 32 - __clz((top - base) | 1u);
  if (list) {
    const int shift = max(bits - 11, 0);
    uint32_t in_bin = rank;
    const uint32_t bin = pick_bin<kThreads>(s_hists[2], in_bin, s_warp, s_out);      // every CTA for itself
    if (s_hists[2][bin] <= kThreads) {
      uint32_t* few = cluster.map_shared_rank(s_hists[0], 0);              // [0]: their number
      uint32_t* keys = cluster.map_shared_rank(s_hists[1], 0);
      const int64_t step = (int64_t)kCluster * kThreads;
      for (int64_t i0 = (int64_t)crank * kThreads + tid; i0 < st.found; i0 += 4 * step) {
        uint32_t k[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) k[u] = i0 + u * step < st.found ? p.list[i0 + u * step] : 0u;
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (i0 + u * step < st.found && ((k[u] - base) >> shift) == bin) keys[atomicAdd(few, 1u)] = k[u];
      }
      cluster.sync();
      if (crank != 0) return;
      const uint32_t left = s_hists[0][0];
      if (tid < (int)left) {              // every key counts the ones above it
        const uint32_t key = s_hists[1][tid];
        uint32_t gt = 0, ge = 0;
        for (uint32_t j = 0; j < left; ++j) {
          gt += s_hists[1][j] > key ? 1u : 0u;
          ge += s_hists[1][j] >= key ? 1u : 0u;
        }
        if (gt <= in_bin && in_bin < ge) *p.thr_out = __uint_as_float(key);    // equal keys write the same
      }
      return;
    }
  }
  for (int i = tid; i < kBins; i += kThreads) s_hists[2][i] = 0;
  cluster.sync();
  // radix select of key - base in [0, top - base], 11 bits at a time from the highest bit in use
  uint32_t prefix = 0, mask = 0;
  const int64_t count = list ? (int64_t)st.found : p.n;
  int pass = 0;
  for (int shift = bits > 11 ? bits - 11 : 0;; shift = shift > 11 ? shift - 11 : 0, ++pass) {
    uint32_t* s_hist = s_hists[pass];
    uint32_t* hist0 = cluster.map_shared_rank(s_hist, 0);
    const int64_t step = (int64_t)kCluster * kThreads;
    for (int64_t i0 = (int64_t)crank * kThreads + tid; i0 < count; i0 += 4 * step) {
      uint32_t k[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t i = i0 + u * step;
        k[u] = i < count ? (list ? p.list[i] : key_at<T>(p, i)) - base : 0xffffffffu;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i0 + u * step < count && (k[u] & mask) == prefix) atomicAdd(&s_hist[(k[u] >> shift) & (kBins - 1)], 1u);
    }
    __syncthreads();
    if (crank != 0)
      for (int i = tid; i < kBins; i += kThreads) if (s_hist[i]) atomicAdd(&hist0[i], s_hist[i]);
    cluster.sync();
    if (crank == 0) pick_bin<kThreads>(s_hist, rank, s_warp, s_out);
    cluster.sync();
    prefix |= out0[0] << shift;
    rank = out0[1];
    mask = 0xffffffffu << shift;
    if (shift == 0) break;            // (the next pass writes s_out behind its own cluster barrier)
  }
  if (crank == 0 && tid == 0) *p.thr_out = __uint_as_float(base + prefix);
  cluster.sync();                     // the first CTA's shared memory is read until here
}

template <typename T>
int launch_one_pass(const OnePassParams& p, bool capturing, cudaStream_t s) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(kCluster, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kCluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = !capturing && cx_pdl_enabled() ? 2 : 1;
  cfg.blockDim = dim3(kBracketThreads, 1, 1);
  cudaError_t e = cudaLaunchKernelEx(&cfg, bracket_kernel<T>, p);
  cfg.blockDim = dim3(kThreads, 1, 1);
  if (e != cudaSuccess) return cx_set_error("bracket_kernel launch", (int)e);
  const int64_t round = (int64_t)kCollectThreads * kCollectEach;
  int grid = cx_sm_count() * kCollectPerSm;
  if (grid > (p.n + round - 1) / round) grid = (int)((p.n + round - 1) / round);
  cx_launch_pdl(collect_kernel<T>, grid, kCollectThreads, 0, s, p, capturing);
  e = cudaLaunchKernelEx(&cfg, exact_finish_kernel<T>, p);
  if (e != cudaSuccess) return cx_set_error("exact_finish_kernel launch", (int)e);
  cx_note_stream(s, true);       // it may read the whole vector behind its trigger
  for (int k = 0; k < 3; ++k) cx_note_launch();
  return cx_check_launch("exact selection kernels");
}

uint32_t candidate_cap(int64_t n) { return (uint32_t)(n / 16 > 65536 ? n / 16 : 65536); }

template <typename T>
int launch_exact(const ExactParams& base, cudaStream_t s) {
  int grid = cx_sm_count() * 6;
  const int64_t need = ((base.n + 3) / 4 + kExactThreads - 1) / kExactThreads;
  if (grid > need) grid = (int)need;
  for (int pass = 0; pass <= 4; ++pass) {
    ExactParams p = base;
    p.pass = pass;
    exact_select_kernel<T><<<pass < 4 ? grid : 1, kExactThreads, 0, s>>>(p);
    cx_note_launch();
  }
  return cx_check_launch("exact_select_kernel");
}

}  // namespace

extern "C" int64_t cx_threshold_workspace_bytes(void) { return 4 * 256 * (int64_t)sizeof(uint32_t); }

extern "C" int64_t cx_threshold_exact_bytes(int64_t n) {
  return cx_threshold_workspace_bytes() + (int64_t)sizeof(ExactState) + 4 * (int64_t)candidate_cap(n);
}

// Host-side part of the rule, in the reference's float arithmetic.
// sample count, stride and rank of the estimate (defined with the host back end)
extern "C" void cx_threshold_plan(int64_t n, float ratio, int default_subsamples,
                                  float subsample_factor, int32_t* samples, int32_t* use_all,
                                  float* stepsize, int32_t* topk_pos);

namespace {

template <typename T, bool FOLD>
int launch_sampled(const ThreshParams* v, int count, unsigned ncta, bool capturing, cudaStream_t s) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  bool small = true;
  for (int i = 0; i < count; ++i) small &= v[i].samples <= kSmallSample;
  cfg.gridDim = dim3(ncta * (unsigned)count, 1, 1);
  cfg.blockDim = dim3(small ? kSmallThreads : kThreads, 1, 1);
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  unsigned na = 0;
  if (ncta > 1) {      // a launch without the attribute costs the host 2 us less
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = ncta;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
  }
  if (!capturing && cx_pdl_enabled()) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  cudaError_t e;
  if (count == 1) {
    ThreshBatch<1> b;
    b.v[0] = v[0];
    e = small ? cudaLaunchKernelEx(&cfg, threshold_small_kernel<T, FOLD, 1>, b) : cudaLaunchKernelEx(&cfg, threshold_kernel<T, FOLD, 1>, b);
  } else {
    ThreshBatch<kVectors> b;
    memcpy(b.v, v, sizeof(ThreshParams) * (size_t)count);
    e = small ? cudaLaunchKernelEx(&cfg, threshold_small_kernel<T, FOLD, kVectors>, b) : cudaLaunchKernelEx(&cfg, threshold_kernel<T, FOLD, kVectors>, b);
  }
  if (e != cudaSuccess) return cx_set_error("threshold_kernel launch", (int)e);
  cx_note_stream(s, true);       // a sample larger than the cache is gathered again behind the trigger
  cx_note_launch();
  return cx_check_launch("threshold_kernel");
}

template <bool FOLD>
int launch_sampled_dtype(int gdtype, const ThreshParams* v, int count, unsigned ncta, bool capturing, cudaStream_t s) {
  switch (gdtype) {
    case CX_F32: return launch_sampled<float, FOLD>(v, count, ncta, capturing, s);
    case CX_BF16: return launch_sampled<__nv_bfloat16, FOLD>(v, count, ncta, capturing, s);
    case CX_F16: return launch_sampled<__half, FOLD>(v, count, ncta, capturing, s);
    default: return cx_set_error("cx_threshold_topk: unsupported dtype on CUDA", 0);
  }
}

void sampled_params(ThreshParams& p, const void* g, const float* r, int64_t n, float ratio, int default_subsamples,
                    float subsample_factor, float* thr_out) {
  memset(&p, 0, sizeof(p));
  p.g = g; p.r = r; p.n = n; p.thr_out = thr_out;
  cx_threshold_plan(n, ratio, default_subsamples, subsample_factor, &p.samples, &p.use_all, &p.stepsize, &p.topk_pos);
  if (n <= 0) { p.samples = 0; p.topk_pos = 0; }
}

// a cluster of 8 CTAs gathers large samples (their keys must fit the first CTA's shared memory)
unsigned cluster_for(const ThreshParams& p) { return (p.samples > kSmallSample && p.samples <= kSmemKeys) ? 8u : 1u; }

bool whole_vector(const ThreshParams& p) { return p.use_all && p.topk_pos > 0 && p.n > kSmemKeys; }

bool exact_wanted(const ThreshParams& p, const void* workspace, int64_t ws_bytes) {
  return whole_vector(p) && workspace && ws_bytes >= cx_threshold_workspace_bytes();
}

}  // namespace

extern "C" int cx_threshold_whole(int64_t n, float ratio, int default_subsamples, float subsample_factor) {
  ThreshParams p;
  sampled_params(p, nullptr, nullptr, n, ratio, default_subsamples, subsample_factor, nullptr);
  return whole_vector(p) ? 1 : 0;
}

int cx_threshold_topk_cuda(int gdtype, const void* g, const float* r, int64_t n, float ratio,
                           int default_subsamples, float subsample_factor, float* thr_out,
                           void* workspace, int64_t ws_bytes, void* stream) {
  if (!g && !r) return cx_set_error("cx_threshold_topk: g and r are both NULL", 0);
  ThreshParams p;
  sampled_params(p, g, r, n, ratio, default_subsamples, subsample_factor, thr_out);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (exact_wanted(p, workspace, ws_bytes) && ws_bytes >= cx_threshold_exact_bytes(n)) {
    OnePassParams q;
    q.g = g; q.r = r; q.n = n; q.rank = (uint32_t)p.topk_pos; q.cap = candidate_cap(n); q.thr_out = thr_out;
    q.st = reinterpret_cast<ExactState*>(reinterpret_cast<char*>(workspace) + cx_threshold_workspace_bytes());
    q.list = reinterpret_cast<uint32_t*>(q.st + 1);
    const double f = (double)p.topk_pos / (double)n, at = f * kBracket, slack = 4.0 * sqrt(at * (1.0 - f)) + 4.0;
    q.hi_rank = at - slack < 0.0 ? ~0u : (uint32_t)(at - slack);
    q.lo_rank = at + slack >= kBracket - 1 ? ~0u : (uint32_t)(at + slack + 1.0);
    const size_t esz = gdtype == CX_F32 ? 4 : 2;
    q.vec = (!r || (reinterpret_cast<uintptr_t>(r) & 15) == 0) && (!g || (reinterpret_cast<uintptr_t>(g) & (4 * esz - 1)) == 0);
    const bool capturing = cx_seq_cell() != nullptr;
    switch (gdtype) {
      case CX_F32: return launch_one_pass<float>(q, capturing, s);
      case CX_BF16: return launch_one_pass<__nv_bfloat16>(q, capturing, s);
      case CX_F16: return launch_one_pass<__half>(q, capturing, s);
      default: return cx_set_error("cx_threshold_topk: unsupported dtype on CUDA", 0);
    }
  }
  if (exact_wanted(p, workspace, ws_bytes)) {
    // exact selection over a vector that does not fit one CTA's shared memory: grid-wide passes
    ExactParams e;
    e.g = g; e.r = r; e.n = n; e.topk_pos = (uint32_t)p.topk_pos; e.pass = 0;
    e.hist = reinterpret_cast<uint32_t*>(workspace); e.thr_out = thr_out;
    const size_t esz = gdtype == CX_F32 ? 4 : 2;
    e.vec = (!r || (reinterpret_cast<uintptr_t>(r) & 15) == 0) && (!g || (reinterpret_cast<uintptr_t>(g) & (4 * esz - 1)) == 0);
    switch (gdtype) {
      case CX_F32: return launch_exact<float>(e, s);
      case CX_BF16: return launch_exact<__nv_bfloat16>(e, s);
      case CX_F16: return launch_exact<__half>(e, s);
      default: return cx_set_error("cx_threshold_topk: unsupported dtype on CUDA", 0);
    }
  }
  return launch_sampled_dtype<false>(gdtype, &p, 1, cluster_for(p), cx_seq_cell() != nullptr, s);
}

// Leading ops of the list that one launch can serve: sampled thresholds of the same element type,
// with the same cluster size, of vectors that are all folded or all plain, into different cells.
// Returns how many were launched (at least one), or a negative error.
int cx_threshold_batch_cuda(const CxOp* ops, int count, void* stream) {
  ThreshParams v[kVectors];
  int k = 0;
  unsigned ncta = 0;
  for (; k < count && k < kVectors; ++k) {
    const CxOp& o = ops[k];
    if (o.kind != CX_OPK_THRESHOLD || o.dev != CX_DEV_CUDA || o.lane != ops[0].lane || o.dtype != ops[0].dtype ||
        (o.fold != nullptr) != (ops[0].fold != nullptr))
      break;
    if (!o.g && !o.r && !o.fold) { if (k) break; return cx_set_error("cx_threshold_topk: g and r are both NULL", 0); }
    bool same_cell = false;
    for (int j = 0; j < k; ++j) same_cell |= v[j].thr_out == o.thr;
    if (same_cell) break;
    sampled_params(v[k], o.g, o.r, o.n, o.ratio, o.default_subsamples, o.subsample_factor, o.thr);
    const bool exact = exact_wanted(v[k], o.workspace, o.ws_bytes);
    if (exact && o.fold) { if (k) break; return cx_set_error("cx_threshold_topk: exact selection reads a plain vector", 0); }
    if (exact || (k && cluster_for(v[k]) != ncta)) {
      if (k) break;
      const int rc = cx_threshold_topk_cuda(o.dtype, o.g, o.r, o.n, o.ratio, o.default_subsamples, o.subsample_factor,
                                            o.thr, o.workspace, o.ws_bytes, stream);
      return rc ? (rc > 0 ? -rc : rc) : 1;
    }
    if (k == 0) ncta = cluster_for(v[0]);
    if (o.fold) v[k].fold = *o.fold;
  }
  const bool capturing = cx_seq_cell() != nullptr;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int rc = ops[0].fold ? launch_sampled_dtype<true>(ops[0].dtype, v, k, ncta, capturing, s)
                             : launch_sampled_dtype<false>(ops[0].dtype, v, k, ncta, capturing, s);
  return rc ? (rc > 0 ? -rc : rc) : k;
}
