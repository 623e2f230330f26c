// Run-length codec on the GPU, fused with the transfer (reference: CompressorRLE,
// src/compressor.hxx:159-532, whose packed-value indexing is wrong for thresholds
// above zero; this is the corrected format of the host codec in host_ref.cpp).
//
// Payload, written straight into the receivers' slots:
//   i32 n | i32 nnz | nnz x f32 values (index order) | i32 nRuns | i32 firstIsYes |
//   nRuns x i32 run lengths, alternating selected / not selected.
// Selection: |r + g| >= thr, except that zeros are never selected at thr == 0.
//
// Send = two launches on one stream, both over the same partition of the vector into one
// contiguous chunk per warp (a CTA's eight chunks are neighbours; one wave of CTAs, so the totals
// are few):
//   1. rle_count:  per chunk: selected elements, run starts, and whether its first element
//                  starts a run.  Only sums leave the warp, no scan is needed,
//   2. rle_emit:   every CTA adds up the totals of the CTAs before it (a few hundred numbers),
//                  then every warp walks its chunk on its own, 256 elements at a time with running
//                  offsets: values and run starts are compacted in shared memory and stored
//                  coalesced at their final position in every target, the residual is updated from
//                  the same registers.  The last CTA writes the two small headers and releases the
//                  sequence number.
// Receive = two launches:
//   1. rle_index:  waits (bounded), checks the headers, sums the run lengths of every block of
//                  kRunBlock runs (one warp per block) and leaves prefixes inside groups of blocks,
//   2. rle_expand: every CTA owns an equal part of the output.  It finds the block of runs its part
//                  starts in, and takes windows of kWindow outputs: the start of every run flips
//                  one bit of a mask in shared memory, the prefix parity of the mask says which
//                  outputs are selected, and counting selected bits gives the index of every value.
//                  The checks (lengths add up to n and nnz) happen before the first store, in every
//                  CTA alike.
// A payload that fails a check sets BAD_HEADER in the status word and leaves `out` untouched.
//
// The expansion used to be prepared by one CTA that scanned all runs of the payload in sequence:
// 2540 us for the 750 k runs of 2^22 elements at top-k 10 %.
#include "cx_device.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kPer = 8;
constexpr int kSeg = 32 * kPer;          // elements a warp takes at a time
constexpr int kSendPerSm = 4;            // resident CTAs of the emit kernel
constexpr int kMaxSend = 1024;           // sending CTAs
constexpr int kGroups = 256;             // groups of run blocks, one per thread of a receiving CTA
constexpr int kRunBlock = 1024;          // runs per block: one warp sums it, one CTA scans it
constexpr int kWindow = 32 * kThreads;   // outputs per window: one mask word per thread

struct ChunkTotals {       // of one warp's chunk, or of a CTA's eight
  int32_t nnz;             // selected elements
  int32_t starts;          // elements that start a run
  int32_t last;            // position of the last run start (-1: none)
  int32_t first;           // 1 if the chunk's first element starts a run
};

struct RleMeta {           // first 256 bytes of the sender's workspace
  uint32_t done;
  int32_t first_yes;
  uint32_t pad[62];
};
struct RleRxMeta {         // first 256 bytes of the receiver's workspace
  int32_t ok;
  int32_t nnz;
  int32_t nruns;
  int32_t first_yes;
  uint32_t pad[60];
};

struct SendParams {
  const void* g;
  float* r;
  int64_t n;
  const float* thr;
  uint64_t seq;
  CxTargets tg;
  RleMeta* meta;
  ChunkTotals* cta;      // [gridDim.x]
  ChunkTotals* chunk;    // [gridDim.x * kWarps]
  int32_t segs;          // segments per chunk
  uint32_t src_rank;
};

__device__ __forceinline__ bool selected(float v, float thr) {
  return fabsf(v) >= thr && !(thr == 0.f && v == 0.f);
}

template <typename T>
__device__ __forceinline__ float value_at(const SendParams& p, int64_t i) {
  float v = p.g ? cx::Elem<T>::to_f(reinterpret_cast<const T*>(p.g)[i]) : 0.f;
  if (p.r) v += p.r[i];
  return v;
}

__device__ __forceinline__ int valid_at(int64_t n, int64_t base) {
  const int64_t left = n - base;
  return left >= kPer ? kPer : (left > 0 ? (int)left : 0);
}

// the thread's 8 consecutive values (zero beyond the vector's end)
template <typename T>
__device__ __forceinline__ void load_values(const SendParams& p, int64_t base, float (&v)[kPer]) {
  const int valid = valid_at(p.n, base);
  const T* g = reinterpret_cast<const T*>(p.g);
  const bool gvec = !g || (reinterpret_cast<uintptr_t>(g) & (4 * sizeof(T) - 1)) == 0;
  const bool rvec = !p.r || (reinterpret_cast<uintptr_t>(p.r) & 15) == 0;
  if (valid == kPer && gvec && rvec) {
    float a[4], b[4];
    if (g) { cx::load4(g + base, a); cx::load4(g + base + 4, b); }
    else { for (int e = 0; e < 4; ++e) a[e] = b[e] = 0.f; }
    if (p.r) {
      float c[4], d[4];
      cx::load4(p.r + base, c); cx::load4(p.r + base + 4, d);
#pragma unroll
      for (int e = 0; e < 4; ++e) { a[e] += c[e]; b[e] += d[e]; }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) { v[e] = a[e]; v[4 + e] = b[e]; }
  } else {
#pragma unroll
    for (int e = 0; e < kPer; ++e) v[e] = e < valid ? value_at<T>(p, base + e) : 0.f;
  }
}

__device__ __forceinline__ uint32_t yes_mask(const float (&v)[kPer], int valid, float thr) {
  uint32_t yes = 0;
#pragma unroll
  for (int e = 0; e < kPer; ++e)
    if (e < valid && selected(v[e], thr)) yes |= 1u << e;
  return yes;
}

// bits of the run starts among the thread's valid elements, given the element in front of them
__device__ __forceinline__ uint32_t start_mask(uint32_t yes, int valid, bool prev_yes) {
  const uint32_t vm = valid >= kPer ? 0xffu : ((1u << valid) - 1u);
  return (yes ^ ((yes << 1) | (prev_yes ? 1u : 0u))) & vm;
}

// Bound by the read of g and r.  The element in front of a lane's share comes from the lane to the
// left; only the first one of a chunk is read from memory (nothing writes r in this kernel).
template <typename T>
__global__ void __launch_bounds__(kThreads) rle_count_kernel(const __grid_constant__ SendParams p) {
  __shared__ ChunkTotals s_chunk[kWarps];
  cx::pdl_wait();
  cx::pdl_trigger();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const float thr = *p.thr;
  const int64_t chunk = (int64_t)blockIdx.x * kWarps + w;
  const int64_t lo = chunk * p.segs * kSeg;
  const int64_t hi = min(lo + (int64_t)p.segs * kSeg, p.n);
  uint32_t tail = 0;
  if (lane == 0 && lo > 0 && lo < hi) tail = selected(value_at<T>(p, lo - 1), thr) ? 1u : 0u;
  int nnz = 0, st = 0, last = -1, first = 0;
#pragma unroll 2
  for (int64_t seg = lo; seg < hi; seg += kSeg) {
    const int64_t base = seg + lane * kPer;
    float v[kPer];
    load_values<T>(p, base, v);
    const int valid = valid_at(p.n, base);
    const uint32_t yes = yes_mask(v, valid, thr);
    const uint32_t edge = yes >> (kPer - 1);
    uint32_t prev = __shfl_up_sync(0xffffffffu, edge, 1);
    if (lane == 0) prev = tail;
    tail = __shfl_sync(0xffffffffu, edge, 31);
    uint32_t starts = start_mask(yes, valid, prev != 0);
    if (base == 0 && valid > 0) {                     // element 0 always starts a run
      starts |= 1u;
      p.meta->first_yes = (int)(yes & 1u);
    }
    if (base == lo) first = (int)(starts & 1u);
    nnz += __popc(yes);
    st += __popc(starts);
    if (starts) last = (int)(base + 31 - __clz(starts));
  }
  if (p.n == 0 && threadIdx.x == 0) p.meta->first_yes = 0;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    nnz += __shfl_xor_sync(0xffffffffu, nnz, d);
    st += __shfl_xor_sync(0xffffffffu, st, d);
    last = max(last, __shfl_xor_sync(0xffffffffu, last, d));
  }
  if (lane == 0) {
    s_chunk[w] = ChunkTotals{nnz, st, last, first};
    p.chunk[chunk] = s_chunk[w];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    ChunkTotals t = s_chunk[0];
    for (int j = 1; j < kWarps; ++j) { t.nnz += s_chunk[j].nnz; t.starts += s_chunk[j].starts; t.last = max(t.last, s_chunk[j].last); }
    p.cta[blockIdx.x] = t;
  }
}

template <typename T>
__global__ void __launch_bounds__(kThreads, kSendPerSm) rle_emit_kernel(const __grid_constant__ SendParams p) {
  __shared__ float s_val[kWarps][kSeg];
  __shared__ int s_start[kWarps][kSeg];
  __shared__ int s_pre[kWarps][5];
  __shared__ uint32_t s_lastblock;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int64_t chunk = (int64_t)blockIdx.x * kWarps + w;
  const int64_t lo = chunk * p.segs * kSeg;
  const int64_t hi = min(lo + (int64_t)p.segs * kSeg, p.n);
  // resident early: the count kernel only reads, so the first segment may be fetched before it ends
  float v[kPer];
  load_values<T>(p, lo + lane * kPer, v);
  cx::pdl_wait();
  const float thr = *p.thr;
  // offsets of this chunk and the totals of all
  int k0 = 0, q0 = 0, prev = -1, nnz_total = 0, nruns = 0;
  for (int c = tid; c < (int)gridDim.x; c += kThreads) {
    const ChunkTotals t = p.cta[c];
    nnz_total += t.nnz;
    nruns += t.starts;
    if (c < (int)blockIdx.x) { k0 += t.nnz; q0 += t.starts; prev = max(prev, t.last); }
  }
  if (tid < kWarps) {                      // the chunks of this CTA, one per thread
    const ChunkTotals t = p.chunk[(int64_t)blockIdx.x * kWarps + tid];
    s_start[0][4 * tid] = t.nnz; s_start[0][4 * tid + 1] = t.starts; s_start[0][4 * tid + 2] = t.last; s_start[0][4 * tid + 3] = t.first;
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    k0 += __shfl_xor_sync(0xffffffffu, k0, d);
    q0 += __shfl_xor_sync(0xffffffffu, q0, d);
    prev = max(prev, __shfl_xor_sync(0xffffffffu, prev, d));
    nnz_total += __shfl_xor_sync(0xffffffffu, nnz_total, d);
    nruns += __shfl_xor_sync(0xffffffffu, nruns, d);
  }
  if (lane == 0) { s_pre[w][0] = k0; s_pre[w][1] = q0; s_pre[w][2] = prev; s_pre[w][3] = nnz_total; s_pre[w][4] = nruns; }
  __syncthreads();
  k0 = q0 = nnz_total = nruns = 0;
  prev = -1;
#pragma unroll
  for (int j = 0; j < kWarps; ++j) {
    k0 += s_pre[j][0]; q0 += s_pre[j][1]; prev = max(prev, s_pre[j][2]); nnz_total += s_pre[j][3]; nruns += s_pre[j][4];
  }
  for (int j = 0; j < w; ++j) { k0 += s_start[0][4 * j]; q0 += s_start[0][4 * j + 1]; prev = max(prev, s_start[0][4 * j + 2]); }
  const bool first_start = s_start[0][4 * w + 3] != 0;
  __syncthreads();
  const size_t runs_off = 8 + 4 * (size_t)nnz_total + 8;
  float* sv = s_val[w];
  int* ss = s_start[w];
  uint32_t tail = 0;           // the last element of the segment before
  for (int64_t seg = lo; seg < hi; seg += kSeg) {
    const int64_t base = seg + lane * kPer;
    const int valid = valid_at(p.n, base);
    const uint32_t yes = yes_mask(v, valid, thr);
    const uint32_t edge = yes >> (kPer - 1);
    uint32_t before = __shfl_up_sync(0xffffffffu, edge, 1);
    if (lane == 0) before = tail;
    tail = __shfl_sync(0xffffffffu, edge, 31);
    uint32_t starts = start_mask(yes, valid, before != 0);
    if (seg == lo && lane == 0) starts = (starts & ~1u) | (first_start ? 1u : 0u);
    // one scan for both counts (at most 256 each)
    const uint32_t mine = (uint32_t)__popc(yes) | ((uint32_t)__popc(starts) << 16);
    uint32_t incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += t;
    }
    const uint32_t tot = __shfl_sync(0xffffffffu, incl, 31);
    uint32_t kv = (incl - mine) & 0xffffu, ks = (incl - mine) >> 16;
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      if ((yes >> e) & 1u) sv[kv++] = v[e];
      if ((starts >> e) & 1u) ss[ks++] = (int)(base + e);
    }
    if (p.r && valid > 0) {
      if (valid == kPer && (reinterpret_cast<uintptr_t>(p.r) & 15) == 0) {
        float a[4], b[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          a[e] = (yes >> e) & 1u ? 0.f : v[e];
          b[e] = (yes >> (4 + e)) & 1u ? 0.f : v[4 + e];
        }
        cx::store4(p.r + base, a);
        cx::store4(p.r + base + 4, b);
      } else {
#pragma unroll
        for (int e = 0; e < kPer; ++e) if (e < valid) p.r[base + e] = (yes >> e) & 1u ? 0.f : v[e];
      }
    }
    if (seg + kSeg < hi) load_values<T>(p, base + kSeg, v);    // the next segment, in flight during the stores
    __syncwarp();
    const int nv = (int)(tot & 0xffffu), ns = (int)(tot >> 16);
    for (int k = 0; k < p.tg.count; ++k) {
      char* pay = reinterpret_cast<char*>(p.tg.ep[k].pairs);
      float* vals = reinterpret_cast<float*>(pay + 8) + k0;
      for (int i = lane; i < nv; i += 32) vals[i] = sv[i];
      int32_t* runs = reinterpret_cast<int32_t*>(pay + runs_off) + q0 - 1;   // start q closes run q - 1
      for (int i = lane; i < ns; i += 32)
        if (q0 + i > 0) runs[i] = ss[i] - (i ? ss[i - 1] : prev);
    }
    if (ns) prev = ss[ns - 1];
    k0 += nv;
    q0 += ns;
    __syncwarp();
  }
  if (lo < hi && hi == p.n && lane < p.tg.count)     // the warp that holds the last element closes the last run
    reinterpret_cast<int32_t*>(reinterpret_cast<char*>(p.tg.ep[lane].pairs) + runs_off)[q0 - 1] = (int)(p.n - prev);
  __syncthreads();       // one thread's trigger counts for its CTA: every warp has read its chunk of g
  cx::pdl_trigger();
  if (!cx::cta_arrive(&p.meta->done, gridDim.x, &s_lastblock)) return;
  if (tid < p.tg.count) {
    const CxEndpoint ep = p.tg.ep[tid];
    int32_t* pay = reinterpret_cast<int32_t*>(ep.pairs);
    pay[0] = (int32_t)p.n;
    pay[1] = nnz_total;
    int32_t* rh = reinterpret_cast<int32_t*>(reinterpret_cast<char*>(ep.pairs) + 8 + 4 * (size_t)nnz_total);
    rh[0] = nruns;
    rh[1] = p.meta->first_yes;
    CxHeader* h = ep.hdr;
    h->bytes = 16 + 4 * (uint64_t)nnz_total + 4 * (uint64_t)nruns;
    h->n = (uint32_t)p.n; h->nnz = (uint32_t)nnz_total; h->nnz_found = (uint32_t)nnz_total;
    h->kind = CX_KIND_RLE; h->threshold = thr; h->nsub = 0; h->src_rank = p.src_rank;
    h->dtype = CX_F32;
    cx::st_release_sys(&h->seq, p.seq);
  }
  if (tid == 0) p.meta->done = 0;
}

// ---- receive ---------------------------------------------------------------------------

struct RunSums {           // of one block of runs, or of one group of blocks
  int32_t len;             // elements covered
  int32_t yes;             // of these: selected
};

struct RecvParams {
  CxEndpoint src;
  uint64_t expect_seq;
  float* out;
  int64_t n;
  int64_t slot_bytes;
  int32_t add;
  RleRxMeta* meta;
  RunSums* group;      // [kGroups]
  int32_t* group_bad;  // [kGroups]
  RunSums* block;      // [blocks of runs]: sums of the blocks before it in its group
  int32_t groups;      // CTAs of the index kernel
  int64_t per_cta;     // outputs per CTA of the expand kernel, a multiple of kWindow
  uint32_t front_wait;  // the kernel in front may be an expansion that still reads the index
  uint32_t* status;
  uint64_t timeout_ns;
};

__device__ __forceinline__ int64_t blocks_per_group(int64_t nruns, int groups) {
  const int64_t blocks = (nruns + kRunBlock - 1) / kRunBlock;
  return (blocks + groups - 1) / groups;
}

__global__ void __launch_bounds__(kThreads) rle_index_kernel(const __grid_constant__ RecvParams p) {
  __shared__ int s_state;
  __shared__ int s_bad;
  __shared__ long long s_sum[kWarps][2];
  cx::pdl_trigger();
  if (p.front_wait) cx::pdl_wait();
  if (threadIdx.x == 0) {
    int st = 0;
    if (!cx::wait_seq(&p.src.hdr->seq, p.expect_seq, p.timeout_ns)) st = CX_ST_TIMEOUT;
    else if (__ldcg(&p.src.hdr->kind) != CX_KIND_RLE || (int64_t)__ldcg(&p.src.hdr->n) != p.n) st = CX_ST_BAD_HEADER;
    s_state = st;
    s_bad = 0;
  }
  __syncthreads();
  int st = s_state;
  const int32_t* pay = reinterpret_cast<const int32_t*>(p.src.pairs);
  int64_t nnz = 0, nruns = 0;
  int first = 0;
  if (!st) {
    nnz = __ldcg(pay + 1);
    if ((int64_t)__ldcg(pay) != p.n || nnz < 0 || nnz > p.n || 16 + 4 * nnz > p.slot_bytes) st = CX_ST_BAD_HEADER;
  }
  const int32_t* rh = nullptr;
  if (!st) {
    rh = reinterpret_cast<const int32_t*>(reinterpret_cast<const char*>(p.src.pairs) + 8 + 4 * nnz);
    nruns = __ldcg(rh);
    first = __ldcg(rh + 1) != 0;
    if (nruns < 0 || nruns > p.n + 1 || 16 + 4 * nnz + 4 * nruns > p.slot_bytes) st = CX_ST_BAD_HEADER;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (st && p.status) atomicOr(p.status, (uint32_t)st);
    p.meta->nnz = (int32_t)nnz;
    p.meta->nruns = (int32_t)nruns;
    p.meta->first_yes = first;
    p.meta->ok = st ? 0 : 1;
  }
  if (threadIdx.x == 0) p.group_bad[blockIdx.x] = st ? 1 : 0;
  if (!st) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int32_t* runs = rh + 2;
    const int64_t nblocks = (nruns + kRunBlock - 1) / kRunBlock;
    const int64_t bpg = blocks_per_group(nruns, p.groups);
    const int64_t b0 = (int64_t)blockIdx.x * bpg, b1 = min(b0 + bpg, nblocks);
    const bool lane_yes = ((lane & 1) == 0) == (first != 0);   // blocks start at even runs
    long long glen = 0, gyes = 0;                              // sums of the group so far
    for (int64_t bb = b0; bb < b1; bb += kWarps) {             // eight blocks at a time, a warp each
      const int64_t b = bb + w;
      int32_t x[kRunBlock / 32];
      long long len = 0;
      bool neg = false;
#pragma unroll
      for (int k = 0; k < kRunBlock / 32; ++k) {
        const int64_t q = b * kRunBlock + k * 32 + lane;
        x[k] = b < b1 && q < nruns ? __ldcg(runs + q) : 0;
      }
#pragma unroll
      for (int k = 0; k < kRunBlock / 32; ++k) { len += x[k]; neg |= x[k] < 0; }
      long long yes = lane_yes ? len : 0;
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) {
        len += __shfl_xor_sync(0xffffffffu, len, d);
        yes += __shfl_xor_sync(0xffffffffu, yes, d);
      }
      // no length is negative, so a block that covers more than n elements cannot be part of a valid payload
      if (__any_sync(0xffffffffu, neg) || len > p.n) {
        if (lane == 0) s_bad = 1;
        len = yes = 0;
      }
      if (lane == 0) { s_sum[w][0] = len; s_sum[w][1] = yes; }
      __syncthreads();
      long long bl = glen, by = gyes;
#pragma unroll
      for (int j = 0; j < kWarps; ++j) {
        if (j < w) { bl += s_sum[j][0]; by += s_sum[j][1]; }
        glen += s_sum[j][0];
        gyes += s_sum[j][1];
      }
      if (lane == 0 && b < b1) p.block[b] = RunSums{(int32_t)bl, (int32_t)by};   // only read when no check fails
      __syncthreads();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      const bool bad = s_bad != 0 || glen > p.n;
      p.group[blockIdx.x] = bad ? RunSums{0, 0} : RunSums{(int32_t)glen, (int32_t)gyes};
      if (bad) p.group_bad[blockIdx.x] = 1;
    }
  }
  cx::pdl_wait();   // launched early behind the sender: do not complete before that grid has
}

// exclusive block-wide sum of x; the total in `tot`.  sm: one word per warp, free to be reused after
// the next barrier
template <typename V>
__device__ __forceinline__ V block_prefix(V x, V& tot, V* sm) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  V inc = x;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const V t = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += t;
  }
  if (lane == 31) sm[w] = inc;
  __syncthreads();
  V pre = 0;
  tot = 0;
#pragma unroll
  for (int j = 0; j < kWarps; ++j) {
    if (j < w) pre += sm[j];
    tot += sm[j];
  }
  return pre + inc - x;
}

// Bound by the output (read and written for `add`).  Looking every output's run up by bisection in
// the scanned block took 40 us for 2^22 elements at top-k 10 %; the mask needs one shared-memory
// atomic per run and two shared-memory reads per four outputs.
__global__ void __launch_bounds__(kThreads, 4) rle_expand_kernel(const __grid_constant__ RecvParams p) {
  __shared__ long long s_l[kWarps];
  __shared__ int s_a[kWarps], s_b[kWarps];
  __shared__ int s_pick[3];
  __shared__ uint32_t s_mask[kThreads];    // run starts of the window, then its selected outputs
  __shared__ int s_base[kThreads];         // index of the word's first value
  cx::pdl_wait();
  cx::pdl_trigger();
  if (!p.meta->ok) return;
  const int nnz = p.meta->nnz, nruns = p.meta->nruns, first = p.meta->first_yes;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int64_t e0 = (int64_t)blockIdx.x * p.per_cta;
  const int64_t e1 = min(e0 + p.per_cta, p.n);
  // every CTA checks the whole payload before any of them writes; group g belongs to thread g
  int64_t blk = 0;
  int at = 0, at_yes = 0;                  // elements and selected elements before block `blk`
  const int64_t nblocks = ((int64_t)nruns + kRunBlock - 1) / kRunBlock;
  {
    const bool have = tid < p.groups;
    const RunSums g = have ? p.group[tid] : RunSums{0, 0};
    const int gbad = have ? p.group_bad[tid] : 0;
    long long total;
    int total_yes;
    const long long gstart = block_prefix<long long>(g.len, total, s_l);
    const int ystart = block_prefix<int>(g.yes, total_yes, s_a);
    const int bad = __syncthreads_or(gbad);
    if (bad || total != p.n || total_yes != nnz) {
      if (blockIdx.x == 0 && tid == 0 && p.status) atomicOr(p.status, (uint32_t)CX_ST_BAD_HEADER);
      return;
    }
    if (e0 >= e1) return;
    // the group, then the block that holds e0 (entries of length zero hold nothing)
    if (have && gstart <= e0 && gstart + g.len > e0) { s_pick[0] = tid; s_pick[1] = (int)gstart; s_pick[2] = ystart; }
    __syncthreads();
    const int64_t bpg = blocks_per_group(nruns, p.groups);
    const int64_t b0 = s_pick[0] * bpg;
    const int count = (int)min(bpg, nblocks - b0);
    const int gs = s_pick[1], gy = s_pick[2];
    __syncthreads();
    for (int i = tid; i < count; i += kThreads) {
      const RunSums x = p.block[b0 + i];
      const int64_t next = i + 1 < count ? (int64_t)gs + p.block[b0 + i + 1].len : (int64_t)p.n;
      if (gs + (int64_t)x.len <= e0 && (i + 1 == count || next > e0)) { s_pick[0] = i; s_pick[1] = gs + x.len; s_pick[2] = gy + x.yes; }
    }
    __syncthreads();
    blk = b0 + s_pick[0];
    at = s_pick[1];
    at_yes = s_pick[2];
  }
  const int32_t* runs = reinterpret_cast<const int32_t*>(reinterpret_cast<const char*>(p.src.pairs) + 16 + 4 * (int64_t)nnz);
  const float* vals = reinterpret_cast<const float*>(reinterpret_cast<const char*>(p.src.pairs) + 8);
  const bool vec = (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
  int vbase = -1;                          // index of the first value at or behind the window's start
  for (int64_t w0 = e0; w0 < e1; w0 += kWindow) {
    const int64_t w1 = min(w0 + kWindow, e1);
    s_mask[tid] = 0;
    // blocks of runs that reach into the window; a run that began earlier counts at its first bit
    for (;;) {
      int len[4], mine = 0, part = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int64_t q = blk * kRunBlock + 4 * tid + k;
        len[k] = q < nruns ? runs[q] : 0;
        mine += len[k];
      }
      int tot;
      int pos = at + block_prefix<int>(mine, tot, s_a);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (blk * kRunBlock + 4 * tid + k < nruns && pos < w1) {
          const int bit = pos > w0 ? (int)(pos - w0) : 0;
          atomicXor(&s_mask[bit >> 5], 1u << (bit & 31));
          const bool yes = ((k & 1) == 0) == (first != 0);
          if (yes && pos < w0) part += (int)(min((int64_t)pos + len[k], w0) - pos);
        }
        pos += len[k];
      }
      if (vbase < 0) {                     // once per CTA: values of this block in front of the window
        int before;
        block_prefix<int>(part, before, s_b);
        vbase = at_yes + before;
      }
      if ((int64_t)at + tot >= w1 || blk + 1 >= nblocks) break;
      at += tot;
      ++blk;
      __syncthreads();                     // s_a is written again
    }
    __syncthreads();
    // word by word: parity of the starts up to every bit, the selected bits, and their number before
    const uint32_t flips = s_mask[tid];
    uint32_t x = flips;
    x ^= x << 1; x ^= x << 2; x ^= x << 4; x ^= x << 8; x ^= x << 16;
    const uint32_t odd = __ballot_sync(0xffffffffu, x >> 31);
    if (lane == 0) s_b[w] = __popc(odd) & 1;
    __syncthreads();
    int carry = __popc(odd & ((1u << lane) - 1u)) & 1;
#pragma unroll
    for (int j = 0; j < kWarps; ++j) if (j < w) carry ^= s_b[j];
    if (carry ^ (first ? 0 : 1)) x = ~x;
    const int64_t left = w1 - w0 - 32 * (int64_t)tid;
    if (left < 32) x &= left <= 0 ? 0u : (1u << left) - 1u;
    int total;
    const int mybase = vbase + block_prefix<int>(__popc(x), total, s_a);
    s_mask[tid] = x;
    s_base[tid] = mybase;
    vbase += total;
    __syncthreads();
#pragma unroll 4
    for (int it = 0; it < kWindow / (4 * kThreads); ++it) {
      const int o = it * 4 * kThreads + 4 * tid;
      const int64_t i0 = w0 + o;
      if (i0 >= w1) continue;
      const uint32_t word = s_mask[o >> 5];
      const uint32_t yes = (word >> (o & 31)) & 0xfu;
      if (p.add && yes == 0) continue;
      int k = s_base[o >> 5] + __popc(word & ((1u << (o & 31)) - 1u));
      float y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int e = 0; e < 4; ++e) if ((yes >> e) & 1u) y[e] = vals[k++];
      if (vec && i0 + 4 <= w1) {
        if (p.add) {
          float z[4];
          cx::load4(p.out + i0, z);
#pragma unroll
          for (int e = 0; e < 4; ++e) y[e] = (yes >> e) & 1u ? z[e] + y[e] : z[e];
        }
        cx::store4(p.out + i0, y);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (i0 + e >= w1) continue;
          if ((yes >> e) & 1u) p.out[i0 + e] = p.add ? p.out[i0 + e] + y[e] : y[e];
          else if (!p.add) p.out[i0 + e] = 0.f;
        }
      }
    }
    __syncthreads();
  }
}

}  // namespace

int64_t cx_rle_slot_bytes(int64_t n) { return (16 + 8 * n + 15) / 16 * 16; }

int64_t cx_rle_workspace_bytes(int64_t n) {
  const int64_t send = 256 + kMaxSend * (1 + kWarps) * (int64_t)sizeof(ChunkTotals);
  const int64_t blocks = (n + 1 + kRunBlock - 1) / kRunBlock;
  const int64_t recv = 256 + kGroups * (int64_t)(sizeof(RunSums) + sizeof(int32_t)) + blocks * (int64_t)sizeof(RunSums);
  return ((send > recv ? send : recv) + 255) / 256 * 256;
}

int cx_rle_send_cuda(int gdtype, const void* g, float* r, int64_t n, const float* thr,
                     int64_t slot_bytes, uint64_t seq, const CxTargets* tg, void* workspace,
                     int64_t ws_bytes, uint32_t src_rank, void* stream) {
  if (!g && !r) return cx_set_error("cx_rle_send: g and r are both NULL", 0);
  if (n < 0 || n > 0x7fffffffLL) return cx_set_error("cx_rle_send: n out of range", 0);
  if (tg->count < 0 || tg->count > CX_MAX_PEERS) return cx_set_error("cx_rle_send: bad target count", 0);
  if (slot_bytes < 16 + 8 * n) return cx_set_error("cx_rle_send: slot smaller than the worst case", 0);
  if (ws_bytes < cx_rle_workspace_bytes(n)) return cx_set_error("cx_rle_send: workspace too small", 0);
  SendParams p;
  p.g = g; p.r = r; p.n = n; p.thr = thr; p.seq = seq; p.tg = *tg; p.src_rank = src_rank;
  // one chunk of whole segments per warp, at most one wave of CTAs
  const int64_t nsegs = n > 0 ? (n + kSeg - 1) / kSeg : 1;
  int64_t wave = (int64_t)cx_sm_count() * kSendPerSm;
  if (wave > kMaxSend) wave = kMaxSend;
  p.segs = (int)((nsegs + wave * kWarps - 1) / (wave * kWarps));
  const int grid = (int)((nsegs + (int64_t)p.segs * kWarps - 1) / ((int64_t)p.segs * kWarps));
  char* ws = reinterpret_cast<char*>(workspace);
  p.meta = reinterpret_cast<RleMeta*>(ws);
  p.cta = reinterpret_cast<ChunkTotals*>(ws + 256);
  p.chunk = p.cta + kMaxSend;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  switch (gdtype) {
    case CX_F32:
      cx_launch_pdl(rle_count_kernel<float>, grid, kThreads, 0, s, p, false);
      cx_launch_pdl(rle_emit_kernel<float>, grid, kThreads, 0, s, p, false);
      break;
    case CX_BF16:
      cx_launch_pdl(rle_count_kernel<__nv_bfloat16>, grid, kThreads, 0, s, p, false);
      cx_launch_pdl(rle_emit_kernel<__nv_bfloat16>, grid, kThreads, 0, s, p, false);
      break;
    case CX_F16:
      cx_launch_pdl(rle_count_kernel<__half>, grid, kThreads, 0, s, p, false);
      cx_launch_pdl(rle_emit_kernel<__half>, grid, kThreads, 0, s, p, false);
      break;
    default: return cx_set_error("cx_rle_send: unsupported dtype on CUDA", 0);
  }
  cx_note_stream(stream, false);
  cx_note_launch();
  cx_note_launch();
  return cx_check_launch("rle send kernels");
}

int cx_rle_recv_cuda(const CxEndpoint* src, uint64_t expect_seq, float* out, int64_t n, int add,
                     int64_t slot_bytes, void* workspace, int64_t ws_bytes, uint32_t* status,
                     uint64_t timeout_ns, void* stream) {
  if (n < 0 || n > 0x7fffffffLL) return cx_set_error("cx_rle_recv: n out of range", 0);
  if (ws_bytes < cx_rle_workspace_bytes(n)) return cx_set_error("cx_rle_recv: workspace too small", 0);
  RecvParams p;
  p.src = *src; p.expect_seq = expect_seq; p.out = out; p.n = n; p.slot_bytes = slot_bytes;
  p.add = add; p.status = status; p.timeout_ns = timeout_ns;
  // index: a warp per block of runs; the number of runs is only known on the device, so the grid
  // follows the densest payload of this length and stays within one wave that may poll together
  int64_t groups = n / (kRunBlock * kWarps) + 1;
  if (groups > kGroups) groups = kGroups;
  p.groups = (int)groups;
  // expand: an equal number of windows per CTA, at most four CTAs per SM
  const int64_t windows = (n + kWindow - 1) / kWindow;
  const int64_t wave = 4 * (int64_t)cx_sm_count();
  p.per_cta = (windows + wave - 1) / wave * kWindow;
  char* ws = reinterpret_cast<char*>(workspace);
  p.meta = reinterpret_cast<RleRxMeta*>(ws);
  p.group = reinterpret_cast<RunSums*>(ws + 256);
  p.group_bad = reinterpret_cast<int32_t*>(p.group + kGroups);
  p.block = reinterpret_cast<RunSums*>(p.group_bad + kGroups);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  p.front_wait = cx_front_wait(stream) ? 1u : 0u;
  cx_note_stream(stream, true);
  cx_launch_pdl(rle_index_kernel, p.groups, kThreads, 0, s, p, false);
  cx_note_launch();
  if (n > 0) {
    const int64_t blocks = (n + p.per_cta - 1) / p.per_cta;
    cx_launch_pdl(rle_expand_kernel, (int)blocks, kThreads, 0, s, p, false);
    cx_note_launch();
  }
  return cx_check_launch("rle receive kernels");
}
