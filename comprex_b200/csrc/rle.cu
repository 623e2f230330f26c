// Run-length codec on the GPU, fused with the transfer (reference: CompressorRLE,
// src/compressor.hxx:159-532, whose packed-value indexing is wrong for thresholds
// above zero; this is the corrected format of the host codec in host_ref.cpp).
//
// Payload, written straight into the receivers' slots:
//   i32 n | i32 nnz | nnz x f32 values (index order) | i32 nRuns | i32 firstIsYes |
//   nRuns x i32 run lengths, alternating selected / not selected.
// Selection: |r + g| >= thr, except that zeros are never selected at thr == 0.
//
// Send = two launches on one stream over the same partition of the vector, one contiguous chunk of whole
// 1024-element sub-tiles per warp (a CTA's eight chunks are neighbours; one wave of CTAs, so the totals
// are few):
//   1. rle_scan:   the only pass over the vector.  Lane l looks at element 32 j + l, so a ballot is 32
//                  bits of the selection in order: the words go to scratch, the selected values, compacted
//                  per chunk, too, the residual is updated.  Totals of every chunk: selected elements, run
//                  starts, the last of them.
//   2. rle_emit:   every CTA adds up the totals of the CTAs before it (a few hundred numbers); then every
//                  warp copies its chunk's values and turns its words into run lengths, coalesced at their
//                  final position in every target.  (The runs lie behind the values, so nobody can write a
//                  run before all values are counted.)  The last CTA writes the two small headers and
//                  releases the sequence number.
// With two passes over the vector (count, then load again and emit, a lane per 8 elements) 2^22 fp32 elements
// at 10 % took 10 + 17 us, 177 and 495 instructions per 256 elements at half of the issue rate.
// Receive = two launches:
//   1. rle_index:  waits (bounded), checks the headers, sums the run lengths of every block of
//                  kRunBlock runs (one warp per block) and leaves prefixes inside groups of blocks,
//   2. rle_expand: every CTA owns an equal part of the output.  It finds the block of runs its part
//                  starts in, and takes windows of kWindow outputs: the start of every run flips
//                  one bit of a mask in shared memory, the prefix parity of the mask says which
//                  outputs are selected, and counting selected bits gives the index of every value.
//                  The first window of `out` is on its way to L2 while the index is made.
//                  The checks (lengths add up to n and nnz) happen before the first store, in every
//                  CTA alike.
// A payload that fails a check sets BAD_HEADER in the status word and leaves `out` untouched.
//
// The expansion used to be prepared by one CTA that scanned all runs of the payload in sequence:
// 2540 us for the 750 k runs of 2^22 elements at top-k 10 %.
#include <type_traits>

#include "cx_device.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kSendPerSm = 4;            // resident CTAs of the scan kernel
constexpr int kRows = 16;                // rows of 32 elements whose loads are in flight together
constexpr int kMaxSend = 1024;           // sending CTAs
constexpr int kGroups = 256;             // groups of run blocks, one per thread of a receiving CTA
constexpr int kRunBlock = 1024;          // runs per block: one warp sums it, one CTA scans it
constexpr int kWindow = 32 * kThreads;   // outputs per window: one mask word per thread
constexpr int kRunsEach = 2 * kRunBlock / kThreads;   // runs a thread takes at a time
constexpr int kBitsOut = 4;             // values of a lane in flight together

struct ChunkTotals {       // of one warp's chunk, or of a CTA's eight.  Whether the first element starts a run is
  int32_t nnz;             // selected elements                        the element's in front to say: not counted
  int32_t starts;          // elements but the first that start a run
  int32_t last;            // position of the last of these (-1: none)
  int32_t ends;            // kFirstYes, kLastYes: the first / last element is selected; kEmpty: no elements
};
constexpr int kFirstYes = 1, kLastYes = 2, kEmpty = 4;

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
  uint32_t* bits;        // [sub-tiles * 32] selected elements
  float* vals;           // [n] selected values, every chunk's from its first element's place on
  int32_t subs;          // sub-tiles per chunk
  uint32_t src_rank;
};

// |v| >= cut selects: like the reference, except that zeros are never selected
__device__ __forceinline__ float cut_of(float thr) { return thr == 0.f ? __uint_as_float(1u) : thr; }

// totals of a, with what follows it; `start`: position of b's first element
__device__ __forceinline__ ChunkTotals append(const ChunkTotals& a, const ChunkTotals& b, int64_t start) {
  if (b.ends & kEmpty) return a;
  ChunkTotals t;
  const bool edge = ((a.ends & kLastYes) != 0) != ((b.ends & kFirstYes) != 0);
  t.nnz = a.nnz + b.nnz;
  t.starts = a.starts + b.starts + (edge ? 1 : 0);
  t.last = b.last >= 0 ? b.last : edge ? (int32_t)start : a.last;
  t.ends = (a.ends & kFirstYes) | (b.ends & kLastYes);
  return t;
}

// One pass: g and r are read, r and the words are written.  A lane holds every 32nd element, so no access
// needs an alignment and the selection of a row is one ballot.
template <typename T, bool HAS_G, bool HAS_R>
__global__ void __launch_bounds__(kThreads, kSendPerSm) rle_scan_kernel(const __grid_constant__ SendParams p) {
  __shared__ ChunkTotals s_chunk[kWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t chunk = (int64_t)blockIdx.x * kWarps + w;
  const int64_t lo = chunk * p.subs * CX_SUBTILE, hi = min(lo + (int64_t)p.subs * CX_SUBTILE, p.n);
  const T* __restrict__ g = reinterpret_cast<const T*>(p.g);
  if (lo + 32 * lane < hi) {           // the first sub-tile starts its way to L2 behind the kernel in front
    if (HAS_R) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.r + lo + 32 * lane));
    if (HAS_G) asm volatile("prefetch.global.L2 [%0];" ::"l"(g + lo + 32 * lane));
  }
  cx::pdl_wait();
  cx::pdl_trigger();
  const float cut = cut_of(*p.thr);
  float* to = p.vals + lo;             // where the next selected value goes (the same in all lanes)
  const uint32_t below = (1u << lane) - 1u;
  uint32_t tail = 0;                   // bit of the element in front
  int st = 0, last = -1, ends = lo < hi ? 0 : kEmpty;
  for (int64_t sub = lo; sub < hi; sub += CX_SUBTILE) {
    const int left = (int)min((int64_t)CX_SUBTILE, hi - sub);
    uint32_t word = 0;                 // elements 32 lane ... of the sub-tile
#pragma unroll 1
    for (int j0 = 0; j0 < CX_SUBTILE / 32; j0 += kRows) {
      const int here = left - 32 * j0 - lane;          // my elements: 32 j < here
      const float* rp = p.r + (sub + 32 * j0 + lane);
      const T* gp = g + (sub + 32 * j0 + lane);
      auto rows = [&](auto whole) {
        constexpr bool WHOLE = decltype(whole)::value;
        float v[kRows], b[kRows];
#pragma unroll
        for (int j = 0; j < kRows; ++j) {
          v[j] = HAS_R && (WHOLE || 32 * j < here) ? rp[32 * j] : 0.f;
          b[j] = HAS_G && (WHOLE || 32 * j < here) ? cx::Elem<T>::to_f(gp[32 * j]) : 0.f;
        }
#pragma unroll
        for (int j = 0; j < kRows; ++j) {
          if (HAS_R && HAS_G) v[j] = b[j] + v[j];
          else if (HAS_G) v[j] = b[j];
          const bool yes = (WHOLE || 32 * j < here) && fabsf(v[j]) >= cut;
          const uint32_t row = __ballot_sync(0xffffffffu, yes);
          if (lane == j0 + j) word = row;
          if (yes) to[__popc(row & below)] = v[j];
          to += __popc(row);
          if (HAS_R && (WHOLE || 32 * j < here)) const_cast<float*>(rp)[32 * j] = yes ? 0.f : v[j];
        }
      };
      if (left >= 32 * (j0 + kRows)) rows(std::true_type());         // (warp-uniform)
      else rows(std::false_type());
    }
    p.bits[(sub >> 5) + lane] = word;
    uint32_t prev = __shfl_up_sync(0xffffffffu, word >> 31, 1);
    if (lane == 0) prev = sub == lo ? word & 1u : tail;          // the chunk's first element: as if it went on
    tail = __shfl_sync(0xffffffffu, word >> 31, 31);
    if (sub == lo) ends |= __shfl_sync(0xffffffffu, word, 0) & 1u ? kFirstYes : 0;
    const int valid = left - 32 * lane;
    uint32_t starts = word ^ (word << 1 | prev);
    if (valid < 32) starts &= valid <= 0 ? 0u : (1u << valid) - 1u;
    st += __popc(starts);
    if (starts) last = (int)(sub + 32 * lane + 31 - __clz(starts));
    if (sub + CX_SUBTILE >= hi) {
      const int end = left - 1;
      ends |= (__shfl_sync(0xffffffffu, word, end >> 5) >> (end & 31)) & 1u ? kLastYes : 0;
    }
  }
  st = __reduce_add_sync(0xffffffffu, st);
  last = __reduce_max_sync(0xffffffffu, last);
  if (lane == 0) {
    s_chunk[w] = ChunkTotals{(int32_t)(to - (p.vals + lo)), st, last, ends};
    p.chunk[chunk] = s_chunk[w];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    ChunkTotals t = s_chunk[0];
    for (int j = 1; j < kWarps; ++j) t = append(t, s_chunk[j], (chunk + j) * p.subs * CX_SUBTILE);
    p.cta[blockIdx.x] = t;
    if (blockIdx.x == 0) p.meta->first_yes = p.n > 0 && (t.ends & kFirstYes) ? 1 : 0;
  }
}

// Bound by latency: totals, words, then the stores of the payload (2^22 elements at 10 %: 4.7 MB).
__global__ void __launch_bounds__(kThreads, kSendPerSm) rle_emit_kernel(const __grid_constant__ SendParams p) {
  __shared__ uint16_t s_start[kWarps][CX_SUBTILE];
  __shared__ int s_pre[kWarps][5];
  __shared__ ChunkTotals s_chunk[kWarps];
  __shared__ uint32_t s_lastblock;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int64_t chunk = (int64_t)blockIdx.x * kWarps + w, span = (int64_t)p.subs * CX_SUBTILE;
  const int64_t lo = chunk * span, hi = min(lo + span, p.n);
  cx::pdl_wait();
  const float thr = *p.thr;
  // my chunk's first words, and the element in front of it
  uint32_t word = lo < hi ? p.bits[(lo >> 5) + lane] : 0u;
  uint32_t tail = lo > 0 && lo < hi ? p.bits[(lo >> 5) - 1] >> 31 : 0u;
  // where this chunk's values and runs go, and the totals of all: CTA c's first element starts a run when the
  // one in front of it differs
  int k0 = 0, q0 = 0, prev = -1, nnz_total = 0, nruns = 0;
  for (int c = tid; c < (int)gridDim.x; c += kThreads) {
    const ChunkTotals t = p.cta[c];
    const bool edge = c == 0 ? p.n > 0 : ((p.cta[c - 1].ends & kLastYes) != 0) != ((t.ends & kFirstYes) != 0);
    const int starts = t.starts + (edge ? 1 : 0);
    nnz_total += t.nnz;
    nruns += starts;
    if (c < (int)blockIdx.x) {
      k0 += t.nnz;
      q0 += starts;
      prev = max(prev, t.last >= 0 ? t.last : edge ? (int)(c * kWarps * span) : -1);
    }
  }
  if (tid < kWarps) s_chunk[tid] = p.chunk[(int64_t)blockIdx.x * kWarps + tid];
  k0 = __reduce_add_sync(0xffffffffu, k0);
  q0 = __reduce_add_sync(0xffffffffu, q0);
  prev = __reduce_max_sync(0xffffffffu, prev);
  nnz_total = __reduce_add_sync(0xffffffffu, nnz_total);
  nruns = __reduce_add_sync(0xffffffffu, nruns);
  if (lane == 0) { s_pre[w][0] = k0; s_pre[w][1] = q0; s_pre[w][2] = prev; s_pre[w][3] = nnz_total; s_pre[w][4] = nruns; }
  __syncthreads();
  k0 = q0 = nnz_total = nruns = 0;
  prev = -1;
#pragma unroll
  for (int j = 0; j < kWarps; ++j) {
    k0 += s_pre[j][0]; q0 += s_pre[j][1]; prev = max(prev, s_pre[j][2]); nnz_total += s_pre[j][3]; nruns += s_pre[j][4];
  }
  {
    // the chunks of this CTA in front of mine; the first one's first element is seen against the CTA before
    uint32_t front = (uint32_t)__shfl_sync(0xffffffffu, tail, 0);
    const int64_t first = (int64_t)blockIdx.x * kWarps * span;
    if (w > 0) front = first > 0 ? p.bits[(first >> 5) - 1] >> 31 : 0u;
    for (int j = 0; j < w; ++j) {
      const ChunkTotals t = s_chunk[j];
      if (t.ends & kEmpty) break;
      const int64_t start = first + j * span;
      const bool edge = start == 0 || (front != 0) != ((t.ends & kFirstYes) != 0);
      k0 += t.nnz;
      q0 += t.starts + (edge ? 1 : 0);
      prev = t.last >= 0 ? t.last : edge ? (int)start : prev;
      front = t.ends & kLastYes ? 1u : 0u;
    }
  }
  const int mine = s_chunk[w].ends & kEmpty ? 0 : s_chunk[w].nnz;
  const size_t runs_off = 8 + 4 * (size_t)nnz_total + 8;
  // the chunk's values
  for (int k = 0; k < p.tg.count; ++k) {
    float* out = reinterpret_cast<float*>(reinterpret_cast<char*>(p.tg.ep[k].pairs) + 8) + k0;
    const float* in = p.vals + lo;
#pragma unroll 4
    for (int i = lane; i < mine; i += 32) out[i] = in[i];
  }
  uint16_t* ss = s_start[w];
  for (int64_t sub = lo; sub < hi; sub += CX_SUBTILE) {
    const int valid = (int)min((int64_t)32, max((int64_t)0, hi - sub - 32 * lane));
    uint32_t front = __shfl_up_sync(0xffffffffu, word >> 31, 1);
    if (lane == 0) front = tail;
    tail = __shfl_sync(0xffffffffu, word >> 31, 31);
    uint32_t starts = word ^ (word << 1 | front);
    if (sub == 0 && lane == 0) starts |= 1u;                    // element 0 always starts a run
    if (valid < 32) starts &= (1u << valid) - 1u;
    if (sub + CX_SUBTILE < hi) word = p.bits[(sub >> 5) + 32 + lane];      // under way during the stores
    const uint32_t number = __popc(starts);
    uint32_t incl = number;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += t;
    }
    const int ns = (int)__shfl_sync(0xffffffffu, incl, 31);
    uint16_t* list = ss + (incl - number);
    for (uint32_t bits = starts; bits; bits &= bits - 1) *list++ = (uint16_t)(32 * lane + __ffs(bits) - 1);
    __syncwarp();
    for (int k = 0; k < p.tg.count; ++k) {
      // start q closes run q - 1
      int32_t* runs = reinterpret_cast<int32_t*>(reinterpret_cast<char*>(p.tg.ep[k].pairs) + runs_off) + q0 - 1;
      for (int i = lane; i < ns; i += 32)
        if (q0 + i > 0) runs[i] = i ? (int)ss[i] - (int)ss[i - 1] : (int)(sub + ss[0] - prev);
    }
    if (ns) prev = (int)(sub + ss[ns - 1]);
    q0 += ns;
    __syncwarp();
  }
  if (lo < hi && hi == p.n && lane < p.tg.count)     // the warp that holds the last element closes the last run
    reinterpret_cast<int32_t*>(reinterpret_cast<char*>(p.tg.ep[lane].pairs) + runs_off)[q0 - 1] = (int)(p.n - prev);
  __syncthreads();
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
  uint32_t front_wait;  // CX_WAIT_*: the kernel in front may be an expansion that still reads the index
  uint32_t* status;
  uint64_t timeout_ns;
};

__device__ __forceinline__ int64_t blocks_per_group(int64_t nruns, int groups) {
  const int64_t blocks = (nruns + kRunBlock - 1) / kRunBlock;
  return (blocks + groups - 1) / groups;
}

__global__ void __launch_bounds__(kThreads) rle_index_kernel(const __grid_constant__ RecvParams p) {
  __shared__ int s_state, s_first;
  __shared__ int64_t s_nnz, s_nruns;
  __shared__ int s_bad;
  __shared__ long long s_sum[kWarps][2];
  cx::pdl_trigger();
  if (p.front_wait == CX_WAIT_START) cx::pdl_wait();   // (the vector is touched by the kernel behind, which waits for this one)
  if (threadIdx.x == 0) {
    int st = 0, first = 0;
    int64_t nnz = 0, nruns = 0;
    if (!cx::wait_seq(&p.src.hdr->seq, p.expect_seq, p.timeout_ns)) st = CX_ST_TIMEOUT;
    if (!st) {
      // one round trip for the header and the first words of the payload (there is room for them in any slot)
      const int32_t* pay = reinterpret_cast<const int32_t*>(p.src.pairs);
      const uint32_t kind = __ldcg(&p.src.hdr->kind), hn = __ldcg(&p.src.hdr->n);
      const int32_t pn = __ldcg(pay);
      nnz = __ldcg(pay + 1);
      if (kind != CX_KIND_RLE || (int64_t)hn != p.n) st = CX_ST_BAD_HEADER;
      else if ((int64_t)pn != p.n || nnz < 0 || nnz > p.n || 16 + 4 * nnz > p.slot_bytes) st = CX_ST_BAD_HEADER;
      if (!st) {
        const int32_t* rh = reinterpret_cast<const int32_t*>(reinterpret_cast<const char*>(p.src.pairs) + 8 + 4 * nnz);
        nruns = __ldcg(rh);
        first = __ldcg(rh + 1) != 0;
        if (nruns < 0 || nruns > p.n + 1 || 16 + 4 * nnz + 4 * nruns > p.slot_bytes) st = CX_ST_BAD_HEADER;
      }
    }
    s_state = st;
    s_first = first;
    s_nnz = nnz;
    s_nruns = nruns;
    s_bad = 0;
  }
  __syncthreads();
  const int st = s_state, first = s_first;
  const int64_t nnz = s_nnz, nruns = s_nruns;
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
    const int32_t* runs = reinterpret_cast<const int32_t*>(reinterpret_cast<const char*>(p.src.pairs) + 16 + 4 * nnz);
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

// Bound by the chain of dependent loads in front of the output, then by the output (read and written for
// `add`).  Looking every output's run up by bisection in the scanned block took 40 us for 2^22 elements at
// top-k 10 %, a mask with one shared-memory atomic per run and four outputs per thread 17 us.  Here two
// blocks of runs are taken at a time (a window of 8192 outputs mostly needs no more), a thread's starts go
// to the mask word by word, and every lane walks the set bits of its own word.
__global__ void __launch_bounds__(kThreads, 4) rle_expand_kernel(const __grid_constant__ RecvParams p) {
  __shared__ long long s_l[kWarps];
  __shared__ int s_a[kWarps], s_b[kWarps];
  __shared__ int s_pick[3];
  __shared__ uint32_t s_mask[kThreads];    // run starts of the window
  // the window of `out` starts its way to L2 while the index is made
  if (p.add) {
    const int64_t i = (int64_t)blockIdx.x * p.per_cta + 32 * threadIdx.x;
    if (i < p.n) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.out + i));
  }
  cx::pdl_wait();
  cx::pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const bool have = tid < p.groups;
  const int ok = p.meta->ok, nnz = p.meta->nnz, nruns = p.meta->nruns, first = p.meta->first_yes;
  const RunSums g = have ? p.group[tid] : RunSums{0, 0};
  const int gbad = have ? p.group_bad[tid] : 0;
  if (!ok) return;
  const int64_t e0 = (int64_t)blockIdx.x * p.per_cta;
  const int64_t e1 = min(e0 + p.per_cta, p.n);
  // every CTA checks the whole payload before any of them writes; group g belongs to thread g
  int64_t blk = 0;
  int at = 0, at_yes = 0;                  // elements and selected elements before block `blk`
  const int64_t nblocks = ((int64_t)nruns + kRunBlock - 1) / kRunBlock;
  {
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
  int vbase = -1;                          // index of the first value at or behind the window's start
  for (int64_t w0 = e0; w0 < e1; w0 += kWindow) {
    const int64_t w1 = min(w0 + kWindow, e1);
    s_mask[tid] = 0;
    // runs that reach into the window, two blocks at a time; a run that began earlier counts at its first bit
    for (;;) {
      int len[kRunsEach], mine = 0, part = 0;
      const int64_t q0 = blk * kRunBlock + kRunsEach * tid;
#pragma unroll
      for (int k = 0; k < kRunsEach; ++k) {
        len[k] = q0 + k < nruns ? runs[q0 + k] : 0;
        mine += len[k];
      }
      int tot;
      int pos = at + block_prefix<int>(mine, tot, s_a);
      uint32_t to = 0, flips = 0;          // starts of one word of the mask, before they go there together
#pragma unroll
      for (int k = 0; k < kRunsEach; ++k) {
        if (q0 + k < nruns && pos < w1) {
          const uint32_t bit = pos > w0 ? (uint32_t)(pos - w0) : 0u;
          if (bit >> 5 != to) {
            if (flips) atomicXor(&s_mask[to], flips);
            to = bit >> 5;
            flips = 0;
          }
          flips ^= 1u << (bit & 31);
          const bool yes = ((k & 1) == 0) == (first != 0);
          if (yes && pos < w0) part += (int)(min((int64_t)pos + len[k], w0) - pos);
        }
        pos += len[k];
      }
      if (flips) atomicXor(&s_mask[to], flips);
      if (vbase < 0) {                     // once per CTA: values of these runs in front of the window
        int before;
        block_prefix<int>(part, before, s_b);
        vbase = at_yes + before;
      }
      if ((int64_t)at + tot >= w1 || blk + 2 >= nblocks) break;
      at += tot;
      blk += 2;
      __syncthreads();                     // s_a is written again
    }
    __syncthreads();
    // word by word: parity of the starts up to every bit, the selected bits, and their number before
    uint32_t x = s_mask[tid];
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
    vbase += total;
    if (!p.add) {                          // zeros first, a row of 32 outputs at a time
      float* row = p.out + (w0 + 32 * (tid & ~31) + lane);
      const int64_t here = w1 - (w0 + 32 * (tid & ~31) + lane);
#pragma unroll
      for (int j = 0; j < 32; ++j) if (32 * j < here) row[32 * j] = 0.f;
      __syncwarp();                        // the other lanes' zeros are in front of this lane's values
    }
    // then every lane the selected outputs of its own word, kBitsOut of them in flight
    float* mine32 = p.out + (w0 + 32 * tid);
    const float* val = vals + mybase;
    while (x) {
      int at32[kBitsOut];
      float y[kBitsOut], z[kBitsOut];
#pragma unroll
      for (int k = 0; k < kBitsOut; ++k) {
        at32[k] = __ffs(x) - 1;            // -1: no more
        x &= x - 1;
        y[k] = at32[k] >= 0 ? val[k] : 0.f;
        z[k] = at32[k] >= 0 && p.add ? mine32[at32[k]] : 0.f;
      }
#pragma unroll
      for (int k = 0; k < kBitsOut; ++k)
        if (at32[k] >= 0) mine32[at32[k]] = p.add ? z[k] + y[k] : y[k];
      val += kBitsOut;
    }
    if (w0 + kWindow < e1) __syncthreads();          // s_a is written again
  }
}

}  // namespace

int64_t cx_rle_slot_bytes(int64_t n) { return (16 + 8 * n + 15) / 16 * 16; }

static int64_t align256(int64_t bytes) { return (bytes + 255) / 256 * 256; }
static int64_t sub_tiles(int64_t n) { return (n + CX_SUBTILE - 1) / CX_SUBTILE; }
constexpr int64_t kSendFixed = 256 + kMaxSend * (1 + kWarps) * (int64_t)sizeof(ChunkTotals);
static_assert(kSendFixed % 256 == 0, "the words behind the totals are aligned");

int64_t cx_rle_recv_workspace_bytes(int64_t n) {
  const int64_t blocks = (n + 1 + kRunBlock - 1) / kRunBlock;
  return align256(256 + kGroups * (int64_t)(sizeof(RunSums) + sizeof(int32_t)) + blocks * (int64_t)sizeof(RunSums));
}
int64_t cx_rle_workspace_bytes(int64_t n) {
  const int64_t send = align256(kSendFixed + sub_tiles(n) * 128 + 4 * n), recv = cx_rle_recv_workspace_bytes(n);
  return send > recv ? send : recv;
}

namespace {
template <typename T>
void launch_send(const SendParams& p, int grid, cudaStream_t s) {
  if (p.g && p.r) cx_launch_pdl(rle_scan_kernel<T, true, true>, grid, kThreads, 0, s, p, false);
  else if (p.r) cx_launch_pdl(rle_scan_kernel<T, false, true>, grid, kThreads, 0, s, p, false);
  else cx_launch_pdl(rle_scan_kernel<T, true, false>, grid, kThreads, 0, s, p, false);
  cx_launch_pdl(rle_emit_kernel, grid, kThreads, 0, s, p, false);
}
}  // namespace

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
  // one chunk of whole sub-tiles per warp, at most one wave of CTAs
  const int64_t nsub = n > 0 ? sub_tiles(n) : 1;
  int64_t wave = (int64_t)cx_sm_count() * kSendPerSm;
  if (wave > kMaxSend) wave = kMaxSend;
  p.subs = (int)((nsub + wave * kWarps - 1) / (wave * kWarps));
  const int grid = (int)((nsub + (int64_t)p.subs * kWarps - 1) / ((int64_t)p.subs * kWarps));
  char* ws = reinterpret_cast<char*>(workspace);
  p.meta = reinterpret_cast<RleMeta*>(ws);
  p.cta = reinterpret_cast<ChunkTotals*>(ws + 256);
  p.chunk = p.cta + kMaxSend;
  p.bits = reinterpret_cast<uint32_t*>(ws + kSendFixed);
  p.vals = reinterpret_cast<float*>(p.bits + 32 * sub_tiles(n));
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  switch (gdtype) {
    case CX_F32: launch_send<float>(p, grid, s); break;
    case CX_BF16: launch_send<__nv_bfloat16>(p, grid, s); break;
    case CX_F16: launch_send<__half>(p, grid, s); break;
    default: return cx_set_error("cx_rle_send: unsupported dtype on CUDA", 0);
  }
  cx_note_sender(stream);
  cx_note_launch();
  cx_note_launch();
  return cx_check_launch("rle send kernels");
}

int cx_rle_recv_cuda(const CxEndpoint* src, uint64_t expect_seq, float* out, int64_t n, int add,
                     int64_t slot_bytes, void* workspace, int64_t ws_bytes, uint32_t* status,
                     uint64_t timeout_ns, void* stream) {
  if (n < 0 || n > 0x7fffffffLL) return cx_set_error("cx_rle_recv: n out of range", 0);
  if (ws_bytes < cx_rle_recv_workspace_bytes(n)) return cx_set_error("cx_rle_recv: workspace too small", 0);
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
  p.front_wait = cx_front_wait(stream);
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
