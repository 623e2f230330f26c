// Fused residual-add / threshold-select / compaction / peer store.
//
// One pass over the vector does what the reference does in
// ThresholdFunction + CompressorIndexPairs::compress_add_update followed by
// SourceBuffer::initTransferPart (src/compressor.hxx:556-611,
// src/comprEx.tpp:176-191):
//
//     r += g ; if |r| > thr { emit (i, r) ; r = 0 }
//
// Work is warp-granular and free of block-wide barriers: a warp owns one
// 1024-element sub-tile at a time, loads it with 16-byte accesses (32
// elements per lane, all loads in flight together), puts the sums into shared memory, ranks the survivors with
// one warp scan, reserves room for them in the pair list with ONE atomicAdd on a counter in this GPU's
// memory, and stores them, picked from shared memory by a list of their places, as coalesced
// 8-byte (index, value) pairs straight into the receive
// slots of up to CX_MAX_PEERS targets (peer GPUs' memory mapped over NVLink,
// or local slots), or once through the switch's multicast mapping.  No warp
// ever waits for another one, so the kernel has no spin loop at all.
//
// The pairs of one sub-tile are contiguous in the list; sub-tiles land in the
// list in the order of their reservations.  Next to the pairs every target
// receives one table entry per sub-tile, {start, count}: receivers use it to
// find, without searching or sorting, the pairs that fall into the part of
// the vector they own, and to apply them in a fixed order.  (The reference's
// wire format lists the pairs in ascending index order; nothing on the
// receiving side depends on that order, each index occurs once per payload.)
//
// Survivors that do not fit into the slot are not emitted and stay in the
// residual, which error feedback makes safe; the count is reported.  The CTA
// that finishes last writes the header and publishes the notification: its
// st.release.sys covers the stores of all CTAs, which were ordered before their
// arrivals at GPU scope (cx::cta_arrive).
#include <stdlib.h>
#include <string.h>

#include "cx_fold.cuh"

namespace {

// 16 warps per SM: each lane keeps a whole sub-tile share of 32 values in registers with all its loads in
// flight, which takes the 128 registers that leaves a thread (no spills without multicast; the folding
// kernel spills 82 to 114 bytes a thread with fp32 momentum, 98 to 226 with 16-bit gradients, most of them at
// tensor borders).  Squeezing more warps onto an SM makes it spill and measured slower at every size (2^24
// elements, 1 %: 55 us with 16 warps, 69 us with 24), and so did an L2 prefetch of the warp's next sub-tile, and
// loads of the next sub-tile issued while this one is stored (2^28 elements 633 -> 650 us).
#ifndef CX_COMPRESS_BULK_DEFAULT
#define CX_COMPRESS_BULK_DEFAULT 0
#endif

// Warps of one CTA wait for one another only at its end, so small CTAs spread a short vector over more
// SMs and let each go as soon as it is done: 65 536 elements 12.3 us with 256 threads, 12.0 with 128 and
// 64; 2^20 elements 15.8, 15.3 and 15.1.  From 6 M elements on it makes no difference.
constexpr int kThreads = 64, kWarpsPerSm = 16;
constexpr int kWarps = kThreads / 32;
constexpr int kPerSm = kWarpsPerSm / kWarps;
constexpr int kChunks = CX_SUBTILE / 128;  // 128 elements = 32 lanes x 4

// -DCX_COMPRESS_TRACE: thread 0 of every CTA stamps %globaltimer at up to eight points of
// compress_kernel (entry, before the loop, after the loop, after the arrival, and in the CTA that
// arrives last: regions summed, headers published, end) into a device array that
// cx_compress_trace copies out; a development aid for the fixed part of the kernel's time, not compiled by default.
#ifdef CX_COMPRESS_TRACE
__device__ unsigned long long g_cx_trace[8 * 2048];
#define CX_TRACE(slot)                                                   \
  do {                                                                   \
    if (threadIdx.x == 0 && blockIdx.x < 2048) {                         \
      unsigned long long t_;                                             \
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_));             \
      g_cx_trace[blockIdx.x * 8 + (slot)] = t_;                          \
    }                                                                    \
  } while (0)
#else
#define CX_TRACE(slot) do { } while (0)
#endif

struct CompressParams {
  const void* g;
  float* r;
  int64_t n;
  const float* thr;
  uint32_t cap;
  uint32_t nsub;
  uint32_t nregions;     // power of two; sub-tile s reserves in region s % nregions
  uint32_t region_size;  // cap / nregions pairs each
  uint32_t early;        // the first sub-tile may be loaded before the kernel in front has finished
  uint32_t vec;          // g and r are aligned for 16-byte (8-byte for 16-bit g) accesses
  uint64_t seq;
  const uint64_t* seq_cell;  // non-NULL inside a captured graph: the sequence number lives there
  CxWorkCounters* ctr;
  CxStats* stats;
  uint32_t src_rank;
  CxTargets tg;
};

// Where the vector that is added to the residual comes from.
enum Input {
  kPlain,      // p.g (or nothing)
  kFold,       // folded from gradient tensors (CxFold), nothing of it kept
  kFoldWrite,  // the same, stored as the new momentum
  kFoldMom     // momentum read, moved on, stored
};
struct FoldCompressParams {
  CompressParams c;
  CxFold f;
  uint32_t chain;   // CX_CHAINED, CX_CHAIN_NEXT
  uint32_t nborder_ctas;
};

// What a warp has seen so far, for the completion.
struct Tally {
  uint32_t found;   // survivors
  bool over;        // some of them did not fit the slot
};

// One aligned, complete sub-tile, one warp, one pass: lane L holds elements {c*128 + 4L + e} in
// registers from the loads to the write-back of the residual.
// gl / rl: where this sub-tile's gradient and residual are read (global memory, or the copy of the
// sub-tile that the copy engine put into shared memory).
template <typename T, bool HAS_G, bool HAS_R>
__device__ __forceinline__ void load_subtile(const T* __restrict__ gl, const float* __restrict__ rl, const int lane,
                                             float (&v)[kChunks][4]) {
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
#pragma unroll
    for (int e = 0; e < 4; ++e) v[c][e] = 0.f;
    if (HAS_R) cx::load4(rl + lane * 4 + c * 128, v[c]);
  }
  if (HAS_G) {
#pragma unroll
    for (int c = 0; c < kChunks; ++c) {
      float b[4];
      cx::load4(gl + lane * 4 + c * 128, b);
#pragma unroll
      for (int e = 0; e < 4; ++e) v[c][e] = v[c][e] + b[e];
    }
  }
}

// The threshold where it is first needed: behind the wait for the kernel in front, which so covers the loads
// ahead of it (that kernel only reads).  Nothing may be stored before get().
struct LateThreshold {
  const float* cell;
  uint32_t chain;
  bool have;
  float thr;
  __device__ __forceinline__ float get() {
    if (!have) {
      if (!(chain & CX_CHAINED)) cx::pdl_wait();
      if (chain & CX_CHAIN_NEXT) cx::pdl_trigger();
      thr = *reinterpret_cast<const volatile float*>(cell);
      have = true;
    }
    return thr;
  }
};
struct KnownThreshold {
  float thr;
  __device__ __forceinline__ float get() const { return thr; }
};

// The same for a folded input: up, mu, coef are the sub-tile's momentum and factors.
template <typename T, Input IN, typename Thr>
__device__ __forceinline__ void load_fold_subtile(const T* __restrict__ gl, const float* __restrict__ rl, float* __restrict__ up,
                                                  const float mu, const float coef, const uint64_t last, const int lane,
                                                  float (&v)[kChunks][4], Thr& late) {
#pragma unroll
  for (int c = 0; c < kChunks; ++c) cx::load4(rl + lane * 4 + c * 128, v[c]);
  // all loads of a group are issued before its first store: the compiler must not move them across
  constexpr int kGroup = IN == kFoldMom && sizeof(T) == 4 ? kChunks / 2 : kChunks;
#pragma unroll
  for (int c0 = 0; c0 < kChunks; c0 += kGroup) {
    typename cx::Raw4<T>::type x[kGroup];
    float y[kGroup][4];
#pragma unroll
    for (int c = 0; c < kGroup; ++c) {
      x[c] = cx::load_hint(reinterpret_cast<const typename cx::Raw4<T>::type*>(gl + lane * 4 + (c0 + c) * 128), last);
      if (IN == kFoldMom) cx::load4(up + lane * 4 + (c0 + c) * 128, y[c]);
    }
    if (IN != kFold && c0 == 0) late.get();      // loads only before, stores from here on
#pragma unroll
    for (int c = 0; c < kGroup; ++c) {
      float t[4];
      cx::Raw4<T>::to_f(x[c], t);
#pragma unroll
      for (int e = 0; e < 4; ++e) t[e] = mu * (IN == kFoldMom ? y[c][e] : 0.f) + coef * t[e];
      if (IN != kFold) cx::store4(up + lane * 4 + (c0 + c) * 128, t);
#pragma unroll
      for (int e = 0; e < 4; ++e) v[c0 + c][e] = v[c0 + c][e] + t[e];
    }
  }
}

// A warp's survivors on their way out: the sub-tile's values, and the places of those that go, in order (more
// than the list holds: one part of them after the other).
constexpr uint32_t kList = 512;
struct Stage {
  float v[CX_SUBTILE];
  uint16_t at[kList];
};

// Selection, compaction and write-back of a loaded sub-tile.  rs: the residual's sub-tile in global
// memory, where the new residual goes.
// A vector of one to three sub-tiles per warp is bound by this chain, not by memory: all warps walk through it
// in step.  So the values go to shared memory first; a lane's survivors are then found by their bits (0.3 of 32 at
// 1 %) instead of by 32 tests with a branch each, and the residual leaves before the reservation is back.
// 2^16 / 2^20 elements 11.9 / 14.9 -> 11.4 / 14.3 us per exchange, 8 x 6.5 M 260 -> 250.
// LONG: many sub-tiles per warp and fp32 gradients.  What counts there is how long the list of a sub-tile with many
// survivors takes: the fullest lane has five or six of them at 10 %, and as many steps; eight steps of four tests,
// with the lanes side by side, are faster then.  fp32, 10 %, added, us per exchange with the bits walked / with tests:
// 30 M 111.2 / 112.1, 50 M 180.7 / 178.5, 100 M 355.5 / 345.6, 128 Mi 475 / 461 (a shorter vector waits for the code:
// 1 Mi 15.4 / 16.0); bf16, 128 Mi 421 / 431.  At 3 % (31 of 1024, few sub-tiles above kMany) there is no difference.
constexpr uint32_t kMany = 48;
template <bool HAS_G, bool HAS_R, bool MC, bool LONG = false>
__device__ __forceinline__ void emit_subtile(const CompressParams& p, const uint32_t sub, const int lane, const float thr,
                                             float* __restrict__ rs, float* sv, uint16_t* sat, float (&v)[kChunks][4],
                                             Tally& tally) {
  // ---- classify: bit c*4+e of mask, strict '>' like the reference; v becomes the new residual -------
#pragma unroll
  for (int c = 0; c < kChunks; ++c) cx::store4(sv + c * 128 + lane * 4, v[c]);
  uint32_t mask = 0;
#pragma unroll
  for (int c = 0; c < kChunks; ++c) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (fabsf(v[c][e]) > thr) {
        mask |= 1u << (4 * c + e);
        v[c][e] = 0.f;
      }
    }
  }

  // ---- rank: lanes in order, each lane's survivors consecutive --------------------
  const uint32_t mine = __popc(mask);
  uint32_t incl = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += t;
  }
  const uint32_t count = __shfl_sync(0xffffffffu, incl, 31);

  // ---- reserve room in the pair list ----------------------------------------------
  // The list is cut into nregions equal regions with one counter each, neighbouring
  // sub-tiles use different regions: atomics on one address are serialised by the L2.
  const uint32_t region = sub & (p.nregions - 1);
  uint32_t base = 0;
  if (count && lane == 0) base = atomicAdd(&p.ctr->region[region][0], count);   // under way until it is asked for

  // ---- residual: zero for every survivor; those that turn out not to fit are put back below ---------
  if (HAS_R) {
    float* wp = rs + lane * 4;
#pragma unroll
    for (int c = 0; c < kChunks; ++c) {
      if (!HAS_G && ((mask >> (4 * c)) & 0xfu) == 0) continue;  // nothing changed in this vector
      cx::store4(wp + c * 128, v[c]);
    }
  }

  // my survivors among the list's entries [w0, w0 + kList)
  auto fill = [&](const uint32_t w0) {
    if (LONG && count > kMany) {
      uint32_t pos = incl - mine - w0;
#pragma unroll 1
      for (uint32_t m = mask, at = lane * 4; m; m >>= 4, at += 128) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (m >> e & 1u) {
            if (pos < kList) sat[pos] = (uint16_t)(at + e);
            ++pos;
          }
        }
      }
      return;
    }
    // two halves of the mask side by side: half the steps of a chain of dependent instructions
    uint32_t low = mask & 0xffffu, high = mask >> 16;
    uint32_t pos = incl - mine - w0, hpos = pos + __popc(low);   // wrap below the window: fail the test
    while (low | high) {
      if (low) {
        const uint32_t b = __ffs(low) - 1;
        if (pos < kList) sat[pos] = (uint16_t)((b >> 2) * 128 + lane * 4 + (b & 3));
        low &= low - 1;
        ++pos;
      }
      if (high) {
        const uint32_t b = __ffs(high) - 1;
        if (hpos < kList) sat[hpos] = (uint16_t)((b >> 2) * 128 + 512 + lane * 4 + (b & 3));
        high &= high - 1;
        ++hpos;
      }
    }
  };
  fill(0);
  base = __shfl_sync(0xffffffffu, base, 0);
  const uint32_t emit = base >= p.region_size ? 0u : min(count, p.region_size - base);  // pairs that fit
  base += region * p.region_size;
  tally.found += count;
  tally.over |= emit < count;
  {
    uint2 entry;
    entry.x = emit ? base : 0u;
    entry.y = emit;
    if (MC) {
      if (lane == 0) cx::mm_st_b64(reinterpret_cast<uint2*>(p.tg.ep[p.tg.count].table) + sub, entry);
    } else if (lane < p.tg.count) {
      reinterpret_cast<uint2*>(p.tg.ep[lane].table)[sub] = entry;
    }
  }
  __syncwarp();

  // ---- coalesced to every target; what does not fit stays in the residual (the barrier above orders that
  //      behind the other lanes' zeros) ------------------------
  const int32_t sub_base = (int32_t)sub * CX_SUBTILE;
  for (uint32_t w0 = 0;;) {
    const uint32_t lim = min(count - w0, kList);
    for (uint32_t i = lane; i < lim; i += 32) {
      const uint32_t e = sat[i];
      CxPair pr;
      pr.idx = sub_base + (int32_t)e;
      pr.val = __float_as_uint(sv[e]);
      if (w0 + i >= emit) {
        if (HAS_R) rs[e] = sv[e];
      } else if (MC) {
        // one store per pair into the multicast mapping: the switch writes every target's slot
        cx::mm_st_b64(p.tg.ep[p.tg.count].pairs + base + w0 + i, make_uint2((uint32_t)pr.idx, pr.val));
      } else {
        for (int k = 0; k < p.tg.count; ++k) p.tg.ep[k].pairs[base + w0 + i] = pr;
      }
    }
    __syncwarp();
    w0 += kList;
    if (w0 >= count) break;                 // all of it, unless the sub-tile is dense
    fill(w0);
    __syncwarp();
  }
}

// Sub-tiles that are partial, not aligned for 16-byte accesses (the last one of a vector, views at
// odd offsets) or folded from several tensors: element 32 j + lane is lane's j-th, kept in a register
// from the load to the write-back, survivors ranked with warp ballots.  No assumption about alignment
// or length.  (Two passes of dependent single loads made a vector of 44 k elements take 13 us.)
template <typename T, bool HAS_G, bool HAS_R, bool MC, Input IN = kPlain, typename Thr = KnownThreshold>
__device__ __forceinline__ void compress_subtile_edge(const CompressParams& p, const uint32_t sub,
                                                      const int lane, Thr&& late,
                                                      const T* __restrict__ g, float* __restrict__ r,
                                                      Tally& tally, const CxFold* f = nullptr) {
  constexpr int kEach = CX_SUBTILE / 32;
  const int64_t sub_base = (int64_t)sub * CX_SUBTILE;
  const int left = (int)min((int64_t)CX_SUBTILE, p.n - sub_base) - lane;   // my elements: 32 j < left
  const int64_t at = sub_base + lane;
  float v[kEach];
#pragma unroll
  for (int j = 0; j < kEach; ++j) v[j] = HAS_R && 32 * j < left ? r[at + 32 * j] : 0.f;
  if (IN == kPlain && HAS_G) {
#pragma unroll
    for (int j = 0; j < kEach; ++j) v[j] = v[j] + (32 * j < left ? cx::Elem<T>::to_f(g[at + 32 * j]) : 0.f);
  }
  if (IN != kPlain) {
    const cx::FoldBlock<T> blk = cx::fold_blocks<T>(*f, sub, lane);
    constexpr int kGroup = IN == kFoldMom ? 16 : 32;     // loads in flight: none of them moves across a store of the momentum
#pragma unroll
    for (int j0 = 0; j0 < kEach; j0 += kGroup) {
      float x[kGroup], y[kGroup];
      uint32_t in = 0;
#pragma unroll
      for (int j = 0; j < kGroup; ++j) {
        const bool t = cx::fold_element<T>(blk, j0 + j, lane, x[j]);
        in |= (t ? 1u : 0u) << j;
        y[j] = IN == kFoldMom && t ? f->u[at + 32 * (j0 + j)] : 0.f;
      }
      if (IN != kFold && j0 == 0) late.get();
#pragma unroll
      for (int j = 0; j < kGroup; ++j) {
        const float t = f->mu * y[j] + __shfl_sync(0xffffffffu, blk.coef, (j0 + j) >> 1) * x[j];
        if (IN != kFold && ((in >> j) & 1u)) f->u[at + 32 * (j0 + j)] = t;
        v[j0 + j] = v[j0 + j] + ((in >> j) & 1u ? t : 0.f);
      }
    }
  }
  const float thr = late.get();
  uint32_t mask = 0, count = 0;
#pragma unroll
  for (int j = 0; j < kEach; ++j) {
    const bool sel = 32 * j < left && fabsf(v[j]) > thr;
    mask |= (sel ? 1u : 0u) << j;
    count += __popc(__ballot_sync(0xffffffffu, sel));
  }
  const uint32_t region = sub & (p.nregions - 1);
  uint32_t base = 0;
  if (count) {
    if (lane == 0) base = atomicAdd(&p.ctr->region[region][0], count);
    base = __shfl_sync(0xffffffffu, base, 0);
  }
  const uint32_t emit = base >= p.region_size ? 0u : min(count, p.region_size - base);
  base += region * p.region_size;
  tally.found += count;
  tally.over |= emit < count;
  {
    uint2 entry;
    entry.x = emit ? base : 0u;
    entry.y = emit;
    if (MC) {
      if (lane == 0) cx::mm_st_b64(reinterpret_cast<uint2*>(p.tg.ep[p.tg.count].table) + sub, entry);
    } else if (lane < p.tg.count) {
      reinterpret_cast<uint2*>(p.tg.ep[lane].table)[sub] = entry;
    }
  }
  uint32_t seen = 0;                       // survivors among the elements before 32 j
#pragma unroll
  for (int j = 0; j < kEach; ++j) {
    const bool sel = (mask >> j) & 1u;
    const uint32_t bal = __ballot_sync(0xffffffffu, sel);
    const uint32_t pos = seen + __popc(bal & ((1u << lane) - 1u));
    float keep = v[j];
    if (sel && pos < emit) {
      CxPair pr;
      pr.idx = (int32_t)(at + 32 * j);
      pr.val = __float_as_uint(v[j]);
      if (MC) {
        cx::mm_st_b64(p.tg.ep[p.tg.count].pairs + base + pos, make_uint2((uint32_t)pr.idx, pr.val));
      } else {
        for (int k = 0; k < p.tg.count; ++k) p.tg.ep[k].pairs[base + pos] = pr;
      }
      keep = 0.f;
    }
    if (HAS_R && 32 * j < left && (HAS_G || keep != v[j])) r[at + 32 * j] = keep;
    seen += __popc(bal);
  }
}

// Completion: every CTA adds its survivors, its arrival and its marks to one 64-bit counter with one
// atomic, whose result tells the CTA that arrives last all it has to know; it writes the headers and
// publishes the notification.  (Reading the 32 region counters back first was 1 us on the end of
// every exchange; they are read only when survivors did not fit.)  `failed`: this CTA could not
// process all its sub-tiles; the payload is then not published (the receivers' bounded waits run
// out) and the status says why.
//
// The fields: 31 bits for the survivors (a vector has fewer than 2^31 elements), 12 for the CTAs that arrived,
// 12 for those whose survivors did not all fit (all of them may say so: a dense residual that is flushed does
// that), 9 for those that failed (only the bulk variant's can, one CTA per SM).  No field may carry into the
// next one: the launches below keep their grids within kMaxGrid and kMaxBulkGrid.
constexpr int kArrived = 31, kOver = 43, kFailed = 55;
constexpr int kMaxGrid = (1 << (kOver - kArrived)) - 1, kMaxBulkGrid = (1 << (64 - kFailed)) - 1;
static_assert(kFailed - kOver >= kOver - kArrived, "every CTA that arrives may have overflowed");

template <int MAX_WARPS>
__device__ __forceinline__ void compress_finish(const CompressParams& p, const int tid, const float thr, const bool failed,
                                                const Tally& tally) {
  __shared__ uint32_t s_found[MAX_WARPS], s_mark[MAX_WARPS];
  __shared__ unsigned long long s_all;
  __shared__ uint32_t s_nnz;
  const int nw = blockDim.x >> 5;
  if ((tid & 31) == 0) {
    s_found[tid >> 5] = tally.found;
    s_mark[tid >> 5] = (tally.over ? 1u : 0u) | (failed ? 2u : 0u);
  }
  __syncthreads();            // all stores of the CTA are issued
  // The receive kernel queued behind this one may become resident now: it polls its flags.  Not before the
  // barrier: one thread's trigger counts for its CTA, and a receiver whose payloads are all there already
  // may write the vector that the CTA's other warps still read.
  cx::pdl_trigger();
  if (tid == 0) {
    uint32_t found = 0, mark = 0;
    for (int w = 0; w < nw; ++w) { found += s_found[w]; mark |= s_mark[w]; }
    const unsigned long long mine = (unsigned long long)found | 1ull << kArrived |
                                    (mark & 1u ? 1ull << kOver : 0ull) | (mark & 2u ? 1ull << kFailed : 0ull);
    s_all = cx::arrive_u64(reinterpret_cast<unsigned long long*>(&p.ctr->done), mine) + mine;   // as in cx::cta_arrive
    s_nnz = 0;
  }
  __syncthreads();
  CX_TRACE(3);
  const unsigned long long all = s_all;
  if (((all >> kArrived) & (uint32_t)kMaxGrid) != gridDim.x) return;
  const uint32_t found = (uint32_t)(all & ((1ull << kArrived) - 1));   // survivors
  const bool over = ((all >> kOver) & ((1u << (kFailed - kOver)) - 1)) != 0, any_failed = (all >> kFailed) != 0;
  uint32_t nnz = found;                   // pairs stored
  if (over) {
    if ((uint32_t)tid < p.nregions)
      atomicAdd(&s_nnz, min(*reinterpret_cast<volatile uint32_t*>(&p.ctr->region[tid][0]), p.region_size));
    __syncthreads();
    nnz = s_nnz;
  }
  CX_TRACE(4);
  if (tid < p.tg.count && !any_failed) {
    CxHeader* h = p.tg.ep[tid].hdr;
    h->bytes = 8ull + 8ull * nnz;
    h->n = (uint32_t)p.n;
    h->nnz = nnz;
    h->nnz_found = found;
    h->kind = CX_KIND_PAIRS;
    h->threshold = thr;
    h->nsub = p.nsub;
    h->src_rank = p.src_rank;
    h->dtype = CX_F32;
    cx::st_release_sys(&h->seq, cx::seq_of(p.seq_cell, p.seq));
  }
  CX_TRACE(5);
  if ((uint32_t)tid < p.nregions) p.ctr->region[tid][0] = 0;
  if (tid == 0) {
    if (p.stats) {
      p.stats->n = (uint32_t)p.n;
      p.stats->nnz = nnz;
      p.stats->nnz_found = found;
      p.stats->status = (found > nnz ? CX_ST_OVERFLOW : 0u) | (any_failed ? CX_ST_TIMEOUT : 0u);
      p.stats->threshold = thr;
    }
    *reinterpret_cast<unsigned long long*>(&p.ctr->done) = 0;
  }
  CX_TRACE(6);
}

// A sub-tile's g and r into L2, a 128-byte line per lane.
template <typename T, bool HAS_G, bool HAS_R>
__device__ __forceinline__ void pull_subtile(const T* __restrict__ g, const float* __restrict__ r, const uint32_t sub, const int lane) {
  const int64_t e0 = (int64_t)sub * CX_SUBTILE;
  if (HAS_R) asm volatile("prefetch.global.L2 [%0];" ::"l"(r + e0 + lane * 32));
  if (HAS_G && lane * (128 / (int)sizeof(T)) < CX_SUBTILE) asm volatile("prefetch.global.L2 [%0];" ::"l"(g + e0 + lane * (128 / (int)sizeof(T))));
}

// T: element type of g.  HAS_G / HAS_R select compress_add_update (both),
// compress_update (r only) and compress (g only).  MC: table and pairs go out once through
// the multicast endpoint tg.ep[tg.count] (multimem.st) instead of once per target; headers and
// notifications are still written target by target.
template <typename T, bool HAS_G, bool HAS_R, bool MC, bool LONG = false>
__global__ void __launch_bounds__(kThreads, kPerSm)
compress_kernel(const __grid_constant__ CompressParams p) {
  __shared__ __align__(16) Stage s_stage[kWarps];

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const T* __restrict__ g = reinterpret_cast<const T*>(p.g);
  float* __restrict__ r = p.r;
  CX_TRACE(0);
  const uint32_t nfull = p.vec ? (uint32_t)(p.n / CX_SUBTILE) : 0u;  // sub-tiles on the fast path
  // Launched with programmatic stream serialization, this grid may be resident while the kernel in
  // front of it still runs.  Behind the threshold estimate, which only reads, the warp's first
  // sub-tile can be loaded right away (1 us off a small exchange); otherwise pull it towards L2, then
  // wait for that kernel to finish before reading its result or touching the residual.
  float v[kChunks][4];
  bool loaded = false;
  {
    const uint32_t sub0 = blockIdx.x * kWarps + warp;
    if (p.early && sub0 < nfull) {
      load_subtile<T, HAS_G, HAS_R>(g + (int64_t)sub0 * CX_SUBTILE, r + (int64_t)sub0 * CX_SUBTILE, lane, v);
      loaded = true;
      // and the second one is on its way to L2 while the threshold is made (25.6 M bf16 elements, whose sample
      // takes 6 us: 56.4 -> 55.2 us; a third one as well: 55.2, and 8 x 6.5 M elements 249 -> 253)
      const uint64_t next = (uint64_t)sub0 + gridDim.x * kWarps;
      if (next < nfull) pull_subtile<T, HAS_G, HAS_R>(g, r, (uint32_t)next, lane);
    } else if (sub0 < p.nsub && lane < 2 * kChunks) {
      const int c = lane >> 1;
      const int64_t e0 = (int64_t)sub0 * CX_SUBTILE + c * 128;
      if (e0 < p.n) {
        const void* a = (lane & 1) ? (HAS_R ? (const void*)(r + e0) : nullptr) : (HAS_G ? (const void*)(g + e0) : nullptr);
        if (a) asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
      }
    }
  }
  cx::pdl_wait();
  const float thr = *p.thr;
  Tally tally = {0, false};
  CX_TRACE(1);
  Stage& stage = s_stage[warp];
  const uint32_t nwarps = gridDim.x * kWarps;

  for (uint32_t sub = blockIdx.x * kWarps + warp; sub < p.nsub; sub += nwarps) {
    if (sub < nfull) {
      const int64_t off = (int64_t)sub * CX_SUBTILE;
      if (!loaded) load_subtile<T, HAS_G, HAS_R>(g + off, r + off, lane, v);
      loaded = false;
      emit_subtile<HAS_G, HAS_R, MC, LONG>(p, sub, lane, thr, r + off, stage.v, stage.at, v, tally);
    }
    else compress_subtile_edge<T, HAS_G, HAS_R, MC>(p, sub, lane, KnownThreshold{thr}, g, r, tally);
  }

#ifdef CX_COMPRESS_TRACE
  __syncthreads();   // the stamp marks the CTA's last warp leaving the loop
#endif
  CX_TRACE(2);
  compress_finish<kWarps>(p, tid, thr, false, tally);
}

// The same for a vector that is folded from gradient tensors on the way (CxFold): what the fold
// kernel would write and this one read again, 8 bytes per element, stays in registers.  Sub-tiles
// that one tensor covers take the register path, the ones at tensor borders the edge path.
// 13.1 M bf16 gradients with momentum: 44 us for the fold and 34 us for the compression as two
// kernels.
template <typename T, bool MC, Input IN, int THREADS>
__global__ void __launch_bounds__(THREADS, kWarpsPerSm * 32 / THREADS)
compress_fold_kernel(const __grid_constant__ FoldCompressParams q) {
  constexpr int WARPS = THREADS / 32;
  __shared__ __align__(16) Stage s_stage[WARPS];
  const CompressParams& p = q.c;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float* __restrict__ r = p.r;
  LateThreshold late = {p.thr, q.chain, false, 0.f};
  // In the small CTAs of a short vector, whose first sub-tiles are all there are, the loads go ahead of the wait
  // for the threshold: descriptors, gradients and residual were complete before that kernel began (LeNet-5 step
  // 20.2 -> 18.7 us).  Longer vectors gain nothing by it.
  if (THREADS != kThreads || !p.early) late.get();
  Tally tally = {0, false};
  if (blockIdx.x < q.nborder_ctas) {
    for (uint32_t b = warp * q.nborder_ctas + blockIdx.x; b < (uint32_t)q.f.nborder; b += q.nborder_ctas * WARPS)
      compress_subtile_edge<T, true, true, MC, IN>(p, (uint32_t)(q.f.border[b] - q.f.base / CX_SUBTILE), lane, late, nullptr, r, tally, &q.f);
  } else {
    const uint32_t nwarps = (gridDim.x - q.nborder_ctas) * WARPS;
    uint32_t sub = (blockIdx.x - q.nborder_ctas) * WARPS + warp;
    cx::FoldWhole<T> cur = {nullptr, 0.f, 0};
    if (sub < p.nsub) cur = cx::fold_whole<T>(q.f, sub);
    while (sub < p.nsub) {
      const int64_t off = (int64_t)sub * CX_SUBTILE;
      const uint32_t next = sub + nwarps;
      cx::FoldWhole<T> ahead = {nullptr, 0.f, 0};
      if (cur.kind == 2) {
        float v[kChunks][4];
        load_fold_subtile<T, IN>(cur.g, r + off, IN == kFold ? nullptr : q.f.u + off, q.f.mu, cur.coef, q.f.keep ? cx::drop_policy() : cx::plain_policy(), lane, v, late);
        if (next < p.nsub) ahead = cx::fold_whole<T>(q.f, next);     // on its way while this one is stored
        emit_subtile<true, true, MC>(p, sub, lane, late.get(), r + off, s_stage[warp].v, s_stage[warp].at, v, tally);
      } else {
        if (next < p.nsub) ahead = cx::fold_whole<T>(q.f, next);
        if (cur.kind == 1) compress_subtile_edge<T, true, true, MC, IN>(p, sub, lane, late, nullptr, r, tally, &q.f);
      }
      cur = ahead;
      sub = next;
    }
  }
  compress_finish<WARPS>(p, tid, late.get(), false, tally);
  if (q.chain & CX_CHAINED) cx::pdl_wait();
}

// ---- the same sub-tile routine fed by the SM's copy engine ------------------------------------
// In compress_kernel a warp has loads in flight only between issuing them and using them; while it
// ranks, reserves and stores, nothing of its next sub-tile is on its way.  Here lane 0 of every
// warp asks the copy engine for the warp's next sub-tiles of r and g (cp.async.bulk into the
// warp's own stages in shared memory, completion counted in bytes on an mbarrier per stage)
// before the warp starts on the current one, so STAGES - 1 sub-tiles per warp are in flight all
// the time without holding a register.  One CTA per SM; the number of warps follows from the
// shared memory a warp needs.  Needs r and g 16-byte aligned; the last, partial sub-tile takes
// the edge path.  Every wait on an mbarrier is bounded; a warp whose copy does not arrive marks
// the call as failed, waits (bounded) for its other copies and joins the completion protocol,
// which then publishes nothing.
#ifndef CX_COMPRESS_BULK_STAGES
#define CX_COMPRESS_BULK_STAGES 2
#endif
constexpr int kBulkMaxWarps = 16;
// bytes per warp beside the stages: the list of survivors, and the sums where no stage holds 32-bit values
template <typename T, bool HAS_R>
__host__ __device__ constexpr uint32_t bulk_extra() { return 2 * kList + (HAS_R || sizeof(T) == 4 ? 0 : 4 * CX_SUBTILE); }

template <typename T, bool HAS_G, bool HAS_R, bool MC, int STAGES>
__global__ void __launch_bounds__(kBulkMaxWarps * 32, 1)
compress_bulk_kernel(const __grid_constant__ CompressParams p) {
  extern __shared__ __align__(128) unsigned char s_dyn[];
  constexpr uint32_t kRB = HAS_R ? (uint32_t)(CX_SUBTILE * sizeof(float)) : 0u;
  constexpr uint32_t kGB = HAS_G ? (uint32_t)(CX_SUBTILE * sizeof(T)) : 0u;
  constexpr uint32_t kStageB = kRB + kGB;
  constexpr uint32_t kWarpB = STAGES * kStageB + bulk_extra<T, HAS_R>();

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const uint32_t nw = blockDim.x >> 5;
  unsigned char* mine = s_dyn + (size_t)warp * kWarpB;
  uint16_t* list = reinterpret_cast<uint16_t*>(mine + STAGES * kStageB);
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_dyn + (size_t)nw * kWarpB) + warp * STAGES;
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < STAGES; ++s) cx::mbar_init(&bars[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncwarp();
  // everything in front of this kernel on the stream is complete and visible after this
  cx::pdl_wait();
  const float thr = *p.thr;
  const T* __restrict__ g = reinterpret_cast<const T*>(p.g);
  float* __restrict__ r = p.r;
  const uint32_t nwarps = gridDim.x * nw;
  const uint32_t nfull = (uint32_t)(p.n / CX_SUBTILE);
  const uint32_t first = blockIdx.x * nw + warp;
  uint32_t issued = 0, consumed = 0;
  bool failed = false;
  Tally tally = {0, false};

  auto issue = [&](uint32_t sub) {   // warp-uniform call; lane 0 talks to the copy engine
    if (lane == 0) {
      unsigned char* dst = mine + (issued % STAGES) * kStageB;
      uint64_t* bar = &bars[issued % STAGES];
      const size_t off = (size_t)sub * CX_SUBTILE;
      cx::mbar_expect_tx(bar, kStageB);
      if (HAS_R) cx::bulk_load(dst, r + off, kRB, bar);
      if (HAS_G) cx::bulk_load(dst + kRB, g + off, kGB, bar);
    }
    ++issued;
  };

#pragma unroll
  for (int t = 0; t < STAGES - 1; ++t) {
    const uint64_t sub = (uint64_t)first + (uint64_t)t * nwarps;
    if (sub < nfull) issue((uint32_t)sub);
  }
  for (uint32_t sub = first; sub < p.nsub; sub += nwarps) {
    const uint64_t ahead = (uint64_t)sub + (uint64_t)(STAGES - 1) * nwarps;
    if (ahead < nfull) issue((uint32_t)ahead);
    if (sub < nfull) {
      const uint32_t s = consumed % STAGES;
      // completion seen by any lane is final: the phase cannot advance again before the next issue()
      if (!__any_sync(0xffffffffu, cx::mbar_wait_bounded(&bars[s], (consumed / STAGES) & 1u))) {
        for (uint32_t c = consumed + 1; c < issued; ++c)
          cx::mbar_wait_bounded(&bars[c % STAGES], (c / STAGES) & 1u);
        failed = true;
        break;
      }
      ++consumed;
      const unsigned char* src = mine + s * kStageB;
      float v[kChunks][4];
      load_subtile<T, HAS_G, HAS_R>(reinterpret_cast<const T*>(src + kRB), reinterpret_cast<const float*>(src), lane, v);
      // the sums go where the copy engine put the residual (or fp32 gradient), each lane's over its own
      float* sums = reinterpret_cast<float*>(HAS_R || sizeof(T) == 4 ? mine + s * kStageB : mine + STAGES * kStageB + 2 * kList);
      emit_subtile<HAS_G, HAS_R, MC>(p, sub, lane, thr, r + (size_t)sub * CX_SUBTILE, sums, list, v, tally);
      // this stage is handed back to the copy engine by a later issue()
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
    } else {
      compress_subtile_edge<T, HAS_G, HAS_R, MC>(p, sub, lane, KnownThreshold{thr}, g, r, tally);
    }
  }
  compress_finish<kBulkMaxWarps>(p, tid, thr, failed, tally);
}

// n == 0: nothing to scan, only the (empty) header and the notification.
__global__ void compress_empty_kernel(const CompressParams p) {
  const int tid = threadIdx.x;
  if (tid < p.tg.count) {
    CxHeader* h = p.tg.ep[tid].hdr;
    h->bytes = 8; h->n = 0; h->nnz = 0; h->nnz_found = 0; h->kind = CX_KIND_PAIRS;
    h->threshold = *p.thr; h->nsub = 0; h->src_rank = p.src_rank; h->dtype = CX_F32;
    __threadfence_system();
    cx::st_release_sys(&h->seq, cx::seq_of(p.seq_cell, p.seq));
  }
  if (tid == 0 && p.stats) {
    p.stats->n = 0; p.stats->nnz = 0; p.stats->nnz_found = 0; p.stats->status = 0;
    p.stats->threshold = *p.thr;
  }
}

template <typename K>
void launch_pdl(K kernel, const CompressParams& p, int grid, cudaStream_t s) {
  cx_launch_pdl(kernel, grid, kThreads, 0, s, p, p.seq_cell != nullptr);
}

// from so many sub-tiles per warp on LONG is the faster one (between 12 and 20)
constexpr uint32_t kLongRounds = 16;

template <typename T, bool MC>
void launch_mode_mc(const CompressParams& p, int grid, cudaStream_t s) {
  if (p.g && p.r && sizeof(T) == 4 && p.nsub > kLongRounds * kWarps * (uint32_t)grid)
    launch_pdl(compress_kernel<T, true, true, MC, sizeof(T) == 4>, p, grid, s);
  else if (p.g && p.r) launch_pdl(compress_kernel<T, true, true, MC>, p, grid, s);
  else if (p.r) launch_pdl(compress_kernel<T, false, true, MC>, p, grid, s);
  else launch_pdl(compress_kernel<T, true, false, MC>, p, grid, s);
}

template <typename T>
void launch_mode(const CompressParams& p, int grid, cudaStream_t s) {
  if (p.tg.pad & CX_TG_MULTICAST) launch_mode_mc<T, true>(p, grid, s);
  else launch_mode_mc<T, false>(p, grid, s);
}

// COMPREX_COMPRESS_BULK=1 (read per call): the copy-engine variant where the alignment allows it.
// Measured equal to or up to 5 % slower than compress_kernel at every size from 2^22 to 2^28
// elements with 2, 3 and 4 stages (the kernel is not bound by its loads in flight), hence opt-in.
bool bulk_wanted() {
  const char* e = getenv("COMPREX_COMPRESS_BULK");
  return e ? atoi(e) != 0 : (CX_COMPRESS_BULK_DEFAULT != 0);
}

template <typename T, bool HAS_G, bool HAS_R, bool MC>
int launch_bulk_one(const CompressParams& p, cudaStream_t s) {
  constexpr int STAGES = CX_COMPRESS_BULK_STAGES;
  constexpr size_t kStageB = (HAS_R ? CX_SUBTILE * sizeof(float) : 0) + (HAS_G ? CX_SUBTILE * sizeof(T) : 0);
  constexpr size_t kWarpB = STAGES * kStageB + bulk_extra<T, HAS_R>() + 8 * STAGES;
  constexpr size_t kBudget = 227 * 1024 - 1024;   // per SM, minus the static part and slack
  int nw = (int)(kBudget / kWarpB);
  if (nw > kBulkMaxWarps) nw = kBulkMaxWarps;
#ifdef CX_COMPRESS_BULK_WARPS
  if (nw > CX_COMPRESS_BULK_WARPS) nw = CX_COMPRESS_BULK_WARPS;
#endif
  if (nw >= 8) nw &= ~3;                          // the same number of warps on every scheduler
  const size_t smem = (size_t)nw * kWarpB;
  auto kern = compress_bulk_kernel<T, HAS_G, HAS_R, MC, STAGES>;
  static bool configured[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cx_set_error("cx_compress: cudaGetDevice", 0);
  if (!configured[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cx_set_error("cx_compress: shared memory opt-in", (int)e);
    configured[dev] = true;
  }
  int grid = cx_sm_count();
  if (grid > kMaxBulkGrid) grid = kMaxBulkGrid;
  const int need = (int)((p.nsub + nw - 1) / nw);
  if (grid > need) grid = need;
  cx_launch_pdl(kern, grid, nw * 32, smem, s, p, p.seq_cell != nullptr);
  return 0;
}

template <typename T, bool MC>
int launch_bulk_mc(const CompressParams& p, cudaStream_t s) {
  if (p.g && p.r) return launch_bulk_one<T, true, true, MC>(p, s);
  if (p.r) return launch_bulk_one<T, false, true, MC>(p, s);
  return launch_bulk_one<T, true, false, MC>(p, s);
}

template <typename T>
int launch_bulk(const CompressParams& p, cudaStream_t s) {
  if (p.tg.pad & CX_TG_MULTICAST) return launch_bulk_mc<T, true>(p, s);
  return launch_bulk_mc<T, false>(p, s);
}

}  // namespace

#ifdef CX_COMPRESS_TRACE
extern "C" int cx_compress_trace(unsigned long long* host, int n) {
  if (n > 8 * 2048) n = 8 * 2048;
  return (int)cudaMemcpyFromSymbol(host, g_cx_trace, sizeof(unsigned long long) * n);
}
#endif

// The only scratch a compressor needs: one zero-initialised CxWorkCounters block.
extern "C" int64_t cx_workspace_bytes(int64_t n) {
  (void)n;
  return (int64_t)sizeof(CxWorkCounters);
}

namespace {

void fill_params(CompressParams& p, const void* g, float* r, int64_t n, const float* thr, uint32_t cap, uint64_t seq,
                 const CxTargets* tg, void* workspace, CxStats* stats, uint32_t src_rank) {
  p.g = g; p.r = r; p.n = n; p.thr = thr; p.cap = cap;
  p.nsub = (uint32_t)((n + CX_SUBTILE - 1) / CX_SUBTILE);
  // at least 8 sub-tiles and 256 pairs per region, so that regions fill evenly
  p.nregions = 1;
  while (p.nregions < CX_MAX_REGIONS && p.nsub / (2 * p.nregions) >= 8 && cap / (2 * p.nregions) >= 256)
    p.nregions *= 2;
  p.region_size = cap / p.nregions;
  p.seq = seq;
  p.seq_cell = cx_seq_cell();
  p.early = (cx_chain_bits() & CX_BEHIND_THRESHOLD) ? 1u : 0u;
  p.ctr = reinterpret_cast<CxWorkCounters*>(workspace);
  p.stats = stats; p.src_rank = src_rank;
  p.tg = *tg;
}

// one wave of CTAs, no more than the completion counter's fields hold
int wave(int per_sm) {
  const int grid = cx_sm_count() * per_sm;
  return grid < kMaxGrid ? grid : kMaxGrid;
}

int grid_for(const CompressParams& p) {
  const int grid = wave(kPerSm);
  const int need = (int)((p.nsub + kWarps - 1) / kWarps);
  return grid < need ? grid : need;
}

template <typename T, Input IN, int THREADS>
void launch_fold_threads(const FoldCompressParams& q, cudaStream_t s) {
  FoldCompressParams p = q;
  int grid;
  p.nborder_ctas = (uint32_t)cx_border_ctas(q.f, q.c.nsub, THREADS / 32, wave(kWarpsPerSm * 32 / THREADS), &grid);
  const bool capturing = q.c.seq_cell != nullptr;
  if (q.c.tg.pad & CX_TG_MULTICAST) cx_launch_pdl(compress_fold_kernel<T, true, IN, THREADS>, grid, THREADS, 0, s, p, capturing);
  else cx_launch_pdl(compress_fold_kernel<T, false, IN, THREADS>, grid, THREADS, 0, s, p, capturing);
}

// Small CTAs for a vector of at most eight sub-tiles per SM (LeNet step 22.1 -> 21.8 us; 1.0 M parameters, us per step
// with 64 / 128 threads: 22.6 / 24.2 fp32, 22.4 / 24.0 bf16).  Then 256 threads, but 128 for gradients that are folded
// into a momentum if they are fp32 or the vector is long; us per step with 128 / 256, 25 MB buckets:
//   bf16, AdamW:     GPT-2 of 30 / 36 / 61 / 124 M parameters 210.0 / 206.0, 250.7 / 242.8, 410 / 399, 803 / 786
//   bf16, momentum:  ResNet of 3.0 / 4.5 / 6.9 M parameters 30.4 / 29.1, 35.9 / 35.3, 41.7 / 41.4,
//                    9.4 / 16 / 25.6 M 47.4 / 47.5, 76.7 / 77.4, 116.5 / 117.2
//   fp32, momentum:  ResNet of 10 / 16 / 25.6 / 27.9 M parameters 68.2 / 69.0, 91.0 / 92.1, 133.3 / 135.2, 142.4 / 144.6,
//                    but 6.9 M, whose second bucket is small, 57.2 / 55.3
constexpr uint32_t kLongFold = 8192;       // sub-tiles
template <typename T, Input IN>
void launch_fold(const FoldCompressParams& q, cudaStream_t s) {
  if (q.c.nsub <= (uint32_t)cx_sm_count() * 8) launch_fold_threads<T, IN, kThreads>(q, s);
  else if (IN == kFoldMom && (sizeof(T) == 4 || q.c.nsub > kLongFold)) launch_fold_threads<T, IN, IN == kFoldMom ? 128 : 256>(q, s);
  else launch_fold_threads<T, IN, IN == kFoldMom && sizeof(T) == 4 ? 128 : 256>(q, s);
}

template <typename T>
void launch_fold_input(const FoldCompressParams& q, cudaStream_t s) {
  if (!q.f.u) launch_fold<T, kFold>(q, s);
  else if (q.f.mu == 0.f) launch_fold<T, kFoldWrite>(q, s);
  else launch_fold<T, kFoldMom>(q, s);
}

}  // namespace

int cx_compress_fold_cuda(int gdtype, const CxFold* fold, float* r, int64_t n, const float* thr, uint32_t cap,
                          uint64_t seq, const CxTargets* tg, void* workspace, int64_t ws_bytes, CxStats* stats,
                          uint32_t src_rank, void* stream) {
  if (!r) return cx_set_error("cx_compress: a folded vector needs a residual", 0);
  if (n <= 0 || n > 0x7fffffffLL) return cx_set_error("cx_compress: n out of range", 0);
  if (tg->count < 0 || tg->count > CX_MAX_PEERS) return cx_set_error("cx_compress: bad target count", 0);
  if ((tg->pad & CX_TG_MULTICAST) && tg->count >= CX_MAX_PEERS)
    return cx_set_error("cx_compress: no room for the multicast endpoint", 0);
  if (ws_bytes < cx_workspace_bytes(n)) return cx_set_error("cx_compress: workspace too small", 0);
  if (!fold->u && fold->mu != 0.f) return cx_set_error("cx_compress: folding with momentum needs the momentum", 0);
  if ((reinterpret_cast<uintptr_t>(r) | reinterpret_cast<uintptr_t>(fold->u)) & 15)
    return cx_set_error("cx_compress: a folded vector needs 16-byte aligned state", 0);
  FoldCompressParams q;
  fill_params(q.c, nullptr, r, n, thr, cap, seq, tg, workspace, stats, src_rank);
  q.f = *fold;
  q.chain = q.c.seq_cell ? 0u : cx_chain_bits();
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  switch (gdtype) {
    case CX_F32: launch_fold_input<float>(q, s); break;
    case CX_BF16: launch_fold_input<__nv_bfloat16>(q, s); break;
    case CX_F16: launch_fold_input<__half>(q, s); break;
    default: return cx_set_error("cx_compress: unsupported dtype on CUDA", 0);
  }
  cx_note_sender(stream);
  cx_note_launch();
  return cx_check_launch("compress_fold_kernel");
}

int cx_compress_cuda(int gdtype, const void* g, float* r, int64_t n, const float* thr,
                     uint32_t cap, uint64_t seq, const CxTargets* tg, void* workspace,
                     int64_t ws_bytes, CxStats* stats, uint32_t src_rank, void* stream) {
  if (!g && !r) return cx_set_error("cx_compress: g and r are both NULL", 0);
  if (n < 0 || n > 0x7fffffffLL) return cx_set_error("cx_compress: n out of range", 0);
  if (tg->count < 0 || tg->count > CX_MAX_PEERS) return cx_set_error("cx_compress: bad target count", 0);
  if ((tg->pad & CX_TG_MULTICAST) && tg->count >= CX_MAX_PEERS)
    return cx_set_error("cx_compress: no room for the multicast endpoint", 0);
  if (ws_bytes < cx_workspace_bytes(n)) return cx_set_error("cx_compress: workspace too small", 0);
  CompressParams p;
  fill_params(p, g, r, n, thr, cap, seq, tg, workspace, stats, src_rank);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (n == 0) {
    compress_empty_kernel<<<1, 32, 0, s>>>(p);
    cx_note_sender(stream);
    cx_note_launch();
    return cx_check_launch("compress_empty_kernel");
  }
  const size_t esz = gdtype == CX_F32 ? 4 : 2;
  p.vec = (!r || (reinterpret_cast<uintptr_t>(r) & 15) == 0) &&
          (!g || (reinterpret_cast<uintptr_t>(g) & (4 * esz - 1)) == 0);
  const bool aligned16 = (!r || (reinterpret_cast<uintptr_t>(r) & 15) == 0) &&
                         (!g || (reinterpret_cast<uintptr_t>(g) & 15) == 0);
  if (bulk_wanted() && aligned16 && n >= CX_SUBTILE) {
    int rc = 0;
    switch (gdtype) {
      case CX_F32: rc = launch_bulk<float>(p, s); break;
      case CX_BF16: rc = launch_bulk<__nv_bfloat16>(p, s); break;
      case CX_F16: rc = launch_bulk<__half>(p, s); break;
      default: return cx_set_error("cx_compress: unsupported dtype on CUDA", 0);
    }
    if (rc) return rc;
    cx_note_sender(stream);
    cx_note_launch();
    return cx_check_launch("compress_bulk_kernel");
  }
  const int grid = grid_for(p);
  switch (gdtype) {
    case CX_F32: launch_mode<float>(p, grid, s); break;
    case CX_BF16: launch_mode<__nv_bfloat16>(p, grid, s); break;
    case CX_F16: launch_mode<__half>(p, grid, s); break;
    default: return cx_set_error("cx_compress: unsupported dtype on CUDA", 0);
  }
  cx_note_sender(stream);
  cx_note_launch();
  return cx_check_launch("compress_kernel");
}
