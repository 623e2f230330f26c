// Receive side: wait for the notifications, then decode the sparse payloads
// of all sources in a fixed source order, fused with averaging and the
// parameter update (reference: CompressorIndexPairs::decompress / add,
// src/compressor.hxx:613-658, called after TargetBuffer::waitForCompletion in
// src/comprEx.tpp:224-246; optimizer math keras/comprex_optimizer.py:150-163).
//
// Ownership instead of atomics: every payload carries, per 1024-element
// sub-tile of the vector, a table entry {start, count} that says where that
// sub-tile's pairs sit in the pair list.  A warp owns one sub-tile at a time,
// looks the ranges of all sources up directly and applies them source after
// source.  Indices are
// unique inside one payload and a sub-tile has a single owner, so no atomic
// is needed and the floating-point sum order is the same on every rank, which
// keeps data-parallel replicas bit-identical.
//
//  * sparse ops (ADD; SGD without weight decay) touch only the addressed
//    elements in global memory, source after source, each rounded on its own;
//  * dense ops (SET, SGD with decay, momentum, AdamW) accumulate the sub-tile
//    in shared memory and then walk it once with 16-byte accesses, so the
//    averaged gradient never exists in global memory.
//
// A wait that runs out of its time budget sets CX_ST_TIMEOUT in the status
// word and the kernel returns without touching the output.
#include <stdlib.h>

#include <type_traits>

#include "cx_fold.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

struct ApplyParams {
  CxSources src;
  CxApplyArgs a;
  int64_t n;
  uint32_t nsub;
  uint32_t vec;  // every dense pointer is 16-byte aligned
  uint32_t* status;
  uint64_t timeout_ns;
  const uint64_t* seq_cell;  // non-NULL inside a captured graph: the waits use its value
  uint32_t front_wait;       // CX_WAIT_*: the kernel in front may be at work on the same vectors
  uint32_t early;            // dense ops: let the kernel behind in at the start
  uint32_t group;            // sparse ops: sub-tiles a warp takes at a time
};

__device__ __forceinline__ CxPair ld_pair(const CxPair* p) {
  const uint2 t = __ldcg(reinterpret_cast<const uint2*>(p));
  CxPair r;
  r.idx = (int32_t)t.x;
  r.val = t.y;
  return r;
}

// At the start of a receive kernel: lets the kernel behind in (`early`) and waits for the one in front as far as
// that has to happen here.
__device__ __forceinline__ void begin_apply(const ApplyParams& p, bool early) {
  if (p.front_wait == CX_WAIT_CHAIN) cx::pdl_wait();
  if (early) cx::pdl_trigger();
  if (p.front_wait == CX_WAIT_START) cx::pdl_wait();
}

// Waits for all sources and validates their headers: the first warp does, lane j for source j.  (Every
// warp for itself would save the barrier, but 7000 warps polling one line cost 5 us.)  Returns false
// (uniformly for the CTA) when the kernel must not touch the output; no table is read before, a
// payload of another length may have a shorter one.  PAIRS: `pairs` is the number of all sources together.
template <bool PAIRS = false>
__device__ __forceinline__ bool wait_sources(const ApplyParams& p, uint64_t* pairs = nullptr) {
  __shared__ uint32_t s_ok;
  __shared__ uint32_t s_pairs[2];
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    uint32_t bad = 0, nnz = 0;
    if (lane < p.src.count) {
      const CxHeader* h = p.src.ep[lane].hdr;
      if (!cx::wait_seq(&h->seq, cx::seq_of(p.seq_cell, p.src.seq[lane]), p.timeout_ns)) {
        bad = CX_ST_TIMEOUT;
      } else {
        const uint32_t kind = *reinterpret_cast<const volatile uint32_t*>(&h->kind);
        const uint32_t hn = *reinterpret_cast<const volatile uint32_t*>(&h->n);
        if (kind != CX_KIND_PAIRS || hn != (uint32_t)p.n) bad = CX_ST_BAD_HEADER;
        if (PAIRS) nnz = *reinterpret_cast<const volatile uint32_t*>(&h->nnz);
      }
      if (bad && p.status) atomicOr(p.status, bad);
    }
    const bool any = __any_sync(0xffffffffu, bad != 0);
    if (PAIRS) {               // in halves: sixteen 32-bit counts
      const uint32_t high = __reduce_add_sync(0xffffffffu, nnz >> 16), low = __reduce_add_sync(0xffffffffu, nnz & 0xffffu);
      if (lane == 0) { s_pairs[0] = low; s_pairs[1] = high; }
    }
    if (lane == 0) s_ok = any ? 0u : 1u;
  }
  __syncthreads();
  if (PAIRS) *pairs = ((uint64_t)s_pairs[1] << 16) + s_pairs[0];
  return s_ok != 0;
}

__device__ __forceinline__ void segment_prefix(int lane, uint32_t a, uint32_t b, uint32_t& pre, uint32_t& total) {
  const uint32_t cnt = b - a;
  uint32_t incl = cnt;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += t;
  }
  pre = incl - cnt;
  total = __shfl_sync(0xffffffffu, incl, 31);
}

__device__ __forceinline__ void table_entry(const ApplyParams& p, uint32_t sub, int lane, uint32_t& a, uint32_t& b) {
  a = 0;
  b = 0;
  if (lane < p.src.count && sub < p.nsub) {
    const uint2 entry = __ldcg(reinterpret_cast<const uint2*>(p.src.ep[lane].table) + sub);
    a = entry.x;
    b = min(entry.x + min(entry.y, (uint32_t)CX_SUBTILE), p.src.cap[lane]);  // never beyond the slot
    a = min(a, b);
  }
}

// The sparse ops: pairs go straight into the vector, source after source.  A warp takes up to 32
// neighbouring sub-tiles at a time: lane l looks sub-tile l up, a scan lays the sub-tiles' pairs end
// to end, and the lanes walk that sequence, AHEAD x 32 pairs in flight.  So a warp is busy whatever
// the density (10 pairs per sub-tile and source at top-k 1 %), and the chain of dependent loads
// (table, pairs, elements) is paid once per group and source: 2^28 elements at 1 %, one source, took
// 165 us with one sub-tile per warp at a time.
// Large groups (many sub-tiles per warp, two rounds or more) take eight rows at a time: 2^28 elements at 1 %
// 653 -> 646 us; the registers that this costs leave fewer warps, 25 M elements at 0.1 % 57 -> 59 us with it.
constexpr int kAhead = 4, kAheadLarge = 8, kLargeGroup = 16;

// What several sources touch has to stay in L2 until the last of them has come to it, so a warp takes fewer
// sub-tiles at a time then: as many as keep the 64-byte pieces that all warps touch within half of L2 (126 MB).
// A vector whose touched pieces fit there anyway is not bound by that; where every source fills a row of
// 32 pairs in every sub-tile, one at a time is best.  2^28 elements, 7 sources, 1 / 2 / 4 / 8 / 19 sub-tiles:
// 0.1 % 344 / 211 / 129 / 98 / 98 us, 1 % 504 / 396 / 488 / 650 / 739, 10 % 1192 / 1479 / 2266 / 2667 / 2641.
// (One sub-tile at a time with all its sources in one round trip, as the batches below do: 166 / 438 / 1729.)
constexpr uint64_t kInL2 = 96ull << 20, kHalfL2 = 63ull << 20;
__device__ __forceinline__ uint32_t group_of_several(const ApplyParams& p, uint64_t pairs, int esize) {
  if (pairs >= (uint64_t)p.nsub * 32 * p.src.count) return 1;
  const uint64_t touched = min((uint64_t)CX_SUBTILE * esize * p.nsub, 64 * pairs);     // of the whole vector
  if (touched <= kInL2) return p.group;
  const uint64_t fit = kHalfL2 * p.nsub / touched / ((uint64_t)gridDim.x * kWarps);
  return max(1u, (uint32_t)min((uint64_t)p.group, fit));
}

template <typename TO, int AHEAD, bool SEVERAL>
__global__ void __launch_bounds__(kThreads) apply_sparse_kernel(const __grid_constant__ ApplyParams p) {
  begin_apply(p, true);
  const int lane = threadIdx.x & 31;
  uint64_t all = 0;
  if (!wait_sources<SEVERAL>(p, &all)) { cx::pdl_wait(); return; }
  const uint32_t group = SEVERAL ? group_of_several(p, all, p.a.op == CX_OP_SGD ? 4 : (int)sizeof(TO)) : p.group;
  const uint32_t nwarps = gridDim.x * kWarps;
  const bool sgd = p.a.op == CX_OP_SGD;
  const float scale = sgd ? -p.a.scale : p.a.scale;
  bool wait = p.front_wait == CX_WAIT_VECTORS;
  uint32_t bad = 0;
  for (uint64_t s0 = (uint64_t)(blockIdx.x * kWarps + (threadIdx.x >> 5)) * group; s0 < p.nsub;
       s0 += (uint64_t)nwarps * group) {
    const uint32_t sub = (uint32_t)s0 + lane;
    const bool have = lane < (int)group && sub < p.nsub;
    uint2 next = have && p.src.count ? __ldcg(reinterpret_cast<const uint2*>(p.src.ep[0].table) + sub) : make_uint2(0, 0);
    for (int j = 0; j < p.src.count; ++j) {
      const uint32_t cap = p.src.cap[j];
      const uint32_t b = min(next.x + min(next.y, (uint32_t)CX_SUBTILE), cap);     // never beyond the slot
      const uint32_t a = min(next.x, b);
      if (have && j + 1 < p.src.count) next = __ldcg(reinterpret_cast<const uint2*>(p.src.ep[j + 1].table) + sub);
      uint32_t pre, total;
      segment_prefix(lane, a, b, pre, total);
      const CxPair* pairs = p.src.ep[j].pairs;
      for (uint32_t f0 = 0; f0 < total; f0 += 32 * AHEAD) {
        CxPair pr[AHEAD];
        uint32_t lo[AHEAD];
        bool in[AHEAD];
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
          const uint32_t f = f0 + 32 * k + lane;
          in[k] = f < total;
          lo[k] = 0;
          pr[k].idx = 0;
          pr[k].val = 0;
          if (f0 + 32 * k >= total) continue;      // warp-uniform
          uint32_t o = 0;          // the last sub-tile whose pairs start at or before f
#pragma unroll
          for (uint32_t d = 16; d > 0; d >>= 1) {
            const uint32_t t = __shfl_sync(0xffffffffu, pre, o + d);
            if (t <= f) o += d;
          }
          const uint32_t off = __shfl_sync(0xffffffffu, a, o) + (f - __shfl_sync(0xffffffffu, pre, o));
          lo[k] = ((uint32_t)s0 + o) * CX_SUBTILE;
          if (in[k]) pr[k] = ld_pair(pairs + off);
        }
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
          if (in[k] && !((uint32_t)pr[k].idx - lo[k] < CX_SUBTILE && (int64_t)pr[k].idx < p.n)) { in[k] = false; bad = CX_ST_BAD_INDEX; }
        }
        if (wait) { cx::pdl_wait(); wait = false; }
        // indices are unique inside one payload: the loads may all go first
        float cur[AHEAD];
        if (sgd) {
          float* w = reinterpret_cast<float*>(p.a.out);
#pragma unroll
          for (int k = 0; k < AHEAD; ++k) cur[k] = in[k] ? w[pr[k].idx] : 0.f;
#pragma unroll
          for (int k = 0; k < AHEAD; ++k) {
            const float nw = cur[k] + scale * __uint_as_float(pr[k].val);
            if (in[k]) w[pr[k].idx] = nw;
            if (in[k] && p.a.shadow) reinterpret_cast<TO*>(p.a.shadow)[pr[k].idx] = cx::Elem<TO>::from_f(nw);
          }
        } else {
          TO* out = reinterpret_cast<TO*>(p.a.out);
#pragma unroll
          for (int k = 0; k < AHEAD; ++k) cur[k] = in[k] ? cx::Elem<TO>::to_f(out[pr[k].idx]) : 0.f;
#pragma unroll
          for (int k = 0; k < AHEAD; ++k)
            if (in[k]) out[pr[k].idx] = cx::Elem<TO>::from_f(cur[k] + scale * __uint_as_float(pr[k].val));
        }
      }
      __syncwarp();  // the next source may address the same elements from other lanes
    }
  }
  if (bad && p.status) atomicOr(p.status, bad);
  cx::pdl_wait();   // launched early behind its sender: do not complete before that grid has
}

// Several sources and few sub-tiles per warp: one chain of dependent loads per source would be most of the
// kernel's time, so the pairs of all sources of a sub-tile are laid end to end and 128 of them at a time are
// fetched in one round trip, the elements they address in a second one.  The additions go source after
// source in shared memory: pairs that address the same element share the slot of one of them.
// ADD, fp32, 7 sources, a group of sub-tiles source after source against this: 2^20 elements at 0.1 / 1 / 10 %
// 16.4 / 18.4 / 21.5 -> 10.3 / 11.3 / 20.5 us, 2^22 18.4 / 20.5 / 27.5 -> 12.3 / 14.5 / 28.7.
constexpr int kBatch = 4;                     // pairs per lane
constexpr uint32_t kBatchPairs = 32 * kBatch;
// Up to one sub-tile per warp (7.2 M elements), and up to two with more than four sources: 12 M elements, 0.1 / 1 %,
// 2 sources 14.3 / 16.4 us in batches and 12.3 / 16.4 in groups, 7 sources 18.5 / 24.6 and 18.5 / 28.7.
inline bool in_batches(uint32_t group, int sources) { return sources > 1 && group <= (sources > 4 ? 2u : 1u); }

template <typename TO>
__global__ void __launch_bounds__(kThreads, 6) apply_sparse_batch_kernel(const __grid_constant__ ApplyParams p) {
  __shared__ uint8_t s_slot[kWarps][CX_SUBTILE];
  __shared__ float s_acc[kWarps][kBatchPairs];
  begin_apply(p, true);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (!wait_sources(p)) { cx::pdl_wait(); return; }
  const uint32_t nwarps = gridDim.x * kWarps;
  const bool sgd = p.a.op == CX_OP_SGD;
  const float scale = sgd ? -p.a.scale : p.a.scale;
  uint8_t* slot = s_slot[warp];
  float* acc = s_acc[warp];
  bool wait = p.front_wait == CX_WAIT_VECTORS;
  uint32_t bad = 0;
  uint32_t sub = blockIdx.x * kWarps + warp, a, b;
  table_entry(p, sub, lane, a, b);
  for (; sub < p.nsub; sub += nwarps) {
    const uint32_t lo = sub * CX_SUBTILE;
    uint32_t na, nb, pre, total;              // the next sub-tile's table entries, in flight meanwhile
    const uint64_t next = (uint64_t)sub + nwarps;
    table_entry(p, next < p.nsub ? (uint32_t)next : p.nsub, lane, na, nb);
    segment_prefix(lane, a, b, pre, total);
    int j0 = 0, j1 = 0;                       // the batch's pairs are of the sources [j0, j1) (warp-uniform)
    for (uint32_t f0 = 0; f0 < total; f0 += kBatchPairs) {
      int src[kBatch];                        // source of the pair, -1: none
      uint32_t off[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; ++k) { src[k] = -1; off[k] = 0; }
      j0 = max(j1 - 1, 0);                    // the last source of the batch before may have more
      for (j1 = j0; j1 < p.src.count; ++j1) {
        const int j = j1;
        const uint32_t pj = __shfl_sync(0xffffffffu, pre, j), aj = __shfl_sync(0xffffffffu, a, j);
        const uint32_t cj = __shfl_sync(0xffffffffu, b, j) - aj;
        if (pj >= f0 + kBatchPairs) break;
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
          const uint32_t f = f0 + 32 * k + lane;
          if (f - pj < cj) { src[k] = j; off[k] = aj + (f - pj); }
        }
      }
      CxPair pr[kBatch];
      uint32_t d[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        pr[k].idx = 0;
        pr[k].val = 0;
        if (src[k] >= 0) pr[k] = ld_pair(p.src.ep[src[k]].pairs + off[k]);
      }
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        d[k] = (uint32_t)pr[k].idx - lo;
        if (src[k] >= 0 && !(d[k] < CX_SUBTILE && (int64_t)pr[k].idx < p.n)) { bad = CX_ST_BAD_INDEX; src[k] = -1; }
        if (src[k] >= 0) slot[d[k]] = (uint8_t)(32 * k + lane);
      }
      if (wait) { cx::pdl_wait(); wait = false; }
      float cur[kBatch];
      if (sgd) {
        const float* w = reinterpret_cast<const float*>(p.a.out);
#pragma unroll
        for (int k = 0; k < kBatch; ++k) cur[k] = src[k] >= 0 ? w[pr[k].idx] : 0.f;
      } else {
        const TO* out = reinterpret_cast<const TO*>(p.a.out);
#pragma unroll
        for (int k = 0; k < kBatch; ++k) cur[k] = src[k] >= 0 ? cx::Elem<TO>::to_f(out[pr[k].idx]) : 0.f;
      }
      __syncwarp();
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        if (src[k] < 0) continue;
        d[k] = slot[d[k]];
        acc[d[k]] = cur[k];                   // the same value from every pair of the element
      }
      __syncwarp();
      for (int j = j0; j < j1; ++j) {         // rounded like the element-by-element path
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
          if (src[k] == j) {
            const float nv = acc[d[k]] + scale * __uint_as_float(pr[k].val);
            acc[d[k]] = sgd ? nv : cx::Elem<TO>::to_f(cx::Elem<TO>::from_f(nv));
          }
        }
        __syncwarp();
      }
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        if (src[k] < 0) continue;
        const float nv = acc[d[k]];
        if (sgd) {
          reinterpret_cast<float*>(p.a.out)[pr[k].idx] = nv;
          if (p.a.shadow) reinterpret_cast<TO*>(p.a.shadow)[pr[k].idx] = cx::Elem<TO>::from_f(nv);
        } else {
          reinterpret_cast<TO*>(p.a.out)[pr[k].idx] = cx::Elem<TO>::from_f(nv);
        }
      }
      __syncwarp();                           // the next batch may address the same elements from other lanes
    }
    a = na;
    b = nb;
  }
  if (bad && p.status) atomicOr(p.status, bad);
  cx::pdl_wait();   // launched early behind its sender: do not complete before that grid has
}

// The update rule on four elements held in registers (g = scale * sum of the payloads).
template <int OP>
__device__ __forceinline__ void rule4(const CxApplyArgs& a, const float (&acc)[4], float (&wv)[4],
                                      float (&mv)[4], float (&vv)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float g = a.scale * acc[e];
    if (OP == CX_OP_SGD) {
      wv[e] = (1.f - a.wd) * wv[e] - g;
    } else if (OP == CX_OP_MOMENTUM) {
      mv[e] = a.momentum * mv[e] + a.lr * g;
      wv[e] = (1.f - a.wd) * wv[e] - mv[e];
    } else {  // AdamW
      // The moments use explicit fused multiply-adds (the host twin calls fmaf in the same
      // places, so m and v agree bit for bit).  The step itself takes the hardware's
      // approximate square root and reciprocal (about 1 ulp each, two instructions instead
      // of two correctly rounded software sequences of ~12 instructions): the kernel is
      // bound by instruction issue, not by memory, and a relative error of 2^-22 in a step
      // that is itself lr-sized is far below the rounding of w.  Every rank runs this same
      // kernel, so replicas stay bit-identical.
      mv[e] = __fmaf_rn(a.beta1, mv[e], (1.f - a.beta1) * g);
      vv[e] = __fmaf_rn(a.beta2, vv[e], ((1.f - a.beta2) * g) * g);
      const float mh = mv[e] * __frcp_rn(a.bc1);   // loop invariants
      const float vh = vv[e] * __frcp_rn(a.bc2);
      float root, inv;
      asm("sqrt.approx.f32 %0, %1;" : "=f"(root) : "f"(vh));
      asm("rcp.approx.f32 %0, %1;" : "=f"(inv) : "f"(root + a.eps));
      wv[e] = __fmaf_rn(-(a.lr * mh), inv, wv[e] * (1.f - a.lr * a.wd));
    }
  }
}

template <int OP, typename TO>
__device__ __forceinline__ void store_state4(const CxApplyArgs& a, int64_t i, const float (&wv)[4],
                                             const float (&mv)[4], const float (&vv)[4]) {
  cx::store4(reinterpret_cast<float*>(a.out) + i, wv);
  if (OP != CX_OP_SGD) cx::store4(a.m + i, mv);
  if (OP == CX_OP_ADAMW) cx::store4(a.v + i, vv);
  if (a.shadow) cx::store4(reinterpret_cast<TO*>(a.shadow) + i, wv);
}

template <int OP, typename TO>
__device__ __forceinline__ void update4(const CxApplyArgs& a, const int64_t n, int64_t i,
                                        const float (&acc)[4], bool vec) {
  if (OP == CX_OP_SET) {
    float o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) o[e] = a.scale * acc[e];
    TO* out = reinterpret_cast<TO*>(a.out);
    if (vec) cx::store4(out + i, o);
    else
      for (int e = 0; e < 4; ++e) if (i + e < n) out[i + e] = cx::Elem<TO>::from_f(o[e]);
    return;
  }
  float* w = reinterpret_cast<float*>(a.out);
  float wv[4], mv[4], vv[4];
  if (vec) {
    cx::load4(w + i, wv);
    if (OP != CX_OP_SGD) cx::load4(a.m + i, mv);
    if (OP == CX_OP_ADAMW) cx::load4(a.v + i, vv);
  } else {
    for (int e = 0; e < 4; ++e) {
      const bool in = i + e < n;
      wv[e] = in ? w[i + e] : 0.f;
      mv[e] = (in && OP != CX_OP_SGD) ? a.m[i + e] : 0.f;
      vv[e] = (in && OP == CX_OP_ADAMW) ? a.v[i + e] : 0.f;
    }
  }
  rule4<OP>(a, acc, wv, mv, vv);
  if (vec) {
    store_state4<OP, TO>(a, i, wv, mv, vv);
  } else {
    for (int e = 0; e < 4; ++e) {
      if (i + e >= n) continue;
      w[i + e] = wv[e];
      if (OP != CX_OP_SGD) a.m[i + e] = mv[e];
      if (OP == CX_OP_ADAMW) a.v[i + e] = vv[e];
      if (a.shadow) reinterpret_cast<TO*>(a.shadow)[i + e] = cx::Elem<TO>::from_f(wv[e]);
    }
  }
}

// the update rule on one element whose state has been loaded
template <int OP>
__device__ __forceinline__ void load_state1(const CxApplyArgs& a, int64_t i, bool in, float& w, float& m, float& v) {
  w = in ? reinterpret_cast<const float*>(a.out)[i] : 0.f;
  m = OP != CX_OP_SGD && in ? a.m[i] : 0.f;
  v = OP == CX_OP_ADAMW && in ? a.v[i] : 0.f;
}
template <int OP, typename TO>
__device__ __forceinline__ void update1(const CxApplyArgs& a, int64_t i, float acc, float w, float m, float v) {
  const float av[4] = {acc, 0.f, 0.f, 0.f};
  float wv[4] = {w, 0.f, 0.f, 0.f}, mv[4] = {m, 0.f, 0.f, 0.f}, vv[4] = {v, 0.f, 0.f, 0.f};
  rule4<OP>(a, av, wv, mv, vv);
  reinterpret_cast<float*>(a.out)[i] = wv[0];
  if (OP != CX_OP_SGD) a.m[i] = mv[0];
  if (OP == CX_OP_ADAMW) a.v[i] = vv[0];
  if (a.shadow) reinterpret_cast<TO*>(a.shadow)[i] = cx::Elem<TO>::from_f(wv[0]);
}

// Sum of all sources' pairs of one sub-tile in shared memory (acc, cleared here).  a, b: lane j holds
// source j's segment of its pair list.  Every source's segment is cut into rows of 32 pairs, and up to
// kRows rows are in flight at a time: one round trip for eight sources of up to 32 pairs each.  The rows are
// summed one after the other, so in source order, and no two lanes of a row meet in an element.  What
// bounds it is the number of instructions: with the segments laid end to end, every lane looking its pair's
// source up by shuffles, a decode of 8 x 65 536 pairs into 25 MB took 12 us at 0.8 of the issue rate while it
// summed; this way 10.4 (8 ranks' exchange 270 -> 259 us, 2^20 elements 17.3 -> 16.1).
// Returns CX_ST_BAD_INDEX or 0.
constexpr int kRows = 8;

__device__ __forceinline__ uint32_t accumulate_subtile(const ApplyParams& p, uint32_t sub, int lane, uint32_t a, uint32_t b,
                                                       float* acc) {
  const uint32_t lo = sub * CX_SUBTILE, span = (uint32_t)min((int64_t)CX_SUBTILE, p.n - lo);
  uint32_t bad = 0;
#pragma unroll
  for (int q = 0; q < CX_SUBTILE / 128; ++q)
    *reinterpret_cast<float4*>(acc + q * 128 + lane * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
  int src = 0;                                   // the next row: pairs [at, at + 32) of this source, up to `end`
  uint32_t at = __shfl_sync(0xffffffffu, a, 0), end = __shfl_sync(0xffffffffu, b, 0);
  while (src < p.src.count) {
    CxPair pr[kRows];
    uint32_t have = 0;                           // bit k: this lane holds a pair of row k
    int rows = 0;
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
      pr[k].idx = (int32_t)lo - 1;
      pr[k].val = 0;
      if (src < p.src.count) {                   // warp-uniform
        if (at + lane < end) {
          pr[k] = ld_pair(p.src.ep[src].pairs + at + lane);
          have |= 1u << k;
        }
        at += 32;
        if (at >= end) {
          ++src;
          at = __shfl_sync(0xffffffffu, a, src & 31);
          end = __shfl_sync(0xffffffffu, b, src & 31);
        }
        rows = k + 1;
      }
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
      if (k < rows) {                            // warp-uniform
        const uint32_t d = (uint32_t)pr[k].idx - lo;
        if (d < span) acc[d] += __uint_as_float(pr[k].val);
        else if (have >> k & 1u) bad = CX_ST_BAD_INDEX;
        __syncwarp();
      }
    }
  }
  return bad;
}

// Variant for the kernel below, which runs few warps per SM and therefore cannot hide one
// memory latency per source: the table entries arrive from the caller (fetched one
// iteration ahead) and the first pair of every source is loaded before any is used.  The
// sums are formed in the same source order as above.
__device__ __forceinline__ uint32_t accumulate_subtile_ahead(const ApplyParams& p, uint32_t sub, int lane,
                                                             uint32_t a, uint32_t b, float* acc) {
  const uint32_t lo = sub * CX_SUBTILE;
  uint32_t bad = 0, have = 0;
  CxPair head[CX_MAX_PEERS];
#pragma unroll
  for (int j = 0; j < CX_MAX_PEERS; ++j) {
    const uint32_t aj = __shfl_sync(0xffffffffu, a, j);
    const uint32_t bj = __shfl_sync(0xffffffffu, b, j);
    head[j].idx = 0;
    head[j].val = 0;
    if (j < p.src.count && aj + lane < bj) {
      head[j] = ld_pair(p.src.ep[j].pairs + aj + lane);
      have |= 1u << j;
    }
  }
#pragma unroll
  for (int q = 0; q < CX_SUBTILE / 128; ++q)
    *reinterpret_cast<float4*>(acc + q * 128 + lane * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncwarp();
#pragma unroll
  for (int j = 0; j < CX_MAX_PEERS; ++j) {
    if (j >= p.src.count) break;
    const uint32_t aj = __shfl_sync(0xffffffffu, a, j);
    const uint32_t bj = __shfl_sync(0xffffffffu, b, j);
    if (aj == bj) continue;            // warp-uniform
    if ((have >> j) & 1u) {
      const uint32_t d = (uint32_t)head[j].idx - lo;
      if (d < CX_SUBTILE && (int64_t)head[j].idx < p.n) acc[d] += __uint_as_float(head[j].val);
      else bad = CX_ST_BAD_INDEX;
    }
    const CxPair* pairs = p.src.ep[j].pairs;
    for (uint32_t i = aj + 32 + lane; i < bj; i += 32) {
      const CxPair pr = ld_pair(pairs + i);
      const uint32_t d = (uint32_t)pr.idx - lo;
      if (d < CX_SUBTILE && (int64_t)pr.idx < p.n) acc[d] += __uint_as_float(pr.val);
      else bad = CX_ST_BAD_INDEX;
    }
    __syncwarp();
  }
  return bad;
}

// ---- bulk-copy (TMA) pipeline for the optimizer state ---------------------------------------
// The dense update streams 12 bytes of state per element in and out (AdamW: w, m, v).  With
// plain vector loads the bytes in flight are bounded by registers.  Here lane 0 of every warp
// asks the copy engine of the SM for the warp's next sub-tile of w / m / v (cp.async.bulk into
// shared memory, completion counted in bytes on an mbarrier) before the warp starts on the
// sparse part of the sub-tile, so the state of up to STAGES sub-tiles per warp is in flight
// without holding a register.  Every wait on an mbarrier is bounded.

using cx::smem_u32;
using cx::mbar_init;
using cx::mbar_expect_tx;
using cx::bulk_load;
using cx::mbar_try_wait;
using cx::mbar_wait_bounded;

template <int OP>
struct StateArrays { static constexpr int n = OP == CX_OP_SGD ? 1 : (OP == CX_OP_MOMENTUM ? 2 : 3); };

constexpr int kBulkMaxThreads = 512;

template <int OP, typename TO, int STAGES>
__global__ void __launch_bounds__(kBulkMaxThreads, 1) apply_dense_bulk_kernel(const ApplyParams p) {
  extern __shared__ __align__(128) unsigned char s_dyn[];
  constexpr int NARR = StateArrays<OP>::n;
  constexpr uint32_t kTileBytes = CX_SUBTILE * sizeof(float);
  constexpr uint32_t kWarpBytes = (1 + STAGES * NARR) * kTileBytes;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  if (!wait_sources(p)) { cx::pdl_wait(); return; }
  const uint32_t nw = blockDim.x >> 5;
  float* acc = reinterpret_cast<float*>(s_dyn + warp * kWarpBytes);
  float* stage0 = acc + CX_SUBTILE;
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_dyn + nw * kWarpBytes) + warp * STAGES;
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < STAGES; ++s) mbar_init(&bars[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncwarp();
  const uint32_t nwarps = gridDim.x * nw;
  const uint32_t nfull = (uint32_t)(p.n / CX_SUBTILE);   // these sub-tiles are copied in bulk
  const uint32_t first = blockIdx.x * nw + warp;
  const float* wsrc = reinterpret_cast<const float*>(p.a.out);
  uint32_t issued = 0, consumed = 0, bad = 0;

  auto issue = [&](uint32_t sub) {   // warp-uniform call; lane 0 talks to the copy engine
    if (lane == 0) {
      const uint32_t s = issued % STAGES;
      float* dst = stage0 + s * NARR * CX_SUBTILE;
      const size_t off = (size_t)sub * CX_SUBTILE;
      mbar_expect_tx(&bars[s], NARR * kTileBytes);
      bulk_load(dst, wsrc + off, kTileBytes, &bars[s]);
      if (NARR > 1) bulk_load(dst + CX_SUBTILE, p.a.m + off, kTileBytes, &bars[s]);
      if (NARR > 2) bulk_load(dst + 2 * CX_SUBTILE, p.a.v + off, kTileBytes, &bars[s]);
    }
    ++issued;
  };

#pragma unroll
  for (int t = 0; t < STAGES - 1; ++t) {
    const uint64_t sub = (uint64_t)first + (uint64_t)t * nwarps;
    if (sub < nfull) issue((uint32_t)sub);
  }
  uint32_t ta, tb;
  table_entry(p, first, lane, ta, tb);
  for (uint32_t sub = first; sub < p.nsub; sub += nwarps) {
    const uint64_t ahead = (uint64_t)sub + (uint64_t)(STAGES - 1) * nwarps;
    if (ahead < nfull) issue((uint32_t)ahead);
    uint32_t na, nb;                                        // the next sub-tile's table entries:
    const uint64_t nxt = (uint64_t)sub + nwarps;            // in flight while this one is summed
    table_entry(p, nxt < p.nsub ? (uint32_t)nxt : p.nsub, lane, na, nb);
    bad |= accumulate_subtile_ahead(p, sub, lane, ta, tb, acc);
    ta = na;
    tb = nb;
    const uint32_t lo = sub * CX_SUBTILE;
    if (sub < nfull) {
      const uint32_t s = consumed % STAGES;
      const uint32_t parity = (consumed / STAGES) & 1u;
      // completion seen by any lane is final: the phase cannot advance again before the next issue()
      if (!__any_sync(0xffffffffu, mbar_wait_bounded(&bars[s], parity))) {
        // give the copies that are still in flight one more bounded chance to land in this
        // CTA's shared memory, report, and leave the output of this warp's tiles untouched
        for (uint32_t c = consumed + 1; c < issued; ++c)
          mbar_wait_bounded(&bars[c % STAGES], (c / STAGES) & 1u);
        if (lane == 0 && p.status) atomicOr(p.status, (uint32_t)CX_ST_TIMEOUT);
        return;
      }
      ++consumed;
      const float* st = stage0 + s * NARR * CX_SUBTILE;
#pragma unroll
      for (int q = 0; q < CX_SUBTILE / 128; ++q) {
        const int e0 = q * 128 + lane * 4;
        float av[4], wv[4], mv[4], vv[4];
        cx::load4(acc + e0, av);
        cx::load4(st + e0, wv);
        if (NARR > 1) cx::load4(st + CX_SUBTILE + e0, mv);
        if (NARR > 2) cx::load4(st + 2 * CX_SUBTILE + e0, vv);
        rule4<OP>(p.a, av, wv, mv, vv);
        store_state4<OP, TO>(p.a, (int64_t)lo + e0, wv, mv, vv);
      }
      // this stage is handed back to the copy engine by a later issue()
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    } else {
#pragma unroll
      for (int q = 0; q < CX_SUBTILE / 128; ++q) {
        const int e0 = q * 128 + lane * 4;
        const int64_t i = (int64_t)lo + e0;
        if (i >= p.n) continue;
        float av[4];
        cx::load4(acc + e0, av);
        update4<OP, TO>(p.a, p.n, i, av, p.vec && i + 3 < p.n);
      }
    }
    __syncwarp();
  }
  if (bad && p.status) atomicOr(p.status, bad);
}

// SET of one source: nothing is summed, so the pairs need not meet in shared memory.  Zeros go straight to the
// sub-tile, then the values to their places (the warp's barrier orders the two).  Only for sub-tiles whose 16-byte
// accesses all work.  A value costs a store of its own and dirties its sector a second time, so a sub-tile with
// more pairs than the limit takes shared memory.  Where a warp has one sub-tile (7.2 M elements) the shorter chain
// counts; behind that the stores do.  us with the sums in shared memory / direct, fp32 destination:
//   pairs per sub-tile     10            31            61            102           154
//   2^20 elements      4.48 / 3.97   4.48 / 3.99   4.48 / 4.22   4.74 / 4.48   4.74 / 4.99
//   2^24               13.4 / 13.2   13.7 / 14.5   14.7 / 16.3   15.2 / 18.3   16.3 / 21.1
//   2^26               52.9 / 53.0   54.7 / 56.2   57.0 / 58.0   57.1 / 64.4   62.6 / 74.4
// bf16 destination, 2^20: 3.97 / 3.71 with 10 pairs, 4.22 / 4.22 with 102; 2^24: 9.60 / 9.09 with 10, 9.60 / 9.85
// with 20; 2^26: 28.6 / 27.5 and 29.8 / 31.0.
constexpr uint32_t kDirectShort = 102, kDirect = 15;
template <typename TO>
__device__ __forceinline__ uint32_t set_subtile(const ApplyParams& p, uint32_t sub, int lane, uint32_t a, uint32_t b, bool& wait) {
  const uint32_t lo = sub * CX_SUBTILE;
  TO* out = reinterpret_cast<TO*>(p.a.out) + lo;
  const CxPair* pairs = p.src.ep[0].pairs;
  constexpr int kAt = 4;
  uint32_t bad = 0;
  CxPair pr[kAt];
#pragma unroll
  for (int k = 0; k < kAt; ++k) {
    pr[k].idx = -1;
    pr[k].val = 0;
    if (a + 32 * k + lane < b) pr[k] = ld_pair(pairs + a + 32 * k + lane);
  }
  if (wait) { cx::pdl_wait(); wait = false; }
  const float zero[4] = {p.a.scale * 0.f, p.a.scale * 0.f, p.a.scale * 0.f, p.a.scale * 0.f};
#pragma unroll
  for (int q = 0; q < CX_SUBTILE / 128; ++q) cx::store4(out + q * 128 + lane * 4, zero);
  __syncwarp();
  while (a < b) {                              // (warp-uniform)
#pragma unroll
    for (int k = 0; k < kAt; ++k) {
      const uint32_t d = (uint32_t)pr[k].idx - lo;
      if (a + 32 * k + lane < b) {
        if (d < CX_SUBTILE) out[d] = cx::Elem<TO>::from_f(p.a.scale * (0.f + __uint_as_float(pr[k].val)));
        else bad = CX_ST_BAD_INDEX;
      }
    }
    a += 32 * kAt;
#pragma unroll
    for (int k = 0; k < kAt; ++k) if (a + 32 * k + lane < b) pr[k] = ld_pair(pairs + a + 32 * k + lane);
  }
  return bad;
}

// CTAs of apply_dense_kernel per SM (registers)
constexpr int dense_per_sm(int op) { return op == CX_OP_MOMENTUM || op == CX_OP_ADAMW ? 5 : 6; }

template <int OP, typename TO>
__global__ void __launch_bounds__(kThreads, dense_per_sm(OP)) apply_dense_kernel(const __grid_constant__ ApplyParams p) {
  __shared__ __align__(16) float s_acc[kWarps][CX_SUBTILE];
  begin_apply(p, p.early);
  const int lane = threadIdx.x & 31;
  if (!wait_sources(p)) { cx::pdl_wait(); return; }
  const int warp = threadIdx.x >> 5;
  const uint32_t nwarps = gridDim.x * kWarps;
  float* acc = s_acc[warp];
  bool wait = p.front_wait == CX_WAIT_VECTORS;
  const uint32_t direct = p.nsub <= nwarps ? kDirectShort : kDirect;
  uint32_t bad = 0;
  uint32_t sub = blockIdx.x * kWarps + warp, a, b;
  table_entry(p, sub, lane, a, b);
  for (; sub < p.nsub; sub += nwarps) {
    const uint32_t lo = sub * CX_SUBTILE;
    uint32_t na, nb;                          // the next sub-tile's table entries, in flight meanwhile
    const uint64_t next = (uint64_t)sub + nwarps;
    table_entry(p, next < p.nsub ? (uint32_t)next : p.nsub, lane, na, nb);
    const bool whole = p.vec && (int64_t)lo + CX_SUBTILE <= p.n;
    if (OP == CX_OP_SET && whole && p.src.count == 1) {
      const uint32_t a0 = __shfl_sync(0xffffffffu, a, 0), b0 = __shfl_sync(0xffffffffu, b, 0);
      if (b0 - a0 <= direct) {
        bad |= set_subtile<TO>(p, sub, lane, a0, b0, wait);
        a = na;
        b = nb;
        continue;
      }
    }
    bad |= accumulate_subtile(p, sub, lane, a, b, acc);
    if (wait) { cx::pdl_wait(); wait = false; }
    a = na;
    b = nb;
    auto walk = [&](auto all) {
      constexpr int kUnroll = decltype(all)::value ? CX_SUBTILE / 128 : 1;
#pragma unroll kUnroll
      for (int q = 0; q < CX_SUBTILE / 128; ++q) {
        const int e0 = q * 128 + lane * 4;
        const int64_t i = (int64_t)lo + e0;
        if (!decltype(all)::value && i >= p.n) continue;
        const float4 t = *reinterpret_cast<const float4*>(acc + e0);
        const float av[4] = {t.x, t.y, t.z, t.w};
        update4<OP, TO>(p.a, p.n, i, av, decltype(all)::value || (p.vec && i + 3 < p.n));
      }
    };
    if (whole) walk(std::true_type());         // without a test per access
    else walk(std::false_type());
    __syncwarp();
  }
  if (bad && p.status) atomicOr(p.status, bad);
  cx::pdl_wait();   // launched early behind its sender: do not complete before that grid has
}

// ---- dense update: the averaged gradient is a plain vector -------------------------------
// After a dense allreduce (or on a single rank, where nothing is exchanged) the gradient is an
// ordinary fp32 vector; the same rule runs over it in one pass with 16-byte accesses.
struct UpdateParams {
  const float* g;
  CxApplyArgs a;
  int64_t n;
  uint32_t vec;
};

template <int OP, typename TO>
__global__ void __launch_bounds__(kThreads) update_dense_kernel(const UpdateParams q) {
  const int64_t gsz = (int64_t)gridDim.x * kThreads;
  const int64_t nv = (q.n + 3) / 4;
  for (int64_t v = (int64_t)blockIdx.x * kThreads + threadIdx.x; v < nv; v += gsz) {
    const int64_t i = v * 4;
    float gv[4];
    const bool vec = q.vec && i + 3 < q.n;
    if (vec) cx::load4(q.g + i, gv);
    else
      for (int e = 0; e < 4; ++e) gv[e] = i + e < q.n ? q.g[i + e] : 0.f;
    update4<OP, TO>(q.a, q.n, i, gv, vec);
  }
}

template <typename TO>
int launch_update(const UpdateParams& q, int grid, cudaStream_t s) {
  switch (q.a.op) {
    case CX_OP_SGD: update_dense_kernel<CX_OP_SGD, TO><<<grid, kThreads, 0, s>>>(q); return 0;
    case CX_OP_MOMENTUM: update_dense_kernel<CX_OP_MOMENTUM, TO><<<grid, kThreads, 0, s>>>(q); return 0;
    case CX_OP_ADAMW: update_dense_kernel<CX_OP_ADAMW, TO><<<grid, kThreads, 0, s>>>(q); return 0;
    default: return cx_set_error("cx_update_dense: op must be an update rule", 0);
  }
}

// The whole step of a rank that exchanges nothing: the folded gradient (CxFold) goes from registers
// into the momentum and the update rule, one pass over gradient, momentum and weights.  A warp takes
// a sub-tile; the ones at tensor borders go element by element.  25.6 M bf16 parameters with momentum:
// 85 us for the fold and 62 us for the update as two kernels.
struct FoldUpdateParams {
  CxFold f;
  CxApplyArgs a;
  int64_t n;
  uint32_t nsub;
  uint32_t nborder_ctas;
};

// KEEP: 0 nothing of the folded vector is kept, 1 it is stored as the momentum, 2 read and stored
template <int OP, typename TO, typename T, int KEEP>
__device__ __forceinline__ void fold_update_border(const FoldUpdateParams& q, uint32_t sub, int lane) {
  const int64_t lo = (int64_t)sub * CX_SUBTILE;
  const cx::FoldBlock<T> blk = cx::fold_blocks<T>(q.f, sub, lane);
  constexpr int kGroup = 4;      // loads in flight: none of them moves across a store
#pragma unroll 1
  for (int j0 = 0; j0 < CX_SUBTILE / 32; j0 += kGroup) {
    float x[kGroup], y[kGroup], w[kGroup], m[kGroup], v[kGroup];
    uint32_t in = 0;
#pragma unroll
    for (int j = 0; j < kGroup; ++j) {
      const int64_t i = lo + 32 * (j0 + j) + lane;
      const bool t = cx::fold_element<T>(blk, j0 + j, lane, x[j]);
      in |= (t ? 1u : 0u) << j;
      y[j] = KEEP == 2 && t ? q.f.u[i] : 0.f;
      load_state1<OP>(q.a, i, i < q.n, w[j], m[j], v[j]);
    }
#pragma unroll
    for (int j = 0; j < kGroup; ++j) {
      const int64_t i = lo + 32 * (j0 + j) + lane;
      const float c = __shfl_sync(0xffffffffu, blk.coef, (j0 + j) >> 1);
      const float t = (in >> j) & 1u ? q.f.mu * y[j] + c * x[j] : 0.f;
      if (KEEP && ((in >> j) & 1u)) q.f.u[i] = t;
      if (i < q.n) update1<OP, TO>(q.a, i, t, w[j], m[j], v[j]);
    }
  }
}

template <int OP, typename TO, typename T, int KEEP>
__global__ void __launch_bounds__(kThreads, 4) fold_update_kernel(const __grid_constant__ FoldUpdateParams q) {
  cx::pdl_wait();
  cx::pdl_trigger();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (blockIdx.x < q.nborder_ctas) {
    for (uint32_t b = warp * q.nborder_ctas + blockIdx.x; b < (uint32_t)q.f.nborder; b += q.nborder_ctas * kWarps)
      fold_update_border<OP, TO, T, KEEP>(q, (uint32_t)(q.f.border[b] - q.f.base / CX_SUBTILE), lane);
    return;
  }
  const uint32_t nwarps = (gridDim.x - q.nborder_ctas) * kWarps;
  uint32_t sub = (blockIdx.x - q.nborder_ctas) * kWarps + warp;
  const uint64_t last = q.f.keep ? cx::drop_policy() : cx::plain_policy();
  cx::FoldWhole<T> cur = {nullptr, 0.f, 0};
  if (sub < q.nsub) cur = cx::fold_whole<T>(q.f, sub);
  while (sub < q.nsub) {
    const int64_t lo = (int64_t)sub * CX_SUBTILE;
    const uint32_t next = sub + nwarps;
    cx::FoldWhole<T> ahead = {nullptr, 0.f, 0};
    if (next < q.nsub) ahead = cx::fold_whole<T>(q.f, next);
    if (cur.kind == 2) {
      constexpr int kGroup = OP == CX_OP_ADAMW ? 1 : 2;     // 128-element rows whose loads are in flight together
#pragma unroll 1
      for (int c0 = 0; c0 < CX_SUBTILE / 128; c0 += kGroup) {
        float x[kGroup][4], y[kGroup][4], wv[kGroup][4], mv[kGroup][4], vv[kGroup][4];
#pragma unroll
        for (int k = 0; k < kGroup; ++k) {
          const int e0 = (c0 + k) * 128 + lane * 4;
          cx::Raw4<T>::to_f(cx::load_hint(reinterpret_cast<const typename cx::Raw4<T>::type*>(cur.g + e0), last), x[k]);
#pragma unroll
          for (int e = 0; e < 4; ++e) y[k][e] = 0.f;
          if (KEEP == 2) cx::load4(q.f.u + lo + e0, y[k]);
          cx::load4(reinterpret_cast<const float*>(q.a.out) + lo + e0, wv[k]);
          if (OP != CX_OP_SGD) cx::load4(q.a.m + lo + e0, mv[k]);
          if (OP == CX_OP_ADAMW) cx::load4(q.a.v + lo + e0, vv[k]);
        }
#pragma unroll
        for (int k = 0; k < kGroup; ++k) {
          const int e0 = (c0 + k) * 128 + lane * 4;
#pragma unroll
          for (int e = 0; e < 4; ++e) y[k][e] = q.f.mu * y[k][e] + cur.coef * x[k][e];
          if (KEEP) cx::store4(q.f.u + lo + e0, y[k]);
          rule4<OP>(q.a, y[k], wv[k], mv[k], vv[k]);
          store_state4<OP, TO>(q.a, lo + e0, wv[k], mv[k], vv[k]);
        }
      }
    } else if (cur.kind == 1) {
      fold_update_border<OP, TO, T, KEEP>(q, sub, lane);    // gradients at an odd address
    }
    cur = ahead;
    sub = next;
  }
}

template <typename TO, typename T, int KEEP>
int launch_fold_update(const FoldUpdateParams& q, int grid, cudaStream_t s) {
  const bool cap = cx_seq_cell() != nullptr;
  switch (q.a.op) {
    case CX_OP_SGD: cx_launch_pdl(fold_update_kernel<CX_OP_SGD, TO, T, KEEP>, grid, kThreads, 0, s, q, cap); return 0;
    case CX_OP_MOMENTUM: cx_launch_pdl(fold_update_kernel<CX_OP_MOMENTUM, TO, T, KEEP>, grid, kThreads, 0, s, q, cap); return 0;
    case CX_OP_ADAMW: cx_launch_pdl(fold_update_kernel<CX_OP_ADAMW, TO, T, KEEP>, grid, kThreads, 0, s, q, cap); return 0;
    default: return cx_set_error("cx_fold_update: op must be an update rule", 0);
  }
}

// ---- verbatim forwarding of a received slot (ring allgather hop) ----------

struct ForwardParams {
  CxEndpoint from;
  uint64_t expect;
  CxTargets tg;
  uint64_t seq;
  uint32_t cap;
  CxWorkCounters* ctr;
  uint32_t* status;
  uint64_t timeout_ns;
};

__global__ void __launch_bounds__(kThreads) forward_kernel(const ForwardParams p) {
  __shared__ uint32_t s_ok, s_last;
  if (threadIdx.x == 0) s_ok = cx::wait_seq(&p.from.hdr->seq, p.expect, p.timeout_ns) ? 1u : 0u;
  __syncthreads();
  // A CTA whose wait ran out copies nothing but still arrives at the completion counter and
  // marks the launch as failed there: the CTA that arrives last then publishes nothing and
  // leaves the counters clean for the next launch, whatever the other CTAs saw.
  const bool ok = s_ok != 0;
  if (!ok && threadIdx.x == 0) {
    if (p.status) atomicOr(p.status, (uint32_t)CX_ST_TIMEOUT);
    atomicOr(&p.ctr->pad[0], 1u);
  }
  CxHeader hv;
  if (!ok) { hv.nnz = 0; hv.nsub = 0; hv.n = 0; hv.nnz_found = 0; hv.kind = CX_KIND_ERROR; hv.threshold = 0.f; hv.src_rank = 0; hv.dtype = 0; }
  else
  {
    const uint4* hp = reinterpret_cast<const uint4*>(p.from.hdr);
    uint4* dp = reinterpret_cast<uint4*>(&hv);
#pragma unroll
    for (int q = 0; q < 4; ++q) dp[q] = __ldcg(hp + q);
  }
  const CxHeader* h = &hv;
  const uint32_t nnz = min(h->nnz, p.cap);
  const uint32_t nsub = h->nsub;
  // a warp per sub-tile: its table entry and its pairs keep their positions
  const int lane = threadIdx.x & 31;
  const uint32_t nwarps = gridDim.x * kWarps;
  for (uint32_t sub = blockIdx.x * kWarps + (threadIdx.x >> 5); sub < nsub; sub += nwarps) {
    uint2 v = __ldcg(reinterpret_cast<const uint2*>(p.from.table) + sub);
    v.y = min(v.y, (uint32_t)CX_SUBTILE);
    if (v.x >= p.cap) v.x = v.y = 0;
    else v.y = min(v.y, p.cap - v.x);
    if (lane < p.tg.count) reinterpret_cast<uint2*>(p.tg.ep[lane].table)[sub] = v;
    for (uint32_t i = lane; i < v.y; i += 32) {
      const uint2 pr = __ldcg(reinterpret_cast<const uint2*>(p.from.pairs + v.x + i));
      for (int k = 0; k < p.tg.count; ++k) *reinterpret_cast<uint2*>(p.tg.ep[k].pairs + v.x + i) = pr;
    }
  }
  if (!cx::cta_arrive(&p.ctr->done, gridDim.x, &s_last)) return;
  const uint32_t failed = *reinterpret_cast<volatile uint32_t*>(&p.ctr->pad[0]);
  if (!failed && (int)threadIdx.x < p.tg.count) {
    CxHeader* o = p.tg.ep[threadIdx.x].hdr;
    o->bytes = 8ull + 8ull * nnz; o->n = h->n; o->nnz = nnz; o->nnz_found = h->nnz_found;
    o->kind = h->kind; o->threshold = h->threshold; o->nsub = nsub; o->src_rank = h->src_rank;
    o->dtype = h->dtype;
    cx::st_release_sys(&o->seq, p.seq);
  }
  __syncthreads();
  if (threadIdx.x == 0) { p.ctr->pad[0] = 0; p.ctr->done = 0; }
}

#ifndef CX_APPLY_STAGES
#define CX_APPLY_STAGES 1
#endif
#ifndef CX_APPLY_WARPS
#define CX_APPLY_WARPS 16
#endif

// COMPREX_APPLY_BULK=1 routes the dense updates through the bulk-copy kernel.  It is off by
// default: AdamW at 2^28 elements and 1 % survivors takes 1336 us in it and 1098 in the register
// kernel (2^24: 179 and 79 us; 10 % survivors: 2784 and 1275 us), because its shared-memory footprint leaves 14 warps per SM to
// cover an instruction-issue-bound update.  The variable is read at every call.
bool bulk_enabled() {
  const char* e = getenv("COMPREX_APPLY_BULK");
  return e && e[0] == '1';
}

// COMPREX_APPLY_STAGES=1|2: sub-tiles of state per warp in flight (more stages, fewer warps per SM)
int bulk_stages() {
  const char* e = getenv("COMPREX_APPLY_STAGES");
  return (e && e[0] == '1') ? 1 : (e && e[0] == '2') ? 2 : CX_APPLY_STAGES;
}

template <int OP, typename TO, int STAGES>
int launch_bulk_stages(const ApplyParams& p, cudaStream_t s) {
  constexpr size_t kWarpBytes = (size_t)(1 + STAGES * StateArrays<OP>::n) * CX_SUBTILE * sizeof(float);
  constexpr size_t kBudget = 227 * 1024 - 1024;      // per SM, minus the static part and slack
  int nw = (int)(kBudget / (kWarpBytes + 8 * STAGES));
  if (nw > CX_APPLY_WARPS) nw = CX_APPLY_WARPS;
  if (nw > kBulkMaxThreads / 32) nw = kBulkMaxThreads / 32;
  const size_t smem = (size_t)nw * (kWarpBytes + 8 * STAGES);
  const int per_sm = (int)(kBudget / (smem + 1024)) > 0 ? (int)(kBudget / (smem + 1024)) : 1;
  auto kern = apply_dense_bulk_kernel<OP, TO, STAGES>;
  static bool configured[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cx_set_error("cx_apply: cudaGetDevice", 0);
  if (!configured[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cx_set_error("cx_apply: shared memory opt-in", (int)e);
    configured[dev] = true;
  }
  int grid = cx_sm_count() * per_sm;
  const int need = (int)((p.nsub + nw - 1) / nw);
  if (grid > need) grid = need;
  kern<<<grid, nw * 32, smem, s>>>(p);
  return 0;
}

template <int OP, typename TO>
int launch_bulk(const ApplyParams& p, cudaStream_t s) {
  return bulk_stages() == 1 ? launch_bulk_stages<OP, TO, 1>(p, s) : launch_bulk_stages<OP, TO, 2>(p, s);
}

template <typename TO>
int launch_apply(const ApplyParams& p, int grid, cudaStream_t s) {
  const int op = p.a.op;
  const bool sparse = op == CX_OP_ADD || (op == CX_OP_SGD && p.a.wd == 0.f);
  if (!sparse && op != CX_OP_SET && p.vec && bulk_enabled()) {
    // optimizer state through the copy engine (16-byte aligned state, full sub-tiles in bulk)
    if (op == CX_OP_SGD) return launch_bulk<CX_OP_SGD, TO>(p, s);
    if (op == CX_OP_MOMENTUM) return launch_bulk<CX_OP_MOMENTUM, TO>(p, s);
    if (op == CX_OP_ADAMW) return launch_bulk<CX_OP_ADAMW, TO>(p, s);
  }
  const bool cap = p.seq_cell != nullptr;
  const bool several = p.src.count > 1;
  if (sparse && in_batches(p.group, p.src.count)) cx_launch_pdl(apply_sparse_batch_kernel<TO>, grid, kThreads, 0, s, p, cap);
  else if (sparse && several) cx_launch_pdl(apply_sparse_kernel<TO, kAhead, true>, grid, kThreads, 0, s, p, cap);
  else if (sparse && p.group >= kLargeGroup) cx_launch_pdl(apply_sparse_kernel<TO, kAheadLarge, false>, grid, kThreads, 0, s, p, cap);
  else if (sparse) cx_launch_pdl(apply_sparse_kernel<TO, kAhead, false>, grid, kThreads, 0, s, p, cap);
  else if (op == CX_OP_SET) cx_launch_pdl(apply_dense_kernel<CX_OP_SET, TO>, grid, kThreads, 0, s, p, cap);
  else if (op == CX_OP_SGD) cx_launch_pdl(apply_dense_kernel<CX_OP_SGD, TO>, grid, kThreads, 0, s, p, cap);
  else if (op == CX_OP_MOMENTUM) cx_launch_pdl(apply_dense_kernel<CX_OP_MOMENTUM, TO>, grid, kThreads, 0, s, p, cap);
  else if (op == CX_OP_ADAMW) cx_launch_pdl(apply_dense_kernel<CX_OP_ADAMW, TO>, grid, kThreads, 0, s, p, cap);
  else return cx_set_error("cx_apply: unknown op", 0);
  return 0;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

int cx_apply_cuda(const CxSources* src, int64_t n, const CxApplyArgs* a, uint32_t* status,
                  uint64_t timeout_ns, void* stream) {
  if (src->count < 0 || src->count > CX_MAX_PEERS) return cx_set_error("cx_apply: bad source count", 0);
  if (n < 0 || n > 0x7fffffffLL) return cx_set_error("cx_apply: n out of range", 0);
  if (!a->out) return cx_set_error("cx_apply: out is NULL", 0);
  if (n == 0) return 0;
  ApplyParams p;
  p.src = *src; p.a = *a; p.n = n;
  p.nsub = (uint32_t)((n + CX_SUBTILE - 1) / CX_SUBTILE);
  p.status = status; p.timeout_ns = timeout_ns; p.seq_cell = cx_seq_cell();
  const bool update = a->op != CX_OP_ADD && a->op != CX_OP_SET;
  if (update && a->op != CX_OP_SGD && !a->m) return cx_set_error("cx_apply: momentum buffer missing", 0);
  if (a->op == CX_OP_ADAMW && !a->v) return cx_set_error("cx_apply: second-moment buffer missing", 0);
  p.vec = aligned16(a->out) && (!a->shadow || aligned16(a->shadow)) && (!a->m || aligned16(a->m)) &&
          (!a->v || aligned16(a->v));
  p.front_wait = cx_chain_bits() & CX_CHAINED ? CX_WAIT_NONE : cx_front_wait(stream);
  // what the first of a chain waits for has to be complete for the others, too
  if (p.front_wait != CX_WAIT_NONE && cx_chain_bits() & CX_CHAIN_NEXT) p.front_wait = CX_WAIT_CHAIN;
  const int dt = update ? (a->shadow ? a->shadow_dtype : CX_F32) : a->out_dtype;
  int grid = cx_sm_count() * dense_per_sm(a->op);      // the sparse ops: as many as for SET
  p.group = 1;
  const bool sparse = a->op == CX_OP_ADD || (a->op == CX_OP_SGD && a->wd == 0.f);
  if (sparse) {
    // as few sub-tiles per warp as fill one wave of warps, then as few waves as 32 per warp allow
    const uint64_t warps = (uint64_t)grid * kWarps;
    const uint64_t waves = (p.nsub + warps * 32 - 1) / (warps * 32);
    p.group = (uint32_t)((p.nsub + warps * waves - 1) / (warps * waves));
  }
  // (the kernels for several sources may take fewer sub-tiles at a time)
  const uint64_t per_cta = (uint64_t)kWarps * (src->count > 1 ? 1u : p.group);
  const int need = (int)((p.nsub + per_cta - 1) / per_cta);
  if (grid > need) grid = need;
  // A dense kernel lets the next one in early when that one is chained to it, or when it leaves most of
  // the GPU free.  Otherwise early CTAs of the next kernel fill the gaps of this one unevenly, and SMs
  // that never run empty keep this kernel's large shared-memory partition: an exchange with exact top-k
  // went from 73 to 84 us, a GPT-2 medium step from 2225 to 2301.  (The sparse kernel has neither
  // problem: 3.7 us less for a ResNet-50 step.)
  p.early = (cx_chain_bits() & CX_CHAIN_NEXT) || grid <= cx_sm_count() ? 1u : 0u;
  cx_note_stream(stream, sparse || p.early);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  int rc;
  switch (dt) {
    case CX_F32: rc = launch_apply<float>(p, grid, s); break;
    case CX_BF16: rc = launch_apply<__nv_bfloat16>(p, grid, s); break;
    case CX_F16: rc = launch_apply<__half>(p, grid, s); break;
    default: return cx_set_error("cx_apply: unsupported dtype on CUDA", 0);
  }
  if (rc) return rc;
  cx_note_launch();
  return cx_check_launch("apply_kernel");
}

int cx_update_dense_cuda(const float* g, int64_t n, const CxApplyArgs* a, void* stream) {
  if (!a->out || !g) return cx_set_error("cx_update_dense: NULL vector", 0);
  if (n < 0 || n > 0x7fffffffLL) return cx_set_error("cx_update_dense: n out of range", 0);
  if (a->op != CX_OP_SGD && a->op != CX_OP_MOMENTUM && a->op != CX_OP_ADAMW)
    return cx_set_error("cx_update_dense: op must be an update rule", 0);
  if (a->op != CX_OP_SGD && !a->m) return cx_set_error("cx_update_dense: momentum buffer missing", 0);
  if (a->op == CX_OP_ADAMW && !a->v) return cx_set_error("cx_update_dense: second-moment buffer missing", 0);
  if (n == 0) return 0;
  UpdateParams q;
  q.g = g; q.a = *a; q.n = n;
  q.vec = aligned16(g) && aligned16(a->out) && (!a->shadow || aligned16(a->shadow)) && (!a->m || aligned16(a->m)) &&
          (!a->v || aligned16(a->v));
  int grid = cx_sm_count() * 8;
  const int need = (int)(((n + 3) / 4 + kThreads - 1) / kThreads);
  if (grid > need) grid = need;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  int rc;
  switch (a->shadow ? a->shadow_dtype : CX_F32) {
    case CX_F32: rc = launch_update<float>(q, grid, s); break;
    case CX_BF16: rc = launch_update<__nv_bfloat16>(q, grid, s); break;
    case CX_F16: rc = launch_update<__half>(q, grid, s); break;
    default: return cx_set_error("cx_update_dense: unsupported dtype on CUDA", 0);
  }
  if (rc) return rc;
  cx_note_launch();
  return cx_check_launch("update_dense_kernel");
}

// The low-precision copy of the weights has the element type of the gradients (both are the model's).
int cx_fold_update_cuda(int gdtype, const CxFold* fold, int64_t n, const CxApplyArgs* a, void* stream) {
  if (!a->out) return cx_set_error("cx_fold_update: NULL vector", 0);
  // all buckets of a model at once: only their sub-tiles are counted in 32 bits
  if (n < 0 || n > (1LL << 40)) return cx_set_error("cx_fold_update: n out of range", 0);
  if (a->op != CX_OP_SGD && a->op != CX_OP_MOMENTUM && a->op != CX_OP_ADAMW)
    return cx_set_error("cx_fold_update: op must be an update rule", 0);
  if (a->op != CX_OP_SGD && !a->m) return cx_set_error("cx_fold_update: momentum buffer missing", 0);
  if (a->op == CX_OP_ADAMW && !a->v) return cx_set_error("cx_fold_update: second-moment buffer missing", 0);
  if (!fold->u && fold->mu != 0.f) return cx_set_error("cx_fold_update: folding with momentum needs the momentum", 0);
  if (a->shadow && a->shadow_dtype != gdtype) return cx_set_error("cx_fold_update: gradients and weights differ in type", 0);
  if (!(aligned16(a->out) && aligned16(fold->u) && aligned16(a->shadow) && aligned16(a->m) && aligned16(a->v)))
    return cx_set_error("cx_fold_update: state must be 16-byte aligned", 0);
  if (n == 0) return 0;
  FoldUpdateParams q;
  q.f = *fold; q.a = *a; q.n = n;
  q.nsub = (uint32_t)((n + CX_SUBTILE - 1) / CX_SUBTILE);
  int grid;
  q.nborder_ctas = (uint32_t)cx_border_ctas(q.f, q.nsub, kWarps, cx_sm_count() * 4, &grid);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int keep = !fold->u ? 0 : fold->mu == 0.f ? 1 : 2;
  int rc;
#define CX_FOLD_UPDATE(T) (keep == 0 ? launch_fold_update<T, T, 0>(q, grid, s) \
                           : keep == 1 ? launch_fold_update<T, T, 1>(q, grid, s) : launch_fold_update<T, T, 2>(q, grid, s))
  switch (gdtype) {
    case CX_F32: rc = CX_FOLD_UPDATE(float); break;
    case CX_BF16: rc = CX_FOLD_UPDATE(__nv_bfloat16); break;
    case CX_F16: rc = CX_FOLD_UPDATE(__half); break;
    default: return cx_set_error("cx_fold_update: unsupported dtype on CUDA", 0);
  }
#undef CX_FOLD_UPDATE
  if (rc) return rc;
  cx_note_stream(stream, true);
  cx_note_launch();
  return cx_check_launch("fold_update_kernel");
}

int cx_forward_cuda(const CxEndpoint* from, uint64_t expect_seq, const CxTargets* tg, uint64_t seq,
                    uint32_t cap, void* counters, uint32_t* status, uint64_t timeout_ns,
                    void* stream) {
  ForwardParams p;
  p.from = *from; p.expect = expect_seq; p.tg = *tg; p.seq = seq; p.cap = cap;
  p.ctr = reinterpret_cast<CxWorkCounters*>(counters);
  p.status = status; p.timeout_ns = timeout_ns;
  // every CTA waits on the same notification, so keep the grid co-resident
  const int grid = cx_sm_count() * 2;
  forward_kernel<<<grid, kThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(p);
  cx_note_sender(stream);
  cx_note_launch();
  return cx_check_launch("forward_kernel");
}
