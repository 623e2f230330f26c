// Elements of a folded vector (CxFold): the gradient tensors autograd produced, scaled by their clip
// factors, plus the momentum, at the positions of the flat parameter buffer.
#pragma once
#include "cx_device.cuh"

namespace cx {

// the tensor that holds flat position `at`, searched from `seg` upwards; nseg when none ends behind it
__device__ __forceinline__ int fold_seek(const CxFold& f, int64_t at, int seg) {
  while (seg < f.nseg && f.seg_end[seg] <= at) ++seg;
  return seg;
}

// value at element i of the range, without moving the momentum on
template <typename T>
__device__ __forceinline__ float fold_at(const CxFold& f, int64_t i) {
  const int64_t at = f.base + i;
  const int seg = fold_seek(f, at, f.sub_seg[i / CX_SUBTILE]);
  if (seg >= f.nseg || f.seg_off[seg] > at) return 0.f;
  const float x = Elem<T>::to_f(reinterpret_cast<const T*>(f.seg_ptr[seg])[at - f.seg_off[seg]]);
  const float y = f.mu != 0.f ? f.u[i] : 0.f;
  return f.mu * y + f.coef[seg] * x;
}

// A sub-tile at tensor borders.  Tensors start at multiples of CX_FOLD_ALIGN = 64 elements, so each
// of its 16 blocks of 64 lies in one tensor (and the gap behind it) or in none: lane b describes
// block b.  The descriptions of the 32 tensors from the first candidate on are loaded side by side
// and handed from lane to lane, so the gradients are two dependent loads away.
template <typename T>
struct FoldBlock {
  const T* g;     // gradient at the block's first element
  float coef;
  int valid;      // elements of the block that belong to the tensor
};
template <typename T>
__device__ __forceinline__ FoldBlock<T> fold_blocks(const CxFold& f, uint32_t sub, int lane) {
  const int s0 = f.sub_seg[sub];
  const int64_t at0 = f.base + (int64_t)sub * CX_SUBTILE;
  const int64_t mine = at0 + CX_FOLD_ALIGN * (int64_t)lane;
  const bool have = s0 + lane < f.nseg;
  int64_t end = have ? f.seg_end[s0 + lane] : (int64_t)1 << 62, off = have ? f.seg_off[s0 + lane] : (int64_t)1 << 62;
  unsigned long long ptr = have ? reinterpret_cast<unsigned long long>(f.seg_ptr[s0 + lane]) : 0ull;
  float coef = have ? f.coef[s0 + lane] : 0.f;
  int k = 0;      // tensors that end at or before my block
#pragma unroll
  for (int b = 0; b < CX_SUBTILE / CX_FOLD_ALIGN; ++b) {
    const uint32_t before = __ballot_sync(0xffffffffu, end <= at0 + CX_FOLD_ALIGN * b);
    if (b == lane) k = __popc(before);
  }
  const int from = k & 31;
  end = __shfl_sync(0xffffffffu, end, from);
  off = __shfl_sync(0xffffffffu, off, from);
  ptr = __shfl_sync(0xffffffffu, ptr, from);
  coef = __shfl_sync(0xffffffffu, coef, from);
  FoldBlock<T> r = {nullptr, 0.f, 0};
  if (lane >= CX_SUBTILE / CX_FOLD_ALIGN) return r;
  if (k == 32) {                               // a row of empty tensors
    const int seg = fold_seek(f, mine, s0 + 32);
    if (seg >= f.nseg) return r;
    end = f.seg_end[seg]; off = f.seg_off[seg]; coef = f.coef[seg];
    ptr = reinterpret_cast<unsigned long long>(f.seg_ptr[seg]);
  }
  if (off > mine) return r;
  const int64_t left = end - mine;
  r.valid = left < CX_FOLD_ALIGN ? (int)left : CX_FOLD_ALIGN;
  r.g = reinterpret_cast<const T*>(ptr) + (mine - off);
  r.coef = coef;
  return r;
}
// element 32 j + lane of the sub-tile (its factor: the coef of lane j / 2): true when a tensor lies there
template <typename T>
__device__ __forceinline__ bool fold_element(const FoldBlock<T>& blk, int j, int lane, float& x) {
  const int b = j >> 1, o = (j & 1) * 32 + lane;
  const T* g = reinterpret_cast<const T*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(blk.g), b));
  const int valid = __shfl_sync(0xffffffffu, blk.valid, b);
  x = o < valid ? Elem<T>::to_f(g[o]) : 0.f;
  return o < valid;
}

// What a whole sub-tile needs to know of the tensor that covers it.  Warp-uniform.
template <typename T>
struct FoldWhole {
  const T* g;
  float coef;
  int kind;       // 0: not covered by one tensor, 1: covered, 2: and four-element accesses work on the address
};
template <typename T>
__device__ __forceinline__ FoldWhole<T> fold_whole(const CxFold& f, uint32_t sub) {
  FoldWhole<T> r = {nullptr, 0.f, 0};
  const int seg = f.sub_seg[sub];
  if (seg >= f.nseg) return r;
  const int64_t at = f.base + (int64_t)sub * CX_SUBTILE, off = f.seg_off[seg], end = f.seg_end[seg];
  r.g = reinterpret_cast<const T*>(f.seg_ptr[seg]) + (at - off);
  r.coef = f.coef[seg];
  if (off <= at && end >= at + CX_SUBTILE) r.kind = (reinterpret_cast<uintptr_t>(r.g) & (4 * sizeof(T) - 1)) == 0 ? 2 : 1;
  return r;
}

}  // namespace cx

// Sub-tiles at tensor borders take several times as long as whole ones (more dependent loads); met
// late in a warp's share they were a tail of 25 us.  The first CTAs of the grid do nothing else, the
// others skip them.  Returns how many: all that are needed while the grid has room, else their share
// of the work, a border sub-tile counted as four whole ones (by its dependent loads; not swept).
inline int cx_border_ctas(const CxFold& f, int64_t nsub, int warps, int room, int* grid) {
  const int64_t nat = (nsub + warps - 1) / warps, bor = (f.nborder + warps - 1) / warps;
  if (nat + bor <= room) { *grid = (int)(nat + bor); return (int)bor; }
  int64_t b = (4 * (int64_t)f.nborder * room + nsub) / (4 * (int64_t)f.nborder + nsub);
  if (b > bor) b = bor;
  if (b > room - 1) b = room - 1;
  if (b < 1 && bor) b = 1;
  *grid = room;
  return (int)b;
}
