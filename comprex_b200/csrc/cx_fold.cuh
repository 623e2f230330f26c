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
// block b, found for all blocks together (three dependent loads per sub-tile; searching element by
// element took 22 us for one sub-tile).
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
  // candidates: the 32 tensors from s0 on, their ends ascend
  const int64_t end = s0 + lane < f.nseg ? f.seg_end[s0 + lane] : (int64_t)1 << 62;
  int seg = 0;
#pragma unroll
  for (int b = 0; b < CX_SUBTILE / CX_FOLD_ALIGN; ++b) {
    const uint32_t before = __ballot_sync(0xffffffffu, end <= at0 + CX_FOLD_ALIGN * b);
    if (b == lane) seg = s0 + __popc(before);
  }
  FoldBlock<T> r = {nullptr, 0.f, 0};
  if (lane >= CX_SUBTILE / CX_FOLD_ALIGN) return r;
  if (seg == s0 + 32) seg = fold_seek(f, mine, seg);       // a row of empty tensors
  if (seg >= f.nseg) return r;
  const int64_t off = f.seg_off[seg];
  if (off > mine) return r;
  const int64_t left = f.seg_end[seg] - mine;
  r.valid = left < CX_FOLD_ALIGN ? (int)left : CX_FOLD_ALIGN;
  r.g = reinterpret_cast<const T*>(f.seg_ptr[seg]) + (mine - off);
  r.coef = f.coef[seg];
  return r;
}
// element 32 j + lane of the sub-tile: true when a tensor lies there
template <typename T>
__device__ __forceinline__ bool fold_element(const FoldBlock<T>& blk, int j, int lane, float& x, float& coef) {
  const int b = j >> 1, o = (j & 1) * 32 + lane;
  const T* g = reinterpret_cast<const T*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(blk.g), b));
  const int valid = __shfl_sync(0xffffffffu, blk.valid, b);
  coef = __shfl_sync(0xffffffffu, blk.coef, b);
  x = o < valid ? Elem<T>::to_f(g[o]) : 0.f;
  return o < valid;
}

// A sub-tile that one tensor covers completely, with the tensor's share at an address four-element
// accesses work on: its gradient and its factor.  Warp-uniform.
template <typename T>
__device__ __forceinline__ bool fold_whole(const CxFold& f, uint32_t sub, const T*& g, float& coef) {
  const int seg = f.sub_seg[sub];
  if (seg >= f.nseg) return false;
  const int64_t at = f.base + (int64_t)sub * CX_SUBTILE, off = f.seg_off[seg];
  if (off > at || f.seg_end[seg] < at + CX_SUBTILE) return false;
  g = reinterpret_cast<const T*>(f.seg_ptr[seg]) + (at - off);
  coef = f.coef[seg];
  return (reinterpret_cast<uintptr_t>(g) & (4 * sizeof(T) - 1)) == 0;
}

}  // namespace cx
