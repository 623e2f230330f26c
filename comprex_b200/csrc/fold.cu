// Gradient fold of the compressed optimizer: per-tensor L2 clipping and the local
// momentum update, straight from the gradient tensors autograd produced into the flat
// fp32 vector that is exchanged (reference: keras/comprex_optimizer.py:101-115 —
// tf.clip_by_norm per tensor, mom = m*mom + lr*g, concat into one blob).
//
// The tensors of a bucket are described once by a static item list (flat offset,
// length, tensor index, offset inside the tensor; large tensors
// are cut into several items for load balance).  Per step only the table
// of gradient pointers changes.
//   1. fold_sumsq:  partial[item][0..8) = sums of squares of the item (fixed order: the
//      result does not depend on scheduling); the CTA that finishes a tensor leaves
//      coef = lr * clip / max(||g_tensor||, clip),
//   2. the kernel that consumes the vector u = mu * u + coef * g computes it where it needs it:
//      the compress kernel (compress.cu), the dense update (apply.cu), or, for the exchanges that
//      want it in memory, fold_apply below.
// With mu = 0, lr = 1 this is the clipped gradient itself in fp32 (AdamW rule).
#include "cx_device.cuh"

namespace {

constexpr int kThreads = 256;

struct FoldParams {
  const void* const* seg_ptr;   // [nseg] gradient base pointers (device memory)
  const int64_t* item_off;      // [nitems] offset in the flat vector
  const int64_t* item_rel;      // [nitems] offset inside the tensor
  const int32_t* item_len;      // [nitems]
  const int32_t* item_seg;      // [nitems]
  const int32_t* seg_first;     // [nseg + 1] first item of every tensor
  float* u;
  float* partial;               // [nitems], or [nitems * 8]: per-warp sums of squares
  float* coef;                  // [nseg]
  uint32_t* count;              // [nseg] arrivals, zero between launches
  int32_t segs;
  int32_t keep;                 // the gradients are to stay in L2 for the kernel that reads them next
  float clip;                   // <= 0: no clipping
  float mu;
  float lr;
};

// Bound by the read of the gradients.  The sum of an item is defined by kSum = 256 strands (strand t:
// the 16-byte groups t, t + 256, ..., in that order), added up warp by warp in a fixed order, so the
// result does not depend on how strands meet CTAs: a CTA takes 128 of them, which spreads even a small
// model over the chip, and leaves the per-warp sums (8 floats per item) to the CTA that arrives last at
// the tensor's counter; that one adds them up.  cx_fold, whose scratch holds one float per item, keeps
// an item in one CTA.  25.6 M bf16 gradients: 15 us with items of 65536 elements and 8-byte loads (eight
// rounds of loads one after the other), plus 2.5 for a kernel that turned the sums into factors.
constexpr int kSum = 256;
constexpr int kSpread = 128;
constexpr int kSumWarps = kSum / 32;
constexpr int kAhead = 8;

// lr times the clip factor of tensor `seg`, by the first kSpread threads of a CTA; valid in all of them.
// W: floats per item.  Thread t adds the items t, t + kSpread, ..., then the threads' sums are added in a
// fixed order.
template <int W>
__device__ __forceinline__ float tensor_coef(const FoldParams& p, int seg, float* s_part) {
  float x = 0.f;
  const int lo = p.seg_first[seg], hi = p.seg_first[seg + 1];
  if (threadIdx.x < kSpread) {
#pragma unroll 2
    for (int i = lo + threadIdx.x; i < hi; i += kSpread) {
      const float* w = p.partial + (size_t)i * W;
      float t = 0.f;
#pragma unroll
      for (int j = 0; j < W; ++j) t += __ldcg(w + j);
      x += t;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) x += __shfl_xor_sync(0xffffffffu, x, d);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = x;
  }
  __syncthreads();
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < kSpread / 32; ++j) ss += s_part[j];
  return p.lr * (p.clip / fmaxf(sqrtf(ss), p.clip));
}

template <typename T, int kStrands>
__global__ void __launch_bounds__(kStrands) fold_sumsq_kernel(const __grid_constant__ FoldParams p) {
  __shared__ float s_w[kSumWarps];
  __shared__ uint32_t s_last;
  cx::pdl_wait();
  cx::pdl_trigger();
  const int item = blockIdx.x / (kSum / kStrands);
  const int strand = blockIdx.x % (kSum / kStrands) * kStrands + threadIdx.x;
  const int len = p.item_len[item], seg = p.item_seg[item];
  const T* g = reinterpret_cast<const T*>(p.seg_ptr[seg]) + p.item_rel[item];
  constexpr int kGroup = 16 / sizeof(T);
  float acc = 0.f;
  const uint64_t first = p.keep ? cx::keep_policy() : cx::plain_policy();
  if ((reinterpret_cast<uintptr_t>(g) & 15) == 0) {
    const uint4* g16 = reinterpret_cast<const uint4*>(g);
    const int nv = len / kGroup;
    for (int q = strand; q < nv; q += kAhead * kSum) {
      uint4 x[kAhead];
#pragma unroll
      for (int k = 0; k < kAhead; ++k) x[k] = q + k * kSum < nv ? cx::load_hint(g16 + q + k * kSum, first) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        const T* e16 = reinterpret_cast<const T*>(&x[k]);
#pragma unroll
        for (int e = 0; e < kGroup; ++e) {
          const float v = cx::Elem<T>::to_f(e16[e]);
          acc += v * v;
        }
      }
    }
    for (int i = nv * kGroup + strand; i < len; i += kSum) {
      const float x = cx::Elem<T>::to_f(g[i]);
      acc += x * x;
    }
  } else {
    for (int i = strand; i < len; i += kSum) {
      const float x = cx::Elem<T>::to_f(g[i]);
      acc += x * x;
    }
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
  if (kStrands < kSum) {
    if ((threadIdx.x & 31) == 0) p.partial[(size_t)item * kSumWarps + (strand >> 5)] = acc;
    const uint32_t ctas = (uint32_t)(p.seg_first[seg + 1] - p.seg_first[seg]) * (kSum / kStrands);
    if (!cx::cta_arrive(p.count + seg, ctas, &s_last)) return;
    const float c = tensor_coef<kSumWarps>(p, seg, s_w);
    if (threadIdx.x == 0) {
      p.coef[seg] = c;
      p.count[seg] = 0;
    }
    return;
  }
  if ((threadIdx.x & 31) == 0) s_w[strand >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < kSumWarps; ++w) t += s_w[w];
    p.partial[item] = t;
  }
}

// without clipping
__global__ void __launch_bounds__(kThreads) fold_coef_kernel(const __grid_constant__ FoldParams p) {
  cx::pdl_wait();
  cx::pdl_trigger();
  const int seg = blockIdx.x * kThreads + threadIdx.x;
  if (seg < p.segs) p.coef[seg] = p.lr;
}

template <typename T>
__global__ void __launch_bounds__(kThreads) fold_apply_kernel(const __grid_constant__ FoldParams p) {
  __shared__ float s_part[kSpread / 32];
  cx::pdl_wait();
  const int item = blockIdx.x;
  const int seg = p.item_seg[item];
  const float a = p.clip > 0.f ? tensor_coef<1>(p, seg, s_part) : p.lr;
  const int len = p.item_len[item];
  const T* g = reinterpret_cast<const T*>(p.seg_ptr[seg]) + p.item_rel[item];
  float* u = p.u + p.item_off[item];
  const bool vec = (reinterpret_cast<uintptr_t>(g) & (4 * sizeof(T) - 1)) == 0 &&
                   (reinterpret_cast<uintptr_t>(u) & 15) == 0;
  const int nv = vec ? len / 4 : 0;
#pragma unroll 4
  for (int q = threadIdx.x; q < nv; q += kThreads) {
    float x[4], y[4] = {0.f, 0.f, 0.f, 0.f};
    cx::load4(g + 4 * q, x);
    if (p.mu != 0.f) cx::load4(u + 4 * q, y);
#pragma unroll
    for (int e = 0; e < 4; ++e) y[e] = p.mu * y[e] + a * x[e];
    cx::store4(u + 4 * q, y);
  }
  for (int i = nv * 4 + threadIdx.x; i < len; i += kThreads) {
    const float y = p.mu != 0.f ? u[i] : 0.f;
    u[i] = p.mu * y + a * cx::Elem<T>::to_f(g[i]);
  }
}

template <typename T, int kStrands>
void launch_sumsq(const FoldParams& p, int items, cudaStream_t s) {
  cx_launch_pdl(fold_sumsq_kernel<T, kStrands>, items * (kSum / kStrands), kStrands, 0, s, p, cx_seq_cell() != nullptr);
  cx_note_launch();
}

template <int kStrands>
int sumsq(int gdtype, const FoldParams& p, int items, cudaStream_t s) {
  switch (gdtype) {
    case CX_F32: launch_sumsq<float, kStrands>(p, items, s); return 0;
    case CX_BF16: launch_sumsq<__nv_bfloat16, kStrands>(p, items, s); return 0;
    case CX_F16: launch_sumsq<__half, kStrands>(p, items, s); return 0;
    default: return cx_set_error("cx_fold: unsupported dtype on CUDA", 0);
  }
}

}  // namespace

int cx_fold_coef_cuda(int gdtype, const CxFoldCoef* f, void* stream) {
  if (f->segs <= 0) return 0;
  FoldParams p = {};
  p.seg_ptr = f->seg_ptr; p.item_rel = f->item_rel; p.item_len = f->item_len; p.item_seg = f->item_seg;
  p.seg_first = f->seg_first; p.partial = f->partial; p.coef = f->coef; p.count = f->count; p.segs = f->segs;
  p.clip = f->clip; p.lr = f->lr;
  p.keep = f->keep;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (f->clip > 0.f) {
    if (const int rc = sumsq<kSpread>(gdtype, p, f->items, s)) return rc;
  } else {
    cx_launch_pdl(fold_coef_kernel, (f->segs + kThreads - 1) / kThreads, kThreads, 0, s, p, cx_seq_cell() != nullptr);
    cx_note_launch();
  }
  cx_note_stream(stream, true);  // the norms read the gradients behind their trigger
  return cx_check_launch("fold kernels");
}

int cx_fold_cuda(int gdtype, const void* const* seg_ptr, const int64_t* item_off,
                 const int64_t* item_rel, const int32_t* item_len, const int32_t* item_seg,
                 const int32_t* seg_first, int nitems, float* u, float* partial, float clip,
                 float mu, float lr, void* stream) {
  if (nitems <= 0) return 0;
  FoldParams p = {};
  p.seg_ptr = seg_ptr; p.item_off = item_off; p.item_rel = item_rel; p.item_len = item_len;
  p.item_seg = item_seg; p.seg_first = seg_first; p.u = u; p.partial = partial;
  p.clip = clip; p.mu = mu; p.lr = lr;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (clip > 0.f)
    if (const int rc = sumsq<kSum>(gdtype, p, nitems, s)) return rc;
  const bool capturing = cx_seq_cell() != nullptr;
  switch (gdtype) {
    case CX_F32: cx_launch_pdl(fold_apply_kernel<float>, nitems, kThreads, 0, s, p, capturing); break;
    case CX_BF16: cx_launch_pdl(fold_apply_kernel<__nv_bfloat16>, nitems, kThreads, 0, s, p, capturing); break;
    case CX_F16: cx_launch_pdl(fold_apply_kernel<__half>, nitems, kThreads, 0, s, p, capturing); break;
    default: return cx_set_error("cx_fold: unsupported dtype on CUDA", 0);
  }
  cx_note_launch();
  return cx_check_launch("fold kernels");
}
