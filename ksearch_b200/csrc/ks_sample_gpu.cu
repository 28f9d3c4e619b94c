// The device half of sampling (crates/ksearch_gemma/src/sample.rs:9-81): which logits can matter at all.
//
// The reference samples on the host from all logits of a step.  A token whose soft-capped logit lies more than
// temperature * ln(1 / min_p) below the largest is dropped by the min-p filter, and the tokens that stay are few, so the
// device finds them (two passes over logits that are still in L2) and the host gets (index, value) pairs instead of a
// megabyte per slot.  The arithmetic of the draw stays the host's, on the same values.
//
// Bound by: two launches.  4 slots x 262144 f32 logits: see the table of timed cases.
#include <cuda_fp16.h>

#include "ks_internal.h"

namespace {

constexpr unsigned CAND_THREADS = 256, CAND_BLOCKS = 64;

__device__ __forceinline__ float ld(const float* p, size_t i) { return p[i]; }
__device__ __forceinline__ float ld(const __half* p, size_t i) { return __half2float(p[i]); }
// floats as integers of the same order (not for NaN)
__device__ __forceinline__ int ordered(float v) {
  const int b = __float_as_int(v);
  return b ^ ((b >> 31) & 0x7FFFFFFF);
}
__device__ __forceinline__ float from_ordered(int o) { return __int_as_float(o ^ ((o >> 31) & 0x7FFFFFFF)); }

__global__ void cand_init_kernel(ks_cand_head* head) {
  ks_pdl_entry();
  ks_cand_head h;
  h.count = 0;
  h.odd = 0;
  h.max_ordered = (int)0x80000000;
  h.pad = 0;
  head[threadIdx.x] = h;
}

template <typename T>
__global__ void __launch_bounds__(CAND_THREADS) cand_max_kernel(const T* logits, size_t n, ks_cand_head* head) {
  ks_pdl_entry();
  const T* row = logits + (size_t)blockIdx.y * n;
  int best = (int)0x80000000;
  bool odd = false;  // an infinity or NaN: the host takes the whole row
  for (size_t i = (size_t)blockIdx.x * CAND_THREADS + threadIdx.x; i < n; i += (size_t)CAND_BLOCKS * CAND_THREADS) {
    const float v = ld(row, i);
    odd |= !(fabsf(v) <= 3.4e38f);
    const int o = ordered(v);
    best = o > best ? o : best;
  }
  __shared__ int sb[CAND_THREADS / 32];
  best = __reduce_max_sync(0xffffffffu, best);
  if ((threadIdx.x & 31u) == 0) sb[threadIdx.x >> 5] = best;
  const int any = __syncthreads_or(odd);
  if (threadIdx.x == 0) {
    for (unsigned w = 1; w < CAND_THREADS / 32; w++) best = sb[w] > best ? sb[w] : best;
    atomicMax(&head[blockIdx.y].max_ordered, best);
    if (any) atomicOr(&head[blockIdx.y].odd, 1u);
  }
}

template <typename T>
__global__ void __launch_bounds__(CAND_THREADS) cand_list_kernel(const T* logits, size_t n, float cap, ks_cand_cut cuts, ks_cand_head* head, ks_cand* list) {
  ks_pdl_entry();
  const unsigned slot = blockIdx.y;
  __shared__ float s_cut;
  if (threadIdx.x == 0) {
    // the smallest logit whose soft-capped value reaches  max - temperature ln(1 / min_p), and a margin of 1e-5 of the cap
    // (or of the value) for what the host's float arithmetic rounds
    const double top = (double)from_ordered(head[slot].max_ordered), below = (double)cuts.below[slot];
    double cut;
    if (cap > 0.0f) {
      const double y = tanh(top / cap) - (below / cap + 1e-5);
      cut = y <= -1.0 ? -3.4e38 : (double)cap * atanh(y);
    } else {
      cut = top - below - 1e-5 * (1.0 + fabs(top));
    }
    s_cut = (float)cut;
  }
  __syncthreads();
  const float cut = s_cut;
  const T* row = logits + (size_t)slot * n;
  for (size_t i = (size_t)blockIdx.x * CAND_THREADS + threadIdx.x; i < n; i += (size_t)CAND_BLOCKS * CAND_THREADS) {
    const float v = ld(row, i);
    if (v >= cut) {
      const unsigned at = atomicAdd(&head[slot].count, 1u);
      if (at < KS_CAND_MAX) list[(size_t)slot * KS_CAND_MAX + at] = ks_cand{(unsigned)i, v};
    }
  }
}

}  // namespace

int ks_launch_candidates(ks_ctx* ctx, ks_dtype act, const void* logits, size_t n, int n_slots, float cap, const ks_cand_cut& cuts, ks_cand_head* head,
                         ks_cand* list) {
  KS_LAUNCH(ctx, cand_init_kernel, 1, (unsigned)n_slots, 0, head);
  int rc = ks_after_launch(ctx, "cand_init");
  if (rc) return rc;
  const dim3 grid(CAND_BLOCKS, (unsigned)n_slots);
  if (act == KS_F32) {
    KS_LAUNCH(ctx, cand_max_kernel<float>, grid, CAND_THREADS, 0, (const float*)logits, n, head);
    if ((rc = ks_after_launch(ctx, "cand_max"))) return rc;
    KS_LAUNCH(ctx, cand_list_kernel<float>, grid, CAND_THREADS, 0, (const float*)logits, n, cap, cuts, head, list);
  } else {
    KS_LAUNCH(ctx, cand_max_kernel<__half>, grid, CAND_THREADS, 0, (const __half*)logits, n, head);
    if ((rc = ks_after_launch(ctx, "cand_max"))) return rc;
    KS_LAUNCH(ctx, cand_list_kernel<__half>, grid, CAND_THREADS, 0, (const __half*)logits, n, cap, cuts, head, list);
  }
  return ks_after_launch(ctx, "cand_list");
}
