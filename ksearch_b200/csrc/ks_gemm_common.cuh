// Shared by the tensor-core GEMM kernels (ks_gemm_q4k.cu, ks_gemm.cu): the f16 image of the token rows, tcgen05 and TMA
// wrappers, and how a launch's work units are dealt to its CTAs.
#pragma once
#include <cuda_fp16.h>

#include "ks_fx.cuh"

constexpr int GM_ROWS = 128;  // weight rows per tile (M of the MMA)

// ---- work units ---------------------------------------------------------------------------------
// The Q4_K kernel cuts a launch into units: one super-block (256 columns) of `nt` neighbouring row tiles of a matrix against one
// block of `tbn` token rows.  Units are numbered column after column inside a work tile (row tiles x token block), the token
// blocks of the same row tiles next to each other, and every CTA gets a run of them: the first `rem` CTAs base + 1, the others
// base.  So no CTA has more than one unit more than another whatever the tile count, and a work tile whose units several CTAs
// share leaves one partial per CTA, in CTA order.  (Plain multiplications on purpose: what the MMA warp derives from them stays
// in uniform registers.)  G == 0: every tile has `splits` partials.
struct ks_gemm_map {
  unsigned G, S;          // CTAs, units per work tile
  unsigned base, rem;
  unsigned nt, tb, tbn;   // row tiles per unit, token blocks, token rows per block
  unsigned splits;
};
__host__ __device__ inline unsigned ks_gemm_first(const ks_gemm_map& m, unsigned cta) { return cta * m.base + (cta < m.rem ? cta : m.rem); }
__host__ __device__ inline unsigned ks_gemm_owner(const ks_gemm_map& m, unsigned u) {
  const unsigned big = m.rem * (m.base + 1u);
  return u < big ? u / (m.base + 1u) : m.rem + (u - big) / m.base;
}
// Partials of row tile `tile` (counted inside its matrix, whose first row-tile group is `group0`) for token row `t`.
__host__ __device__ inline unsigned ks_gemm_slots(const ks_gemm_map& m, unsigned group0, unsigned tile, unsigned t) {
  if (m.G == 0) return m.splits;
  const unsigned w = (group0 + tile / m.nt) * m.tb + t / m.tbn;
  return ks_gemm_owner(m, w * m.S + m.S - 1u) - ks_gemm_owner(m, w * m.S) + 1u;
}

namespace {

// 1 in exactly one lane of a converged warp.
__device__ __forceinline__ unsigned elect_one() {
  unsigned pred;
  asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(pred));
  return pred;
}
__device__ __forceinline__ uint32_t pack_h2(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
// Eight f32 values -> 16 bytes of hi and 16 bytes of lo halves (hi = rn(v), lo = rn(v - hi)).
__device__ __forceinline__ void split8(const float (&w)[8], uint4& hi, uint4& lo) {
  uint32_t h[4], l[4];
#pragma unroll
  for (int e = 0; e < 4; e++) {
    const __half2 hh = __floats2half2_rn(w[2 * e], w[2 * e + 1]);
    const float2 hf = __half22float2(hh);
    h[e] = pack_h2(hh);
    l[e] = pack_h2(__floats2half2_rn(w[2 * e] - hf.x, w[2 * e + 1] - hf.y));
  }
  hi = make_uint4(h[0], h[1], h[2], h[3]);
  lo = make_uint4(l[0], l[1], l[2], l[3]);
}
// The B image: chunk c (8 k), part p (0 hi, 1 lo), token t, 8 halves.  A chunk's hi and lo rows are neighbours, so one MMA
// can take both as 2 NP rows of B.  Two forms:
//   plain (Q6_K weights)   chunk = k / 8, elements in order;
//   q4k                    36 chunks per 256 k.  Chunks 0..31 are the values, elements 1 and 2 of every four swapped: the
//                          order in which masking the packed nibbles in place leaves the weights.  Chunks 32..35 carry the
//                          sub-block sums the minima multiply: chunk 32 + g holds, with S = 2^-5 (sum of a 32-value
//                          sub-block), (S_hi, S_hi', S_lo, S_lo', S_hi, S_hi', 0, 0) of sub-blocks 2 g and 2 g + 1.
//                          Token rows come in blocks of `tbn`, each an image like this of its own, one behind the other.
__device__ __forceinline__ void put_split8(__half* xt, unsigned np, unsigned tbn, unsigned t, unsigned ck, unsigned chunks, const float (&v)[8], bool q4k) {
  unsigned at = ck;
  if (q4k) {
    at = (ck >> 5) * 36u + (ck & 31u);
    const unsigned blk = t / tbn;
    t -= blk * tbn;
    xt += (size_t)(chunks / 32u * 36u) * 2u * (blk * tbn) * 8u;
    np = tbn;
    const float w[8] = {v[0], v[2], v[1], v[3], v[4], v[6], v[5], v[7]};
    uint4 hi, lo;
    split8(w, hi, lo);
    __half* base = xt + (size_t)at * 2u * np * 8u + (size_t)t * 8u;
    *reinterpret_cast<uint4*>(base) = hi;
    *reinterpret_cast<uint4*>(base + (size_t)np * 8u) = lo;
    // four neighbouring lanes hold a sub-block (all 32 lanes call: a row is a multiple of 256 values)
    float s = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    const float s1 = __shfl_xor_sync(0xffffffffu, s, 4);
    if ((ck & 7u) < 2u) {
      uint4 e = make_uint4(0u, 0u, 0u, 0u);
      if ((ck & 7u) == 0u) {
        const __half2 h = __floats2half2_rn(s * 0.03125f, s1 * 0.03125f);
        const float2 hf = __half22float2(h);
        e.x = pack_h2(h);
        e.y = pack_h2(__floats2half2_rn(s * 0.03125f - hf.x, s1 * 0.03125f - hf.y));
        e.z = e.x;
      }
      __half* ext = xt + (size_t)((ck >> 5) * 36u + 32u + ((ck & 31u) >> 3)) * 2u * np * 8u + (size_t)t * 8u;
      *reinterpret_cast<uint4*>(ext + ((ck & 7u) ? (size_t)np * 8u : 0)) = e;  // lane 1 clears the lo row
    }
    return;
  }
  uint4 hi, lo;
  split8(v, hi, lo);
  __half* base = xt + (size_t)at * 2u * np * 8u + (size_t)t * 8u;
  *reinterpret_cast<uint4*>(base) = hi;
  *reinterpret_cast<uint4*>(base + (size_t)np * 8u) = lo;
}

// The same for passes of many rows: a warp holds 64 columns (chunks ck0 .. ck0 + 7, ck0 a multiple of 8) of four neighbouring token
// rows, lane = row t0 + lane % 4 (t0 a multiple of 4), chunk ck0 + lane / 4.  A chunk's four rows are then 64 neighbouring bytes of
// the q4k image; one row per block leaves a warp's 16-byte stores in 32 lines, 4 KB apart.  The sums are added in the order of put_split8.
__device__ __forceinline__ void put_split8_rows4(__half* xt, unsigned tbn, unsigned t0, unsigned ck0, unsigned chunks, const float (&v)[8]) {
  const unsigned lane = threadIdx.x & 31u, c = lane >> 2, ck = ck0 + c, blk = t0 / tbn, t = t0 - blk * tbn + (lane & 3u);
  xt += (size_t)(chunks / 32u * 36u) * 2u * (blk * tbn) * 8u + (size_t)t * 8u;
  const float w[8] = {v[0], v[2], v[1], v[3], v[4], v[6], v[5], v[7]};
  uint4 hi, lo;
  split8(w, hi, lo);
  __half* base = xt + (size_t)((ck >> 5) * 36u + (ck & 31u)) * 2u * tbn * 8u;
  *reinterpret_cast<uint4*>(base) = hi;
  *reinterpret_cast<uint4*>(base + (size_t)tbn * 8u) = lo;
  float s = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
  s += __shfl_xor_sync(0xffffffffu, s, 4);
  s += __shfl_xor_sync(0xffffffffu, s, 8);
  const float s1 = __shfl_xor_sync(0xffffffffu, s, 16);
  if (c < 2u) {
    uint4 e = make_uint4(0u, 0u, 0u, 0u);
    if (c == 0u) {
      const __half2 h = __floats2half2_rn(s * 0.03125f, s1 * 0.03125f);
      const float2 hf = __half22float2(h);
      e.x = pack_h2(h);
      e.y = pack_h2(__floats2half2_rn(s * 0.03125f - hf.x, s1 * 0.03125f - hf.y));
      e.z = e.x;
    }
    __half* ext = xt + (size_t)((ck0 >> 5) * 36u + 32u + ((ck0 & 31u) >> 3)) * 2u * tbn * 8u;
    *reinterpret_cast<uint4*>(ext + (c ? (size_t)tbn * 8u : 0)) = e;  // chunk 1's lanes clear the lo row
  }
}

// Range.  f16 ends at 65504 and loses its low term below ~1e-3 (the low half of a small value is a denormal);
// activations do neither.  Every token row is therefore stored as x * 2^-e with e = exponent(largest magnitude) - 14,
// so the scaled row peaks in [2^14, 2^15), and the GEMM multiplies that token's outputs by 2^e (both exact).
// The factors 2^e sit behind the image, one float per (padded) token row; an all-zero row keeps e = 0.
__device__ __host__ __forceinline__ size_t xt_scale_off(unsigned cols, unsigned np) { return (size_t)(cols / 256u * 288u) * np * 2u; }  // in halves; either form
__device__ __forceinline__ float row_scale_down(float row_max, float* scale_up) {
  int e = 0;
  if (row_max > 0.0f && row_max < 3.0e38f) {
    e = (int)((__float_as_uint(row_max) >> 23) & 0xFFu) - 127 - 14;
    e = e < -100 ? -100 : e;  // 2^-e must stay a float
  }
  *scale_up = __uint_as_float((unsigned)(127 + e) << 23);
  return __uint_as_float((unsigned)(127 - e) << 23);
}
__device__ __forceinline__ float block_max_f(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = (lane < nwarp) ? red[lane] : 0.0f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, o));
  return t;
}
__device__ __forceinline__ float absmax8(const float (&v)[8]) {
  return fmaxf(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))),
               fmaxf(fmaxf(fabsf(v[4]), fabsf(v[5])), fmaxf(fabsf(v[6]), fabsf(v[7]))));
}

// ---- tcgen05 wrappers ---------------------------------------------------------------------------
__device__ __forceinline__ void tc_alloc(uint32_t slot_smem, unsigned cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_smem), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(uint32_t taddr, unsigned cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// D[tmem] (+)= A[smem desc] . B[smem desc]^T, f16 inputs, f32 accumulation; one thread issues.
__device__ __forceinline__ void tc_mma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The same with A in tensor memory (lane = row, column = two neighbouring k).
__device__ __forceinline__ void tc_mma_f16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_st8(uint32_t taddr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]),
               "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
__device__ __forceinline__ void tc_st4(uint32_t taddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 4 or 16 consecutive f32 columns of this warp's 32 lanes; the values are there after tc_wait_ld16, which names the registers so
// that nothing that reads them moves in front of it.
__device__ __forceinline__ void tc_ld4(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                 "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tc_wait_ld16(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                 "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}
// A box of a 2-D tensor map into shared memory (x in elements of the map, here bytes: a multiple of 16).
__device__ __forceinline__ void tma_in_2d(uint32_t dst, const void* map, unsigned x, unsigned y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
               "l"(map), "r"(x), "r"(y), "r"(bar)
               : "memory");
}
// 8 consecutive f32 columns of this warp's 32 lanes.
__device__ __forceinline__ void tc_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// Shared-memory operand descriptor, K-major, no swizzle: 8-row x 16-byte core matrices; `lbo` = bytes between the
// two 8-k chunks of one MMA, `sbo` = bytes between 8-row groups.
__device__ __forceinline__ uint64_t tc_desc(uint32_t smem_addr, unsigned lbo, unsigned sbo) {
  return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) | ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) |
         (1ull << 46);
}

}  // namespace
