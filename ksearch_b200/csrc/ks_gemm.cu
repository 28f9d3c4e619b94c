// Q6_K weights x a batch of 9..256 token rows on the tensor cores (tcgen05), the images of the token rows and the
// epilogues of both GEMM kernels (Q4_K weights: ks_gemm_q4k.cu).
//
// The reference routes matvec_batch with more than 8 rows (crates/ksearch_kernels/src/lib.rs:1414) to its
// mul_mm kernel (crates/ksearch_codegen/src/render.rs:1073-1291: 64x32 tiles, weights dequantised to half in
// threadgroup memory, simdgroup 8x8 MMA).  Here one CTA owns 128 weight rows and ALL token rows:
//   D[weight row, token] (f32, in tensor memory)  +=  A[128 rows, 16 k] . B[tokens, 16 k]^T
// with the weight rows as the M side of the MMA, so 9 tokens cost as little tensor work as the instruction
// allows (N = 16) and 256 tokens fill it (N = 256).
//   * B (token rows) is prepared once per call by x_split_kernel: every f32 x is split into two f16 terms
//     (hi = rn(x), lo = rn(x - hi)) and stored k-step by k-step in exactly the shared-memory image the MMA wants
//     (8x8 core matrices, K-major, no swizzle; per 8-k chunk the hi rows of all tokens, then the lo rows), so a
//     k-step of B is ONE cp.async.bulk into the stage.
//   * A (weights) is dequantised by the CTA's 512 threads, a quarter of a row's k-step (16 weights) each, in half2
//     arithmetic straight from the packed bytes (gguf_impl.rs:761-791; see dequant_to_stage): two f16 terms that add up
//     to the f32 weight (times 2^6, exact) to 2^-17, stored as core matrices.
//   * Products: Ahi.Bhi + Ahi.Blo + Alo.Bhi; the dropped lo.lo term is below 2^-22 relative, so the result matches
//     f32 arithmetic (the reference's single half operands give ~1e-3).  Up to 128 token rows the first two are ONE
//     MMA over 2 NP rows of B (the hi and lo rows of a chunk are neighbours): the accumulator has 2 NP columns, the
//     epilogue adds the halves, and the tensor core fetches the A tile twice per 16 k instead of three times.
//   * Warp-specialised: 16 warps dequantise into two A stages and signal each one full on an mbarrier (one arrival
//     per warp); the first lane of a 17th warp waits for both operands of a step, issues its MMAs and lets
//     tcgen05.commit release the step's A and B stage on one mbarrier; the first lane of an 18th warp requests the
//     token rows (ring of two or four stages) as those mbarriers complete.  No block-wide barrier inside the k
//     loop; the packed weights are fetched two k-steps ahead into registers.  The accumulator is read back with
//     tcgen05.ld, scaled by 2^-6 and stored coalesced along the weight-row index.
// Every wait is bounded; on expiry the CTA raises the context's status word, waits (bounded) for what it has in
// flight, frees its tensor memory and returns.
#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include <cstdlib>

#include "ks_gemm.h"

namespace {

constexpr int GM_KSTEP = 64;        // k per stage: half of a Q6_K 128-run
constexpr int GM_THREADS = 512;     // dequantising threads: four per weight row and k-step (two more warps: MMAs, copies)
constexpr unsigned GM_A_BYTES = 2u * 8u * GM_ROWS * 16u;  // hi + lo, 8 k-chunks, 128 rows, 16 bytes: 32 KB
constexpr unsigned GM_WAIT = 1u << 20;
constexpr float GM_SCALE = 64.0f;   // weights carry 2^6: keeps the low f16 term of small weights out of the denormal
                                    // range and the high term finite up to |w| = 1000

struct GemmArgs {
  // up to three matrices over the same columns and token rows in one launch (q, k, v; gate, up): matrix i owns
  // the row tiles [tile0[i], tile0[i + 1])
  const uint8_t* W[3];
  float* y[3];            // y[i][token * ldy[i] + row]
  size_t ldy[3];
  size_t part_stride[3];  // floats between the outputs of consecutive k splits
  unsigned rows[3], tile0[4];
  size_t row_bytes;
  const __half* xt;   // [chunks of 8 k][2][NP][8] halves
  unsigned cols, n_tok, np;        // np: token count padded to a multiple of 16 (<= 256)
  unsigned tmem_cols;              // power of two >= max(32, accumulator columns)
  unsigned ksteps_per;             // k-steps per CTA (grid.y splits the k range)
  unsigned nb;                     // stages (2..4) of the A ring and of the B ring
  unsigned wait_limit;             // polls before a wait inside the kernel gives up
  unsigned test_stall;             // test hook: the token rows of k-step test_stall - 1 of every CTA are never requested
  unsigned* err;
};

// x[token, k] (f32, row stride ldx) -> the B image.  One block per (padded) token row; rows past n_tok become zeros.
__device__ __forceinline__ void x_chunk(const float* row, unsigned ck, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(row + (size_t)ck * 8u), b = *reinterpret_cast<const float4*>(row + (size_t)ck * 8u + 4u);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
// ONE: a thread per chunk, which it reads once (rows of up to 8192 values: one trip to memory, and no more warps than there is work for;
// with the partial counts of the sums behind it worked out early, 55 rows against 4096x1536 in three launches 12.9 -> 10.6 us).
template <bool ONE>
__global__ void __launch_bounds__(1024) x_split_kernel(const float* x, size_t ldx, unsigned n_tok, unsigned np, unsigned tbn, unsigned cols, __half* xt, int q4k) {
  ks_pdl_entry();
  __shared__ float red[32];
  const unsigned t = blockIdx.x, chunks = cols / 8u;
  const bool live = t < n_tok;
  const float* row = x + (size_t)t * ldx;
  float m = 0.0f, v[8];
#pragma unroll
  for (int e = 0; e < 8; e++) v[e] = 0.0f;
  if (live) {
    if constexpr (ONE) {
      x_chunk(row, threadIdx.x, v);
      m = absmax8(v);
    } else {
      for (unsigned ck = threadIdx.x; ck < chunks; ck += blockDim.x) {
        x_chunk(row, ck, v);
        m = fmaxf(m, absmax8(v));
      }
    }
  }
  m = block_max_f(m, red);
  float up;
  const float down = row_scale_down(m, &up);
  if (threadIdx.x == 0) reinterpret_cast<float*>(xt + xt_scale_off(cols, np))[t] = up;
  for (unsigned ck = threadIdx.x; ck < chunks; ck += blockDim.x) {
    if (!ONE && live) x_chunk(row, ck, v);
    float w[8];
#pragma unroll
    for (int e = 0; e < 8; e++) w[e] = v[e] * down;  // (zeros past n_tok)
    put_split8(xt, np, tbn, t, ck, chunks, w, q4k != 0);
  }
}

// The packed bytes one thread needs for one k-step, fetched two steps ahead of their use.  Thread (row, quarter qd)
// owns weights [64 ks + 16 qd, +16) of its row: chunks 2 qd and 2 qd + 1 of the stage.
struct Raw {
  uint32_t ql[4], qh[4];  // the 16 bytes that hold the quarter's nibbles, the 16 bytes that hold its bit pairs
  float ds;               // 2^6 d sc of the quarter's 16-run
};

// A read-only load the compiler must issue where it is written (it may not sink it towards the first use, which is
// two k-steps later): the weights have to be in flight while the steps before them are converted.
__device__ __forceinline__ uint32_t ldg_now32(const void* p) {
  uint32_t v;
  asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
// 16 bytes from a 2-byte-aligned address: five aligned words, shifted into place (the fifth lies inside the same
// 210-byte block wherever this is used).
__device__ __forceinline__ void load16_a2(const uint8_t* p, uint32_t (&o)[4]) {
  const unsigned sh = 8u * (unsigned)((uintptr_t)p & 3u);
  const uint32_t* q = reinterpret_cast<const uint32_t*>(p - (sh >> 3));
  const uint32_t x0 = ldg_now32(q), x1 = ldg_now32(q + 1), x2 = ldg_now32(q + 2), x3 = ldg_now32(q + 3), x4 = ldg_now32(q + 4);
  o[0] = __funnelshift_r(x0, x1, sh);
  o[1] = __funnelshift_r(x1, x2, sh);
  o[2] = __funnelshift_r(x2, x3, sh);
  o[3] = __funnelshift_r(x3, x4, sh);
}
// Q6_K: block = ql[128] qh[64] scales[16] d; a 128-run holds four groups g of 32 (gguf_impl.rs:761-791):
// group g takes nibble g >> 1 of ql[32 (g & 1) + l] and bits 2g, 2g + 1 of qh[l]; scale index 2g + (l >> 4).
__device__ __forceinline__ void load_raw(const uint8_t* W, size_t row_bytes, unsigned row, unsigned qd, unsigned ks, Raw& w) {
  const uint8_t* blk = W + (size_t)row * row_bytes + (size_t)(ks >> 2) * 210u;  // blocks are 2-byte aligned
  const unsigned n = (ks >> 1) & 1u, g = 2u * (ks & 1u) + (qd >> 1), sub = qd & 1u;
  load16_a2(blk + 64u * n + 32u * (g & 1u) + 16u * sub, w.ql);
  load16_a2(blk + 128u + 32u * n + 16u * sub, w.qh);
  const int8_t sc = *reinterpret_cast<const int8_t*>(blk + 192u + 8u * n + 2u * g + sub);
  w.ds = __half2float(*reinterpret_cast<const __half*>(blk + 208u)) * GM_SCALE * (float)sc;
}

// The thread's 16 weights into chunks 2 qd, 2 qd + 1 of the A stage (hi and lo halves).
__device__ __forceinline__ void dequant_to_stage(const Raw& w, bool live, unsigned qd, unsigned ks, unsigned char* A, unsigned r) {
  uint4* Ahi = reinterpret_cast<uint4*>(A) + (size_t)(2u * qd) * GM_ROWS + r;
  uint4* Alo = Ahi + (size_t)8u * GM_ROWS;
  if (!live) {  // rows past the matrix: zeros (their outputs are not stored)
#pragma unroll
    for (int cc = 0; cc < 2; cc++) {
      Ahi[(size_t)cc * GM_ROWS] = make_uint4(0, 0, 0, 0);
      Alo[(size_t)cc * GM_ROWS] = make_uint4(0, 0, 0, 0);
    }
    return;
  }
  // (2^6 d sc) q in half2 arithmetic: the f32 scale A is cut into A1 = A rounded to 6 significant bits (A1 q is
  // exact in f16 for q in -32..31) and A2 = A - A1 (at most 11 significant bits: exact in f16); q + 32 comes out of
  // the packed bytes as the half 0x5400 | (q + 32) << 4 = 64 + (q + 32) by one byte permute and one OR; one exact
  // add makes it q, and two multiplies give hi = A1 q (exact) and lo = rn(A2 q): hi + lo is A q to 2^-17.
  const unsigned g = 2u * (ks & 1u) + (qd >> 1);
  const __half a1 = __float2half_rn(__uint_as_float((__float_as_uint(w.ds) + 0x00020000u) & 0xFFFC0000u));
  const __half2 s1 = __half2half2(a1), s2 = __half2half2(__float2half_rn(w.ds - __half2float(a1)));
  const __half2 bias = __float2half2_rn(-96.0f);
  const unsigned shl = 4u * (1u - (g >> 1)), shh = 2u * g;
  uint32_t hi[8], lo[8];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t tl = (w.ql[k] << shl) & 0xF0F0F0F0u;   // the nibble at bits 4..7 of its byte
    const uint32_t th = (w.qh[k] >> shh) & 0x03030303u;   // the bit pair at bits 0..1: bits 8..9 of the half
    const __half2 p0 = __hadd2(as_h2(__byte_perm(tl, th, 0x5140u) | 0x54005400u), bias);
    const __half2 p1 = __hadd2(as_h2(__byte_perm(tl, th, 0x7362u) | 0x54005400u), bias);
    hi[2 * k] = pack_h2(__hmul2(p0, s1));
    hi[2 * k + 1] = pack_h2(__hmul2(p1, s1));
    lo[2 * k] = pack_h2(__hmul2(p0, s2));
    lo[2 * k + 1] = pack_h2(__hmul2(p1, s2));
  }
#pragma unroll
  for (int cc = 0; cc < 2; cc++) {
    Ahi[(size_t)cc * GM_ROWS] = make_uint4(hi[4 * cc], hi[4 * cc + 1], hi[4 * cc + 2], hi[4 * cc + 3]);
    Alo[(size_t)cc * GM_ROWS] = make_uint4(lo[4 * cc], lo[4 * cc + 1], lo[4 * cc + 2], lo[4 * cc + 3]);
  }
}

// grid = (row tiles, k splits): CTA (bx, by) multiplies rows [128 bx, +128) over k-steps [by * per, (by + 1) * per)
// and stores its sums at y + by * part_stride (a partial when there is more than one split).
// Warps 0..15 dequantise; an elected lane of warp 16 issues the MMAs; an elected lane of warp 17 requests the token rows.  Step i uses
// stage i % nb of the A ring and of the B ring (nb = 2..4); its MMAs commit to free[i % nb], which releases both.
__global__ void __launch_bounds__(GM_THREADS + 64, 2) gemm_q6k_tc_kernel(const GemmArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  // [0,32): mbarriers fullB[4]; [32,64): free[4]; [64,72): done; [72,104): fullA[4]; [104,108): tensor-memory address;
  // [108,112): failure flag; from 1024: the A stages, then the B stages
  const uint32_t bars = sm32(smem);
  const uint32_t bar_free = bars + 32u, bar_done = bars + 64u, bar_fullA = bars + 72u;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + 104);
  volatile unsigned* fail = reinterpret_cast<volatile unsigned*>(smem + 108);  // a bounded wait gave up somewhere in the CTA
  const unsigned b_bytes = a.np * 256u;                 // 8 chunks, hi + lo, np tokens, 16 bytes
  unsigned char* A0 = smem + 1024;
  const unsigned nb = a.nb;
  unsigned char* B0 = A0 + (size_t)nb * GM_A_BYTES;
  const unsigned tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
  // a producer warp takes 8 rows x 4 quarters: its 32 loads of a k-step fall into 8 runs of contiguous bytes, and the
  // 8 lanes that store together (same quarter) write 128 contiguous bytes
  const unsigned r = ((warp << 3) | (tid & 7u)) & (GM_ROWS - 1), qd = (tid >> 3) & 3u;
  // which matrix this row tile belongs to (selects, no dynamic indexing of the parameter arrays)
  const unsigned bx = blockIdx.x;
  const int seg = (bx >= a.tile0[1]) + (bx >= a.tile0[2]);
  const uint8_t* W = seg == 0 ? a.W[0] : seg == 1 ? a.W[1] : a.W[2];
  const unsigned seg_rows = seg == 0 ? a.rows[0] : seg == 1 ? a.rows[1] : a.rows[2];
  const size_t ldy = seg == 0 ? a.ldy[0] : seg == 1 ? a.ldy[1] : a.ldy[2];
  const size_t part_stride = seg == 0 ? a.part_stride[0] : seg == 1 ? a.part_stride[1] : a.part_stride[2];
  const unsigned row_base = (bx - (seg == 0 ? a.tile0[0] : seg == 1 ? a.tile0[1] : a.tile0[2])) * GM_ROWS;
  const unsigned row = row_base + r;
  const bool live = row < seg_rows;
  const unsigned ks0 = blockIdx.y * a.ksteps_per, ks1 = min(ks0 + a.ksteps_per, a.cols / GM_KSTEP);
  const unsigned ksteps = ks1 - ks0;
  float* yout = (seg == 0 ? a.y[0] : seg == 1 ? a.y[1] : a.y[2]) + (size_t)blockIdx.y * part_stride;

  // weights do not depend on the kernels before this one: the first two k-steps are fetched right away
  const bool producer = warp < GM_THREADS / 32;
  Raw raw0, raw1;
  if (producer && live) {
    load_raw(W, a.row_bytes, row, qd, ks0, raw0);
    if (ksteps > 1) load_raw(W, a.row_bytes, row, qd, ks0 + 1, raw1);
  }
  if (tid == 0) {
    for (int i = 0; i < 9; i++) mb_init(bars + 8u * i, 1);                    // fullB[4], free[4], done: one arrival each
    for (int i = 0; i < 4; i++) mb_init(bar_fullA + 8u * i, GM_THREADS / 32);  // fullA[4]: one arrival per producer warp
    *fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tc_alloc(sm32(tslot), a.tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  ks_pdl_entry();  // the B image comes from the kernel before this one

  if (producer) {
    // ---- 16 warps: packed weights -> two f16 terms -> A stage; no block-wide barrier inside the loop
    for (unsigned i = 0; i < ksteps; i++) {
      const unsigned ks = ks0 + i, s = i % nb;
      unsigned char* A = A0 + (size_t)s * GM_A_BYTES;
      if (i >= nb && !mb_wait(bar_free + 8u * s, (i / nb - 1u) & 1u, a.wait_limit)) {  // the MMAs of step i - nb still read this stage
        *fail = 1;
        break;
      }
      const Raw cur = raw0;
      raw0 = raw1;
      if (live && i + 2 < ksteps) load_raw(W, a.row_bytes, row, qd, ks + 2, raw1);  // in flight while two steps are converted
      dequant_to_stage(cur, live, qd, ks, A, r);
      __syncwarp();
      if (lane == 0) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the warp's generic-proxy stores of A, then the tensor core's reads
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_fullA + 8u * s) : "memory");
      }
    }
  } else if (warp == GM_THREADS / 32) {
    // ---- the MMAs of a step as soon as both operands are there.  The whole warp runs the loop, converged, and one
    // elected lane issues: the loop state and the 64-bit descriptors then live in uniform registers, which is where
    // tcgen05.mma reads them (computed inside a one-lane branch they are moved there one by one, ~150 cycles per MMA).
    const unsigned leader = elect_one();
    const uint32_t idesc = (1u << 4) | ((a.np >> 3) << 17) | ((unsigned)(GM_ROWS >> 4) << 24);  // f32 accumulate, f16 x f16, K-major both
    // up to 128 token rows: the hi and lo rows of B go through ONE instruction as 2 NP rows (columns [0, NP) take
    // Ahi.Bhi, columns [NP, 2 NP) Ahi.Blo), so the tensor core fetches the A tile twice per 16 k instead of three times
    const bool cat = a.np <= 128u;
    const uint32_t idesc2 = (1u << 4) | ((a.np >> 2) << 17) | ((unsigned)(GM_ROWS >> 4) << 24);
    // descriptors of the first chunk pair of stage 0; the address field counts 16-byte units and shared memory ends
    // below its 14 bits, so the other stages and chunks are plain additions
    const uint64_t a_desc0 = tc_desc(sm32(A0), GM_ROWS * 16u, 128u), b_desc0 = tc_desc(sm32(B0), 2u * a.np * 16u, 128u);
    bool ok = true;
    for (unsigned i = 0; i < ksteps; i++) {
      const unsigned t = i % nb, s = t;
      const bool got = mb_wait(bars + 8u * t, (i / nb) & 1u, a.wait_limit) && mb_wait(bar_fullA + 8u * s, (i / nb) & 1u, a.wait_limit);
      if (!__all_sync(0xffffffffu, got)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const uint64_t a_hi = a_desc0 + (uint64_t)(s * (GM_A_BYTES >> 4)), b_hi = b_desc0 + (uint64_t)(t * (b_bytes >> 4));
      if (leader) {
#pragma unroll
        for (unsigned j = 0; j < 4; j++) {  // 16 k each: chunks 2j, 2j+1
          const uint64_t ah = a_hi + (uint64_t)(2u * j * GM_ROWS);
          const uint64_t al = ah + (uint64_t)(8u * GM_ROWS);
          const uint64_t bh = b_hi + (uint64_t)(4u * j * a.np);  // chunk 2j: 2 NP rows of 16 bytes each
          if (cat) {
            tc_mma_f16(tmem, ah, bh, idesc2, (i | j) ? 1u : 0u);
          } else {
            tc_mma_f16(tmem, ah, bh, idesc, (i | j) ? 1u : 0u);
            tc_mma_f16(tmem, ah, bh + (uint64_t)a.np, idesc, 1u);
          }
          tc_mma_f16(tmem, al, bh, idesc, 1u);
        }
        tc_commit(bar_free + 8u * t);
        if (i + 1 == ksteps) tc_commit(bar_done);
      }
      __syncwarp();
    }
    if (!ok) {
      // every MMA issued so far must finish before shared and tensor memory go away (bounded): a fresh commit tracks them all
      if (leader) {
        *fail = 1;
        tc_commit(bar_done);
      }
      __syncwarp();
      mb_wait(bar_done, 0u, a.wait_limit);
    }
  } else if (warp == GM_THREADS / 32 + 1) {
    // ---- token rows of step j into B stage j % nb, as soon as the MMAs of step j - nb are done (whole warp in the
    // loop, one elected lane issues)
    const unsigned leader = elect_one();
    unsigned issued = 0;
    for (unsigned j = 0; j < ksteps; j++) {
      const bool got = j < nb || mb_wait(bar_free + 8u * (j % nb), (j / nb - 1u) & 1u, a.wait_limit);
      if (!__all_sync(0xffffffffu, got)) {
        if (leader) *fail = 1;
        break;
      }
      const bool withheld = a.test_stall && j + 1 == a.test_stall;  // test hook: this step's token rows never arrive
      if (leader) {
        const uint32_t fb = bars + 8u * (j % nb);
        mb_expect(fb, b_bytes);
        if (!withheld) bulk_in(sm32(B0 + (size_t)(j % nb) * b_bytes), a.xt + (size_t)(ks0 + j) * (b_bytes / 2u), b_bytes, fb);
      }
      if (withheld) break;  // nothing to wait for at the end either
      issued++;
      __syncwarp();
    }
    // the copies must have landed before this CTA's shared memory goes away (bounded; all done already unless a wait gave up)
    for (unsigned j = issued > nb ? issued - nb : 0u; j < issued; j++) mb_wait(bars + 8u * (j % nb), (j / nb) & 1u, a.wait_limit);
  }
  __syncthreads();
  bool ok = *fail == 0;
  // all MMAs done (tcgen05.commit tracks every MMA issued before it)
  if (ok && !mb_wait(bar_done, 0u, a.wait_limit)) ok = false;
  tc_fence_after();
  if (ok && producer) {
    // warp w reads lanes 32 (w % 4) .. +31; the four warps of a lane quarter take every fourth 8-column group
    const unsigned lane_base = (warp & 3u) * 32u;
    const unsigned out_row = row_base + lane_base + lane;
    const float* up = reinterpret_cast<const float*>(a.xt + xt_scale_off(a.cols, a.np));  // 2^e of every token row
    for (unsigned c0 = (warp >> 2) * 8u; c0 < a.np; c0 += 32u) {
      uint32_t v[8], v2[8];
      tc_ld8(tmem + (lane_base << 16) + c0, v);
      if (a.np <= 128u) {
        tc_ld8(tmem + (lane_base << 16) + a.np + c0, v2);  // the columns that took Ahi.Blo
      } else {
#pragma unroll
        for (unsigned e = 0; e < 8; e++) v2[e] = 0u;
      }
      if (out_row < seg_rows) {
#pragma unroll
        for (unsigned e = 0; e < 8; e++)
          if (c0 + e < a.n_tok)
            yout[(size_t)(c0 + e) * ldy + out_row] = (__uint_as_float(v[e]) + __uint_as_float(v2[e])) * ((1.0f / GM_SCALE) * up[c0 + e]);
      }
    }
  } else if (!ok && tid == 0) {
    atomicOr(a.err, 8u);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tc_dealloc(tmem, a.tmem_cols);
}

// Sum of the k-split partials in split order (the result does not depend on how the CTAs were scheduled) into y[i], for up
// to three matrices.
struct FinishArgs {
  const float* P[3];
  float* y[3];
  size_t ldy[3], part_stride[3];
  unsigned rows[3], tile0[3], group0[3], n_seg, n_tok;
  ks_gemm_map map;
};
// One block per row tile and a few token rows (the tile's partial count is the block's); a thread sums four neighbouring rows
// where row counts and addresses allow 16-byte accesses, else one.
template <int V>
struct FinVec {
  float v[V];
};
template <int V>
__device__ __forceinline__ FinVec<V> sum_slots(const float* P, size_t stride, unsigned n, size_t at) {
  FinVec<V> g;
#pragma unroll
  for (int k = 0; k < V; k++) g.v[k] = 0.0f;
#pragma unroll 4
  for (unsigned s = 0; s < n; s++) {
    const float* p = P + (size_t)s * stride + at;
    if constexpr (V == 4) {
      const float4 a = *reinterpret_cast<const float4*>(p);
      g.v[0] += a.x; g.v[1] += a.y; g.v[2] += a.z; g.v[3] += a.w;
    } else {
      g.v[0] += *p;
    }
  }
  return g;
}
template <int V>
__global__ void __launch_bounds__(256) gemm_finish_kernel(const FinishArgs f) {
  constexpr unsigned PER = GM_ROWS / V, TOK = 256u / PER;  // threads per token row, token rows per block
  const unsigned bx = blockIdx.x, seg = (bx >= f.tile0[1]) + (bx >= f.tile0[2]);
  const unsigned rows = seg == 0 ? f.rows[0] : seg == 1 ? f.rows[1] : f.rows[2];
  const unsigned tile0 = seg == 0 ? f.tile0[0] : seg == 1 ? f.tile0[1] : f.tile0[2];
  const float* P = seg == 0 ? f.P[0] : seg == 1 ? f.P[1] : f.P[2];
  const size_t ps = seg == 0 ? f.part_stride[0] : seg == 1 ? f.part_stride[1] : f.part_stride[2];
  const size_t ldy = seg == 0 ? f.ldy[0] : seg == 1 ? f.ldy[1] : f.ldy[2];
  float* y = seg == 0 ? f.y[0] : seg == 1 ? f.y[1] : f.y[2];
  const unsigned t = blockIdx.y * TOK + threadIdx.x / PER, r = (bx - tile0) * GM_ROWS + (threadIdx.x % PER) * V;
  if (t >= f.n_tok || r >= rows) return;
  const size_t at = (size_t)t * rows + r;  // partials are dense [split][token][row]
  const unsigned group0 = seg == 0 ? f.group0[0] : seg == 1 ? f.group0[1] : f.group0[2];
  const unsigned slots = ks_gemm_slots(f.map, group0, bx - tile0, t);  // (half a dozen divisions: in front of the wait)
  ks_pdl_entry();
  const FinVec<V> g = sum_slots<V>(P, ps, slots, at);
  float* o = y + (size_t)t * ldy + r;
  if constexpr (V == 4) *reinterpret_cast<float4*>(o) = make_float4(g.v[0], g.v[1], g.v[2], g.v[3]);
  else *o = g.v[0];
}

}  // namespace

namespace {
// The sum of a matrix's k-split partials straight into what consumes it, one block per token row:
//   y = sum of partials;  x = res + rms(y) * w_post (lower.rs:3926-4077, the residual update of lib.rs:539);
//   the image of rms(x) * w_norm for the next GEMM.
// The f32 normed vector is not stored: on this path only a GEMM reads it.  Rows past n_tok become zeros.
// Eight neighbouring rows of a token's partials, FLY partials in flight at a time: read one after the other, the partials of a
// down-projection (12 row tiles over 148 CTAs: 13 each) cost 13 trips to L2, 9 us a launch instead of 5.
template <unsigned FLY>
__device__ __forceinline__ void sum8(const float* p, size_t stride, unsigned n, float (&y)[8]) {
#pragma unroll
  for (int i = 0; i < 8; i++) y[i] = 0.0f;
  for (unsigned s = 0; s < n; s += FLY) {
    float4 a[FLY], b[FLY];
#pragma unroll
    for (unsigned k = 0; k < FLY; k++)
      if (s + k < n) {
        a[k] = *reinterpret_cast<const float4*>(p + (size_t)(s + k) * stride);
        b[k] = *reinterpret_cast<const float4*>(p + (size_t)(s + k) * stride + 4);
      }
#pragma unroll
    for (unsigned k = 0; k < FLY; k++)
      if (s + k < n) {
        y[0] += a[k].x; y[1] += a[k].y; y[2] += a[k].z; y[3] += a[k].w;
        y[4] += b[k].x; y[5] += b[k].y; y[6] += b[k].z; y[7] += b[k].w;
      }
  }
}
struct EpiNormArgs {
  const float* P;
  size_t part_stride;
  ks_gemm_map map;
  unsigned n_tok, np, tbn, rows;  // np, tbn: blocks of the image written
  int q4k;      // its form
  const float *res, *w_post, *w_norm;
  float eps;
  float* out_x;
  __half* xt;
};
constexpr size_t GM_NORM_AHEAD = 3u << 18;  // values of a launch up to which the weights come early
constexpr size_t GM_NORM_MOST = 8 * 1024;  // the longest rows: eight values per thread
// THREADS: at most; more than 512 have half the registers each.  AHEAD: the norm weights are asked for with the first partials: with few
// rows that hides two trips to memory, with many it costs the registers that more blocks per SM need.  A layer with its two launches, us,
// ahead / without: 1536 values 128 rows 80.5 / 84.1, 512 160.2 / 164.5, 768 203.1 / 201.8 (one launch of 2047 19.4 / 17); 2560 values 256 rows 171.0 /
// 175.7, 300 208.7 / 209.1, 384 226.8 / 223.7, 1536 730 / 724; 4096 values 128 rows 126.9 / 130.2, 200 181.5 / 179.3, 512 322.9 / 314.4.
template <unsigned THREADS, bool AHEAD>
__global__ void __launch_bounds__(THREADS, AHEAD ? 1 : 1024 / THREADS) gemm_finish_norm_split_kernel(const EpiNormArgs e) {
  __shared__ float red[32];
  const unsigned t = blockIdx.x, ck = threadIdx.x, chunks = e.rows / 8u;
  const bool live = ck < chunks && t < e.n_tok;
  const unsigned slots = live ? ks_gemm_slots(e.map, 0u, 8u * ck / GM_ROWS, t) : 0u;  // (half a dozen divisions: in front of the wait)
  ks_pdl_entry();
  float y[8];
  const size_t at = (size_t)t * e.rows + 8u * ck;
  // everything that does not depend on the sums is requested first
  float4 r0{}, r1{}, p0{}, p1{}, n0{}, n1{};
  if (live) {
    r0 = *reinterpret_cast<const float4*>(e.res + at);
    r1 = *reinterpret_cast<const float4*>(e.res + at + 4);
    if constexpr (AHEAD) {
      p0 = *reinterpret_cast<const float4*>(e.w_post + 8u * ck);
      p1 = *reinterpret_cast<const float4*>(e.w_post + 8u * ck + 4);
      n0 = *reinterpret_cast<const float4*>(e.w_norm + 8u * ck);
      n1 = *reinterpret_cast<const float4*>(e.w_norm + 8u * ck + 4);
    }
  }
  sum8<AHEAD ? 4 : 2>(e.P + at, e.part_stride, slots, y);
  float ss = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; i++) ss = fmaf(y[i], y[i], ss);
  ss = block_sum_f(ss, red);
  const float inv = 1.0f / sqrtf(ss / (float)e.rows + e.eps);
  float v[8], ss2 = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; i++) v[i] = 0.0f;
  if (live) {
    if constexpr (!AHEAD) {
      p0 = *reinterpret_cast<const float4*>(e.w_post + 8u * ck);
      p1 = *reinterpret_cast<const float4*>(e.w_post + 8u * ck + 4);
    }
    const float rr[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w}, pp[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = __fadd_rn(rr[i], __fmul_rn(__fmul_rn(y[i], inv), pp[i]));
    *reinterpret_cast<float4*>(e.out_x + at) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(e.out_x + at + 4) = make_float4(v[4], v[5], v[6], v[7]);
  }
#pragma unroll
  for (int i = 0; i < 8; i++) ss2 = fmaf(v[i], v[i], ss2);
  ss2 = block_sum_f(ss2, red);
  const float inv2 = 1.0f / sqrtf(ss2 / (float)e.rows + e.eps);
  float xn[8];
#pragma unroll
  for (int i = 0; i < 8; i++) xn[i] = 0.0f;
  if (live) {
    if constexpr (!AHEAD) {
      n0 = *reinterpret_cast<const float4*>(e.w_norm + 8u * ck);
      n1 = *reinterpret_cast<const float4*>(e.w_norm + 8u * ck + 4);
    }
    const float nn[8] = {n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, n1.z, n1.w};
#pragma unroll
    for (int i = 0; i < 8; i++) xn[i] = __fmul_rn(__fmul_rn(v[i], inv2), nn[i]);
  }
  float up;
  const float down = row_scale_down(block_max_f(absmax8(xn), red), &up);
  if (threadIdx.x == 0) reinterpret_cast<float*>(e.xt + xt_scale_off(e.rows, e.np))[t] = up;
  if (ck < chunks) {
#pragma unroll
    for (int i = 0; i < 8; i++) xn[i] *= down;
    put_split8(e.xt, e.np, e.tbn, t, ck, chunks, xn, e.q4k != 0);
  }
}

constexpr int GM_ROW_THREADS = 1024;  // threads of a block that writes one token row of an image
// gelu(sum of gate partials) * (sum of up partials) (lib.rs:953) straight into the image the down GEMM reads.  A cluster of four
// blocks per (padded) token row, 8 values per thread: the row maximum that scales the image meets in distributed shared memory,
// and few token rows still make enough blocks (8 rows of 10240 values: 64 blocks instead of 16).
constexpr unsigned GM_GELU_CL = 4, GM_GELU_THREADS = 512;
constexpr size_t GM_GELU_MOST = 8 * GM_GELU_CL * GM_GELU_THREADS;
__global__ void __cluster_dims__(GM_GELU_CL, 1, 1) __launch_bounds__(GM_GELU_THREADS)
    gemm_finish_gelu_split_kernel(const float* P0, const float* P1, size_t part_stride, ks_gemm_map map, unsigned n_tok, unsigned np, unsigned tbn,
                                  unsigned rows, __half* xt) {
  __shared__ float red[32], maxima[GM_GELU_CL];
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  cluster.barrier_arrive();  // (a block's shared memory is there once it has started)
  const unsigned rank = blockIdx.x % GM_GELU_CL, t = blockIdx.x / GM_GELU_CL, chunks = rows / 8u, ck = rank * blockDim.x + threadIdx.x;
  // how many partials (divisions: in front of the wait)
  const unsigned tile = 8u * ck / GM_ROWS, groups = map.G ? ((rows + GM_ROWS - 1u) / GM_ROWS + map.nt - 1u) / map.nt : 0u;
  const unsigned ng = ks_gemm_slots(map, 0u, tile, t), nu = ks_gemm_slots(map, groups, tile, t);
  ks_pdl_entry();
  float v[8];
#pragma unroll
  for (int k = 0; k < 8; k++) v[k] = 0.0f;
  if (t < n_tok && ck < chunks) {
    float g[8], u[8];
    const size_t at = (size_t)t * rows + 8u * ck;
    sum8<4>(P0 + at, part_stride, ng, g);
    sum8<4>(P1 + at, part_stride, nu, u);
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = gelu_mul(g[k], u[k]);
  }
  // gelu(gate) * up is where a random-weight model leaves the f16 range
  const float m = block_max_f(absmax8(v), red);
  cluster.barrier_wait();
  if (threadIdx.x < GM_GELU_CL) *cluster.map_shared_rank(&maxima[rank], threadIdx.x) = m;
  cluster.sync();
  float row_max = maxima[0];
#pragma unroll
  for (unsigned k = 1; k < GM_GELU_CL; k++) row_max = fmaxf(row_max, maxima[k]);
  float up;
  const float down = row_scale_down(row_max, &up);
  if (rank == 0 && threadIdx.x == 0) reinterpret_cast<float*>(xt + xt_scale_off(rows, np))[t] = up;
  if (ck < chunks) {
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] *= down;
    put_split8(xt, np, tbn, t, ck, chunks, v, true);  // a down-projection is always Q4_K
  }
}

// The same for passes of many rows: a cluster of eight blocks per FOUR token rows, two steps of 64 columns per warp
// (put_split8_rows4).  Bound by loads in flight: all first partials are requested before anything is waited for, and 64 registers
// keep five blocks of 192 threads on an SM (with 94 and three: 60 us instead of 47; with the second partials requested early as well
// it spills: 51).  The partial counts, half a dozen divisions each, are a lane's work each (31 to 24 million instructions).
// 2047 rows of 6144 values, 113 MB read and 57 written: 84 us with a cluster of four per row, 45 here; 1530 rows of 10240: 121, 61.
constexpr unsigned GM_R4_CL = 8, GM_R4_S = 2, GM_R4_WARPS = 16;  // blocks of a cluster, steps of a warp, warps at most
// From so many rows and more values than so many, a cluster per row / per four rows, each launch alone behind flushed caches: 129 rows of 6144
// values 10.4 / 9.0 us, of 10240 15.9 / 10.7, of 3072 6.6 / 6.0, of 2048 6.1 / 5.5; 128 of 2048 6.1 / 7.7; 256 of 1024 6.3 / 7.7, 257 7.7 / 5.7.  (4096
// values from 129 to 192 rows are on the wrong side: 7.2 / 7.9 to 7.7 / 8.5.)
constexpr int GM_R4_ROWS = 128;
constexpr size_t GM_R4_VALUES = 1u << 18;
static_assert(GM_GELU_MOST <= GM_R4_CL * GM_R4_S * GM_R4_WARPS * 64, "the longest rows fit");
__device__ __forceinline__ void ld8(const float* p, float (&v)[8]) {
  *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(p);
  *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(p + 4);
}
// Partials 1 .. n - 1 on top of the first.
__device__ __forceinline__ void add_slots(const float* p, size_t stride, unsigned n, float (&v)[8]) {
  for (unsigned k = 1; k < n; k++) {
    float x[8];
    ld8(p + (size_t)k * stride, x);
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] += x[i];
  }
}
__global__ void __cluster_dims__(GM_R4_CL, 1, 1) __launch_bounds__(GM_R4_WARPS * 32, 2)
    gemm_finish_gelu_rows_kernel(const float* P0, const float* P1, size_t part_stride, ks_gemm_map map, unsigned n_tok, unsigned np, unsigned tbn,
                                 unsigned rows, __half* xt) {
  ks_pdl_entry();
  __shared__ float red[GM_R4_WARPS][4], maxima[GM_R4_CL][4];
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  cluster.barrier_arrive();  // (a block's shared memory is there once it has started)
  const unsigned rank = blockIdx.x % GM_R4_CL, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const unsigned t0 = blockIdx.x / GM_R4_CL * 4u, t = t0 + (lane & 3u);
  const unsigned steps = rows / 64u, per = (steps + GM_R4_CL - 1u) / GM_R4_CL, first = rank * per, end = min(first + per, steps);
  const unsigned groups = map.G ? ((rows + GM_ROWS - 1u) / GM_ROWS + map.nt - 1u) / map.nt : 0u;
  float v[GM_R4_S][8], u[GM_R4_S][8];
#pragma unroll
  for (unsigned s = 0; s < GM_R4_S; s++) {
    const unsigned st = first + warp + s * warps;
#pragma unroll
    for (int k = 0; k < 8; k++) v[s][k] = u[s][k] = 0.0f;
    if (st < end && t < n_tok) {
      const size_t at = (size_t)t * rows + 64u * st + 8u * (lane >> 2);
      ld8(P0 + at, v[s]);
      ld8(P1 + at, u[s]);
    }
  }
  const unsigned my_slots = ks_gemm_slots(map, lane & 1u ? groups : 0u, 64u * (first + warp + (lane >> 1) % GM_R4_S * warps) / GM_ROWS, t0);
  float m = 0.0f;
#pragma unroll
  for (unsigned s = 0; s < GM_R4_S; s++) {
    const unsigned st = first + warp + s * warps, ng = __shfl_sync(0xffffffffu, my_slots, 2 * s), nu = __shfl_sync(0xffffffffu, my_slots, 2 * s + 1);
    if (st < end && t < n_tok) {
      const size_t at = (size_t)t * rows + 64u * st + 8u * (lane >> 2);
      add_slots(P0 + at, part_stride, ng, v[s]);
      add_slots(P1 + at, part_stride, nu, u[s]);
#pragma unroll
      for (int k = 0; k < 8; k++) v[s][k] = gelu_mul(v[s][k], u[s][k]);
      m = fmaxf(m, absmax8(v[s]));
    }
  }
  // the rows' largest values: over the warp's lanes, the block, the cluster
#pragma unroll
  for (int o = 4; o <= 16; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane < 4u) red[warp][lane] = m;
  __syncthreads();
  m = 0.0f;
#pragma unroll 4
  for (unsigned w = 0; w < warps; w++) m = fmaxf(m, red[w][lane & 3u]);
  cluster.barrier_wait();
  if (threadIdx.x < 4u * GM_R4_CL) cluster.map_shared_rank(&maxima[rank][0], threadIdx.x >> 2)[lane & 3u] = m;
  cluster.sync();
  float row_max = maxima[0][lane & 3u];
#pragma unroll
  for (unsigned k = 1; k < GM_R4_CL; k++) row_max = fmaxf(row_max, maxima[k][lane & 3u]);
  float up;
  const float down = row_scale_down(row_max, &up);
  if (rank == 0 && threadIdx.x < 4u) reinterpret_cast<float*>(xt + xt_scale_off(rows, np))[t] = up;
#pragma unroll
  for (unsigned s = 0; s < GM_R4_S; s++) {
    const unsigned st = first + warp + s * warps;
    if (st < end) {
#pragma unroll
      for (int k = 0; k < 8; k++) v[s][k] *= down;
      put_split8_rows4(xt, tbn, t0, 8u * st, rows / 8u, v[s]);
    }
  }
}

// The q, k and v partials of a token through per-head RMS norm, RoPE and the Q4_0 pack of K and V (lower.rs:4231-4702), one warp
// per (token, head).  A lane holds HD / 64 neighbouring dims of each half of the head, so RoPE partners sit in one lane and a
// 32-value block in 8 (16) neighbouring lanes.
struct EpiQkvArgs {
  const float* P[3];
  size_t part_stride[3];
  unsigned rows[3], group0[3];
  ks_gemm_map map;
  unsigned n_tok, n_q, n_kv;
  float eps;
  const float *qw, *kw, *rope;
  const int *pos, *row_slot;
  float* q_out;
  uint8_t *kv_k, *kv_v;
  size_t slot_stride;
};
template <int HD>
__global__ void __launch_bounds__(256) gemm_finish_qkv_kernel(const EpiQkvArgs e) {
  constexpr int V = HD / 64, LPB = 32 / V;  // values per lane and half, lanes per 32-value block
  constexpr unsigned ROWB = HD / 32 * KS_Q40_BLOCK_BYTES;
  const unsigned lane = threadIdx.x & 31u, jobs = e.n_q + 2u * e.n_kv, id = blockIdx.x * 8u + (threadIdx.x >> 5);
  if (id >= e.n_tok * jobs) return;
  const unsigned tok = id / jobs, job = id - tok * jobs;
  const int seg = (job >= e.n_q) + (job >= e.n_q + e.n_kv);
  const unsigned head = seg == 0 ? job : seg == 1 ? job - e.n_q : job - e.n_q - e.n_kv;
  const float* P = seg == 0 ? e.P[0] : seg == 1 ? e.P[1] : e.P[2];
  const size_t ps = seg == 0 ? e.part_stride[0] : seg == 1 ? e.part_stride[1] : e.part_stride[2];
  const unsigned rows = seg == 0 ? e.rows[0] : seg == 1 ? e.rows[1] : e.rows[2], g0 = seg == 0 ? e.group0[0] : seg == 1 ? e.group0[1] : e.group0[2];
  // (half a head is one row tile, or within one; how many partials it has takes half a dozen divisions: a lane each, in front of the wait)
  const unsigned my_slots = ks_gemm_slots(e.map, g0, (head * HD + (lane & 1u) * (HD / 2)) / GM_ROWS, tok);
  ks_pdl_entry();
  const size_t p = (size_t)e.pos[tok];
  const float* cs = e.rope + p * HD;
  float c[V], sn[V], w[2][V], x[2][V];
#pragma unroll
  for (int k = 0; k < V; k++) {
    const unsigned d = lane * V + k;
    c[k] = cs[d];
    sn[k] = cs[HD / 2 + d];
    w[0][k] = seg == 0 ? e.qw[d] : seg == 1 ? e.kw[d] : 1.0f;
    w[1][k] = seg == 0 ? e.qw[HD / 2 + d] : seg == 1 ? e.kw[HD / 2 + d] : 1.0f;
  }
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const unsigned row = head * HD + (unsigned)h * (HD / 2) + lane * V, n = __shfl_sync(0xffffffffu, my_slots, h);
    const float* src = P + (size_t)tok * rows + row;
#pragma unroll
    for (int k = 0; k < V; k++) x[h][k] = 0.0f;
#pragma unroll 4
    for (unsigned s = 0; s < n; s++)
      if constexpr (V == 4) {
        const float4 a = *reinterpret_cast<const float4*>(src + (size_t)s * ps);
        x[h][0] += a.x; x[h][1] += a.y; x[h][2] += a.z; x[h][3] += a.w;
      } else {
        const float2 a = *reinterpret_cast<const float2*>(src + (size_t)s * ps);
        x[h][0] += a.x; x[h][1] += a.y;
      }
  }
  float ss = 0.0f;
#pragma unroll
  for (int k = 0; k < V; k++) ss = fmaf(x[0][k], x[0][k], fmaf(x[1][k], x[1][k], ss));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const float inv = 1.0f / sqrtf(ss / (float)HD + e.eps);
  float y[2][V];
#pragma unroll
  for (int k = 0; k < V; k++) {
    const float u = __fmul_rn(__fmul_rn(x[0][k], inv), w[0][k]), v = __fmul_rn(__fmul_rn(x[1][k], inv), w[1][k]);
    y[0][k] = seg == 2 ? u : __fsub_rn(__fmul_rn(u, c[k]), __fmul_rn(v, sn[k]));
    y[1][k] = seg == 2 ? v : __fadd_rn(__fmul_rn(u, sn[k]), __fmul_rn(v, c[k]));
  }
  if (seg == 0) {
    float* o = e.q_out + (size_t)tok * e.rows[0] + head * HD + lane * V;
#pragma unroll
    for (int h = 0; h < 2; h++)
      if constexpr (V == 4) *reinterpret_cast<float4*>(o + h * (HD / 2)) = make_float4(y[h][0], y[h][1], y[h][2], y[h][3]);
      else *reinterpret_cast<float2*>(o + h * (HD / 2)) = make_float2(y[h][0], y[h][1]);
    return;
  }
  uint8_t* dst = (seg == 1 ? e.kv_k : e.kv_v) + (size_t)(e.row_slot ? (unsigned)e.row_slot[tok] : tok) * e.slot_stride + (p * e.n_kv + head) * ROWB;
#pragma unroll
  for (int h = 0; h < 2; h++) {
    float amax = 0.0f, val[V];
#pragma unroll
    for (int k = 0; k < V; k++) {
      val[k] = __half2float(__float2half_rn(y[h][k]));  // values pass through f16 before packing (render.rs:1046)
      amax = fmaxf(amax, fabsf(val[k]));
    }
#pragma unroll
    for (int o = LPB / 2; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float scale = amax > 0.0f ? amax / 7.0f : 1.0f, is = 1.0f / scale;
    unsigned q = 0;
#pragma unroll
    for (int k = 0; k < V; k++) {
      int i = (int)roundf(__fmul_rn(val[k], is)) + 8;
      i = i < 0 ? 0 : i > 15 ? 15 : i;
      q |= (unsigned)i << (8 * k);
    }
    q |= __shfl_down_sync(0xffffffffu, q, LPB / 2) << 4;  // the block's second sixteen go to the high nibbles
    const unsigned l = lane % LPB;
    uint8_t* blk = dst + ((unsigned)h * (HD / 64) + lane / LPB) * KS_Q40_BLOCK_BYTES;
    if (l < LPB / 2) {
      unsigned short* o = reinterpret_cast<unsigned short*>(blk + 2 + l * V);
      o[0] = (unsigned short)q;
      if constexpr (V == 4) o[1] = (unsigned short)(q >> 16);
    }
    if (l == 0) *reinterpret_cast<__half*>(blk) = __float2half_rn(scale);
  }
}
}  // namespace

namespace {
// Token rows of the Q6_K kernel, padded to what its MMAs take.
unsigned gemm_np(int n_tok) { return n_tok > 128 ? ((unsigned)n_tok + 31u) / 32u * 32u : ((unsigned)n_tok + 15u) / 16u * 16u; }
// Shared memory of one CTA and its stage count (A and B rings have the same depth): two stages when that lets two
// CTAs share an SM (measured: a third stage that still lets them does not pay), else as many (up to four) as one CTA fits.
size_t gemm_smem(const ks_ctx* ctx, unsigned np, unsigned* nb_out) {
  const size_t stage = (size_t)GM_A_BYTES + (size_t)np * 256, per_sm = ctx->smem_optin + 1024;  // the SM holds 1 KB more than a CTA may ask for
  auto bytes = [&](size_t n) { return 1024 + n * stage; };
  auto two_fit = [&](size_t n) { return 2 * (bytes(n) + 1024) <= per_sm; };  // each resident CTA costs 1 KB on top
  if (bytes(2) > ctx->smem_optin) return 0;
  size_t nb = 2;
  if (!two_fit(2))
    while (nb < 4 && bytes(nb + 1) <= ctx->smem_optin) nb++;
  if (nb_out) *nb_out = (unsigned)nb;
  return bytes(nb);
}
// k splits of a launch over `tiles` row tiles: the count that minimises rounds x (k-steps per CTA + a fixed
// start-up and epilogue cost of about three k-steps); two CTAs that share an SM cost each other about a fifth.
unsigned gemm_splits(const ks_ctx* ctx, size_t rows, size_t cols, int n_tok) {
  const unsigned tiles = (unsigned)((rows + GM_ROWS - 1) / GM_ROWS), ksteps = (unsigned)(cols / GM_KSTEP);
  const size_t smem = gemm_smem(ctx, gemm_np(n_tok), nullptr);
  const unsigned cps = smem && 2 * (smem + 1024) <= ctx->smem_optin + 1024 ? 2u : 1u;
  const unsigned sms = (unsigned)ctx->sm_count, slots = sms * cps;
  if (const char* f = getenv("KSEARCH_GEMM_SPLITS")) {  // measurement override
    const unsigned s = (unsigned)atoi(f);
    if (s >= 1 && s <= 16 && s * 2 <= (ksteps < 2 ? 2 : ksteps)) return s;
  }
  unsigned best = 1;
  double best_cost = 1e30;
  for (unsigned s = 1; s <= 16 && s * 2 <= (ksteps < 2 ? 2 : ksteps); s++) {
    const unsigned per = (ksteps + s - 1) / s, real = (ksteps + per - 1) / per;
    if (real != s) continue;  // this count leaves a split empty
    const unsigned ctas = tiles * s, rounds = (ctas + slots - 1) / slots;
    const double cost = (double)rounds * (per + 3) * (cps == 2 && ctas > sms ? 1.2 : 1.0);
    if (cost < best_cost * 0.97) {
      best_cost = cost;
      best = s;
    }
  }
  return best;
}
typedef ks_gemm_blocks Blocks;
// Q4_K: the fewest blocks of at most `most` rows, all alike, a multiple of 16.
Blocks gemm_blocks(int n_tok, unsigned most = 128u) {
  const unsigned tb = ((unsigned)n_tok + most - 1u) / most, tbn = (((unsigned)n_tok + tb - 1) / tb + 15u) / 16u * 16u;
  return {tbn, tb * tbn};
}
ks_gemm_map gemm_map(const ks_ctx* ctx, ks_dtype wdtype, const size_t* rows, int n_seg, size_t cols, int n_tok, Blocks b, bool plain) {
  ks_gemm_map m{};
  size_t total_rows = 0;
  for (int i = 0; i < n_seg; i++) total_rows += rows[i];
  if (wdtype == KS_Q4K && n_tok <= KS_GEMM_SKINNY && (m.splits = ks_gemm_skinny_splits(ctx, total_rows, (unsigned)cols)) != 0) return m;
  if (wdtype == KS_Q4K) return ks_gemm_q4k_map(ctx, rows, n_seg, (unsigned)cols, b.np, b.tbn, plain);
  if (n_tok <= KS_GEMM_SKINNY && n_seg == 1 && ks_gemm_q6k_skinny_covers(ctx, total_rows, (unsigned)cols)) {
    m.splits = 1;
    return m;
  }
  const unsigned ksteps = (unsigned)(cols / GM_KSTEP), s = gemm_splits(ctx, total_rows, cols, n_tok), per = (ksteps + s - 1) / s;
  m.splits = (ksteps + per - 1) / per;
  return m;
}
// The most partials a work tile of the launch leaves.
unsigned map_slots(const ks_gemm_map& map, unsigned groups) {
  unsigned slots = map.G ? 0 : map.splits;
  for (unsigned w = 0; map.G && w < groups * map.tb; w++) {
    const unsigned n = ks_gemm_owner(map, w * map.S + map.S - 1u) - ks_gemm_owner(map, w * map.S) + 1u;
    slots = n > slots ? n : slots;
  }
  return slots;
}
bool gemm_covers(ks_dtype wdtype, size_t cols, int n_tok) {
  return (wdtype == KS_Q4K || wdtype == KS_Q6K) && cols % 256 == 0 && n_tok >= 1 && n_tok <= (wdtype == KS_Q4K ? KS_GEMM_ROWS : 256);
}
}  // namespace

bool ks_gemm_few_rows_q6k(const ks_ctx* ctx, size_t rows, size_t cols) { return ks_gemm_q6k_skinny_covers(ctx, rows, (unsigned)cols); }
// Q4_K matrices against more than 64 token rows: pairs of row tiles against blocks of up to 128 read the token rows half as
// often; where that leaves few units for the SMs, single tiles against blocks of up to 64 are four times as many.  By the
// estimate both maps are chosen by; with an epilogue behind it (sums always read once more) only where it promises a tenth: a
// whole E2B layer of 256 rows took 142 us with wide blocks, 145 with the four small ones the bare estimate picks, 139 with this
// line; of 128 rows 117 with wide blocks and 105 with small ones, of the tiny shape 87 and 60.
ks_gemm_blocks ks_gemm_pick(const ks_ctx* ctx, ks_dtype wdtype, int n_seg, const size_t* rows, size_t cols, int n_tok, bool plain) {
  if (wdtype != KS_Q4K) return {gemm_np(n_tok), gemm_np(n_tok)};
  const Blocks wide = gemm_blocks(n_tok);
  if (wide.tbn <= 64u) return wide;
  const Blocks small = gemm_blocks(n_tok, 64u);
  double cw, cs;
  ks_gemm_q4k_map(ctx, rows, n_seg, (unsigned)cols, wide.np, wide.tbn, plain, &cw);
  ks_gemm_q4k_map(ctx, rows, n_seg, (unsigned)cols, small.np, small.tbn, plain, &cs);
  return cs < (plain ? cw : 0.9 * cw) ? small : wide;
}
bool ks_gemm_layers_cover(size_t hidden, size_t ffn, size_t q_cols) {
  return hidden % 256 == 0 && ffn % 256 == 0 && q_cols % 256 == 0 && hidden <= GM_NORM_MOST && ffn <= GM_GELU_MOST;
}

// Bytes of the B image of n_tok rows of `cols` values (hi + lo halves, token count padded to 16).
size_t ks_gemm_xt_bytes(size_t cols, int n_tok) {  // image + one factor per row, whatever the blocks
  const size_t np = n_tok > 128 ? ((size_t)n_tok + 127) / 128 * 128 : n_tok > 64 ? 128 : gemm_np(n_tok);
  return cols / 256 * 288 * np * 4 + np * 4;
}

// x[t * ldx + k] (f32) -> the B image in xt.
int ks_launch_gemm_split(ks_ctx* ctx, ks_dtype wdtype, const float* x, size_t ldx, int n_tok, size_t cols, void* xt, ks_gemm_blocks b) {
  if (cols % 256 || n_tok < 1 || n_tok > KS_GEMM_ROWS || ldx % 4) return ks_fail(ctx, KS_ERR_INVALID, "gemm: bad operand shape");
  const bool one = cols <= 8u * GM_ROW_THREADS;
  KS_LAUNCH(ctx, (one ? x_split_kernel<true> : x_split_kernel<false>), b.np, one ? (unsigned)(cols / 8) : (unsigned)GM_ROW_THREADS, 0, x, ldx, (unsigned)n_tok, b.np, b.tbn,
            (unsigned)cols, (__half*)xt, (int)(wdtype == KS_Q4K));
  return ks_after_launch(ctx, "x_split");
}

// Up to three matrices over the same columns in one launch.  With one k split matrix i's result goes straight to
// y[i] (row stride ldy[i]); otherwise the partials go to P (dense [split][token][row] per matrix, matrix after
// matrix) and a second launch sums them in split order into y, or takes them through an epilogue.  `xt` is the image of the token rows in these blocks.
int ks_launch_gemm_segs(ks_ctx* ctx, ks_dtype wdtype, int n_seg, const uint8_t* const* W, const size_t* rows, size_t cols, const void* xt,
                        int n_tok, float* const* y, const size_t* ldy, float* P, int mode, const ks_gemm_epi* epi, ks_gemm_blocks blocks) {
  if (!gemm_covers(wdtype, cols, n_tok) || n_seg < 1 || n_seg > 3) return ks_fail(ctx, KS_ERR_UNSUPPORTED, "gemm: shape not covered");
  if ((mode == KS_GEMM_NORM_SPLIT && (n_seg != 1 || !epi || rows[0] % 8 || rows[0] > GM_NORM_MOST)) ||
      (mode == KS_GEMM_QKV && (n_seg != 3 || !epi || (epi->hd != 128 && epi->hd != 256) || rows[0] != (size_t)epi->n_q * epi->hd ||
                               rows[1] != (size_t)epi->n_kv * epi->hd || rows[2] != rows[1])) ||
      (mode == KS_GEMM_GELU_SPLIT && (n_seg != 2 || !epi || rows[0] != rows[1] || rows[0] % 8 || rows[0] > GM_GELU_MOST || rows[0] % 256)))
    return ks_fail(ctx, KS_ERR_INVALID, "gemm: bad epilogue arguments");
  const unsigned np = blocks.np;
  const ks_gemm_map map = gemm_map(ctx, wdtype, rows, n_seg, cols, n_tok, blocks, mode == KS_GEMM_PLAIN);
  unsigned tiles = 0, tile0[4], groups = 0, group0[3] = {0, 0, 0};
  size_t total_rows = 0;
  for (int i = 0; i < 3; i++) {
    tile0[i] = i < n_seg ? tiles : 0xFFFFFFFFu;  // no tile reaches an absent matrix
    if (i >= n_seg) continue;
    const unsigned n = (unsigned)((rows[i] + GM_ROWS - 1) / GM_ROWS);
    group0[i] = groups;
    tiles += n;
    groups += map.G ? (n + map.nt - 1) / map.nt : 0;
    total_rows += rows[i];
  }
  tile0[3] = tiles;
  const unsigned slots = map_slots(map, groups);
  const bool direct = slots == 1 && mode == KS_GEMM_PLAIN;
  FinishArgs f{};
  float* out[3] = {nullptr, nullptr, nullptr};
  size_t ldo[3] = {0, 0, 0}, part_stride[3] = {0, 0, 0}, poff = 0;
  for (int i = 0; i < n_seg; i++) {
    if (direct) {
      out[i] = y[i];
      ldo[i] = ldy[i];
    } else {
      out[i] = P + poff;
      ldo[i] = rows[i];
      part_stride[i] = (size_t)n_tok * rows[i];
      f.P[i] = out[i];
      f.part_stride[i] = part_stride[i];
      f.rows[i] = (unsigned)rows[i];
      f.y[i] = y[i];  // null where an epilogue takes the sums
      f.ldy[i] = ldy[i];
      poff += (size_t)slots * n_tok * rows[i];
    }
  }
  int rc;
  const bool skinny6 = wdtype == KS_Q6K && n_tok <= KS_GEMM_SKINNY && n_seg == 1 && direct && ((uintptr_t)W[0] & 15) == 0 &&
                       ks_gemm_q6k_skinny_covers(ctx, rows[0], (unsigned)cols);
  if (wdtype == KS_Q4K || skinny6) {
    ks_gemm_job job{};
    job.n_seg = n_seg;
    for (int i = 0; i < n_seg; i++) {
      job.W[i] = W[i];
      job.rows[i] = rows[i];
      job.y[i] = out[i];
      job.ldy[i] = ldo[i];
      job.part_stride[i] = part_stride[i];
    }
    job.cols = (unsigned)cols;
    job.n_tok = (unsigned)n_tok;
    job.np = np;
    job.xt = (const __half*)xt;
    job.map = map;
    rc = skinny6 ? ks_launch_gemm_q6k_skinny(ctx, job) : map.G ? ks_launch_gemm_q4k(ctx, job) : ks_launch_gemm_skinny(ctx, job);
  } else {
    GemmArgs a{};
    for (int i = 0; i < 3; i++) {
      a.tile0[i] = tile0[i];
      if (i >= n_seg) continue;
      a.W[i] = W[i];
      a.rows[i] = (unsigned)rows[i];
      a.y[i] = out[i];
      a.ldy[i] = ldo[i];
      a.part_stride[i] = part_stride[i];
    }
    a.tile0[3] = tiles;
    a.row_bytes = cols / 256 * KS_Q6K_BLOCK_BYTES;
    a.xt = (const __half*)xt;
    a.cols = (unsigned)cols;
    a.n_tok = (unsigned)n_tok;
    a.np = np;
    a.tmem_cols = 32;  // the accumulator: 2 NP columns up to 128 token rows (hi and lo products side by side), NP beyond
    while (a.tmem_cols < (a.np <= 128 ? 2 * a.np : a.np)) a.tmem_cols <<= 1;
    const unsigned ksteps = (unsigned)(cols / GM_KSTEP);
    a.ksteps_per = (ksteps + map.splits - 1) / map.splits;
    a.err = (unsigned*)ctx->ws + KS_WS_ERR_WORD;
    a.wait_limit = GM_WAIT;
    if (const char* t = getenv("KSEARCH_GEMM_TEST_STALL")) {  // exercises the give-up path: short waits, one operand withheld
      a.test_stall = (unsigned)atoi(t);
      if (a.test_stall) a.wait_limit = 4000;
    }
    const size_t smem = gemm_smem(ctx, a.np, &a.nb);
    if (!smem) return ks_fail(ctx, KS_ERR_UNSUPPORTED, "gemm: %u token rows do not fit the shared memory", a.np);
    static size_t smem_set[16] = {0};
    size_t& set = smem_set[ctx->device & 15];
    if (smem > set) {
      cudaError_t e = cudaFuncSetAttribute(gemm_q6k_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return ks_fail(ctx, KS_ERR_CUDA, "gemm: cannot set %zu B shared memory: %s", smem, cudaGetErrorString(e));
      set = smem;
    }
    KS_LAUNCH(ctx, gemm_q6k_tc_kernel, dim3(tiles, map.splits), GM_THREADS + 64, smem, a);
    rc = ks_after_launch(ctx, "gemm_q6k_tc");
  }
  if (rc || direct) return rc;
  if (mode == KS_GEMM_NORM_SPLIT) {
    EpiNormArgs e{};
    e.P = out[0];
    e.part_stride = part_stride[0];
    e.map = map;
    e.n_tok = (unsigned)n_tok;
    e.np = epi->next.np;
    e.tbn = epi->next.tbn;
    e.q4k = epi->next_dtype == KS_Q4K;
    e.rows = (unsigned)rows[0];
    e.res = epi->res;
    e.w_post = epi->w_post;
    e.w_norm = epi->w_norm;
    e.eps = epi->eps;
    e.out_x = epi->out_x;
    e.xt = (__half*)epi->xt_out;
    const unsigned threads = (unsigned)((rows[0] / 8 + 31) / 32 * 32);
    if (threads > 512u) KS_LAUNCH(ctx, (gemm_finish_norm_split_kernel<1024, false>), e.np, threads, 0, e);
    else if ((size_t)n_tok * rows[0] <= GM_NORM_AHEAD) KS_LAUNCH(ctx, (gemm_finish_norm_split_kernel<512, true>), e.np, threads, 0, e);
    else KS_LAUNCH(ctx, (gemm_finish_norm_split_kernel<512, false>), e.np, threads, 0, e);
    return ks_after_launch(ctx, "gemm_finish_norm_split");
  }
  if (mode == KS_GEMM_QKV) {
    EpiQkvArgs e{};
    for (int i = 0; i < 3; i++) {
      e.P[i] = out[i];
      e.part_stride[i] = part_stride[i];
      e.rows[i] = (unsigned)rows[i];
      e.group0[i] = group0[i];
    }
    e.map = map;
    e.n_tok = (unsigned)n_tok;
    e.n_q = epi->n_q;
    e.n_kv = epi->n_kv;
    e.eps = epi->eps;
    e.qw = epi->qw;
    e.kw = epi->kw;
    e.rope = epi->rope;
    e.pos = epi->pos;
    e.row_slot = epi->row_slot;
    e.q_out = epi->out_x;
    e.kv_k = epi->kv_k;
    e.kv_v = epi->kv_v;
    e.slot_stride = epi->slot_stride;
    const unsigned grid = (e.n_tok * (e.n_q + 2 * e.n_kv) + 7) / 8;
    if (epi->hd == 256) KS_LAUNCH(ctx, (gemm_finish_qkv_kernel<256>), grid, 256, 0, e);
    else KS_LAUNCH(ctx, (gemm_finish_qkv_kernel<128>), grid, 256, 0, e);
    return ks_after_launch(ctx, "gemm_finish_qkv");
  }
  if (mode == KS_GEMM_GELU_SPLIT) {
    if (n_tok >= GM_R4_ROWS && (size_t)n_tok * rows[0] > GM_R4_VALUES) {
      const unsigned per = ((unsigned)rows[0] / 64u + GM_R4_CL - 1u) / GM_R4_CL, warps = (per + GM_R4_S - 1u) / GM_R4_S;
      KS_LAUNCH(ctx, gemm_finish_gelu_rows_kernel, epi->next.np / 4u * GM_R4_CL, warps * 32u, 0, (const float*)out[0], (const float*)out[1], part_stride[0], map,
                (unsigned)n_tok, epi->next.np, epi->next.tbn, (unsigned)rows[0], (__half*)epi->xt_out);
      return ks_after_launch(ctx, "gemm_finish_gelu_rows");
    }
    // whole warps per block: a 32-value sub-block of the image is four neighbouring lanes of one
    const unsigned threads = ((unsigned)rows[0] / 8u / GM_GELU_CL + 31u) / 32u * 32u;
    KS_LAUNCH(ctx, (gemm_finish_gelu_split_kernel), epi->next.np * GM_GELU_CL, threads, 0, (const float*)out[0], (const float*)out[1], part_stride[0], map,
              (unsigned)n_tok, epi->next.np, epi->next.tbn, (unsigned)rows[0], (__half*)epi->xt_out);
    return ks_after_launch(ctx, "gemm_finish_gelu_split");
  }
  f.n_seg = (unsigned)n_seg;
  f.map = map;
  for (int i = 0; i < 3; i++) {
    f.tile0[i] = tile0[i];
    f.group0[i] = group0[i];
  }
  f.n_tok = (unsigned)n_tok;
  bool vec = true;
  for (int i = 0; i < n_seg; i++) {
    vec = vec && rows[i] % 4 == 0 && ((uintptr_t)out[i] & 15) == 0 && ((uintptr_t)f.y[i] & 15) == 0 && f.ldy[i] % 4 == 0;
  }
  const unsigned tok = vec ? 8u : 2u;
  const dim3 grid(tiles, ((unsigned)n_tok + tok - 1) / tok);
  if (vec) KS_LAUNCH(ctx, (gemm_finish_kernel<4>), grid, 256, 0, f);
  else KS_LAUNCH(ctx, (gemm_finish_kernel<1>), grid, 256, 0, f);
  return ks_after_launch(ctx, "gemm_finish");
}

// Floats of partials ks_launch_gemm_segs writes for these matrices and token rows.
size_t ks_gemm_part_floats(const ks_ctx* ctx, ks_dtype wdtype, int n_seg, const size_t* rows, size_t cols, int n_tok, bool plain) {
  const ks_gemm_map m = gemm_map(ctx, wdtype, rows, n_seg, cols, n_tok, ks_gemm_pick(ctx, wdtype, n_seg, rows, cols, n_tok, plain), plain);
  size_t total = 0;
  unsigned groups = 0;
  for (int i = 0; i < n_seg; i++) {
    total += rows[i];
    if (m.G) groups += (unsigned)(((rows[i] + GM_ROWS - 1) / GM_ROWS + m.nt - 1) / m.nt);
  }
  return (size_t)map_slots(m, groups) * (size_t)n_tok * total;
}

// Scratch of ks_launch_gemm_kq: the image and the partials of that one launch.
size_t ks_gemm_kq_bytes(const ks_ctx* ctx, ks_dtype wdtype, size_t rows, size_t cols, int n_tok) {
  const ks_gemm_map m = gemm_map(ctx, wdtype, &rows, 1, cols, n_tok, ks_gemm_pick(ctx, wdtype, 1, &rows, cols, n_tok, true), true);
  const size_t slots = m.G ? (m.S + m.base - 1) / m.base + 1 : m.splits;
  return ks_gemm_xt_bytes(cols, n_tok) + 4 * slots * n_tok * rows;
}

// y[t * ldy + r] = sum_k W[r, k] x[t * ldx + k] for t < n_tok (Q4_K: up to KS_GEMM_ROWS, Q6_K: 256), f32 x and y: operand split, GEMM and, when
// the k range was split, the ordered sum of the partials.  `scratch`: ks_gemm_kq_bytes.
int ks_launch_gemm_kq(ks_ctx* ctx, ks_dtype wdtype, size_t rows, size_t cols, const uint8_t* W, const float* x, size_t ldx, float* y,
                      size_t ldy, int n_tok, void* scratch) {
  if (!gemm_covers(wdtype, cols, n_tok) || ldx % 4) return 1;
  const Blocks b = ks_gemm_pick(ctx, wdtype, 1, &rows, cols, n_tok, true);
  int rc = ks_launch_gemm_split(ctx, wdtype, x, ldx, n_tok, cols, scratch, b);
  if (rc) return rc;
  float* P = (float*)((char*)scratch + ks_gemm_xt_bytes(cols, n_tok));
  return ks_launch_gemm_segs(ctx, wdtype, 1, &W, &rows, cols, scratch, n_tok, &y, &ldy, P, KS_GEMM_PLAIN, nullptr, b);
}
