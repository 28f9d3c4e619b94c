// Q4_K weights x a batch of token rows on the tensor cores (tcgen05), weights dequantised into TENSOR memory.
//
// The reference's op is mul_mm (crates/ksearch_codegen/src/render.rs:1073-1291, reached from
// crates/ksearch_kernels/src/lib.rs:1414).  A Q4_K weight is  d sc q - dmin m  with an 11-bit d, 6-bit sc and m and a 4-bit q
// (crates/ksearch_gguf/src/gguf_impl.rs:690-721).  What goes to the tensor core is the integer  sc q  (at most 945: exact
// in ONE f16), so a super-block of 256 k costs two products (x_hi, x_lo) where a split weight would cost three, and the
// f32 result of each super-block is multiplied by its d on the way out of tensor memory:
//   y[row, t] = sum over super-blocks of  s ( sum_k (sc q p) x[t, k]  -  sum_sub (mu m) S[t, sub] ),   s = d 2^j, p = 2^-j
// with S the sub-block sums of x (2^-5 scaled, in the B image) and mu = 32 dmin / s as two f16 terms: the minima ride along as
// 32 more k.  j = 0 unless dmin > 32 d, where it keeps mu m inside f16; sc q 2^-j stays exact.
//
// Per unit (128 rows x one super-block):
//   * the packed rows come by ONE 2-D TMA box (128 rows x 144 bytes; 144-byte row pitch: 16-byte reads of 8 rows hit 8
//     different bank groups) into a ring; the token rows by bulk copies of 32, 96 or 288 k into another;
//   * 16 warps: warp w owns the 32 rows of tensor-memory lane quadrant w % 4 and the 64 weights g = w / 4 of each: one
//     LOP3 and one HFMA2 make two weights out of packed nibbles ((1024 + q) sc - 1024 sc, exact), tcgen05.st puts them where
//     the MMA reads A.  Shared memory then carries only packed weights and B: A never passes through it;
//   * one elected lane issues the MMAs; after a super-block tcgen05.commit hands the accumulator to the warps that fold it into
//     registers (s times) while the next super-block's MMAs run in the other accumulator.
// Token rows come in blocks (the image has one part per block), two kernels by the block's rows:
//   up to 64   one row tile per unit, the same 16 warps convert and fold, x_hi and x_lo are ONE MMA of 2 tbn columns;
//   65 to 128  two row tiles per unit share the block's token rows, converting and folding in warps of their own.
// Tensor memory (512 columns): A ring of three half super-blocks (3 x 64) and blocks of minima (16 each) below 224 or 256, two
// accumulators of up to 128 columns above.
// One CTA per SM walks its units (ks_gemm_map) without a gap between tiles: the copies of the next tile are in flight while
// the last one is written out.
//
// Bound by: few token rows, the packed weights from memory and the issue slots of the dequantisation (about 1.7 instructions
// per weight and lane of 16 warps); blocks of 128, the tensor core (20480 x 2560 x 256 rows: 93 % busy inside a work tile, at the 1.4
// GHz that the power limit leaves; 132 -> 72 us against the kernel that wrote split weights to shared memory); few tiles, the latency
// of one unit and of the launches around it.
// Every wait is bounded; on expiry the CTA raises the context's status word, waits (bounded) for what it has in flight, frees
// its tensor memory and returns.
#include <cuda.h>

#include <cstdlib>
#include <cstring>

#include "ks_gemm_common.cuh"
#include "ks_gemm.h"

namespace {

constexpr unsigned Q_WARPS = 16, Q_THREADS = (Q_WARPS + 3) * 32;  // workers, MMA, packed rows, token rows
constexpr unsigned Q_RAW = GM_ROWS * KS_Q4K_BLOCK_BYTES;          // bytes of a unit's packed rows
constexpr unsigned Q_EXT = 192;                                   // tensor-memory column of the first block of minima
constexpr unsigned Q_WAIT = 1u << 20;
constexpr unsigned Q_MAX_RAW = 6, Q_MAX_B = 6;

struct __align__(64) Q4Args {
  CUtensorMap w[3];        // matrix i: rows[i] rows of row_bytes bytes
  float* y[3];             // y[i] + slot * part_stride[i] + token * ldy[i] + row
  size_t ldy[3], part_stride[3];
  unsigned rows[3], group0[3];
  ks_gemm_map map;
  const __half* xt;        // the q4k form of the B image
  unsigned cols, n_tok, np;
  unsigned n_raw, n_b;     // ring depths
  unsigned head;           // bytes in front of the rings: barriers, scale factors, wide: s of the last tiles' rows
  unsigned wait_limit, test_stall;
  unsigned* err;
};

// barriers (8 bytes each) at the start of shared memory
enum { QB_RAW_FULL = 0, QB_RAW_FREE = QB_RAW_FULL + Q_MAX_RAW, QB_B_FULL = QB_RAW_FREE + Q_MAX_RAW, QB_B_FREE = QB_B_FULL + Q_MAX_B,
       QB_A_FULL = QB_B_FREE + Q_MAX_B, QB_A_FREE = QB_A_FULL + 3, QB_D_FULL = QB_A_FREE + 3, QB_D_FREE = QB_D_FULL + 2, QB_DONE = QB_D_FREE + 2,
       QB_UP, QB_COUNT };
constexpr unsigned Q_HEAD = 512;  // barriers; behind them the token rows' scale factors
static_assert(QB_COUNT * 8 + 16 <= 512, "barriers fit the head of shared memory");

__device__ __forceinline__ void mb_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t and_or(uint32_t w, uint32_t mask, uint32_t bits) { return (w & mask) | bits; }

// What a thread needs of its row's super-block header: the two sub-blocks 2 g and 2 g + 1 (g uniform in a warp).
struct Q4Hdr {
  __half2 sc[2], cc[2];     // sub-block 2 g: sc p, -1024 sc p;  2 g + 1: sc p / 16, -64 sc p
  uint32_t mhi, mlo;        // -(mu m) of both, two f16 terms
  float s;
};
__device__ __forceinline__ __half2 small_int_h2(unsigned v) {  // v < 1024 in both halves: 1024 + v by its bits, then an exact subtract
  return __hsub2(as_h2(v * 0x00010001u | 0x64006400u), __float2half2_rn(1024.0f));
}
__device__ __forceinline__ void q4_header(const uint4 h, unsigned g, Q4Hdr& o) {
  const __half2 dd = *reinterpret_cast<const __half2*>(&h.x);
  const float d = __low2float(dd), dm = __high2float(dd);
  // bytes 2 g', 2 g' + 1 (g' = g & 1) of the three groups of four scale bytes; g < 2: sc and m lie in the low six bits of the
  // first two, else nibbles of the third and the top bits of the first two
  const unsigned sh = 16u * (g & 1u);
  const unsigned y = h.y >> sh, z = h.z >> sh, w = h.w >> sh;
  unsigned sc0, sc1, m0, m1;
  if (g < 2u) {
    sc0 = y & 63u;
    sc1 = (y >> 8) & 63u;
    m0 = z & 63u;
    m1 = (z >> 8) & 63u;
  } else {
    sc0 = (w & 15u) | ((y >> 2) & 48u);
    sc1 = ((w >> 8) & 15u) | ((y >> 10) & 48u);
    m0 = ((w >> 4) & 15u) | ((z >> 2) & 48u);
    m1 = ((w >> 12) & 15u) | ((z >> 10) & 48u);
  }
  const float ad = fabsf(d), am = fabsf(dm);
  __half2 s0 = small_int_h2(sc0), s1 = small_int_h2(sc1);
  float s = d, mu = ad > 0.0f ? __fdividef(32.0f * dm, d) : 0.0f;
  if (am > 32.0f * ad && (h.z | (h.w & 0xF0F0F0F0u)) != 0u) {  // (a block without minima has nothing to make room for, whatever its dmin)
    // j: the smallest power of two with dmin <= 32 d 2^j; beyond 2^20 (or d = 0) the d part is below the last bit of the minima
    float p = 0.0f;
    if (am <= 32.0f * 1048576.0f * ad) {
      const unsigned e = (__float_as_uint(__fdividef(am, 32.0f * ad)) >> 23) - 127u + 1u;  // 1..21
      p = __uint_as_float((127u - e) << 23);
      s = d * __uint_as_float((127u + e) << 23);
      mu *= p;
    } else {
      s = dm * 0.03125f;
      mu = 1024.0f;
    }
    s0 = __hmul2(s0, __float2half2_rn(p));
    s1 = __hmul2(s1, __float2half2_rn(p));
  }
  o.sc[0] = s0;
  o.cc[0] = __hmul2(s0, __float2half2_rn(-1024.0f));
  o.sc[1] = __hmul2(s1, __float2half2_rn(0.0625f));
  o.cc[1] = __hmul2(s1, __float2half2_rn(-64.0f));
  const float v0 = -mu * (float)m0, v1 = -mu * (float)m1;
  const __half2 mh = __floats2half2_rn(v0, v1);
  const float2 mf = __half22float2(mh);
  o.mhi = pack_h2(mh);
  o.mlo = pack_h2(__floats2half2_rn(v0 - mf.x, v1 - mf.y));
  o.s = s;
}
// 16 packed bytes (16 weights of sub-block 2 g in the low nibbles, 16 of 2 g + 1 in the high ones) -> 8 + 8 words of A.
__device__ __forceinline__ void q4_words(const uint4 q, const Q4Hdr& h, uint32_t (&lo)[8], uint32_t (&hi)[8]) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint32_t v = w[i] >> 8;
    lo[2 * i] = pack_h2(__hfma2(as_h2(and_or(w[i], 0x000F000Fu, 0x64006400u)), h.sc[0], h.cc[0]));
    lo[2 * i + 1] = pack_h2(__hfma2(as_h2(and_or(v, 0x000F000Fu, 0x64006400u)), h.sc[0], h.cc[0]));
    hi[2 * i] = pack_h2(__hfma2(as_h2(and_or(w[i], 0x00F000F0u, 0x64006400u)), h.sc[1], h.cc[1]));
    hi[2 * i + 1] = pack_h2(__hfma2(as_h2(and_or(v, 0x00F000F0u, 0x64006400u)), h.sc[1], h.cc[1]));
  }
}

struct Seg {  // one matrix of the launch, picked without dynamic indexing of the parameters
  unsigned rows, group0;
  float* y;
  size_t ldy, part;
};
__device__ __forceinline__ Seg pick_seg(const Q4Args& a, unsigned grp) {
  const int i = (grp >= a.group0[1]) + (grp >= a.group0[2]);
  Seg s;
  s.rows = i == 0 ? a.rows[0] : i == 1 ? a.rows[1] : a.rows[2];
  s.group0 = i == 0 ? a.group0[0] : i == 1 ? a.group0[1] : a.group0[2];
  s.y = i == 0 ? a.y[0] : i == 1 ? a.y[1] : a.y[2];
  s.ldy = i == 0 ? a.ldy[0] : i == 1 ? a.ldy[1] : a.ldy[2];
  s.part = i == 0 ? a.part_stride[0] : i == 1 ? a.part_stride[1] : a.part_stride[2];
  return s;
}

// Token rows in blocks of up to 64.  TQ: token rows per worker thread at most (tbn / 4: the four warps of a lane quadrant share the
// accumulator's columns).
template <int TQ>
__global__ void __launch_bounds__(Q_THREADS, 1) gemm_q4k_tc_kernel(const __grid_constant__ Q4Args a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t bars = sm32(smem);
  auto bar = [&](unsigned i) { return bars + 8u * i; };
  uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + QB_COUNT * 8);
  volatile unsigned* fail = reinterpret_cast<volatile unsigned*>(smem + QB_COUNT * 8 + 8);
  const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  constexpr unsigned Q_D = 224;                     // first accumulator
  const unsigned tbn = a.map.tbn;                   // token rows of a unit
  const unsigned b_group = 4u * 2u * tbn * 16u, b_stage = 9u * b_group;
  float* up_s = reinterpret_cast<float*>(smem + Q_HEAD);   // 2^e of every token row
  const uint32_t raw0 = bars + a.head, b0 = raw0 + a.n_raw * Q_RAW;
  const unsigned u0 = ks_gemm_first(a.map, blockIdx.x), n_units = a.map.base + (blockIdx.x < a.map.rem ? 1u : 0u);

  if (threadIdx.x == 0) {
    for (unsigned i = 0; i < a.n_raw; i++) {
      mb_init(bar(QB_RAW_FULL + i), 1);
      mb_init(bar(QB_RAW_FREE + i), Q_WARPS);
    }
    for (unsigned i = 0; i < a.n_b; i++) {
      mb_init(bar(QB_B_FULL + i), 1);
      mb_init(bar(QB_B_FREE + i), 1);
    }
    for (unsigned i = 0; i < 3; i++) {
      mb_init(bar(QB_A_FULL + i), Q_WARPS / 2);
      mb_init(bar(QB_A_FREE + i), 1);
    }
    for (unsigned i = 0; i < 2; i++) {
      mb_init(bar(QB_D_FULL + i), 1);
      mb_init(bar(QB_D_FREE + i), Q_WARPS);
    }
    mb_init(bar(QB_DONE), 1);
    mb_init(bar(QB_UP), 1);
    *fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 0) tc_alloc(sm32(tslot), 512);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (*tslot != 0u && threadIdx.x == 0) *fail = 1;  // all 512 columns were asked for: they start at 0
  constexpr uint32_t tmem = 0;

  if (warp < Q_WARPS) {
    // ---- workers
    const unsigned quad = warp & 3u, g = warp >> 2, half = g >> 1;
    const uint32_t tlane = tmem + ((quad * 32u) << 16);
    const unsigned row = quad * 32u + lane;
    const unsigned tq = tbn >> 2;                // tokens of this thread: [g * tq, + tq) of the unit's
    float acc[TQ], s_prev = 0.0f;
#pragma unroll
    for (int i = 0; i < TQ; i++) acc[i] = 0.0f;
    bool ok = true;
    unsigned wt = u0 / a.map.S, sb = u0 - wt * a.map.S, prev_wt = 0;   // work tile and super-block of the unit
    unsigned rs = 0, rph = 0;  // ring stage of the packed rows and its phase
    uint4 hraw = {}, qa = {}, qb = {};
    // the packed bytes of this thread, read one unit ahead: the reads overlap the accumulator's way out
    auto fetch = [&]() {
      const bool got = __all_sync(0xffffffffu, mb_wait(bar(QB_RAW_FULL + rs), rph, a.wait_limit));
      if (got) {
        const uint32_t blk = raw0 + rs * Q_RAW + row * KS_Q4K_BLOCK_BYTES;
        hraw = lds128(blk);
        qa = lds128(blk + 16u + 32u * g);
        qb = lds128(blk + 32u + 32u * g);
        __syncwarp();
        if (lane == 0) mb_arrive(bar(QB_RAW_FREE + rs));
        if (++rs == a.n_raw) {
          rs = 0;
          rph ^= 1u;
        }
      }
      return got;
    };
    if (n_units) ok = fetch();
    for (unsigned i = 0; i <= n_units && ok; i++) {
      // does the unit before this one end a work tile, or this CTA's share of one?
      const bool last = i == n_units || (i > 0 && sb == 0);
      float s_cur = 0.0f;
      // the first unit's weights need nothing of the kernels before this one; the waits below depend on the image, and what is
      // written at the end may still be read by them
      if (i == 1) asm volatile("griddepcontrol.wait;" ::: "memory");
      if (i < n_units) {
        Q4Hdr h;
        q4_header(hraw, g, h);
        s_cur = h.s;
        const unsigned n = 2u * i + half, slot = n % 3u;
        if (n >= 3u && !__all_sync(0xffffffffu, mb_wait(bar(QB_A_FREE + slot), (n / 3u - 1u) & 1u, a.wait_limit))) { ok = false; break; }
        tc_fence_after();
        const uint32_t at = tlane + slot * 64u + (g & 1u) * 32u;
        uint32_t lo[8], hi[8];
        q4_words(qa, h, lo, hi);
        tc_st8(at, lo);
        tc_st8(at + 16u, hi);
        q4_words(qb, h, lo, hi);
        tc_st8(at + 8u, lo);
        tc_st8(at + 24u, hi);
        tc_st4(tlane + Q_EXT + (i & 1u) * 16u + 4u * g, h.mhi, h.mhi, h.mlo, 0u);
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mb_arrive(bar(QB_A_FULL + slot));
        if (i + 1u < n_units && !fetch()) { ok = false; break; }
      }
      if (i > 0) {  // fold the previous super-block's accumulator
        const unsigned j = i - 1u, buf = j & 1u;
        if (!__all_sync(0xffffffffu, mb_wait(bar(QB_D_FULL + buf), (j >> 1) & 1u, a.wait_limit))) { ok = false; break; }
        tc_fence_after();
        const uint32_t dcol = tlane + Q_D + buf * 2u * tbn + g * tq;
        uint32_t d0[16], d1[16];
        if (TQ >= 16 && tq == 16u) {
          tc_ld16(dcol, d0);
          tc_ld16(dcol + tbn, d1);
        } else {
#pragma unroll
          for (int k = 0; k < TQ; k += 4)
            if ((unsigned)k < tq) {
              tc_ld4(dcol + k, d0 + k);
              tc_ld4(dcol + tbn + k, d1 + k);
            }
        }
        tc_wait_ld16(d0);
        tc_wait_ld16(d1);
#pragma unroll
        for (int k = 0; k < TQ; k++)
          if ((unsigned)(k & ~3) < tq) acc[k] = fmaf(s_prev, __uint_as_float(d0[k]) + __uint_as_float(d1[k]), acc[k]);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mb_arrive(bar(QB_D_FREE + buf));
        if (last) {
          const unsigned grp = prev_wt / a.map.tb, tok0 = (prev_wt - grp * a.map.tb) * tbn + g * tq;
          const Seg sg = pick_seg(a, grp);
          const unsigned out_row = (grp - sg.group0) * GM_ROWS + row;
          const unsigned pslot = blockIdx.x - ks_gemm_owner(a.map, prev_wt * a.map.S);
          float* y = sg.y + (size_t)pslot * sg.part + out_row;
          const bool live = out_row < sg.rows;
          if (!__all_sync(0xffffffffu, mb_wait(bar(QB_UP), 0u, a.wait_limit))) { ok = false; break; }
#pragma unroll
          for (int k = 0; k < TQ; k++) {
            const unsigned tok = tok0 + k;
            if ((unsigned)k < tq && tok < a.n_tok && live) y[(size_t)tok * sg.ldy] = acc[k] * up_s[tok];
            acc[k] = 0.0f;
          }
        }
      }
      s_prev = s_cur;
      prev_wt = wt;
      if (++sb == a.map.S) {
        sb = 0;
        wt++;
      }
    }
    if (!ok && lane == 0) *fail = 1;
  } else if (warp == Q_WARPS) {
    // ---- MMAs: the whole warp runs the loop, converged, and one elected lane issues (loop state and descriptors then stay in
    // uniform registers)
    const unsigned leader = elect_one();
    const unsigned ncol = 2u * tbn;   // x_hi and x_lo side by side
    const uint32_t idesc = (1u << 4) | ((ncol >> 3) << 17) | ((unsigned)(GM_ROWS >> 4) << 24);  // f32 accumulate, f16 x f16, K-major both
    const uint64_t bdesc0 = tc_desc(b0, 2u * tbn * 16u, 128u);
    const unsigned chunk2 = 4u * tbn;   // in descriptor units of 16 bytes: two chunks of 8 k
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // What an MMA takes has to be in uniform registers when it issues.  It gets there by itself only while the compiler can see
    // that the warp stays together: loop bounds from launch parameters and blockIdx, no value out of memory (hence the
    // constant tensor-memory base), one way out.  Otherwise every MMA waits for five register moves, about 200 cycles.
    bool ok = false;
    unsigned bs = 0, bph = 0;   // B stage and its phase
    unsigned sl = 0, sph = 0;   // A slot and its phase: the slots are taken in the order the MMAs go
    for (unsigned i = 0; i < n_units; i++) {
      const unsigned buf = i & 1u;
      const uint32_t d = tmem + Q_D + buf * ncol;
#pragma unroll
      for (unsigned hf = 0; hf < 2; hf++) {
        bool got = true;
        if (hf == 0 && i >= 2u) got = mb_wait(bar(QB_D_FREE + buf), ((i >> 1) - 1u) & 1u, a.wait_limit);
        got = got && mb_wait(bar(QB_A_FULL + sl), sph, a.wait_limit);
        if (hf == 0) got = got && mb_wait(bar(QB_B_FULL + bs), bph, a.wait_limit);
        if (!__all_sync(0xffffffffu, got)) goto out;
        tc_fence_after();
        if (leader) {
          const uint64_t bd = bdesc0 + (uint64_t)(bs * (b_stage >> 4)) + (uint64_t)((hf ? 4u : 0u) * (b_group >> 4));
#pragma unroll
          for (unsigned kg = 0; kg < 4u + hf; kg++) {  // groups of 32 k; the fifth: the minima
            const uint32_t at = kg == 4u ? tmem + Q_EXT + (i & 1u) * 16u : tmem + sl * 64u + kg * 16u;
            const uint64_t b = bd + (uint64_t)(kg * (b_group >> 4));
            tc_mma_f16_ta(d, at, b, idesc, (hf | kg) ? 1u : 0u);
            tc_mma_f16_ta(d, at + 8u, b + chunk2, idesc, 1u);
          }
          tc_commit(bar(QB_A_FREE + sl));
          if (hf) {
            tc_commit(bar(QB_B_FREE + bs));
            tc_commit(bar(QB_D_FULL + buf));
          }
        }
        __syncwarp();
        if (++sl == 3u) {
          sl = 0;
          sph ^= 1u;
        }
      }
      if (++bs == a.n_b) {
        bs = 0;
        bph ^= 1u;
      }
    }
    ok = true;
  out:
    // every MMA issued must finish before shared and tensor memory go away (bounded): a last commit tracks them all
    if (leader) {
      if (!ok) *fail = 1;
      tc_commit(bar(QB_DONE));
    }
    __syncwarp();
    mb_wait(bar(QB_DONE), 0u, Q_WAIT);
  } else if (warp == Q_WARPS + 1) {
    // ---- packed rows: they depend on no kernel before this one
    const unsigned leader = elect_one();
    unsigned issued = 0, st = 0, ph = 1, wt = u0 / a.map.S, sb = u0 - wt * a.map.S;
    for (unsigned i = 0; i < n_units; i++) {
      const bool got = i < a.n_raw || mb_wait(bar(QB_RAW_FREE + st), ph, a.wait_limit);
      if (!__all_sync(0xffffffffu, got)) {
        if (leader) *fail = 1;
        break;
      }
      if (leader) {
        const unsigned grp = wt / a.map.tb;
        const int k = (grp >= a.group0[1]) + (grp >= a.group0[2]);
        const unsigned g0 = k == 0 ? a.group0[0] : k == 1 ? a.group0[1] : a.group0[2];
        mb_expect(bar(QB_RAW_FULL + st), Q_RAW);  // rows past the matrix come as zeros and count
        tma_in_2d(raw0 + st * Q_RAW, k == 0 ? &a.w[0] : k == 1 ? &a.w[1] : &a.w[2], sb * KS_Q4K_BLOCK_BYTES, (grp - g0) * GM_ROWS,
                  bar(QB_RAW_FULL + st));
      }
      issued++;
      if (++st == a.n_raw) {
        st = 0;
        ph ^= 1u;
      }
      if (++sb == a.map.S) {
        sb = 0;
        wt++;
      }
      __syncwarp();
    }
    for (unsigned j = issued > a.n_raw ? issued - a.n_raw : 0u; j < issued; j++) mb_wait(bar(QB_RAW_FULL + j % a.n_raw), (j / a.n_raw) & 1u, a.wait_limit);
  } else {
    // ---- token rows
    const unsigned leader = elect_one();
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the image comes from the kernel before this one
    const float* up = reinterpret_cast<const float*>(a.xt + xt_scale_off(a.cols, a.np));
    if (leader) {
      mb_expect(bar(QB_UP), a.np * 4u);  // np: a multiple of 16
      bulk_in(sm32(up_s), up, a.np * 4u, bar(QB_UP));
    }
    __syncwarp();
    unsigned issued = 0, wt = u0 / a.map.S, sb = u0 - wt * a.map.S, st = 0, ph = 1;
    for (unsigned j = 0; j < n_units; j++) {  // a super-block each
      const bool got = j < a.n_b || mb_wait(bar(QB_B_FREE + st), ph, a.wait_limit);
      if (!__all_sync(0xffffffffu, got)) {
        if (leader) *fail = 1;
        break;
      }
      if (a.test_stall && j + 1u == a.test_stall) break;  // test hook: this unit's token rows never arrive
      if (leader) {
        mb_expect(bar(QB_B_FULL + st), b_stage);
        const size_t at = ((size_t)(wt % a.map.tb) * a.map.S + sb) * b_stage;
        bulk_in(b0 + st * b_stage, reinterpret_cast<const unsigned char*>(a.xt) + at, b_stage, bar(QB_B_FULL + st));
      }
      issued++;
      if (++st == a.n_b) {
        st = 0;
        ph ^= 1u;
      }
      if (++sb == a.map.S) {
        sb = 0;
        wt++;
      }
      __syncwarp();
    }
    for (unsigned j = issued > a.n_b ? issued - a.n_b : 0u; j < issued; j++) mb_wait(bar(QB_B_FULL + j % a.n_b), (j / a.n_b) & 1u, a.wait_limit);
    mb_wait(bar(QB_UP), 0u, a.wait_limit);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x == 0 && *fail) atomicOr(a.err, 8u);
  if (warp == 0) tc_dealloc(tmem, 512);
}

// Token rows in blocks of 65 to 128.  A unit is a super-block of TWO row tiles: the token rows of a half super-block
// (4 groups of 32 k, or 5 with the minima's) are brought in once and the MMAs of the tiles alternate between two accumulators,
//   (tile 0, half 0) (tile 1, half 0) (tile 0, half 1) (tile 1, half 1),
// which halves the traffic of B from L2 (one tile against 256 rows at once read B at 8.9 TB/s and could not go faster).
// Converting and folding are different warps: with the same 16 warps doing both, the MMAs waited 60 % of the time for an
// accumulator whose folders stood before a slot of A (13.4k cycles per unit, MMAs 4.5k).  Eight warps convert (32 rows x 128 k
// each), eight fold (32 rows x half the tokens of both tiles: 128 sums per thread, hence the register split 56 / 168 / 32 of the
// 96 a thread is launched with).
constexpr unsigned QW_THREADS = 640;  // 5 groups of 4 warps
constexpr unsigned QW_D = 256;
__global__ void __launch_bounds__(QW_THREADS, 1) gemm_q4k_wide_kernel(const __grid_constant__ Q4Args a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const uint32_t bars = sm32(smem);
  auto bar = [&](unsigned i) { return bars + 8u * i; };
  uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + QB_COUNT * 8);
  volatile unsigned* fail = reinterpret_cast<volatile unsigned*>(smem + QB_COUNT * 8 + 8);
  const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const unsigned tbn = a.map.tbn;
  const unsigned b_group = 4u * 2u * tbn * 16u, b_stage = 5u * b_group;
  float* s_s = reinterpret_cast<float*>(smem + Q_HEAD);    // [4][128]: s of the rows of the last tiles, converters to folders
  float* up_s = s_s + 4 * GM_ROWS;                         // 2^e of every token row
  const uint32_t raw0 = bars + a.head, b0 = raw0 + a.n_raw * Q_RAW;
  const unsigned u0 = ks_gemm_first(a.map, blockIdx.x), n_units = a.map.base + (blockIdx.x < a.map.rem ? 1u : 0u);

  if (threadIdx.x == 0) {
    for (unsigned i = 0; i < a.n_raw; i++) {
      mb_init(bar(QB_RAW_FULL + i), 1);
      mb_init(bar(QB_RAW_FREE + i), 8);
    }
    for (unsigned i = 0; i < a.n_b; i++) {
      mb_init(bar(QB_B_FULL + i), 1);
      mb_init(bar(QB_B_FREE + i), 1);
    }
    for (unsigned i = 0; i < 3; i++) {
      mb_init(bar(QB_A_FULL + i), 4);
      mb_init(bar(QB_A_FREE + i), 1);
    }
    for (unsigned i = 0; i < 2; i++) {
      mb_init(bar(QB_D_FULL + i), 1);
      mb_init(bar(QB_D_FREE + i), 8);
    }
    mb_init(bar(QB_DONE), 1);
    mb_init(bar(QB_UP), 1);
    *fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 0) tc_alloc(sm32(tslot), 512);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (*tslot != 0u && threadIdx.x == 0) *fail = 1;  // all 512 columns were asked for: they start at 0
  constexpr uint32_t tmem = 0;

  if (warp < 8u) {
    // ---- converters
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    const unsigned quad = warp & 3u, half = warp >> 2, row = quad * 32u + lane;
    const uint32_t tlane = tmem + ((quad * 32u) << 16);
    bool ok = true;
    unsigned rs = 0, rph = 0;                        // ring stage of the packed rows and its phase
    unsigned n = 2u * half, slot = n, sph = 1;       // A slot and the phase in which it is free
    for (unsigned v = 0; v < 2u * n_units && ok; v++) {  // row tiles of units
      if (!__all_sync(0xffffffffu, mb_wait(bar(QB_RAW_FULL + rs), rph, a.wait_limit))) { ok = false; break; }
      const uint32_t blk = raw0 + rs * Q_RAW + row * KS_Q4K_BLOCK_BYTES;
      const uint4 hraw = lds128(blk);
      if (n >= 3u && !__all_sync(0xffffffffu, mb_wait(bar(QB_A_FREE + slot), sph, a.wait_limit))) { ok = false; break; }
      tc_fence_after();
#pragma unroll
      for (unsigned gg = 0; gg < 2; gg++) {
        const unsigned g = 2u * half + gg;
        const uint4 qa = lds128(blk + 16u + 32u * g), qb = lds128(blk + 32u + 32u * g);
        Q4Hdr h;
        q4_header(hraw, g, h);
        if (g == 0) s_s[(v & 3u) * 128u + row] = h.s;
        const uint32_t at = tlane + slot * 64u + gg * 32u;
        uint32_t lo[8], hi[8];
        q4_words(qa, h, lo, hi);
        tc_st8(at, lo);
        tc_st8(at + 16u, hi);
        q4_words(qb, h, lo, hi);
        tc_st8(at + 8u, lo);
        tc_st8(at + 24u, hi);
        tc_st4(tlane + Q_EXT + (v & 3u) * 16u + 4u * g, h.mhi, h.mhi, h.mlo, 0u);
      }
      __syncwarp();
      if (lane == 0) mb_arrive(bar(QB_RAW_FREE + rs));  // the packed bytes are in registers (and used)
      if (++rs == a.n_raw) {
        rs = 0;
        rph ^= 1u;
      }
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mb_arrive(bar(QB_A_FULL + slot));
      // slots go 4 i + t + 2 half: one on from tile 0 to tile 1, three (the same slot) to the next unit's tile 0
      const unsigned step = (v & 1u) ? 3u : 1u;
      n += step;
      slot += step;
      if (slot >= 3u) {
        slot -= 3u;
        sph ^= 1u;
      }
    }
    if (!ok && lane == 0) *fail = 1;
  } else if (warp < 16u) {
    // ---- folders
    asm volatile("setmaxnreg.inc.sync.aligned.u32 168;");
    const unsigned quad = warp & 3u, th = (warp >> 2) & 1u, row = quad * 32u + lane, tq = tbn >> 1;  // tokens [th * tq, + tq) of the unit's
    const uint32_t tlane = tmem + ((quad * 32u) << 16);
    float acc[2][64];
#pragma unroll
    for (int t = 0; t < 2; t++)
#pragma unroll
      for (int k = 0; k < 64; k++) acc[t][k] = 0.0f;
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the kernels before this one may still read what is written here
    bool ok = true;
    unsigned wt = u0 / a.map.S, sb = u0 - wt * a.map.S;
    for (unsigned i = 0; i < n_units && ok; i++) {
      const bool last = i + 1u == n_units || sb + 1u == a.map.S;  // the work tile, or this CTA's share of it, ends here
#pragma unroll
      for (unsigned t = 0; t < 2; t++) {
        if (!__all_sync(0xffffffffu, mb_wait(bar(QB_D_FULL + t), i & 1u, a.wait_limit))) { ok = false; break; }
        tc_fence_after();
        const float s = s_s[((2u * i + t) & 3u) * 128u + row];
        const uint32_t dcol = tlane + QW_D + t * tbn + th * tq;
#pragma unroll
        for (int c = 0; c < 64; c += 16) {
          if ((unsigned)c < tq) {
            uint32_t d0[16];
            if ((unsigned)c + 16u <= tq) {
              tc_ld16(dcol + c, d0);
            } else {
              tc_ld4(dcol + c, d0);
              tc_ld4(dcol + c + 4, d0 + 4);
            }
            tc_wait_ld16(d0);
#pragma unroll
            for (int k = 0; k < 16; k++)
              if (k < 8 || (unsigned)c + 16u <= tq) acc[t][c + k] = fmaf(s, __uint_as_float(d0[k]), acc[t][c + k]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mb_arrive(bar(QB_D_FREE + t));
        if (last) {
          const unsigned grp = wt / a.map.tb, tblk = wt - grp * a.map.tb;
          const Seg sg = pick_seg(a, grp);
          const unsigned out_row = ((grp - sg.group0) * 2u + t) * GM_ROWS + row, tok0 = tblk * tbn + th * tq;
          const unsigned pslot = blockIdx.x - ks_gemm_owner(a.map, wt * a.map.S);
          float* y = sg.y + (size_t)pslot * sg.part + (size_t)tok0 * sg.ldy + out_row;
          const unsigned n_tok = out_row < sg.rows ? a.n_tok : 0u;
          if (!__all_sync(0xffffffffu, mb_wait(bar(QB_UP), 0u, a.wait_limit))) { ok = false; break; }
#pragma unroll
          for (int k = 0; k < 64; k++) {
            if ((unsigned)k < tq && tok0 + k < n_tok) *y = acc[t][k] * up_s[tok0 + k];
            y += sg.ldy;
            acc[t][k] = 0.0f;
          }
        }
      }
      if (++sb == a.map.S) {
        sb = 0;
        wt++;
      }
    }
    if (!ok && lane == 0) *fail = 1;
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
    if (warp == 16u) {
    // ---- MMAs: see above
    const unsigned leader = elect_one();
    const uint32_t idesc = (1u << 4) | ((tbn >> 3) << 17) | ((unsigned)(GM_ROWS >> 4) << 24);  // f32 accumulate, f16 x f16, K-major both
    const uint64_t bdesc0 = tc_desc(b0, 2u * tbn * 16u, 128u);
    const unsigned chunk2 = 4u * tbn, lo_rows = tbn;   // in descriptor units of 16 bytes: two chunks of 8 k, the hi rows
    asm volatile("griddepcontrol.wait;" ::: "memory");
    bool ok = false;
    unsigned bs = 0, bph = 0;   // B stage and its phase
    unsigned sl = 0, sph = 0;   // A slot and its phase: the slots are taken in the order the MMAs go
    for (unsigned i = 0; i < n_units; i++) {
#pragma unroll
      for (unsigned hf = 0; hf < 2; hf++) {
#pragma unroll
        for (unsigned t = 0; t < 2; t++) {
          const uint32_t d = tmem + QW_D + t * tbn;
          bool got = true;
          if (hf == 0 && i >= 1u) got = mb_wait(bar(QB_D_FREE + t), (i - 1u) & 1u, a.wait_limit);
          got = got && mb_wait(bar(QB_A_FULL + sl), sph, a.wait_limit);
          if (t == 0) got = got && mb_wait(bar(QB_B_FULL + bs), bph, a.wait_limit);
          if (!__all_sync(0xffffffffu, got)) goto out;
          tc_fence_after();
          if (leader) {
            const uint64_t bd = bdesc0 + (uint64_t)(bs * (b_stage >> 4));
#pragma unroll
            for (unsigned kg = 0; kg < 4u + hf; kg++) {  // groups of 32 k; the fifth: the minima
              const bool ext = kg == 4u;
              const uint32_t at = ext ? tmem + Q_EXT + ((2u * i + t) & 3u) * 16u : tmem + sl * 64u + kg * 16u;
              const uint64_t b = bd + (uint64_t)(kg * (b_group >> 4));
              tc_mma_f16_ta(d, at, b, idesc, (hf | kg) ? 1u : 0u);
              if (!ext) tc_mma_f16_ta(d, at, b + lo_rows, idesc, 1u);
              tc_mma_f16_ta(d, at + 8u, b + chunk2, idesc, 1u);
              if (!ext) tc_mma_f16_ta(d, at + 8u, b + chunk2 + lo_rows, idesc, 1u);
            }
            tc_commit(bar(QB_A_FREE + sl));
            if (t) tc_commit(bar(QB_B_FREE + bs));
            if (hf) tc_commit(bar(QB_D_FULL + t));
          }
          __syncwarp();
          if (++sl == 3u) {
            sl = 0;
            sph ^= 1u;
          }
        }
        if (++bs == a.n_b) {
          bs = 0;
          bph ^= 1u;
        }
      }
    }
    ok = true;
  out:
    // every MMA issued must finish before shared and tensor memory go away (bounded): a last commit tracks them all
    if (leader) {
      if (!ok) *fail = 1;
      tc_commit(bar(QB_DONE));
    }
    __syncwarp();
    mb_wait(bar(QB_DONE), 0u, Q_WAIT);
    } else if (warp == 17u) {
    // ---- packed rows: they depend on no kernel before this one
    const unsigned leader = elect_one();
    unsigned issued = 0, st = 0, ph = 1, wt = u0 / a.map.S, sb = u0 - wt * a.map.S, t = 0;
    for (unsigned i = 0; i < 2u * n_units; i++) {
      const bool got = i < a.n_raw || mb_wait(bar(QB_RAW_FREE + st), ph, a.wait_limit);
      if (!__all_sync(0xffffffffu, got)) {
        if (leader) *fail = 1;
        break;
      }
      if (leader) {
        const unsigned grp = wt / a.map.tb;
        const int k = (grp >= a.group0[1]) + (grp >= a.group0[2]);
        const unsigned g0 = k == 0 ? a.group0[0] : k == 1 ? a.group0[1] : a.group0[2];
        mb_expect(bar(QB_RAW_FULL + st), Q_RAW);  // rows past the matrix come as zeros and count
        tma_in_2d(raw0 + st * Q_RAW, k == 0 ? &a.w[0] : k == 1 ? &a.w[1] : &a.w[2], sb * KS_Q4K_BLOCK_BYTES, ((grp - g0) * 2u + t) * GM_ROWS,
                  bar(QB_RAW_FULL + st));
      }
      issued++;
      if (++st == a.n_raw) {
        st = 0;
        ph ^= 1u;
      }
      if (++t == 2u) {
        t = 0;
        if (++sb == a.map.S) {
          sb = 0;
          wt++;
        }
      }
      __syncwarp();
    }
    for (unsigned j = issued > a.n_raw ? issued - a.n_raw : 0u; j < issued; j++) mb_wait(bar(QB_RAW_FULL + j % a.n_raw), (j / a.n_raw) & 1u, a.wait_limit);
    } else if (warp == 18u) {
    // ---- token rows
    const unsigned leader = elect_one();
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the image comes from the kernel before this one
    const float* up = reinterpret_cast<const float*>(a.xt + xt_scale_off(a.cols, a.np));
    if (leader) {
      mb_expect(bar(QB_UP), a.np * 4u);  // np: a multiple of 16
      bulk_in(sm32(up_s), up, a.np * 4u, bar(QB_UP));
    }
    __syncwarp();
    unsigned issued = 0, wt = u0 / a.map.S, sb = u0 - wt * a.map.S, hf = 0, st = 0, ph = 1;
    for (unsigned j = 0; j < 2u * n_units; j++) {  // halves of a super-block: 4 and 5 groups
      const bool got = j < a.n_b || mb_wait(bar(QB_B_FREE + st), ph, a.wait_limit);
      if (!__all_sync(0xffffffffu, got)) {
        if (leader) *fail = 1;
        break;
      }
      if (a.test_stall && j / 2u + 1u == a.test_stall) break;  // test hook: this unit's token rows never arrive
      if (leader) {
        const unsigned tblk = wt % a.map.tb, bytes = (4u + hf) * b_group;
        const size_t at = (((size_t)tblk * a.map.S + sb) * 9u + 4u * hf) * b_group;
        mb_expect(bar(QB_B_FULL + st), bytes);
        bulk_in(b0 + st * b_stage, reinterpret_cast<const unsigned char*>(a.xt) + at, bytes, bar(QB_B_FULL + st));
      }
      issued++;
      if (++st == a.n_b) {
        st = 0;
        ph ^= 1u;
      }
      if (++hf == 2u) {
        hf = 0;
        if (++sb == a.map.S) {
          sb = 0;
          wt++;
        }
      }
      __syncwarp();
    }
    for (unsigned j = issued > a.n_b ? issued - a.n_b : 0u; j < issued; j++) mb_wait(bar(QB_B_FULL + j % a.n_b), (j / a.n_b) & 1u, a.wait_limit);
    mb_wait(bar(QB_UP), 0u, a.wait_limit);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x == 0 && *fail) atomicOr(a.err, 8u);
  if (warp == 0) tc_dealloc(tmem, 512);
}

typedef CUresult (*encode_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                              const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
encode_fn tensor_map_encoder() {
  static encode_fn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
    return reinterpret_cast<encode_fn>(p);
  }();
  return fn;
}

// Ring depths: two B stages at least, then packed rows up to the four units that cover the latency of memory, then whatever
// of either still fits.
size_t q4_rings(const ks_ctx* ctx, unsigned tbn, unsigned nt, unsigned np, Q4Args& a) {
  a.head = (Q_HEAD + (nt == 1 ? 0u : 4u * GM_ROWS * 4u) + np * 4u + 1023u) & ~1023u;
  const size_t room = ctx->smem_optin - a.head, stage = (size_t)(nt == 1 ? 9 : 5) * tbn * 128u;
  unsigned n_raw = 2, n_b = 2;
  auto fits = [&](unsigned r, unsigned b) { return r <= Q_MAX_RAW && b <= Q_MAX_B && b * stage + r * Q_RAW <= room; };
  while (n_raw < 4 && fits(n_raw + 1, n_b)) ++n_raw;
  while (fits(n_raw, n_b + 1)) ++n_b;
  while (fits(n_raw + 1, n_b)) ++n_raw;
  a.n_raw = n_raw;
  a.n_b = n_b;
  return a.head + n_b * stage + n_raw * Q_RAW;
}
}  // namespace

// How many CTAs a launch takes, by an estimate in us.  A CTA's time is its units and writing its shares of work tiles; sums that
// several CTAs share are then read once more by a second launch.  The constants are fitted to 300..18363 rows x 512..10240
// columns x 70..256 token rows, measured with single tiles and with pairs: choosing between the two by this estimate loses
// 0.5 % against the better one.
ks_gemm_map ks_gemm_q4k_map(const ks_ctx* ctx, const size_t* rows, int n_seg, unsigned cols, unsigned np, unsigned tbn, bool plain,
                            double* cost_out) {
  ks_gemm_map m{};
  m.S = cols / 256u;
  m.tbn = tbn;
  m.tb = np / m.tbn;
  m.nt = tbn > 64u ? 2u : 1u;
  unsigned wtiles = 0;
  for (int i = 0; i < n_seg; i++) wtiles += (unsigned)(((rows[i] + GM_ROWS - 1) / GM_ROWS + m.nt - 1) / m.nt);
  wtiles *= m.tb;
  const unsigned U = wtiles * m.S, most = (unsigned)ctx->sm_count < U ? (unsigned)ctx->sm_count : U;
  // the choice of the last few shapes is kept (a call asks three to seven times: 0.6 us each)
  struct Kept {
    unsigned most = 0, wtiles = 0, S = 0, tbn = 0, plain = 0, G = 0;
    double cost = 0;
  };
  static thread_local Kept kept[64];
  Kept& k = kept[(wtiles * 31u + m.S * 7u + m.tbn / 8u + plain) % 64u];
  if (k.most != most || k.wtiles != wtiles || k.S != m.S || k.tbn != m.tbn || k.plain != (unsigned)plain) {
    const double t_u = m.nt == 2 ? 0.95 + m.tbn * 0.0316 : 1.0 + m.tbn * 0.011, t_w = (0.15 + m.tbn * 0.0075) * m.nt, start = m.nt == 2 ? 2.0 : 0.0;
    double best = 1e30;
    for (unsigned G = 1; G <= most; G++) {
      if (G < most && wtiles % G && G * 4u < most * 3u) continue;
      const bool whole = plain && wtiles % G == 0;  // no work tile is shared
      const unsigned per = (U + G - 1) / G, shares = whole ? wtiles / G : (per + m.S - 2) / m.S + 1;
      const double again = whole ? 0.0 : 2.5 + ((double)G / wtiles + 2.0) * wtiles * m.nt * m.tbn * (GM_ROWS * 4e-6 / 4.0);
      const double cost = start + per * t_u + shares * t_w + again;
      if (cost < best) {
        best = cost;
        m.G = G;
      }
    }
    k = {most, wtiles, m.S, m.tbn, (unsigned)plain, m.G, best};
  }
  m.G = k.G;
  m.base = U / m.G;
  m.rem = U % m.G;
  if (cost_out) *cost_out = k.cost;
  return m;
}

int ks_launch_gemm_q4k(ks_ctx* ctx, const ks_gemm_job& job) {
  encode_fn enc = tensor_map_encoder();
  if (!enc) return ks_fail(ctx, KS_ERR_CUDA, "gemm: cuTensorMapEncodeTiled is not available");
  Q4Args a;
  memset(&a, 0, sizeof a);
  const cuuint64_t row_bytes = (cuuint64_t)job.cols / 256 * KS_Q4K_BLOCK_BYTES;
  unsigned groups = 0;
  for (int i = 0; i < 3; i++) {
    a.group0[i] = i < job.n_seg ? groups : 0xFFFFFFFFu;  // no unit reaches an absent matrix
    if (i >= job.n_seg) continue;
    a.rows[i] = (unsigned)job.rows[i];
    a.y[i] = job.y[i];
    a.ldy[i] = job.ldy[i];
    a.part_stride[i] = job.part_stride[i];
    groups += (unsigned)(((job.rows[i] + GM_ROWS - 1) / GM_ROWS + job.map.nt - 1) / job.map.nt);
    const cuuint64_t dims[2] = {row_bytes, (cuuint64_t)job.rows[i]}, strides[1] = {row_bytes};
    const cuuint32_t box[2] = {KS_Q4K_BLOCK_BYTES, GM_ROWS}, es[2] = {1, 1};
    if (enc(&a.w[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(job.W[i]), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return ks_fail(ctx, KS_ERR_INVALID, "gemm: the packed rows cannot be described to TMA (base must be 16-byte aligned)");
  }
  a.map = job.map;
  a.xt = job.xt;
  a.cols = job.cols;
  a.n_tok = job.n_tok;
  a.np = job.np;
  const unsigned tbn = job.map.tbn;
  const int c = tbn <= 16 ? 0 : tbn <= 32 ? 1 : tbn <= 64 ? 2 : 3;
  const size_t smem = q4_rings(ctx, job.map.tbn, job.map.nt, job.np, a);
  a.err = (unsigned*)ctx->ws + KS_WS_ERR_WORD;
  a.wait_limit = Q_WAIT;
  if (const char* t = getenv("KSEARCH_GEMM_TEST_STALL")) {  // exercises the give-up path: short waits, one operand withheld
    a.test_stall = (unsigned)atoi(t);
    if (a.test_stall) a.wait_limit = 4000;
  }
  void (*kern)(Q4Args) = c == 0 ? gemm_q4k_tc_kernel<4> : c == 1 ? gemm_q4k_tc_kernel<8> : c == 2 ? gemm_q4k_tc_kernel<16> : gemm_q4k_wide_kernel;
  static size_t set[4][16] = {{0}};
  size_t& have = set[c][ctx->device & 15];
  if (smem > have) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return ks_fail(ctx, KS_ERR_CUDA, "gemm: cannot set %zu B shared memory: %s", smem, cudaGetErrorString(e));
    have = smem;
  }
  KS_LAUNCH(ctx, kern, dim3(job.map.G), c == 3 ? QW_THREADS : Q_THREADS, smem, a);
  return ks_after_launch(ctx, "gemm_q4k_tc");
}
