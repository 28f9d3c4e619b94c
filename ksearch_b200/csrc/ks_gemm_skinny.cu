// Q4_K weights x 1..8 token rows on the tensor cores (mma.sync m16n8k16): the matrices of a decode step of several slots.
//
// The reference's op is the batch matvec (crates/ksearch_kernels/src/lib.rs:1414).  With so few rows the tcgen05 kernel is a
// chain of short hand-overs (packed rows -> tensor memory -> MMA -> fold: 2 us per 18 KB of weights); here a warp owns 128
// columns (half a super-block) for ALL the row tiles of its block:
//   * its share of the token rows, two f16 terms of each value, sits in 32 registers as B fragments and is loaded once;
//   * packed rows come by cp.async into a ring of the warp's own (16 rows x 80 bytes per tile), requested before the wait for
//     the previous kernel; no warp waits for another inside a tile;
//   * A is q - 8 as f16, exact, by one LOP3 and one HADD2 (HFMA2) per two weights.  Tokens are the 8 columns; their second and
//     first terms go into the same f32 sums of a 32-column sub-block, the small ones first, which then take the sub-block's
//     scale in f32.  The eights and the minima are two more mmas: A = scales, minima, B = the image's sub-block sums.
//     (The nibble masked in place is the f16 subnormal q 2^-24 and saves the HADD2, but products seem to be aligned by their
//     operands' exponents, not by their own leading bits: the error against 64 bits was 4 times the matvec's on normal rows and
//     20 to 40 times on rows with outliers.  Centred operands keep the sums as small as the result.);
//   * the warps' sums of a tile meet in shared memory, four tiles at a time, in warp order.
// The block's columns are one of `splits` shares of the row (at most 20 warps of 128); every share leaves one partial.
// Bound by instructions (about 190 per warp and tile of 16 x 128 weights) where there are many rows, else by the latency of
// the ring and the launch.
#include <cstdlib>

#include "ks_gemm.h"

namespace {

constexpr unsigned SK_RING = 4, SK_ROW = 96, SK_ITEM = 16 * SK_ROW;  // stages per warp; bytes per row (80 used: conflict-free reads)
constexpr unsigned SK_GROUP = 4;                                      // tiles whose sums meet at once
constexpr unsigned SK_MAX_WARPS = 20;

struct SkinnyArgs {
  const uint8_t* W[3];
  float* y[3];
  size_t ldy[3], part_stride[3];
  unsigned rows[3], tile0[4];   // 16-row tiles
  unsigned row_bytes, cols, n_tok, np;
  unsigned warps, splits, per_split;  // blocks per split
  const __half* xt;
};

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// The four scales and the four minima (6 bits each, one per byte) of half a super-block's sub-blocks (get_scale_min_k4,
// gguf_impl.rs:563-573).
__device__ __forceinline__ void header_half(const uint4 h, unsigned half, uint32_t& sc, uint32_t& mn) {
  if (half == 0) {
    sc = h.y & 0x3F3F3F3Fu;
    mn = h.z & 0x3F3F3F3Fu;
  } else {
    sc = (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
    mn = ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u);
  }
}
// The nibbles 0 (1) of bytes 0 and 2 as two halves n - 8.
__device__ __forceinline__ uint32_t nib_lo(uint32_t w) { return pack_h2(__hadd2(as_h2((w & 0x000F000Fu) | 0x64006400u), __float2half2_rn(-1032.0f))); }
__device__ __forceinline__ uint32_t nib_hi(uint32_t w) {
  return pack_h2(__hfma2(as_h2((w & 0x00F000F0u) | 0x64006400u), __float2half2_rn(0.0625f), __float2half2_rn(-72.0f)));
}
// Two of four bytes below 64 as halves (sel: 0x4140 the first two, 0x4342 the last two).
__device__ __forceinline__ uint32_t bytes_h2(uint32_t v, uint32_t sel) {
  return pack_h2(__hsub2(as_h2(__byte_perm(v, 0x64646464u, sel)), __float2half2_rn(1024.0f)));
}
// Byte j of v as a float.
__device__ __forceinline__ float byte_f(uint32_t v, unsigned j) { return __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7540u + j)) - 8388608.0f; }

__global__ void __launch_bounds__(SK_MAX_WARPS * 32, 1) gemm_q4k_skinny_kernel(const __grid_constant__ SkinnyArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3u;
  const unsigned split = blockIdx.x / a.per_split, b = blockIdx.x - split * a.per_split;
  const unsigned tiles = a.tile0[3], base = tiles / a.per_split, rem = tiles - base * a.per_split;
  const unsigned first = b * base + min(b, rem), n = base + (b < rem ? 1u : 0u);
  const unsigned hidx = split * a.warps + warp, sb = hidx >> 1, half = hidx & 1u;  // this warp's super-block and half of it
  const unsigned char* stage0 = smem + warp * (SK_RING * SK_ITEM);
  const uint32_t ring = sm32(stage0);
  float* psum = reinterpret_cast<float*>(smem + a.warps * (SK_RING * SK_ITEM));    // [2][SK_GROUP][warps][16 rows][8 tokens]

  // ---- packed rows: lane copies chunks lane, lane + 32, lane + 64 of the 80 16-byte chunks of a tile (chunk = row * 5 + part)
  unsigned cr[3], cin[3];
  uint32_t cdst[3];
#pragma unroll
  for (unsigned i = 0; i < 3; i++) {
    const unsigned c = lane + 32u * i, part = c % 5u;
    cr[i] = c / 5u;
    cin[i] = part ? 16u * part + 64u * half : 0u;
    cdst[i] = ring + cr[i] * SK_ROW + part * 16u;
  }
  auto fetch = [&](unsigned k) {
    if (k < n) {
      const unsigned tile = first + k;
      const int seg = (tile >= a.tile0[1]) + (tile >= a.tile0[2]);
      const uint8_t* W = seg == 0 ? a.W[0] : seg == 1 ? a.W[1] : a.W[2];
      const unsigned rows = seg == 0 ? a.rows[0] : seg == 1 ? a.rows[1] : a.rows[2];
      const unsigned r0 = (tile - (seg == 0 ? a.tile0[0] : seg == 1 ? a.tile0[1] : a.tile0[2])) * 16u, last = rows - 1u - r0;
      const uint8_t* src = W + (size_t)r0 * a.row_bytes + sb * KS_Q4K_BLOCK_BYTES;
      const uint32_t to = (k % SK_RING) * SK_ITEM;
#pragma unroll
      for (unsigned i = 0; i < 3; i++)
        if (i < 2u || lane < 16u)
          asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(cdst[i] + to), "l"(src + (min(cr[i], last) * a.row_bytes + cin[i])) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (unsigned k = 0; k < SK_RING - 1u; k++) fetch(k);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the image comes from the kernel before this one

  // ---- this warp's columns of the token rows (the q4k form of the image): B fragments and sub-block sums
  uint4 bh[4], bl[4];   // sub-blocks 4 half + j: tokens' first and second terms, column g
  uint32_t bs;          // lanes t = 0, 1: first terms of the sums of sub-blocks 2t, 2t + 1; t = 2, 3: their second terms
  {
    const __half* x = a.xt + (size_t)sb * 36u * 2u * a.np * 8u;
#pragma unroll
    for (unsigned j = 0; j < 4; j++) {
      const __half* c = x + (size_t)((4u * half + j) * 4u + t) * 2u * a.np * 8u + g * 8u;
      bh[j] = *reinterpret_cast<const uint4*>(c);
      bl[j] = *reinterpret_cast<const uint4*>(c + (size_t)a.np * 8u);
    }
    bs = *reinterpret_cast<const uint32_t*>(x + (size_t)(32u + 2u * half + (t & 1u)) * 2u * a.np * 8u + g * 8u + 2u * (t >> 1));
  }
  const float* up = reinterpret_cast<const float*>(a.xt + xt_scale_off(a.cols, a.np));
  const uint32_t msel = (t & 1u) ? 0x4342u : 0x4140u;  // this lane's two scales and minima
  unsigned buf = 0;

  for (unsigned k0 = 0; k0 < n; k0 += SK_GROUP) {
    const unsigned kn = min(SK_GROUP, n - k0);
    for (unsigned kk = 0; kk < kn; kk++) {
      const unsigned k = k0 + kk;
      fetch(k + SK_RING - 1u);  // into the stage the warp left one tile ago
      asm volatile("cp.async.wait_group %0;" ::"n"(SK_RING - 1) : "memory");
      __syncwarp();
      const unsigned char* ra = stage0 + (k % SK_RING) * SK_ITEM + g * SK_ROW;
      const unsigned char* rb = ra + 8u * SK_ROW;
      const uint4 ha = *reinterpret_cast<const uint4*>(ra), hb = *reinterpret_cast<const uint4*>(rb);
      uint32_t sca, mna, scb, mnb;
      header_half(ha, half, sca, mna);
      header_half(hb, half, scb, mnb);
      float cm[4] = {0.f, 0.f, 0.f, 0.f}, cs[4] = {0.f, 0.f, 0.f, 0.f}, tot[4];
      mma16816(cm, bytes_h2(mna, msel), bytes_h2(mnb, msel), 0u, 0u, bs, 0u);
      mma16816(cs, bytes_h2(sca, msel), bytes_h2(scb, msel), 0u, 0u, bs, 0u);
#pragma unroll
      for (unsigned uu = 0; uu < 2; uu++) {
        const uint2 qa = *reinterpret_cast<const uint2*>(ra + 8u * t + 16u + 32u * uu), qb = *reinterpret_cast<const uint2*>(rb + 8u * t + 16u + 32u * uu);
        const uint32_t a8 = qa.x >> 8, b8 = qb.x >> 8, a9 = qa.y >> 8, b9 = qb.y >> 8;
#pragma unroll
        for (unsigned hn = 0; hn < 2; hn++) {
          const unsigned j = 2u * uu + hn;
          const uint32_t xa = hn ? nib_hi(qa.x) : nib_lo(qa.x), xb = hn ? nib_hi(qb.x) : nib_lo(qb.x), xa8 = hn ? nib_hi(a8) : nib_lo(a8),
                         xb8 = hn ? nib_hi(b8) : nib_lo(b8);
          const uint32_t ya = hn ? nib_hi(qa.y) : nib_lo(qa.y), yb = hn ? nib_hi(qb.y) : nib_lo(qb.y), ya8 = hn ? nib_hi(a9) : nib_lo(a9),
                         yb8 = hn ? nib_hi(b9) : nib_lo(b9);
          float c[4] = {0.f, 0.f, 0.f, 0.f};
          mma16816(c, xa, xb, xa8, xb8, bl[j].x, bl[j].y);
          mma16816(c, ya, yb, ya8, yb8, bl[j].z, bl[j].w);
          mma16816(c, xa, xb, xa8, xb8, bh[j].x, bh[j].y);
          mma16816(c, ya, yb, ya8, yb8, bh[j].z, bh[j].w);
          const float fa = byte_f(sca, j), fb = byte_f(scb, j);
          tot[0] = j ? fmaf(fa, c[0], tot[0]) : fa * c[0];
          tot[1] = j ? fmaf(fa, c[1], tot[1]) : fa * c[1];
          tot[2] = j ? fmaf(fb, c[2], tot[2]) : fb * c[2];
          tot[3] = j ? fmaf(fb, c[3], tot[3]) : fb * c[3];
        }
      }
      float2 da = __half22float2(as_h2(ha.x)), db = __half22float2(as_h2(hb.x));  // (d, dmin)
      da.y *= 32.0f; db.y *= 32.0f;                                               // the sums carry 2^-5
#pragma unroll
      for (int e = 0; e < 4; e++) tot[e] = fmaf(256.0f, cs[e], tot[e]);
      float* ps = psum + (size_t)((buf + kk) * a.warps + warp) * 128u + g * 8u + 2u * t;
      *reinterpret_cast<float2*>(ps) = make_float2(da.x * tot[0] - da.y * cm[0], da.x * tot[1] - da.y * cm[1]);
      *reinterpret_cast<float2*>(ps + 64) = make_float2(db.x * tot[2] - db.y * cm[2], db.x * tot[3] - db.y * cm[3]);
      __syncwarp();  // every lane is done with the stage
    }
    __syncthreads();
    for (unsigned i = threadIdx.x; i < kn * 128u; i += blockDim.x) {
      const unsigned kk = i >> 7, r = (i >> 3) & 15u, tok = i & 7u;
      float v = 0.0f;
      for (unsigned w = 0; w < a.warps; w++) v += psum[(size_t)((buf + kk) * a.warps + w) * 128u + (i & 127u)];
      const unsigned tile = first + k0 + kk;
      const int seg = (tile >= a.tile0[1]) + (tile >= a.tile0[2]);
      const unsigned row = (tile - (seg == 0 ? a.tile0[0] : seg == 1 ? a.tile0[1] : a.tile0[2])) * 16u + r;
      float* y = (seg == 0 ? a.y[0] : seg == 1 ? a.y[1] : a.y[2]) + (size_t)split * (seg == 0 ? a.part_stride[0] : seg == 1 ? a.part_stride[1] : a.part_stride[2]);
      if (row < (seg == 0 ? a.rows[0] : seg == 1 ? a.rows[1] : a.rows[2]) && tok < a.n_tok)
        y[(size_t)tok * (seg == 0 ? a.ldy[0] : seg == 1 ? a.ldy[1] : a.ldy[2]) + row] = v * up[tok];
    }
    buf ^= SK_GROUP;  // two buffers: whoever writes this one again has met the barrier of the group between
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// ---- Q6_K (the head) ------------------------------------------------------------------------------------------------------
// One matrix, direct output.  A tile is 16 whole rows: 3360 bytes per 256 columns, contiguous and a multiple of 16, so one bulk
// copy brings it into a ring of `stages` (rows of 210-byte blocks start on any even address: words are read aligned and shifted
// into place).  A = q - 32 as f16, exact; a 16-column run (one scale) is one k step, its two mmas (the tokens' two terms) share
// f32 sums that then take the scale.  Bound by instructions, about 350 per warp and tile of 16 x 128 weights, most on the
// integer pipe: 262144 x 2560 x 8 rows 204 us where the bytes take 84 (the tcgen05 kernel, which spends its time on hand-overs:
// 450 us).
constexpr unsigned S6_PITCH = 10, S6_PSUM = 16 * S6_PITCH, S6_GROUP = 2, S6_MAX_STAGES = 6;
constexpr unsigned S6_TILE = 16u * 210u;  // bytes of a tile per 256 columns
constexpr unsigned S6_WAIT = 1u << 20;
constexpr unsigned S6_PAIR_WARPS = 12;    // 80 registers a thread: two such blocks fill an SM's 65536

struct Skinny6Args {
  const uint8_t* W;
  float* y;
  size_t ldy;
  unsigned rows, cols, n_tok, np, warps, stages, wait_limit, test_stall;
  const __half* xt;
  unsigned* err;
};

// The word at an even address whose aligned word and shift (0 or 16) are given.
__device__ __forceinline__ uint32_t word_even(const unsigned char* al, unsigned sh) {
  return __funnelshift_r(reinterpret_cast<const uint32_t*>(al)[0], reinterpret_cast<const uint32_t*>(al)[1], sh);
}
// Signed byte j of v (given with its sign bits flipped) as a float.
__device__ __forceinline__ float sbyte_f(uint32_t v, unsigned j) { return __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7540u + j)) - 8388736.0f; }

// WARPS: the most a block may have; PER_SM: blocks an SM must have registers for.
template <unsigned WARPS, unsigned PER_SM>
__global__ void __launch_bounds__(WARPS * 32, PER_SM) gemm_q6k_skinny_kernel(const Skinny6Args a) {
  extern __shared__ __align__(128) unsigned char smem[];
  // [0, 64): mbarriers; [64, 68): failure flag; from 128: the ring, then the sums [2][S6_GROUP][warps][16 rows, pitch 10]
  const uint32_t bars = sm32(smem);
  volatile unsigned* fail = reinterpret_cast<volatile unsigned*>(smem + 64);
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3u, sb = warp >> 1, half = warp & 1u;
  const unsigned nblk = a.cols / 256u, row_bytes = nblk * 210u, tile_bytes = nblk * S6_TILE;
  const unsigned char* stage0 = smem + 128u;
  const uint32_t ring = bars + 128u;
  float* psum = reinterpret_cast<float*>(smem + 128u + (size_t)a.stages * tile_bytes);
  const unsigned tiles = (a.rows + 15u) / 16u, base = tiles / gridDim.x, rem = tiles - base * gridDim.x, b = blockIdx.x;
  const unsigned first = b * base + min(b, rem), n = base + (b < rem ? 1u : 0u);

  auto request = [&](unsigned k) {  // one thread
    const unsigned s = k % a.stages, r0 = (first + k) * 16u, bytes = min(16u, a.rows - r0) * row_bytes;
    mb_expect(bars + 8u * s, bytes);
    if (a.test_stall != k + 1u) bulk_in(ring + s * tile_bytes, a.W + (size_t)r0 * row_bytes, bytes, bars + 8u * s);
  };
  unsigned requested = 0;
  if (threadIdx.x == 0) {
    for (unsigned i = 0; i < a.stages; i++) mb_init(bars + 8u * i, 1);
    *fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (; requested < a.stages && requested < n; requested++) request(requested);  // the weights do not depend on the kernels before
  }
  __syncthreads();
  ks_pdl_entry();  // the image does

  // ---- this warp's columns of the token rows (the plain form of the image): run r of 16 columns, this lane's four of token g
  uint2 bh[8], bl[8];
  {
    const __half* x = a.xt + (size_t)(sb * 32u + half * 16u + (t >> 1)) * 2u * a.np * 8u + g * 8u + 4u * (t & 1u);
#pragma unroll
    for (unsigned r = 0; r < 8; r++) {
      const uint2 h = *reinterpret_cast<const uint2*>(x + (size_t)(2u * r) * 2u * a.np * 8u);
      const uint2 l = *reinterpret_cast<const uint2*>(x + (size_t)(2u * r) * 2u * a.np * 8u + (size_t)a.np * 8u);
      // elements (0, 2) and (1, 3): the order in which masking leaves the weights
      bh[r] = make_uint2(__byte_perm(h.x, h.y, 0x5410u), __byte_perm(h.x, h.y, 0x7632u));
      bl[r] = make_uint2(__byte_perm(l.x, l.y, 0x5410u), __byte_perm(l.x, l.y, 0x7632u));
    }
  }
  const float* up = reinterpret_cast<const float*>(a.xt + xt_scale_off(a.cols, a.np));
  const __half2 bias = __float2half2_rn(-1056.0f);
  unsigned buf = 0;
  bool ok = true;

  for (unsigned k0 = 0; k0 < n; k0 += S6_GROUP) {
    const unsigned kn = min(S6_GROUP, n - k0);
    for (unsigned kk = 0; kk < kn; kk++) {
      const unsigned k = k0 + kk, s = k % a.stages;
      if (!__all_sync(0xffffffffu, mb_wait(bars + 8u * s, (k / a.stages) & 1u, a.wait_limit))) {
        *fail = 1;
        break;
      }
      uint32_t ql[2][4], qh[2][2], sc[2][2];
      float d[2], tot[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (unsigned i = 0; i < 2; i++) {
        const unsigned off = s * tile_bytes + (g + 8u * i) * row_bytes + sb * 210u, sh = (off & 2u) * 8u;
        const unsigned char* al = stage0 + (off & ~3u);
        const unsigned char *lo = al + 64u * half + 4u * t, *hi = al + 32u * half + 4u * t;
#pragma unroll
        for (unsigned w = 0; w < 4; w++) ql[i][w] = word_even(lo + 16u * w, sh);
#pragma unroll
        for (unsigned w = 0; w < 2; w++) qh[i][w] = word_even(hi + 128u + 16u * w, sh);
        const uint32_t* sp = reinterpret_cast<const uint32_t*>(al + 8u * half + 192u);
        const uint32_t s0 = sp[0], s1 = sp[1], s2 = sp[2];
        sc[i][0] = __funnelshift_r(s0, s1, sh) ^ 0x80808080u;
        sc[i][1] = __funnelshift_r(s1, s2, sh) ^ 0x80808080u;
        d[i] = __half2float(*reinterpret_cast<const __half*>(al + (off & 2u) + 208u));
      }
#pragma unroll
      for (unsigned r = 0; r < 8; r++) {  // group r >> 1 of 32 columns, its half r & 1 (gguf_impl.rs:761-791)
        const unsigned grp = r >> 1, w = 2u * (grp & 1u) + (r & 1u);
        uint32_t f[2][2];
#pragma unroll
        for (unsigned i = 0; i < 2; i++) {
          const uint32_t q = ql[i][w] >> (4u * (grp >> 1)), h = grp == 3u ? qh[i][r & 1u] >> 2 : qh[i][r & 1u] << (4u - 2u * grp);
          const uint32_t q8 = q >> 8, h8 = grp == 3u ? qh[i][r & 1u] >> 10 : grp == 2u ? qh[i][r & 1u] >> 8 : qh[i][r & 1u] >> (4u + 2u * grp);
          f[i][0] = pack_h2(__hadd2(as_h2((q & 0x000F000Fu) | 0x64006400u | (h & 0x00300030u)), bias));
          f[i][1] = pack_h2(__hadd2(as_h2((q8 & 0x000F000Fu) | 0x64006400u | (h8 & 0x00300030u)), bias));
        }
        float c[4] = {0.f, 0.f, 0.f, 0.f};
        mma16816(c, f[0][0], f[1][0], f[0][1], f[1][1], bh[r].x, bh[r].y);
        mma16816(c, f[0][0], f[1][0], f[0][1], f[1][1], bl[r].x, bl[r].y);
        const float fa = sbyte_f(sc[0][r >> 2], r & 3u), fb = sbyte_f(sc[1][r >> 2], r & 3u);
        tot[0] = fmaf(fa, c[0], tot[0]);
        tot[1] = fmaf(fa, c[1], tot[1]);
        tot[2] = fmaf(fb, c[2], tot[2]);
        tot[3] = fmaf(fb, c[3], tot[3]);
      }
      float* ps = psum + (size_t)((buf + kk) * a.warps + warp) * S6_PSUM + g * S6_PITCH + 2u * t;
      *reinterpret_cast<float2*>(ps) = make_float2(d[0] * tot[0], d[0] * tot[1]);
      *reinterpret_cast<float2*>(ps + 8u * S6_PITCH) = make_float2(d[1] * tot[2], d[1] * tot[3]);
    }
    __syncthreads();  // the sums are there, and the group's stages are free
    if (*fail) {
      ok = false;
      break;
    }
    if (threadIdx.x == 0)
      for (; requested < n && requested < k0 + kn + a.stages; requested++) request(requested);
    for (unsigned i = threadIdx.x; i < kn * 128u; i += blockDim.x) {
      const unsigned kk = i >> 7, r = i & 15u, tok = (i >> 4) & 7u, row = (first + k0 + kk) * 16u + r;
      const float* ps = psum + (size_t)(buf + kk) * a.warps * S6_PSUM + r * S6_PITCH + tok;
      float v = 0.0f;
#pragma unroll 4
      for (unsigned w = 0; w < a.warps; w++) v += ps[w * S6_PSUM];
      if (row < a.rows && tok < a.n_tok) a.y[(size_t)tok * a.ldy + row] = v * up[tok];
    }
    buf ^= S6_GROUP;  // two buffers: whoever writes this one again has met the barrier of the group between
  }
  if (!ok && threadIdx.x == 0) {
    // the copies in flight must have landed before the shared memory goes away (bounded)
    for (unsigned k = requested > a.stages ? requested - a.stages : 0u; k < requested; k++)
      if (a.test_stall != k + 1u) mb_wait(bars + 8u * (k % a.stages), (k / a.stages) & 1u, a.wait_limit);
    atomicOr(a.err, 8u);
  }
}

size_t skinny6_psum(unsigned warps) { return (size_t)2 * S6_GROUP * warps * S6_PSUM * 4; }
// Stages of a block of `warps` warps (2 warps per 256 columns) when `per_sm` blocks share an SM; 0: too few to overlap.
unsigned skinny6_stages(const ks_ctx* ctx, unsigned warps, unsigned per_sm) {
  const size_t room = (ctx->smem_optin + 1024) / per_sm - 1024, fixed = 128 + skinny6_psum(warps), tile = (size_t)warps / 2 * S6_TILE;
  if (room < fixed) return 0;
  const size_t n = (room - fixed) / tile;
  return n < S6_GROUP + 1 ? 0 : n > S6_MAX_STAGES ? S6_MAX_STAGES : (unsigned)n;
}

size_t skinny_smem(unsigned warps) { return (size_t)warps * (SK_RING * SK_ITEM + 2u * SK_GROUP * 512u); }
// Blocks of at most ten warps share an SM.
unsigned skinny_cps(unsigned warps) { return warps <= 10u ? 2u : 1u; }
}  // namespace

// Shares of a row's columns: a divisor of its half super-blocks that leaves at most 20 warps a block; of those, the one whose
// blocks' rounds of tiles take least (a round: the warps of an SM, plus a fixed cost for its latency).
unsigned ks_gemm_skinny_splits(const ks_ctx* ctx, size_t rows, unsigned cols) {
  const unsigned halves = cols / 128u, tiles = (unsigned)((rows + 15) / 16), sms = (unsigned)ctx->sm_count;
  unsigned best = 0;
  double best_cost = 0;
  for (unsigned s = 1; s <= halves; s++) {
    if (halves % s || halves / s > SK_MAX_WARPS) continue;
    const unsigned w = halves / s, cps = skinny_cps(w), per = sms * cps / s;
    if (per == 0 || (w < 4u && best)) continue;
    const double cost = (double)((tiles + per - 1) / per) * (w * cps + 8.0);
    if (!best || cost < best_cost * 0.99) {
      best = s;
      best_cost = cost;
    }
  }
  return best;  // 0: not covered
}

int ks_launch_gemm_skinny(ks_ctx* ctx, const ks_gemm_job& job) {
  SkinnyArgs a{};
  unsigned tiles = 0;
  for (int i = 0; i < 3; i++) {
    a.tile0[i] = i < job.n_seg ? tiles : 0xFFFFFFFFu;
    if (i >= job.n_seg) continue;
    if ((uintptr_t)job.W[i] & 15) return ks_fail(ctx, KS_ERR_INVALID, "gemm: packed rows must start on a 16-byte boundary");
    a.W[i] = job.W[i];
    a.rows[i] = (unsigned)job.rows[i];
    a.y[i] = job.y[i];
    a.ldy[i] = job.ldy[i];
    a.part_stride[i] = job.part_stride[i];
    tiles += (unsigned)((job.rows[i] + 15) / 16);
  }
  a.tile0[3] = tiles;
  a.row_bytes = job.cols / 256u * KS_Q4K_BLOCK_BYTES;
  a.cols = job.cols;
  a.n_tok = job.n_tok;
  a.np = job.np;
  a.xt = job.xt;
  a.splits = job.map.splits;
  a.warps = job.cols / 128u / a.splits;
  a.per_split = (unsigned)ctx->sm_count * skinny_cps(a.warps) / a.splits;
  if (a.per_split > tiles) a.per_split = tiles;
  const size_t smem = skinny_smem(a.warps);
  static size_t set[16] = {0};
  size_t& have = set[ctx->device & 15];
  if (smem > have) {
    cudaError_t e = cudaFuncSetAttribute(gemm_q4k_skinny_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return ks_fail(ctx, KS_ERR_CUDA, "gemm: cannot set %zu B shared memory: %s", smem, cudaGetErrorString(e));
    have = smem;
  }
  KS_LAUNCH(ctx, gemm_q4k_skinny_kernel, a.per_split * a.splits, a.warps * 32u, smem, a);
  return ks_after_launch(ctx, "gemm_q4k_skinny");
}

// Whole rows of at most 20 warps' columns, and tiles that end on a 16-byte boundary.
bool ks_gemm_q6k_skinny_covers(const ks_ctx* ctx, size_t rows, unsigned cols) {
  return cols / 128u <= SK_MAX_WARPS && rows % 8 == 0 && skinny6_stages(ctx, cols / 128u, 1) != 0;
}

int ks_launch_gemm_q6k_skinny(ks_ctx* ctx, const ks_gemm_job& job) {
  Skinny6Args a{};
  a.W = job.W[0];
  a.y = job.y[0];
  a.ldy = job.ldy[0];
  a.rows = (unsigned)job.rows[0];
  a.cols = job.cols;
  a.n_tok = job.n_tok;
  a.np = job.np;
  a.warps = job.cols / 128u;
  a.xt = job.xt;
  a.err = (unsigned*)ctx->ws + KS_WS_ERR_WORD;
  a.wait_limit = S6_WAIT;
  if (const char* t = getenv("KSEARCH_GEMM_TEST_STALL")) {  // exercises the give-up path: short waits, one tile withheld
    a.test_stall = (unsigned)atoi(t);
    if (a.test_stall) a.wait_limit = 4000;
  }
  // two blocks per SM where registers and at least three stages each allow it: one's barriers fall into the other's work
  const unsigned per_sm = a.warps <= S6_PAIR_WARPS && skinny6_stages(ctx, a.warps, 2) ? 2u : 1u;
  void (*kern)(Skinny6Args) = per_sm == 2 ? gemm_q6k_skinny_kernel<S6_PAIR_WARPS, 2> : gemm_q6k_skinny_kernel<SK_MAX_WARPS, 1>;
  a.stages = skinny6_stages(ctx, a.warps, per_sm);
  const size_t smem = 128 + (size_t)a.stages * (a.cols / 256u) * S6_TILE + skinny6_psum(a.warps);
  static size_t set[2][16] = {{0}};
  size_t& have = set[per_sm - 1][ctx->device & 15];
  if (smem > have) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return ks_fail(ctx, KS_ERR_CUDA, "gemm: cannot set %zu B shared memory: %s", smem, cudaGetErrorString(e));
    have = smem;
  }
  const unsigned tiles = (a.rows + 15u) / 16u, most = (unsigned)ctx->sm_count * per_sm;
  KS_LAUNCH(ctx, kern, tiles < most ? tiles : most, a.warps * 32u, smem, a);
  return ks_after_launch(ctx, "gemm_q6k_skinny");
}
