// Q4_K weights x 1..8 token rows on the tensor cores (mma.sync m16n8k16): the matrices of a decode step of several slots.
//
// The reference's op is the batch matvec (crates/ksearch_kernels/src/lib.rs:1414).  With so few rows the tcgen05 kernel is a
// chain of short hand-overs (packed rows -> tensor memory -> MMA -> fold: 2 us per 18 KB of weights); here a warp owns 128
// columns (half a super-block) for ALL the row tiles of its block:
//   * its share of the token rows, two f16 terms of each value, sits in 32 registers as B fragments and is loaded once;
//   * packed rows come by cp.async into a ring of the warp's own (16 rows x 80 bytes per tile), requested before the wait for
//     the previous kernel; no warp waits for another inside a tile;
//   * A is the packed nibble itself: masked in place it is the f16 subnormal q 2^-24 (q 2^-20 in the high half), which the
//     tensor core multiplies exactly, so two weights cost one LOP3.  Tokens are the 8 columns; their first and second terms
//     go into the same f32 sums of a 32-column sub-block, which then take the sub-block's scale in f32.  The minima are one
//     more mma: A = m 2^-24, B = the image's sub-block sums;
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
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
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
// Byte j of v as a float.
__device__ __forceinline__ float byte_f(uint32_t v, unsigned j) { return __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7540u + j)) - 8388608.0f; }

__global__ void __launch_bounds__(SK_MAX_WARPS * 32, 1) gemm_q4k_skinny_kernel(const __grid_constant__ SkinnyArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3u;
  const unsigned split = blockIdx.x / a.per_split, b = blockIdx.x - split * a.per_split;
  const unsigned tiles = a.tile0[3], base = tiles / a.per_split, rem = tiles - base * a.per_split;
  const unsigned first = b * base + min(b, rem), n = base + (b < rem ? 1u : 0u);
  const unsigned hidx = split * a.warps + warp, sb = hidx >> 1, half = hidx & 1u;  // this warp's super-block and half of it
  const uint32_t ring = sm32(smem) + warp * (SK_RING * SK_ITEM);
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
  const uint32_t msel = (t & 1u) ? 0x4342u : 0x4140u;  // this lane's two minima as halves
  unsigned buf = 0;

  for (unsigned k0 = 0; k0 < n; k0 += SK_GROUP) {
    const unsigned kn = min(SK_GROUP, n - k0);
    for (unsigned kk = 0; kk < kn; kk++) {
      const unsigned k = k0 + kk;
      fetch(k + SK_RING - 1u);  // into the stage the warp left one tile ago
      asm volatile("cp.async.wait_group %0;" ::"n"(SK_RING - 1) : "memory");
      __syncwarp();
      const uint32_t ra = ring + (k % SK_RING) * SK_ITEM + g * SK_ROW, rb = ra + 8u * SK_ROW;
      const uint4 ha = lds128(ra), hb = lds128(rb);
      uint32_t sca, mna, scb, mnb;
      header_half(ha, half, sca, mna);
      header_half(hb, half, scb, mnb);
      float cm[4] = {0.f, 0.f, 0.f, 0.f}, tot[4];
      mma16816(cm, __byte_perm(mna, 0u, msel), __byte_perm(mnb, 0u, msel), 0u, 0u, bs, 0u);
#pragma unroll
      for (unsigned uu = 0; uu < 2; uu++) {
        const uint2 qa = lds64(ra + 16u + 32u * uu + 8u * t), qb = lds64(rb + 16u + 32u * uu + 8u * t);
        const uint32_t a8 = qa.x >> 8, b8 = qb.x >> 8, a9 = qa.y >> 8, b9 = qb.y >> 8;
#pragma unroll
        for (unsigned hn = 0; hn < 2; hn++) {
          constexpr uint32_t LO = 0x000F000Fu;
          const uint32_t M = hn ? LO << 4 : LO;
          const unsigned j = 2u * uu + hn;
          float c[4] = {0.f, 0.f, 0.f, 0.f};
          mma16816(c, qa.x & M, qb.x & M, a8 & M, b8 & M, bh[j].x, bh[j].y);
          mma16816(c, qa.y & M, qb.y & M, a9 & M, b9 & M, bh[j].z, bh[j].w);
          mma16816(c, qa.x & M, qb.x & M, a8 & M, b8 & M, bl[j].x, bl[j].y);
          mma16816(c, qa.y & M, qb.y & M, a9 & M, b9 & M, bl[j].z, bl[j].w);
          const float fa = byte_f(sca, j) * (hn ? 0.0625f : 1.0f), fb = byte_f(scb, j) * (hn ? 0.0625f : 1.0f);
          tot[0] = j ? fmaf(fa, c[0], tot[0]) : fa * c[0];
          tot[1] = j ? fmaf(fa, c[1], tot[1]) : fa * c[1];
          tot[2] = j ? fmaf(fb, c[2], tot[2]) : fb * c[2];
          tot[3] = j ? fmaf(fb, c[3], tot[3]) : fb * c[3];
        }
      }
      float2 da = __half22float2(as_h2(ha.x)), db = __half22float2(as_h2(hb.x));  // (d, dmin)
      da.x *= 16777216.0f; db.x *= 16777216.0f;      // the weights' 2^24
      da.y *= 536870912.0f; db.y *= 536870912.0f;    // and 2^5 of the sums
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
