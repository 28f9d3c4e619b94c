// Attention of a prompt chunk: many token rows of one slot, or of several, against their Q4_0 caches, causal (and windowed) by row.
//
// The reference runs its decode attention once per prompt row (forward_prefill_chunk, crates/ksearch_gemma/src/
// gemma_prim.rs:1463-1472, over crates/ksearch_codegen/src/lower.rs:4897-6088), so every row reads the whole context again.
// Here the tiles of 64 positions that the rows see are decoded ONCE into an image (kv_image_kernel: K as positions x dims, V as dims x
// positions, each value d (n - 8) exactly as two f16 terms, in the layout shared memory wants), and a block takes 128 query rows that
// share a KV head (128 / G tokens x the head's G query heads), brings tile after tile in by bulk copies and multiplies on tcgen05 (f16
// in, f32 out) without giving up f32 accuracy: q (scaled per row by a power of two) and the probabilities are two f16 terms each as
// well, a product is hi hi + hi lo + lo hi.
//   * q's first term and the probabilities lie in TENSOR memory as the A operand, q's second term and the tile in shared memory; scores
//     and a tile's values are the accumulators (HD = 256 fills the 512 columns);
//   * eight warps own half a row per thread: they add the values of the tile before, scaled as the maximum moved, to f32 registers while
//     the scores of this one are made, then mask, running maximum (the two threads of a row trade theirs), probabilities;
//   * one warp issues the products, one the copies.
// The sums leave tensor memory after every tile and small terms come first, because the accumulator truncates: against 64 bits the
// result is off by 1.3..1.8e-7 (2-norm) whatever the context, where accumulating on gave 3e-6 over 2047 positions, 1e-5 over 4000.
// The context is split over blockIdx.z; (m, l, O) records go to `tmp` as the decode kernels leave them and
// sdpa_merge_split_kernel folds them straight into the operand image of the output projection.
//
// Bound by the chain of a tile: scores (48 MMAs), probabilities, values (12 MMAs of 256 columns), 3.2 us for 128 x 64.  When eight warps
// of every block decoded its tiles it was 5.7 us, 2.2 of them waiting for keys; one thread per row of scores: 3.7.  A block takes another
// 8 us: q 3.6, records 2, setting up 2.  Launches with their image, back to back: 2047 rows of 8 heads (128 blocks of up to 32 tiles) 118
// us, in two splits 76 (decoding in every block 205 and 118); 2000 rows behind 2000 positions, 2 KV heads (126 blocks of up to 63 tiles)
// 213, in two splits 188 (387 and 343); 300 rows in three splits 23.5 (30).
#include "ks_gemm_common.cuh"

namespace {

constexpr int CH_BM = 128, CH_BN = 64;                 // query rows, positions of a tile
constexpr int CH_WORK_WARPS = 8, CH_THREADS = (CH_WORK_WARPS + 4) * 32;
constexpr unsigned CH_WAIT = 1u << 20;
constexpr float CH_P = 256.0f;                         // probabilities carry 2^8
constexpr unsigned CH_K_MOST = 0x6FFFu;                // the largest scale with 8 d in f16, 8188
constexpr float kNegInit = -1.0e30f;

// barriers: the tile's K and V there (copies), its probabilities, its O taken (workers), products ready (commits: scores done = K
// free; values done = V and P free)
enum { CB_K_FULL, CB_V_FULL, CB_P_FULL, CB_O_FREE, CB_S_FULL, CB_K_FREE, CB_V_FREE, CB_DONE, CB_COUNT };

template <int HD>
struct ChunkSmem {
  static constexpr unsigned slot = 64, row = 128;     // tensor-memory address, failure flag; per row: scale, first, past the last position, then
                                                      // the maxima and the sums of the two threads that share it, of two tiles
  static constexpr unsigned ql = 4096, kh = ql + CH_BM * HD * 2, kl = kh + CH_BN * HD * 2, vh = kl + CH_BN * HD * 2,
                            vl = vh + CH_BN * HD * 2, total = vl + CH_BN * HD * 2;
  static_assert(row + CH_BM * 28 <= ql, "the rows' words fit in front of the operands");
  static constexpr unsigned o = ql, OP = HD + 4;      // the result on its way out: rows of OP floats
  static_assert(o + CH_BM * OP * 4 <= total, "the result fits the operands");
  // tensor memory: first term of q, scores, the probabilities' two terms, O
  static constexpr unsigned t_q = 0, t_s = HD / 2, t_ph = t_s + CH_BN, t_pl = t_ph + CH_BN / 2, t_o = t_pl + CH_BN / 2;
  static_assert(t_o + HD <= 512, "tensor memory");
};

__device__ __forceinline__ void mb_arrive1(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
// `threads` threads (whole warps) meet at barrier `id`; true if every one of them says so.
__device__ __forceinline__ bool meet_all(unsigned id, unsigned threads, bool ok) {
  unsigned r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.and.pred q, %2, %3, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((unsigned)ok), "r"(id), "r"(threads)
      : "memory");
  return r != 0;
}
// d (n - 8) of two values as two f16 terms, exactly.
__device__ __forceinline__ void split_d(__half2 n, __half2 d, uint32_t& hi, uint32_t& lo) {
  const __half2 x = __hmul2(n, d);
  hi = pack_h2(x);
  lo = pack_h2(__hfma2(n, d, __hneg2(x)));
}
__device__ __forceinline__ __half2 nib_h2(uint32_t w) { return __hsub2(as_h2((w & 0x000F000Fu) | 0x64006400u), __float2half2_rn(1032.0f)); }  // nibbles 0 of bytes 0 and 2

struct ChunkParts {  // part p: rows from row0[p] on, row tiles from tile0[p] on; its decoded tiles start at image0[p] of the image
  unsigned n, row0[65], tile0[65], slot[64], image0[64];
};
// Decoded tile t of KV head h in the image: K's first and second terms, V's, each as the kernel wants it in shared memory; behind all
// tiles, what their scores are multiplied by.
template <int HD>
struct ChunkImage {
  static constexpr unsigned HALF = 2 * CH_BN * HD * 2, TILE = 2 * HALF;  // bytes of a tile's K (V), and of both
};

// The tiles of 64 positions that some row of a part sees, decoded once for all its query tiles.  grid = (tiles, 4 n_kv, parts): a block
// takes K or V of a tile, half the dims.
template <int HD>
__global__ void __launch_bounds__(256) kv_image_kernel(const __grid_constant__ ChunkParts parts, size_t slot_stride, unsigned n_kv, const uint8_t* K, const uint8_t* V,
                                                        const float* meta, unsigned char* img, float* img_up) {
  ks_pdl_entry();
  constexpr unsigned NB = HD / 32, ROWB = NB * KS_Q40_BLOCK_BYTES;
  const unsigned tid = threadIdx.x, part = blockIdx.z, kvh = blockIdx.y >> 2, half = blockIdx.y & 1u;
  const float *m0 = meta + (size_t)parts.row0[part] * 4u, *m1 = meta + (size_t)(parts.row0[part + 1u] - 1u) * 4u;  // starts and ends grow with the row
  const unsigned end = (unsigned)((int)m1[0] + (int)m1[1]), tile = (unsigned)(int)m0[1] / CH_BN + blockIdx.x, p0 = tile * CH_BN;
  if (p0 >= end) return;
  const size_t at = (size_t)(parts.image0[part] + tile) * n_kv + kvh;
  unsigned char* out = img + at * ChunkImage<HD>::TILE;
  const bool vals = (blockIdx.y & 2u) != 0u;
  const uint8_t* src = (vals ? V : K) + parts.slot[part] * slot_stride + (size_t)kvh * ROWB;
  auto row = [&](unsigned p) { return src + (size_t)min(p0 + p, end - 1u) * n_kv * ROWB; };  // (rows past the end repeat the last: their scores are masked)
  if (!vals) {
    // a tile with a scale whose products leave f16 is decoded at an eighth and its scores are multiplied by 8; what that rounds off
    // (2^-22 of a value at most) is nothing beside a value of 57000
    bool over = false;
    for (unsigned i = tid; i < CH_BN * NB; i += 256u)
      over |= (*reinterpret_cast<const unsigned short*>(row(i % CH_BN) + i / CH_BN * KS_Q40_BLOCK_BYTES) & 0x7FFFu) > CH_K_MOST;
    const float up = __syncthreads_or(over) ? 8.0f : 1.0f;
    if (tid == 0 && half == 0) img_up[at] = up;
    const __half2 down = __float2half2_rn(1.0f / up);
    for (unsigned job = tid; job < CH_BN * NB / 2u; job += 256u) {  // a block of a row
      const unsigned p = job % CH_BN, b = half * (NB / 2u) + job / CH_BN;
      const uint8_t* x = row(p) + b * KS_Q40_BLOCK_BYTES;
      const __half2 d = __hmul2(__half2half2(__ushort_as_half(*reinterpret_cast<const unsigned short*>(x))), down);
      uint32_t w[4];
#pragma unroll
      for (int k = 0; k < 4; k++)
        w[k] = *reinterpret_cast<const unsigned short*>(x + 2 + 4 * k) | (uint32_t)*reinterpret_cast<const unsigned short*>(x + 4 + 4 * k) << 16;
#pragma unroll
      for (int hn = 0; hn < 2; hn++)  // dims 0..15 of the block are the low nibbles
#pragma unroll
        for (int c = 0; c < 2; c++) {
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int k = 0; k < 2; k++) {
            const uint32_t v = hn ? w[2 * c + k] >> 4 : w[2 * c + k];
            split_d(nib_h2(__byte_perm(v, 0u, 0x4140)), d, hi[2 * k], lo[2 * k]);
            split_d(nib_h2(__byte_perm(v, 0u, 0x4342)), d, hi[2 * k + 1], lo[2 * k + 1]);
          }
          unsigned char* o = out + ((4u * b + 2u * hn + c) * CH_BN + p) * 16u;
          *reinterpret_cast<uint4*>(o) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<uint4*>(o + ChunkImage<HD>::HALF / 2u) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
    }
    return;
  }
  out += ChunkImage<HD>::HALF;
  for (unsigned job = tid; job < 16u * (NB / 2u) * (CH_BN / 8); job += 256u) {  // byte j of a block in eight neighbouring rows
    const unsigned j = job % 16u, b = half * (NB / 2u) + job / 16u % (NB / 2u), pg = job / (16u * (NB / 2u));
    uint32_t hl[4], ll[4], hh[4], lh[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint8_t *x = row(8u * pg + 2u * k) + b * KS_Q40_BLOCK_BYTES, *y = row(8u * pg + 2u * k + 1u) + b * KS_Q40_BLOCK_BYTES;
      const uint32_t n = x[2 + j] | (uint32_t)y[2 + j] << 16;
      const __half2 d = as_h2(*reinterpret_cast<const unsigned short*>(x) | (uint32_t)*reinterpret_cast<const unsigned short*>(y) << 16);
      split_d(nib_h2(n), d, hl[k], ll[k]);
      split_d(nib_h2(n >> 4), d, hh[k], lh[k]);
    }
    unsigned char* o = out + (pg * HD + 32u * b + j) * 16u;
    *reinterpret_cast<uint4*>(o) = make_uint4(hl[0], hl[1], hl[2], hl[3]);
    *reinterpret_cast<uint4*>(o + 256u) = make_uint4(hh[0], hh[1], hh[2], hh[3]);
    *reinterpret_cast<uint4*>(o + ChunkImage<HD>::HALF / 2u) = make_uint4(ll[0], ll[1], ll[2], ll[3]);
    *reinterpret_cast<uint4*>(o + ChunkImage<HD>::HALF / 2u + 256u) = make_uint4(lh[0], lh[1], lh[2], lh[3]);
  }
}

template <int HD>
__global__ void __launch_bounds__(CH_THREADS, 1)
sdpa_chunk_kernel(const __grid_constant__ ChunkParts parts, unsigned n_q, unsigned n_kv, float scale, const float* q, const float* meta, float* tmp, unsigned n_splits,
                  const unsigned char* img, const float* img_up, unsigned* err) {
  using S = ChunkSmem<HD>;
  using Image = ChunkImage<HD>;
  extern __shared__ __align__(1024) unsigned char smem[];
  ks_pdl_entry();
  const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const unsigned G = n_q / n_kv, kvh = blockIdx.y, split = blockIdx.z;
  const unsigned bx = gridDim.x - 1u - blockIdx.x;  // the last rows see the most: they start first
  unsigned part_id = 0;
  while (part_id + 1u < parts.n && bx >= parts.tile0[part_id + 1u]) part_id++;
  const unsigned row0 = (bx - parts.tile0[part_id]) * CH_BM, first_tok = parts.row0[part_id], n_tok = parts.row0[part_id + 1u] - first_tok;
  q += (size_t)first_tok * n_q * HD;  // from here on rows are counted inside the part
  meta += (size_t)first_tok * 4u;
  tmp += (size_t)first_tok * n_q * n_splits * (HD + 2);
  const uint32_t sb = sm32(smem);
  auto bar = [&](unsigned i) { return sb + 8u * i; };
  uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + S::slot);
  volatile unsigned* fail = reinterpret_cast<volatile unsigned*>(smem + S::slot + 8);
  float* row_scale = reinterpret_cast<float*>(smem + S::row);
  int* row_first = reinterpret_cast<int*>(smem + S::row + CH_BM * 4);
  int* row_end = reinterpret_cast<int*>(smem + S::row + CH_BM * 8);
  float* row_max = reinterpret_cast<float*>(smem + S::row + CH_BM * 12);  // [2 tiles][2 halves][CH_BM]

  // ---- the block's rows: row r is query head kvh G + r % G of token (row0 + r) / G; positions they see at all
  const unsigned tok_a = row0 / G, tok_b = min((row0 + CH_BM - 1u) / G, n_tok - 1u);
  const int pmin = (int)meta[tok_a * 4 + 1] & ~(CH_BN - 1);                         // starts and ends grow with the token; tiles start at multiples of 64
  const int pmax = (int)meta[tok_b * 4 + 0] + (int)meta[tok_b * 4 + 1];
  const int span = (pmax - pmin + CH_BN - 1) / CH_BN, per = (span + (int)n_splits - 1) / (int)n_splits;
  const int t_begin = pmin + (int)split * per * CH_BN, t_end = min(pmin + (int)(split + 1u) * per * CH_BN, pmax);
  const unsigned n_tiles = t_begin < t_end ? (unsigned)((t_end - t_begin + CH_BN - 1) / CH_BN) : 0u;
  if (n_tiles == 0u) {  // an empty record is all the merge needs
    for (unsigned r = tid; r < CH_BM; r += CH_THREADS) {
      const unsigned t = (row0 + r) / G, head = kvh * G + (row0 + r) % G;
      if (t < n_tok) *reinterpret_cast<float2*>(tmp + (((size_t)t * n_q + head) * n_splits + split) * (HD + 2)) = make_float2(kNegInit, 0.0f);
    }
    return;
  }
  const size_t img_at = (size_t)(parts.image0[part_id] + (unsigned)t_begin / CH_BN) * n_kv + kvh;  // tiles are n_kv apart

  if (tid == 0) {
    mb_init(bar(CB_K_FULL), 1);
    mb_init(bar(CB_V_FULL), 1);
    mb_init(bar(CB_P_FULL), CH_WORK_WARPS);
    mb_init(bar(CB_O_FREE), CH_WORK_WARPS);
    for (unsigned i = CB_S_FULL; i < CB_COUNT; i++) mb_init(bar(i), 1);
    *fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == CH_WORK_WARPS) tc_alloc(sm32(tslot), 512);

  // ---- q: a worker warp takes twice eight rows, lane = row lane % 8, chunk of 8 dims lane / 8 (+ 4 a step): a load touches 128 neighbouring
  // bytes of eight rows, a store 128 bytes of a chunk; all loads come first (one trip instead of two: 5.7 -> 3.6 us a block).  The row
  // maximum sets a power of two, then two f16 terms per value: the second stays in shared memory as core matrices, the first passes
  // through there (K's place) to tensor memory.
  if (warp < CH_WORK_WARPS) {
    constexpr int STEPS = HD / 32, GROUPS = CH_BM / 8 / CH_WORK_WARPS;
    float v[GROUPS][STEPS][8], first_pos[GROUPS], length[GROUPS];
#pragma unroll
    for (int p = 0; p < GROUPS; p++) {
      const unsigned r = (warp * GROUPS + p) * 8u + (lane & 7u), t = (row0 + r) / G, head = kvh * G + (row0 + r) % G;
      const float* src = q + ((size_t)t * n_q + head) * HD + 8u * (lane >> 3);
      const bool in = t < n_tok;
      length[p] = in ? meta[t * 4] : 0.0f;
      first_pos[p] = in ? meta[t * 4 + 1] : 0.0f;
#pragma unroll
      for (int k = 0; k < STEPS; k++) {
        const float4 a = in ? *reinterpret_cast<const float4*>(src + 32 * k) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 b = in ? *reinterpret_cast<const float4*>(src + 32 * k + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[p][k][0] = a.x; v[p][k][1] = a.y; v[p][k][2] = a.z; v[p][k][3] = a.w;
        v[p][k][4] = b.x; v[p][k][5] = b.y; v[p][k][6] = b.z; v[p][k][7] = b.w;
      }
    }
#pragma unroll
    for (int p = 0; p < GROUPS; p++) {
      const unsigned r = (warp * GROUPS + p) * 8u + (lane & 7u);
      float m = 0.0f;
#pragma unroll
      for (int k = 0; k < STEPS; k++) m = fmaxf(m, absmax8(v[p][k]));
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
      float up;
      const float down = row_scale_down(m, &up);
      if (lane < 8u) {
        row_scale[r] = up * scale;
        row_first[r] = (int)first_pos[p];
        row_end[r] = (int)first_pos[p] + (int)length[p];
      }
#pragma unroll
      for (int k = 0; k < STEPS; k++) {
#pragma unroll
        for (int e = 0; e < 8; e++) v[p][k][e] *= down;
        uint4 hi, lo;
        split8(v[p][k], hi, lo);
        const unsigned at = ((4u * k + (lane >> 3)) * CH_BM + r) * 16u;
        *reinterpret_cast<uint4*>(smem + S::kh + at) = hi;
        *reinterpret_cast<uint4*>(smem + S::ql + at) = lo;
      }
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();
  const uint32_t tmem = *tslot;
  if (tmem != 0u && tid == 0) *fail = 1;  // all 512 columns were asked for: they start at 0
  const unsigned quad = warp & 3u, half = warp >> 2 & 1u, row = quad * 32u + lane;  // workers: half the columns of a row
  const uint32_t tlane = quad << 21;      // 32 rows per warp, in the address bits of the lane
  if (warp < CH_WORK_WARPS) {
#pragma unroll
    for (unsigned k = 0; k < HD / 16u; k += 2u) {
      const unsigned c = half * (HD / 16u) + k;
      const uint4 a = *reinterpret_cast<const uint4*>(smem + S::kh + (c * CH_BM + row) * 16u), b = *reinterpret_cast<const uint4*>(smem + S::kh + ((c + 1u) * CH_BM + row) * 16u);
      const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      tc_st8(tlane + S::t_q + c * 4u, w);
    }
    tc_wait_st();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // K's place has been read: the first copy may write it
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (warp < CH_WORK_WARPS) {
    // ---- half a row per thread: the tile before's values into f32 registers, then this tile's scores -> probabilities
    asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
    constexpr unsigned HALF = HD / 2;
    const float sc = row_scale[row];
    const int first = row_first[row], end = row_end[row];
    float acc[HALF], ref = kNegInit, l = 0.0f, alpha = 1.0f;
#pragma unroll
    for (unsigned c = 0; c < HALF; c++) acc[c] = 0.0f;
    auto fold = [&] {
      tc_fence_after();
#pragma unroll
      for (unsigned c = 0; c < HALF; c += 32u) {
        uint32_t o[2][16];
        tc_ld16(tlane + S::t_o + half * HALF + c, o[0]);
        tc_ld16(tlane + S::t_o + half * HALF + c + 16u, o[1]);
        tc_wait_ld16(o[0]);
        tc_wait_ld16(o[1]);
#pragma unroll
        for (unsigned e = 0; e < 32u; e++) acc[c + e] = fmaf(acc[c + e], alpha, __uint_as_float(o[e / 16u][e % 16u]));
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mb_arrive1(bar(CB_O_FREE));
    };
    bool ok = true;
    for (unsigned i = 0; i < n_tiles; i++) {
      const float up = img_up[img_at + (size_t)i * n_kv];
      if (i > 0) {  // the scores of this tile are made meanwhile
        ok = __all_sync(0xffffffffu, mb_wait(bar(CB_V_FREE), (i - 1u) & 1u, CH_WAIT));
        if (ok) fold();
      }
      ok = ok && __all_sync(0xffffffffu, mb_wait(bar(CB_S_FULL), i & 1u, CH_WAIT));
      float mx = -INFINITY;
      uint32_t s[2][16];
      if (ok) {
        tc_fence_after();
        tc_ld16(tlane + S::t_s + half * 32u, s[0]);
        tc_ld16(tlane + S::t_s + half * 32u + 16u, s[1]);
        tc_wait_ld16(s[0]);
        tc_wait_ld16(s[1]);
        const int p0 = t_begin + (int)i * CH_BN + (int)half * 32, a = first - p0, b = min(end, t_end) - p0;  // columns [a, b) are seen
        const float st = sc * up;
        if (__all_sync(0xffffffffu, a <= 0 && b >= 32)) {
#pragma unroll
          for (int j = 0; j < 32; j++) {
            const float x = __uint_as_float(s[j / 16][j % 16]) * st;
            s[j / 16][j % 16] = __float_as_uint(x);
            mx = fmaxf(mx, x);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; j++) {
            const float x = j >= a && j < b ? __uint_as_float(s[j / 16][j % 16]) * st : -INFINITY;
            s[j / 16][j % 16] = __float_as_uint(x);
            mx = fmaxf(mx, x);
          }
        }
        row_max[((i & 1u) * 2u + half) * CH_BM + row] = mx;
      }
      if (!meet_all(1u + quad, 64u, ok)) { ok = false; break; }  // the two warps that share 32 query rows
      mx = fmaxf(fmaxf(mx, row_max[((i & 1u) * 2u + (half ^ 1u)) * CH_BM + row]), ref);
      alpha = __expf(ref - mx);
      ref = mx;
      float sum = 0.0f;
#pragma unroll
      for (int k = 0; k < 2; k++) {
        uint32_t ph[8], pl[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {  // a masked score is -infinity: its probability is 0 whatever the maximum
          const float x = __expf(__uint_as_float(s[k][2 * j]) - ref), y = __expf(__uint_as_float(s[k][2 * j + 1]) - ref);
          sum += x + y;
          const __half2 h = __floats2half2_rn(x * CH_P, y * CH_P);
          const float2 f = __half22float2(h);
          ph[j] = pack_h2(h);
          pl[j] = pack_h2(__floats2half2_rn(x * CH_P - f.x, y * CH_P - f.y));
        }
        tc_st8(tlane + S::t_ph + half * 16u + 8u * k, ph);
        tc_st8(tlane + S::t_pl + half * 16u + 8u * k, pl);
      }
      l = l * alpha + sum;
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mb_arrive1(bar(CB_P_FULL));
    }
    ok = ok && __all_sync(0xffffffffu, mb_wait(bar(CB_V_FREE), (n_tiles - 1u) & 1u, CH_WAIT));
    if (!ok && lane == 0) *fail = 1;
    if (ok) {  // the rows through shared memory, so that they leave in whole lines; every product that read it is done
      fold();
      float* out = reinterpret_cast<float*>(smem + S::o) + row * S::OP + half * HALF;
#pragma unroll
      for (unsigned c = 0; c < HALF; c += 4u)
        *reinterpret_cast<float4*>(out + c) = make_float4(acc[c] * (1.0f / CH_P), acc[c + 1] * (1.0f / CH_P), acc[c + 2] * (1.0f / CH_P), acc[c + 3] * (1.0f / CH_P));
      row_max[((n_tiles & 1u) * 2u + half) * CH_BM + row] = l;  // (the tile before's maxima have been read by both)
      if (half == 0) row_scale[row] = ref;
    }
    if (meet_all(5u, CH_WORK_WARPS * 32u, ok)) {
      // here, where the registers are: four rows of a warp's in flight at a time (one after the other, in twelve warps, they took 5.5 us)
      constexpr unsigned FLY = 4, PER = HD / 64;
      const float* sums = row_max + (n_tiles & 1u) * 2u * CH_BM;
#pragma unroll 1
      for (unsigned r0 = warp; r0 < CH_BM; r0 += CH_WORK_WARPS * FLY) {
        float2 o[FLY][PER];
#pragma unroll
        for (unsigned f = 0; f < FLY; f++)
#pragma unroll
          for (unsigned k = 0; k < PER; k++) o[f][k] = (reinterpret_cast<const float2*>(smem + S::o) + (r0 + f * CH_WORK_WARPS) * (S::OP / 2))[lane + 32u * k];
#pragma unroll
        for (unsigned f = 0; f < FLY; f++) {
          const unsigned r = r0 + f * CH_WORK_WARPS, t = (row0 + r) / G, head = kvh * G + (row0 + r) % G;
          if (t >= n_tok) continue;
          float* rec = tmp + (((size_t)t * n_q + head) * n_splits + split) * (HD + 2);
#pragma unroll
          for (unsigned k = 0; k < PER; k++) *reinterpret_cast<float2*>(rec + 2 + 2u * (lane + 32u * k)) = o[f][k];
          if (lane == 0) *reinterpret_cast<float2*>(rec) = make_float2(row_scale[r], sums[r] + sums[CH_BM + r]);
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 24;");
    if (warp == CH_WORK_WARPS) {
    // ---- products: the whole warp runs the loop, one elected lane issues; the trip count out of a warp reduction, so that it and
    // the descriptors stay in uniform registers
    const unsigned leader = elect_one(), tiles = __reduce_max_sync(0xffffffffu, n_tiles);
    constexpr uint32_t idesc_s = (1u << 4) | ((CH_BN >> 3) << 17) | ((CH_BM >> 4) << 24), idesc_o = (1u << 4) | ((HD >> 3) << 17) | ((CH_BM >> 4) << 24);
    const uint64_t d_ql = tc_desc(sb + S::ql, CH_BM * 16u, 128u), d_kh = tc_desc(sb + S::kh, CH_BN * 16u, 128u), d_kl = tc_desc(sb + S::kl, CH_BN * 16u, 128u),
                   d_vh = tc_desc(sb + S::vh, HD * 16u, 128u), d_vl = tc_desc(sb + S::vl, HD * 16u, 128u);
    bool ok = false;
    // Within a tile the small terms come first: the accumulator drops bits below its largest term at every step.
    for (unsigned i = 0; i < tiles; i++) {
      if (!__all_sync(0xffffffffu, mb_wait(bar(CB_K_FULL), i & 1u, CH_WAIT))) goto out;
      tc_fence_after();
      if (leader) {
#pragma unroll
        for (unsigned ks = 0; ks < HD / 16u; ks++) {  // (address fields count 16 bytes; two chunks a step)
          tc_mma_f16_ta(S::t_s, S::t_q + 8u * ks, d_kl + (uint64_t)(2u * ks * CH_BN), idesc_s, ks ? 1u : 0u);
          tc_mma_f16(S::t_s, d_ql + (uint64_t)(2u * ks * CH_BM), d_kh + (uint64_t)(2u * ks * CH_BN), idesc_s, 1u);
        }
#pragma unroll
        for (unsigned ks = 0; ks < HD / 16u; ks++) tc_mma_f16_ta(S::t_s, S::t_q + 8u * ks, d_kh + (uint64_t)(2u * ks * CH_BN), idesc_s, 1u);
        tc_commit(bar(CB_S_FULL));
        tc_commit(bar(CB_K_FREE));
      }
      __syncwarp();
      {
        const bool got = mb_wait(bar(CB_V_FULL), i & 1u, CH_WAIT) && (i == 0u || mb_wait(bar(CB_O_FREE), (i - 1u) & 1u, CH_WAIT)) &&
                         mb_wait(bar(CB_P_FULL), i & 1u, CH_WAIT);
        if (!__all_sync(0xffffffffu, got)) goto out;
      }
      tc_fence_after();
      if (leader) {
#pragma unroll
        for (unsigned ks = 0; ks < CH_BN / 16u; ks++) {
          tc_mma_f16_ta(S::t_o, S::t_pl + 8u * ks, d_vh + (uint64_t)(2u * ks * HD), idesc_o, ks ? 1u : 0u);
          tc_mma_f16_ta(S::t_o, S::t_ph + 8u * ks, d_vl + (uint64_t)(2u * ks * HD), idesc_o, 1u);
        }
#pragma unroll
        for (unsigned ks = 0; ks < CH_BN / 16u; ks++) tc_mma_f16_ta(S::t_o, S::t_ph + 8u * ks, d_vh + (uint64_t)(2u * ks * HD), idesc_o, 1u);
        tc_commit(bar(CB_V_FREE));
      }
      __syncwarp();
    }
    ok = true;
  out:
    if (leader) {  // every product issued must finish before shared and tensor memory go away (bounded)
      if (!ok) *fail = 1;
      tc_commit(bar(CB_DONE));
    }
    __syncwarp();
    mb_wait(bar(CB_DONE), 0u, CH_WAIT);
    } else if (warp == CH_WORK_WARPS + 1) {
    // ---- decoded tiles: K of the next one when its scores are made, V when its values are
    const unsigned leader = elect_one();
    constexpr unsigned BYTES = Image::HALF;
    const unsigned char* src = img + img_at * Image::TILE;
    unsigned ks = 0, vs = 0;  // copies sent
    for (unsigned i = 0; i < n_tiles; i++) {
      if (i > 0 && !__all_sync(0xffffffffu, mb_wait(bar(CB_K_FREE), (i - 1u) & 1u, CH_WAIT))) break;
      if (leader) {
        mb_expect(bar(CB_K_FULL), BYTES);
        bulk_in(sb + S::kh, src, BYTES, bar(CB_K_FULL));
      }
      ks++;
      if (i > 0 && !__all_sync(0xffffffffu, mb_wait(bar(CB_V_FREE), (i - 1u) & 1u, CH_WAIT))) break;
      if (leader) {
        mb_expect(bar(CB_V_FULL), BYTES);
        bulk_in(sb + S::vh, src + BYTES, BYTES, bar(CB_V_FULL));
      }
      vs++;
      src += (size_t)n_kv * Image::TILE;
      __syncwarp();
    }
    if ((ks < n_tiles || vs < n_tiles) && leader) *fail = 1;
    // the copies must have landed before this block's shared memory goes away (bounded)
    if (ks) mb_wait(bar(CB_K_FULL), (ks - 1u) & 1u, CH_WAIT);
    if (vs) mb_wait(bar(CB_V_FULL), (vs - 1u) & 1u, CH_WAIT);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (tid == 0 && *fail) atomicOr(err, 8u);
  if (warp == CH_WORK_WARPS) tc_dealloc(tmem, 512);
}

// The (m, l, O) records of a token's heads -> the image the output projection reads its rows from (lower.rs:5897-6088 and
// the operand split in one).  One block per (padded) token row, 8 neighbouring dims per thread and step.  The first splits' O are
// requested before the (m, l) pairs are looked at; a warp makes the factors of a head.
constexpr unsigned MG_FLY = 4;
__global__ void __launch_bounds__(512) sdpa_merge_split_kernel(unsigned n_tok, unsigned np, unsigned tbn, unsigned n_q, unsigned hd, const float* tmp, unsigned n_splits,
                                                               __half* xt) {
  ks_pdl_entry();
  extern __shared__ float fac[];  // [n_q][n_splits]: exp(m - M) / L, 0 for an empty split (which may have left no O)
  __shared__ float red[32];
  const unsigned t = blockIdx.x, chunks = n_q * hd / 8u, lane = threadIdx.x & 31u;
  const float* rec_t = tmp + (size_t)t * n_q * n_splits * (hd + 2u);
  constexpr int MOST = 2;
  float v[MOST][8];
  float2 o[MG_FLY][4];
  auto request = [&](const float* rec, unsigned d, unsigned s0) {
#pragma unroll
    for (unsigned k = 0; k < MG_FLY; k++)
#pragma unroll
      for (int e = 0; e < 4; e++)
        o[k][e] = s0 + k < n_splits ? *reinterpret_cast<const float2*>(rec + (size_t)(s0 + k) * (hd + 2u) + 2 + d + 2 * e) : make_float2(0.f, 0.f);
  };
  auto place = [&](unsigned ck, const float*& rec, unsigned& head, unsigned& d) {
    head = ck * 8u / hd;
    d = ck * 8u - head * hd;
    rec = rec_t + (size_t)head * n_splits * (hd + 2u);
  };
  const float* rec;
  unsigned head, d;
  if (t < n_tok && threadIdx.x < chunks) {
    place(threadIdx.x, rec, head, d);
    request(rec, d, 0);
  }
  if (t < n_tok)
    for (unsigned h = threadIdx.x >> 5; h < n_q; h += blockDim.x >> 5) {
      const float* r = rec_t + (size_t)h * n_splits * (hd + 2u);
      float M = kNegInit, L = 0.0f;
      for (unsigned s = lane; s < n_splits; s += 32u) M = fmaxf(M, r[(size_t)s * (hd + 2u)]);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
      for (unsigned s = lane; s < n_splits; s += 32u) {
        const float l = r[(size_t)s * (hd + 2u) + 1], f = l != 0.0f ? __expf(r[(size_t)s * (hd + 2u)] - M) : 0.0f;
        L = fmaf(l, f, L);
        fac[h * n_splits + s] = f;
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) L += __shfl_xor_sync(0xffffffffu, L, off);
      for (unsigned s = lane; s < n_splits; s += 32u) fac[h * n_splits + s] /= L;
    }
  __syncthreads();
  float m = 0.0f;
#pragma unroll
  for (int kk = 0; kk < MOST; kk++) {
    const unsigned ck = threadIdx.x + (unsigned)kk * blockDim.x;
#pragma unroll
    for (int e = 0; e < 8; e++) v[kk][e] = 0.0f;
    if (t < n_tok && ck < chunks) {
      place(ck, rec, head, d);
      for (unsigned s0 = 0; s0 < n_splits; s0 += MG_FLY) {
        if (kk || s0) request(rec, d, s0);
#pragma unroll
        for (unsigned k = 0; k < MG_FLY; k++) {
          const float f = s0 + k < n_splits ? fac[head * n_splits + s0 + k] : 0.0f;
          if (f != 0.0f)
#pragma unroll
            for (int e = 0; e < 4; e++) {
              v[kk][2 * e] = fmaf(o[k][e].x, f, v[kk][2 * e]);
              v[kk][2 * e + 1] = fmaf(o[k][e].y, f, v[kk][2 * e + 1]);
            }
        }
      }
      m = fmaxf(m, absmax8(v[kk]));
    }
  }
  float up;
  const float down = row_scale_down(block_max_f(m, red), &up);
  if (threadIdx.x == 0) reinterpret_cast<float*>(xt + xt_scale_off(n_q * hd, np))[t] = up;
#pragma unroll
  for (int kk = 0; kk < MOST; kk++) {
    const unsigned ck = threadIdx.x + (unsigned)kk * blockDim.x;
    if (ck < chunks) {
#pragma unroll
      for (int e = 0; e < 8; e++) v[kk][e] *= down;
      put_split8(xt, np, tbn, t, ck, chunks, v[kk], true);
    }
  }
}

template <int HD>
int launch_chunk(ks_ctx* ctx, dim3 grid, const ChunkParts& parts, size_t slot_stride, unsigned n_q, unsigned n_kv, float scale, const float* q, const uint8_t* K, const uint8_t* V,
                 const float* meta, float* tmp, unsigned n_splits, const ks_kv_image& image) {
  constexpr size_t smem = ChunkSmem<HD>::total;
  static bool set[16] = {false};
  if (!set[ctx->device & 15]) {
    cudaError_t e = cudaFuncSetAttribute(sdpa_chunk_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return ks_fail(ctx, KS_ERR_CUDA, "sdpa_chunk: cannot set %zu B shared memory: %s", smem, cudaGetErrorString(e));
    set[ctx->device & 15] = true;
  }
  unsigned char* img = (unsigned char*)image.base;
  float* img_up = (float*)(img + image.tiles * n_kv * (size_t)ChunkImage<HD>::TILE);
  KS_LAUNCH(ctx, (kv_image_kernel<HD>), dim3(image.span, 4u * n_kv, parts.n), 256, 0, parts, slot_stride, n_kv, K, V, meta, img, img_up);
  const int rc = ks_after_launch(ctx, "kv_image");
  if (rc) return rc;
  KS_LAUNCH(ctx, sdpa_chunk_kernel<HD>, grid, CH_THREADS, smem, parts, n_q, n_kv, scale, q, meta, tmp, n_splits, (const unsigned char*)img, (const float*)img_up,
            (unsigned*)ctx->ws + KS_WS_ERR_WORD);
  return ks_after_launch(ctx, "sdpa_chunk");
}
}  // namespace

// Context splits of a chunk: enough blocks for every SM, at least two tiles each.  A nearly empty second wave costs more than fewer
// splits, except against one: the later rows see most of the context, and half a chip waits for them (2047 rows of 8 heads, 128
// blocks: 118 us, twice as many halves 76, three times as many thirds 95; 64 blocks in halves 44, thirds 46; 19 blocks 31, 26 and 23.5; 126
// blocks behind as many positions 213, 188 and 187).  `ctx_len` may exceed what the rows see.
int ks_sdpa_chunk_splits(const ks_ctx* ctx, int n_tok, size_t n_q, size_t n_kv, size_t ctx_len, int most) {
  const size_t blocks = ((size_t)n_tok * (n_q / n_kv) + CH_BM - 1) / CH_BM * n_kv;
  size_t s = ((size_t)ctx->sm_count + blocks - 1) / blocks;
  if (s > 2 && s * blocks > (size_t)ctx->sm_count + (size_t)ctx->sm_count / 8) s--;
  const size_t by_len = (ctx_len + 2 * CH_BN - 1) / (2 * CH_BN);
  if (s > by_len) s = by_len;
  if (s > (size_t)most) s = most;
  return s < 1 ? 1 : (int)s;
}

bool ks_sdpa_merge_split_covers(size_t n_q, size_t hd) { return n_q * hd <= 8192 && n_q * hd % 256 == 0 && n_q <= 64; }
// Groups of query heads: those of decode attention.
bool ks_sdpa_chunk_covers(size_t n_q, size_t n_kv, size_t hd, const void* K, const void* V) {
  const size_t G = n_q / n_kv;
  return (hd == 256 || hd == 128) && G <= 16 && CH_BM % G == 0 && ks_sdpa_merge_split_covers(n_q, hd) && (((uintptr_t)K | (uintptr_t)V) & 3u) == 0;
}

size_t ks_kv_image_bytes(size_t tiles, size_t n_kv, size_t hd) { return tiles * n_kv * (hd == 256 ? ChunkImage<256>::TILE : ChunkImage<128>::TILE) + tiles * n_kv * sizeof(float); }
unsigned ks_kv_image_tiles(size_t positions) { return (unsigned)((positions + CH_BN - 1) / CH_BN); }

// q [n_tok, n_q hd] f32, meta [n_tok][4] = (tlen, start, -, -) with both ends growing along the rows of a slot
// -> records in tmp [n_tok][n_q][n_splits][hd + 2].
int ks_launch_sdpa_chunk(ks_ctx* ctx, int n_tok, size_t n_q, size_t n_kv, size_t hd, float scale, const float* q, const uint8_t* K, const uint8_t* V,
                         const float* meta, float* tmp, int n_splits, const ks_kv_image& image, const ks_row_parts* parts, size_t slot_stride) {
  ChunkParts cp{};
  cp.n = parts ? parts->n : 1u;
  unsigned tiles = 0;
  for (unsigned p = 0; p < cp.n; p++) {
    cp.row0[p] = parts ? parts->row0[p] : 0u;
    cp.row0[p + 1] = parts ? parts->row0[p + 1] : (unsigned)n_tok;
    cp.slot[p] = parts ? parts->slot[p] : 0u;
    cp.image0[p] = parts ? parts->image0[p] : 0u;
    cp.tile0[p] = tiles;
    tiles += (unsigned)(((cp.row0[p + 1] - cp.row0[p]) * (n_q / n_kv) + CH_BM - 1) / CH_BM);
  }
  cp.tile0[cp.n] = tiles;
  const dim3 grid(tiles, (unsigned)n_kv, (unsigned)n_splits);
  return hd == 256 ? launch_chunk<256>(ctx, grid, cp, slot_stride, (unsigned)n_q, (unsigned)n_kv, scale, q, K, V, meta, tmp, (unsigned)n_splits, image)
                   : launch_chunk<128>(ctx, grid, cp, slot_stride, (unsigned)n_q, (unsigned)n_kv, scale, q, K, V, meta, tmp, (unsigned)n_splits, image);
}

// Records of n_tok rows -> the Q4_K form of the operand image (rows past n_tok as zeros).
int ks_launch_sdpa_merge_split(ks_ctx* ctx, int n_tok, ks_gemm_blocks b, size_t n_q, size_t hd, const float* tmp, int n_splits, void* xt) {
  const unsigned chunks = (unsigned)(n_q * hd / 8), threads = chunks < 512u ? (chunks + 31u) / 32u * 32u : 512u;
  KS_LAUNCH(ctx, sdpa_merge_split_kernel, b.np, threads, (size_t)n_q * n_splits * sizeof(float), (unsigned)n_tok, b.np, b.tbn, (unsigned)n_q, (unsigned)hd, tmp, (unsigned)n_splits, (__half*)xt);
  return ks_after_launch(ctx, "sdpa_merge_split");
}

// Chunk attention alone, for tests.
extern "C" int ks_debug_sdpa_chunk(ks_ctx* ctx, size_t n_q, size_t n_kv, size_t hd, size_t max_t, float scale, int n_parts, const int* row0, const int* slots,
                                   size_t slot_stride_bytes, const ks_buf* q, const ks_buf* K, const ks_buf* V, const ks_buf* meta, ks_buf* tmp, int n_splits) {
  if (!ctx) return KS_ERR_INVALID;
  KS_REQUIRE(ctx, n_q > 0 && n_kv > 0 && n_q % n_kv == 0 && hd % 32 == 0 && max_t > 0 && n_splits >= 1 && n_splits < 65536, "sdpa_chunk: bad shape");
  KS_REQUIRE(ctx, n_parts >= 1 && n_parts <= 64 && row0 && slots && row0[0] == 0 && slot_stride_bytes % 4 == 0, "sdpa_chunk: bad parts");
  const size_t cache = max_t * n_kv * (hd / 32) * KS_Q40_BLOCK_BYTES;
  ks_row_parts parts{};
  parts.n = (unsigned)n_parts;
  size_t last = 0;
  for (int p = 0; p < n_parts; p++) {
    KS_REQUIRE(ctx, row0[p + 1] > row0[p] && row0[p + 1] <= KS_GEMM_ROWS && slots[p] >= 0, "sdpa_chunk: bad parts");
    parts.row0[p + 1] = (unsigned)row0[p + 1];
    parts.slot[p] = (unsigned)slots[p];
    parts.image0[p] = (unsigned)p * ks_kv_image_tiles(max_t);
    last = (size_t)slots[p] > last ? (size_t)slots[p] : last;
  }
  const size_t n = (size_t)row0[n_parts], need = last * slot_stride_bytes + cache;
  KS_REQUIRE(ctx, ks_fits(K, 0, need) && ks_fits(V, 0, need) && ks_fits(q, 0, n * n_q * hd * 4) && ks_fits(meta, 0, n * 16) &&
             ks_fits(tmp, 0, n * n_q * (size_t)n_splits * (hd + 2) * 4), "sdpa_chunk: a buffer is too small");
  if (!ks_sdpa_chunk_covers(n_q, n_kv, hd, K->dptr, V->dptr)) return ks_fail(ctx, KS_ERR_UNSUPPORTED, "sdpa_chunk: shape not covered");
  ks_kv_image image{};
  image.span = ks_kv_image_tiles(max_t);
  image.tiles = (size_t)n_parts * image.span;
  const int rc = ks_ctx_gemm_scratch(ctx, ks_kv_image_bytes(image.tiles, n_kv, hd), &image.base);
  if (rc) return rc;
  return ks_launch_sdpa_chunk(ctx, (int)n, n_q, n_kv, hd, scale, (const float*)q->dptr, (const uint8_t*)K->dptr, (const uint8_t*)V->dptr, (const float*)meta->dptr,
                              (float*)tmp->dptr, n_splits, image, &parts, slot_stride_bytes);
}
