// Attention of a prompt chunk: many token rows of one slot, or of several, against their Q4_0 caches, causal (and windowed) by row.
//
// The reference runs its decode attention once per prompt row (forward_prefill_chunk, crates/ksearch_gemma/src/
// gemma_prim.rs:1463-1472, over crates/ksearch_codegen/src/lower.rs:4897-6088), so every row reads the whole context again.
// Here a block takes 128 query rows that share a KV head (128 / G tokens x the head's G query heads), brings each tile of 64
// positions in once and multiplies on tcgen05 (f16 in, f32 out) without giving up f32 accuracy: q (scaled per row by a power of
// two), the cached values d (n - 8), exactly, and the probabilities are two f16 terms each, a product is hi hi + hi lo + lo hi.
//   * q's first term and the probabilities lie in TENSOR memory as the A operand, q's second term and the decoded tile in shared
//     memory; scores and a tile's values are the accumulators (HD = 256 fills the 512 columns);
//   * four warps own a row of scores per thread: mask, running maximum, probabilities;
//   * eight decode: K as positions x dims, V as dims x positions (a thread takes one byte of eight neighbouring rows), and add each
//     tile's values, scaled as the maximum moved, to f32 registers, half a row per thread (184 registers);
//   * one issues.  The scores of the next tile follow the values of this one in the tensor pipe, and meanwhile the decoders work;
//     what the pipe waits for is the probabilities.
// The sums leave tensor memory after every tile and small terms come first, because the accumulator truncates: against 64 bits the
// result is off by 1.3..1.8e-7 (2-norm) whatever the context, where accumulating on gave 3e-6 over 2047 positions, 1e-5 over 4000.
// The context is split over blockIdx.z; (m, l, O) records go to `tmp` as the decode kernels leave them and
// sdpa_merge_split_kernel folds them straight into the operand image of the output projection.
//
// Bound by the decoders, who turn a tile's values, fold the one before and turn the next one's keys in a row: 5.7 us for 128 x 64,
// 1.2 of them MMAs (2047 rows, 2 splits: tensor pipe 21 %, issue slots 38 %).  A block takes another 18 us for its start, q and
// records.  Back to back: one block of 64 tiles 381 us; 2047 rows of 8 heads (128 blocks of up to 32 tiles) 205 us, in two splits 118;
// 2000 rows behind 2000 positions, 2 KV heads (126 blocks of up to 63 tiles) 388, in two splits 344.  On mma.sync (64 rows a block) the
// last two took 336 and 809.
#include "ks_gemm_common.cuh"

namespace {

constexpr int CH_BM = 128, CH_BN = 64;                 // query rows, positions of a tile
constexpr int CH_ROW_WARPS = 4, CH_DEC_WARPS = 8, CH_WORK = (CH_ROW_WARPS + CH_DEC_WARPS) * 32, CH_THREADS = CH_WORK + 128;
constexpr unsigned CH_WAIT = 1u << 20;
constexpr float CH_P = 256.0f;                         // probabilities carry 2^8
constexpr unsigned CH_K_MOST = 0x6FFFu;                // the largest scale with 8 d in f16, 8188
constexpr float kNegInit = -1.0e30f;

// barriers: operands ready (decoders, row warps), the tile's O taken (decoders), products ready (commits: scores done = K free;
// values done = V and P free)
enum { CB_K_FULL, CB_V_FULL, CB_P_FULL, CB_O_FREE, CB_S_FULL, CB_K_FREE, CB_V_FREE, CB_DONE, CB_COUNT };

template <int HD>
struct ChunkSmem {
  static constexpr unsigned NB = HD / 32, ROWB = NB * KS_Q40_BLOCK_BYTES, RP = ROWB + 4;
  static constexpr unsigned slot = 64, row = 128;     // tensor-memory address, failure flag; per row: scale, first, past the last position, maximum,
                                                      // then what the sums so far are multiplied by, of two tiles
  static constexpr unsigned up = row + CH_BM * 24;    // of two tiles: what their scores are multiplied by
  static constexpr unsigned raw = 4096;
  static_assert(up + 8 <= raw, "the rows' words fit in front of the packed rows");
  static constexpr unsigned ql = (raw + 2 * CH_BN * RP + 1023u) & ~1023u, kh = ql + CH_BM * HD * 2, kl = kh + CH_BN * HD * 2, vh = kl + CH_BN * HD * 2,
                            vl = vh + CH_BN * HD * 2, total = vl + CH_BN * HD * 2;
  static constexpr unsigned o = ql, OP = HD + 4;      // the result on its way out: rows of OP floats
  static_assert(o + CH_BM * OP * 4 <= total, "the result fits the operands");
  // tensor memory: first term of q, scores, the probabilities' two terms, O
  static constexpr unsigned t_q = 0, t_s = HD / 2, t_ph = t_s + CH_BN, t_pl = t_ph + CH_BN / 2, t_o = t_pl + CH_BN / 2;
  static_assert(t_o + HD <= 512, "tensor memory");
};

__device__ __forceinline__ void mb_arrive1(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void cp4(uint32_t dst, const void* src) { asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory"); }
// The decoders meet; true if every one of them says so.
__device__ __forceinline__ bool dec_all(bool ok) {
  unsigned r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.and.pred q, 1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((unsigned)ok), "n"(CH_DEC_WARPS * 32)
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

struct ChunkParts {  // part p: rows from row0[p] on, row tiles from tile0[p] on
  unsigned n, row0[65], tile0[65], slot[64];
};

template <int HD>
__global__ void __launch_bounds__(CH_THREADS, 1)
sdpa_chunk_kernel(const __grid_constant__ ChunkParts parts, size_t slot_stride, unsigned n_q, unsigned n_kv, float scale, const float* q, const uint8_t* K,
                  const uint8_t* V, const float* meta, float* tmp, unsigned n_splits, unsigned* err) {
  using S = ChunkSmem<HD>;
  constexpr unsigned NB = S::NB, RP = S::RP, ROWB = S::ROWB;
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
  K += parts.slot[part_id] * slot_stride;
  V += parts.slot[part_id] * slot_stride;
  const uint32_t sb = sm32(smem);
  auto bar = [&](unsigned i) { return sb + 8u * i; };
  uint32_t* tslot = reinterpret_cast<uint32_t*>(smem + S::slot);
  volatile unsigned* fail = reinterpret_cast<volatile unsigned*>(smem + S::slot + 8);
  float* row_scale = reinterpret_cast<float*>(smem + S::row);
  int* row_first = reinterpret_cast<int*>(smem + S::row + CH_BM * 4);
  int* row_end = reinterpret_cast<int*>(smem + S::row + CH_BM * 8);
  unsigned* row_max = reinterpret_cast<unsigned*>(smem + S::row + CH_BM * 12);
  float* row_alpha = reinterpret_cast<float*>(smem + S::row + CH_BM * 16);
  float* tile_up = reinterpret_cast<float*>(smem + S::up);

  // ---- the block's rows: row r is query head kvh G + r % G of token (row0 + r) / G; positions they see at all
  const unsigned tok_a = row0 / G, tok_b = min((row0 + CH_BM - 1u) / G, n_tok - 1u);
  const int pmin = (int)meta[tok_a * 4 + 1];                                        // starts and ends grow with the token
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
  const bool decoder = warp >= CH_ROW_WARPS && warp < CH_ROW_WARPS + CH_DEC_WARPS;
  const unsigned dt = tid - CH_ROW_WARPS * 32;  // decoders: 0..255
  auto fetch = [&](int t0) {  // the packed rows of positions t0 .. +64 (rows past the end repeat the last, their scores are masked)
    for (unsigned r = dt >> 5; r < 2u * CH_BN; r += CH_DEC_WARPS) {
      const int pos = min(t0 + (int)(r & (CH_BN - 1u)), pmax - 1);
      const uint8_t* src = (r < CH_BN ? K : V) + ((size_t)pos * n_kv + kvh) * ROWB;
      const uint32_t dst = sb + S::raw + r * RP;
      for (unsigned w = lane; w < ROWB / 4u; w += 32u) cp4(dst + 4u * w, src + 4u * w);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // The largest scale (its f16 bits) of the K rows this thread copied.  Block b's scale is half of word 18 b / 4, and those words are
  // all among a lane's first.
  static_assert((NB - 1u) * KS_Q40_BLOCK_BYTES < 128u, "scales lie in the first 32 words of a row");
  const unsigned scale_at = (lane * 4u + KS_Q40_BLOCK_BYTES - 1u) / KS_Q40_BLOCK_BYTES * KS_Q40_BLOCK_BYTES;
  const bool has_scale = scale_at < lane * 4u + 4u && scale_at < ROWB;
  const unsigned scale_off = S::raw + ((warp - CH_ROW_WARPS) & (CH_DEC_WARPS - 1u)) * RP + (has_scale ? scale_at : lane * 4u);
  auto most_scale = [&] {
    unsigned m = 0;
#pragma unroll
    for (unsigned k = 0; k < CH_BN / CH_DEC_WARPS; k++) {
      const unsigned d = *reinterpret_cast<const unsigned short*>(smem + scale_off + k * CH_DEC_WARPS * RP) & 0x7FFFu;
      m = d > m ? d : m;
    }
    return has_scale ? m : 0u;
  };
  if (decoder) fetch(t_begin);

  if (tid == 0) {
    mb_init(bar(CB_K_FULL), CH_DEC_WARPS);
    mb_init(bar(CB_V_FULL), CH_DEC_WARPS);
    mb_init(bar(CB_P_FULL), CH_ROW_WARPS);
    mb_init(bar(CB_O_FREE), CH_DEC_WARPS);
    for (unsigned i = CB_S_FULL; i < CB_COUNT; i++) mb_init(bar(i), 1);
    *fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (tid < CH_BM) row_max[tid] = 0u;
  if (warp == CH_ROW_WARPS + CH_DEC_WARPS) tc_alloc(sm32(tslot), 512);
  __syncthreads();

  // ---- q: a thread takes every third chunk of 8 dims of a row; the row maximum sets a power of two, then two f16 terms per value.
  // The second term stays in shared memory as core matrices, the first passes through there (K's place) to tensor memory.
  {
    constexpr unsigned PARTS = CH_WORK / CH_BM, PER = (HD / 8 + PARTS - 1) / PARTS;
    const unsigned r = tid % CH_BM, part = tid / CH_BM, t = (row0 + r) / G, head = kvh * G + (row0 + r) % G;
    float v[PER][8];
    float m = 0.0f;
    if (tid < CH_WORK) {
      const float* src = q + ((size_t)t * n_q + head) * HD;
#pragma unroll
      for (unsigned k = 0; k < PER; k++) {
        const unsigned c = part + k * PARTS;
        const bool in = c < HD / 8u && t < n_tok;
        const float4 a = in ? *reinterpret_cast<const float4*>(src + 8u * c) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 b = in ? *reinterpret_cast<const float4*>(src + 8u * c + 4u) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[k][0] = a.x; v[k][1] = a.y; v[k][2] = a.z; v[k][3] = a.w;
        v[k][4] = b.x; v[k][5] = b.y; v[k][6] = b.z; v[k][7] = b.w;
        m = fmaxf(m, absmax8(v[k]));
      }
      atomicMax(row_max + r, __float_as_uint(m));
    }
    __syncthreads();
    if (tid < CH_WORK) {
      float up;
      const float down = row_scale_down(__uint_as_float(row_max[r]), &up);
      if (part == 0) {
        row_scale[r] = up * scale;
        row_first[r] = t < n_tok ? (int)meta[t * 4 + 1] : 0;
        row_end[r] = t < n_tok ? (int)meta[t * 4 + 1] + (int)meta[t * 4 + 0] : 0;
      }
#pragma unroll
      for (unsigned k = 0; k < PER; k++) {
        const unsigned c = part + k * PARTS;
        if (c < HD / 8u) {
#pragma unroll
          for (int e = 0; e < 8; e++) v[k][e] *= down;
          uint4 hi, lo;
          split8(v[k], hi, lo);
          *reinterpret_cast<uint4*>(smem + S::kh + (c * CH_BM + r) * 16u) = hi;
          *reinterpret_cast<uint4*>(smem + S::ql + (c * CH_BM + r) * 16u) = lo;
        }
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  const uint32_t tmem = *tslot;
  if (tmem != 0u && tid == 0) *fail = 1;  // all 512 columns were asked for: they start at 0
  const uint32_t tlane = (warp & 3u) << 21;   // 32 rows per warp, in the address bits of the lane
  if (warp < CH_ROW_WARPS) {
#pragma unroll
    for (unsigned c = 0; c < HD / 8u; c += 2u) {
      const uint4 a = *reinterpret_cast<const uint4*>(smem + S::kh + (c * CH_BM + tid) * 16u), b = *reinterpret_cast<const uint4*>(smem + S::kh + ((c + 1u) * CH_BM + tid) * 16u);
      const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      tc_st8(tlane + S::t_q + c * 4u, w);
    }
    tc_wait_st();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (warp < CH_ROW_WARPS) {
    // ---- a row of scores per thread
    asm volatile("setmaxnreg.dec.sync.aligned.u32 120;");
    const float sc = row_scale[tid];
    const int first = row_first[tid], end = row_end[tid];
    float ref = kNegInit, l = 0.0f;
    bool ok = true;
    for (unsigned i = 0; i < n_tiles; i++) {
      if (!__all_sync(0xffffffffu, mb_wait(bar(CB_S_FULL), i & 1u, CH_WAIT))) { ok = false; break; }
      tc_fence_after();
      uint32_t s[4][16];
#pragma unroll
      for (int k = 0; k < 4; k++) tc_ld16(tlane + S::t_s + 16u * k, s[k]);
#pragma unroll
      for (int k = 0; k < 4; k++) tc_wait_ld16(s[k]);
      const int p0 = t_begin + (int)i * CH_BN, a = first - p0, b = min(end, t_end) - p0;  // columns [a, b) are seen
      const float st = sc * tile_up[i & 1u];
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < CH_BN; j++) {
        const float x = j >= a && j < b ? __uint_as_float(s[j / 16][j % 16]) * st : -INFINITY;
        s[j / 16][j % 16] = __float_as_uint(x);
        mx = fmaxf(mx, x);
      }
      mx = fmaxf(mx, ref);
      const float alpha = __expf(ref - mx);
      ref = mx;
      row_alpha[(i & 1u) * CH_BM + tid] = alpha;
      if (i > 0) {  // P is free
        if (!__all_sync(0xffffffffu, mb_wait(bar(CB_V_FREE), (i - 1u) & 1u, CH_WAIT))) { ok = false; break; }
        tc_fence_after();
      }
      float sum = 0.0f;
#pragma unroll
      for (int k = 0; k < 4; k++) {
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
        tc_st8(tlane + S::t_ph + 8u * k, ph);
        tc_st8(tlane + S::t_pl + 8u * k, pl);
      }
      l = l * alpha + sum;
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mb_arrive1(bar(CB_P_FULL));
    }
    if (!ok && lane == 0) *fail = 1;
    row_scale[tid] = ref;
    reinterpret_cast<float*>(row_max)[tid] = l;
  } else if (decoder) {
    // ---- packed rows -> two f16 terms of K (positions x dims) and of V transposed (dims x positions); a tile's values are added to
    // half a row per thread
    asm volatile("setmaxnreg.inc.sync.aligned.u32 184;");
    constexpr unsigned HALF = HD / 2;
    const unsigned orow = (warp & 3u) * 32u + lane, ocol = (warp >> 2 & 1u) * HALF;  // (warps 4..7 and 8..11)
    float acc[HALF];
#pragma unroll
    for (unsigned c = 0; c < HALF; c++) acc[c] = 0.0f;
    auto fold = [&](unsigned i) {
      tc_fence_after();
      const float alpha = row_alpha[(i & 1u) * CH_BM + orow];
#pragma unroll
      for (unsigned c = 0; c < HALF; c += 16u) {
        uint32_t o[16];
        tc_ld16(tlane + S::t_o + ocol + c, o);
        tc_wait_ld16(o);
#pragma unroll
        for (unsigned e = 0; e < 16u; e++) acc[c + e] = fmaf(acc[c + e], alpha, __uint_as_float(o[e]));
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mb_arrive1(bar(CB_O_FREE));
    };
    bool ok = true;
    for (unsigned i = 0; i < n_tiles; i++) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      const bool fits = most_scale() <= CH_K_MOST;
      if (i > 0) ok = mb_wait(bar(CB_K_FREE), (i - 1u) & 1u, CH_WAIT);
      // The raw rows are there, K is free.  A tile with a scale whose products leave f16 is decoded at an eighth and its scores are
      // multiplied by 8; what that rounds off (2^-22 of a value at most) is nothing beside a value of 57000.  Every thread looks at
      // the scales that it copied itself.
      float tile = 1.0f;
      if (!dec_all(ok && fits)) {
        if (!dec_all(ok)) { ok = false; break; }
        tile = 8.0f;
      }
      const __half2 down = __float2half2_rn(1.0f / tile);
#pragma unroll 1
      for (unsigned job = dt; job < CH_BN * NB; job += CH_DEC_WARPS * 32) {  // a block of a row
        const unsigned p = job % CH_BN, b = job / CH_BN;
        const unsigned char* src = smem + S::raw + p * RP + b * KS_Q40_BLOCK_BYTES;
        const __half2 d = __hmul2(__half2half2(__ushort_as_half(*reinterpret_cast<const unsigned short*>(src))), down);
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; k++)
          w[k] = *reinterpret_cast<const unsigned short*>(src + 2 + 4 * k) | (uint32_t)*reinterpret_cast<const unsigned short*>(src + 4 + 4 * k) << 16;
#pragma unroll 1
        for (int half = 0; half < 2; half++)  // dims 0..15 of the block are the low nibbles
#pragma unroll
          for (int c = 0; c < 2; c++) {
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int k = 0; k < 2; k++) {
              const uint32_t x = half ? w[2 * c + k] >> 4 : w[2 * c + k];
              split_d(nib_h2(__byte_perm(x, 0u, 0x4140)), d, hi[2 * k], lo[2 * k]);
              split_d(nib_h2(__byte_perm(x, 0u, 0x4342)), d, hi[2 * k + 1], lo[2 * k + 1]);
            }
            const unsigned at = ((4u * b + 2u * half + c) * CH_BN + p) * 16u;
            *reinterpret_cast<uint4*>(smem + S::kh + at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4*>(smem + S::kl + at) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
          }
      }
      if (dt == 0) tile_up[i & 1u] = tile;
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mb_arrive1(bar(CB_K_FULL));
      if (i > 0) ok = mb_wait(bar(CB_V_FREE), (i - 1u) & 1u, CH_WAIT);
      if (!dec_all(ok)) { ok = false; break; }
      if (i > 0) fold(i - 1u);
#pragma unroll 1
      for (unsigned job = dt; job < 16u * NB * (CH_BN / 8); job += CH_DEC_WARPS * 32) {  // byte j of a block in eight neighbouring rows
        const unsigned j = job % 16u, b = job / 16u % NB, pg = job / (16u * NB);
        const unsigned char* src = smem + S::raw + (CH_BN + 8u * pg) * RP + b * KS_Q40_BLOCK_BYTES;
        uint32_t hl[4], ll[4], hh[4], lh[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const unsigned char *x = src + 2 * k * RP, *y = x + RP;
          const uint32_t n = x[2 + j] | (uint32_t)y[2 + j] << 16;
          const __half2 d = as_h2(*reinterpret_cast<const unsigned short*>(x) | (uint32_t)*reinterpret_cast<const unsigned short*>(y) << 16);
          split_d(nib_h2(n), d, hl[k], ll[k]);
          split_d(nib_h2(n >> 4), d, hh[k], lh[k]);
        }
        const unsigned at = (pg * HD + 32u * b + j) * 16u;
        *reinterpret_cast<uint4*>(smem + S::vh + at) = make_uint4(hl[0], hl[1], hl[2], hl[3]);
        *reinterpret_cast<uint4*>(smem + S::vl + at) = make_uint4(ll[0], ll[1], ll[2], ll[3]);
        *reinterpret_cast<uint4*>(smem + S::vh + at + 256u) = make_uint4(hh[0], hh[1], hh[2], hh[3]);
        *reinterpret_cast<uint4*>(smem + S::vl + at + 256u) = make_uint4(lh[0], lh[1], lh[2], lh[3]);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mb_arrive1(bar(CB_V_FULL));
      if (!dec_all(true)) break;  // (meets only: the raw rows are used up)
      if (i + 1u < n_tiles) fetch(t_begin + (int)(i + 1u) * CH_BN);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    ok = ok && __all_sync(0xffffffffu, mb_wait(bar(CB_V_FREE), (n_tiles - 1u) & 1u, CH_WAIT));
    if (!ok && lane == 0) *fail = 1;
    if (ok) {  // the rows through shared memory, so that they leave in whole lines; every product that read it is done
      fold(n_tiles - 1u);
      float* out = reinterpret_cast<float*>(smem + S::o) + orow * S::OP + ocol;
#pragma unroll
      for (unsigned c = 0; c < HALF; c += 4u)
        *reinterpret_cast<float4*>(out + c) = make_float4(acc[c] * (1.0f / CH_P), acc[c + 1] * (1.0f / CH_P), acc[c + 2] * (1.0f / CH_P), acc[c + 3] * (1.0f / CH_P));
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 24;");
    if (warp == CH_ROW_WARPS + CH_DEC_WARPS) {
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
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (*fail) {
    if (tid == 0) atomicOr(err, 8u);
  } else {
    for (unsigned r = warp; r < CH_BM; r += CH_THREADS / 32) {
      const unsigned t = (row0 + r) / G, head = kvh * G + (row0 + r) % G;
      if (t >= n_tok) continue;
      float* rec = tmp + (((size_t)t * n_q + head) * n_splits + split) * (HD + 2);
      const float2* o = reinterpret_cast<const float2*>(smem + S::o) + r * (S::OP / 2);
      for (unsigned d = lane; d < HD / 2u; d += 32u) *reinterpret_cast<float2*>(rec + 2 + 2u * d) = o[d];
      if (lane == 0) *reinterpret_cast<float2*>(rec) = make_float2(row_scale[r], reinterpret_cast<float*>(row_max)[r]);
    }
  }
  __syncthreads();
  if (warp == CH_ROW_WARPS + CH_DEC_WARPS) tc_dealloc(tmem, 512);
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
                 const float* meta, float* tmp, unsigned n_splits) {
  constexpr size_t smem = ChunkSmem<HD>::total;
  static bool set[16] = {false};
  if (!set[ctx->device & 15]) {
    cudaError_t e = cudaFuncSetAttribute(sdpa_chunk_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return ks_fail(ctx, KS_ERR_CUDA, "sdpa_chunk: cannot set %zu B shared memory: %s", smem, cudaGetErrorString(e));
    set[ctx->device & 15] = true;
  }
  KS_LAUNCH(ctx, sdpa_chunk_kernel<HD>, grid, CH_THREADS, smem, parts, slot_stride, n_q, n_kv, scale, q, K, V, meta, tmp, n_splits,
            (unsigned*)ctx->ws + KS_WS_ERR_WORD);
  return ks_after_launch(ctx, "sdpa_chunk");
}
}  // namespace

// Context splits of a chunk: enough blocks for every SM, at least two tiles each.  A nearly empty second wave costs more than fewer
// splits, except against one: the later rows see most of the context, and half a chip waits for them (2047 rows of 8 heads, 128
// blocks: 205 us, twice as many halves 118, three times as many thirds 151).  `ctx_len` may exceed what the rows see.
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

// q [n_tok, n_q hd] f32, meta [n_tok][4] = (tlen, start, -, -) with both ends growing along the rows of a slot
// -> records in tmp [n_tok][n_q][n_splits][hd + 2].
int ks_launch_sdpa_chunk(ks_ctx* ctx, int n_tok, size_t n_q, size_t n_kv, size_t hd, float scale, const float* q, const uint8_t* K, const uint8_t* V,
                         const float* meta, float* tmp, int n_splits, const ks_row_parts* parts, size_t slot_stride) {
  ChunkParts cp{};
  cp.n = parts ? parts->n : 1u;
  unsigned tiles = 0;
  for (unsigned p = 0; p < cp.n; p++) {
    cp.row0[p] = parts ? parts->row0[p] : 0u;
    cp.row0[p + 1] = parts ? parts->row0[p + 1] : (unsigned)n_tok;
    cp.slot[p] = parts ? parts->slot[p] : 0u;
    cp.tile0[p] = tiles;
    tiles += (unsigned)(((cp.row0[p + 1] - cp.row0[p]) * (n_q / n_kv) + CH_BM - 1) / CH_BM);
  }
  cp.tile0[cp.n] = tiles;
  const dim3 grid(tiles, (unsigned)n_kv, (unsigned)n_splits);
  return hd == 256 ? launch_chunk<256>(ctx, grid, cp, slot_stride, (unsigned)n_q, (unsigned)n_kv, scale, q, K, V, meta, tmp, (unsigned)n_splits)
                   : launch_chunk<128>(ctx, grid, cp, slot_stride, (unsigned)n_q, (unsigned)n_kv, scale, q, K, V, meta, tmp, (unsigned)n_splits);
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
    last = (size_t)slots[p] > last ? (size_t)slots[p] : last;
  }
  const size_t n = (size_t)row0[n_parts], need = last * slot_stride_bytes + cache;
  KS_REQUIRE(ctx, ks_fits(K, 0, need) && ks_fits(V, 0, need) && ks_fits(q, 0, n * n_q * hd * 4) && ks_fits(meta, 0, n * 16) &&
             ks_fits(tmp, 0, n * n_q * (size_t)n_splits * (hd + 2) * 4), "sdpa_chunk: a buffer is too small");
  if (!ks_sdpa_chunk_covers(n_q, n_kv, hd, K->dptr, V->dptr)) return ks_fail(ctx, KS_ERR_UNSUPPORTED, "sdpa_chunk: shape not covered");
  return ks_launch_sdpa_chunk(ctx, (int)n, n_q, n_kv, hd, scale, (const float*)q->dptr, (const uint8_t*)K->dptr, (const uint8_t*)V->dptr, (const float*)meta->dptr,
                              (float*)tmp->dptr, n_splits, &parts, slot_stride_bytes);
}
