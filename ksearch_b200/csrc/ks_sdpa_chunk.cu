// Attention of a prompt chunk: many token rows of one slot against its Q4_0 cache, causal (and windowed) by row.
//
// The reference runs its decode attention once per prompt row (forward_prefill_chunk, crates/ksearch_gemma/src/
// gemma_prim.rs:1463-1472, over crates/ksearch_codegen/src/lower.rs:4897-6088), so every row reads the whole context again.
// Here a block takes 64 query rows that share a KV head (64 / G tokens x the head's G query heads), brings each tile of 64
// positions in once and multiplies on the tensor cores (mma.sync m16n8k16, f16 in, f32 out) without giving up f32 accuracy:
//   scores   a cached K value is d (n - 8) with a 4-bit n: the integer n - 8 is exact in f16, q is split into two f16 terms
//            (scaled per row by a power of two), and each 32-dim block's integer product is multiplied by its d in f32;
//   values   d (n - 8) has 15 significant bits: two f16 terms hold it exactly; the probabilities are split the same way and
//            p_hi v_hi + p_lo v_hi + p_hi v_lo leaves out 2^-22.
// Eight warps: warp (r, h) owns rows 16 r .. +16; it scores half h of the tile's positions and gathers half h of the
// dims.  Probabilities cross between the two through shared memory; the running maximum does too.
// The context is split over blockIdx.z; (m, l, O) records go to `tmp` as the decode kernels leave them and
// sdpa_chunk_merge_kernel folds them straight into the operand image of the output projection.
//
// Bound by shared-memory reads of the operands (about 4300 cycles per 64 x 64 tile) and mma issue (about 5100 cycles at
// 1024 MAC per cycle and SM); decoding the cache is a tenth of that.
#include "ks_gemm_common.cuh"

namespace {

constexpr int CH_BM = 64, CH_BN = 64, CH_THREADS = 256;
constexpr float kNegInit = -1.0e30f;

template <int HD>
struct ChunkSmem {
  static constexpr unsigned NB = HD / 32, ROWB = NB * KS_Q40_BLOCK_BYTES, RP = ROWB + 4;
  static constexpr unsigned LD = HD + 8;            // halves per row of q, K, V: 16 bytes off a multiple of 128
  static constexpr unsigned LP = CH_BN + 8;         // halves per row of p
  static constexpr unsigned qh = 0, ql = qh + CH_BM * LD * 2, k = ql + CH_BM * LD * 2, vh = k + CH_BN * LD * 2, vl = vh + CH_BN * LD * 2,
                            ph = vl + CH_BN * LD * 2, pl = ph + CH_BM * LP * 2, dk = pl + CH_BM * LP * 2, raw = dk + NB * CH_BN * 4,
                            row = raw + 2 * CH_BN * RP,   // per row: scale, first, past the last position
                            red = row + CH_BM * 12, total = red + 4 * CH_BM * 4;
};

__device__ __forceinline__ void ldsm4(uint32_t a, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldsm4t(uint32_t a, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cp4(uint32_t dst, const void* src) { asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory"); }

// Two neighbouring Q4_0 blocks (36 bytes, nine words) -> their scales and 2 x 32 values n - 8 as half2 pairs in dim order.
struct Pair40 {
  __half d[2];
  __half2 v[2][16];
};
__device__ __forceinline__ void decode_pair(const uint32_t* w, Pair40& o) {
  uint32_t q[2][4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    q[0][i] = __funnelshift_r(w[i], w[i + 1], 16);
    q[1][i] = w[5 + i];
  }
  o.d[0] = __ushort_as_half((unsigned short)(w[0] & 0xFFFFu));
  o.d[1] = __ushort_as_half((unsigned short)(w[4] >> 16));
  const __half2 off = __float2half2_rn(1032.0f);
#pragma unroll
  for (int b = 0; b < 2; b++)
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t lo = q[b][i] & 0x0F0F0F0Fu, hi = (q[b][i] >> 4) & 0x0F0F0F0Fu;  // dims 4 i .. +3 and 16 + 4 i .. +3
      o.v[b][2 * i] = __hsub2(as_h2(__byte_perm(lo, 0, 0x4140) | 0x64006400u), off);
      o.v[b][2 * i + 1] = __hsub2(as_h2(__byte_perm(lo, 0, 0x4342) | 0x64006400u), off);
      o.v[b][8 + 2 * i] = __hsub2(as_h2(__byte_perm(hi, 0, 0x4140) | 0x64006400u), off);
      o.v[b][8 + 2 * i + 1] = __hsub2(as_h2(__byte_perm(hi, 0, 0x4342) | 0x64006400u), off);
    }
}

template <int HD>
__global__ void __launch_bounds__(CH_THREADS, 1)
sdpa_chunk_kernel(unsigned n_tok, unsigned n_q, unsigned n_kv, float scale, const float* q, const uint8_t* K, const uint8_t* V, const float* meta,
                  float* tmp, unsigned n_splits) {
  using S = ChunkSmem<HD>;
  constexpr unsigned NB = S::NB, LD = S::LD, LP = S::LP, RP = S::RP, ROWB = S::ROWB;
  constexpr int NT = HD / 16;   // 8-dim output tiles of a warp (half the head)
  extern __shared__ __align__(128) unsigned char smem[];
  ks_pdl_entry();
  const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, rg = warp >> 1, h = warp & 1u;
  const unsigned G = n_q / n_kv, kvh = blockIdx.y, split = blockIdx.z;
  const unsigned row0 = (gridDim.x - 1u - blockIdx.x) * CH_BM;  // the last rows see the most: they start first
  const uint32_t sb = sm32(smem);
  float* row_scale = reinterpret_cast<float*>(smem + S::row);
  int* row_first = reinterpret_cast<int*>(smem + S::row + CH_BM * 4);
  int* row_end = reinterpret_cast<int*>(smem + S::row + CH_BM * 8);
  float* red = reinterpret_cast<float*>(smem + S::red);
  float* dk = reinterpret_cast<float*>(smem + S::dk);

  // ---- the block's rows: row r is query head kvh G + r % G of token (row0 + r) / G; positions they see at all
  const unsigned tok_a = row0 / G, tok_b = min((row0 + CH_BM - 1u) / G, n_tok - 1u);
  const int pmin = (int)meta[tok_a * 4 + 1];                                        // starts and ends grow with the token
  const int pmax = (int)meta[tok_b * 4 + 0] + (int)meta[tok_b * 4 + 1];
  const int span = (pmax - pmin + CH_BN - 1) / CH_BN, per = (span + (int)n_splits - 1) / (int)n_splits;
  const int t_begin = pmin + (int)split * per * CH_BN, t_end = min(pmin + (int)(split + 1u) * per * CH_BN, pmax);

  auto fetch = [&](int t0) {  // the packed rows of positions t0 .. +64 (zeros past the end are masked, rows are clamped)
    for (unsigned r = warp; r < 2u * CH_BN; r += CH_THREADS / 32) {
      const unsigned p = r & (CH_BN - 1u);
      const int pos = min(t0 + (int)p, pmax - 1);
      const uint8_t* src = (r < CH_BN ? K : V) + ((size_t)pos * n_kv + kvh) * ROWB;
      const uint32_t dst = sb + S::raw + r * RP;
      for (unsigned w = lane; w < ROWB / 4u; w += 32u) cp4(dst + 4u * w, src + 4u * w);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (t_begin < t_end) fetch(t_begin);

  for (unsigned r = warp; r < CH_BM; r += CH_THREADS / 32) {
    const unsigned t = (row0 + r) / G, head = kvh * G + (row0 + r) % G;
    float v[HD / 32];
    float m = 0.0f;
#pragma unroll
    for (int j = 0; j < HD / 32; j++) {
      v[j] = t < n_tok ? q[((size_t)t * n_q + head) * HD + lane * (HD / 32) + j] : 0.0f;
      m = fmaxf(m, fabsf(v[j]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    float up;
    const float down = row_scale_down(m, &up);
    uint32_t hi[HD / 64], lo[HD / 64];
#pragma unroll
    for (int j = 0; j < HD / 64; j++) {
      const float a = v[2 * j] * down, b = v[2 * j + 1] * down;
      const __half2 hh = __floats2half2_rn(a, b);
      const float2 hf = __half22float2(hh);
      hi[j] = pack_h2(hh);
      lo[j] = pack_h2(__floats2half2_rn(a - hf.x, b - hf.y));
    }
    uint32_t* dh = reinterpret_cast<uint32_t*>(smem + S::qh + (size_t)r * LD * 2) + lane * (HD / 64);
    uint32_t* dl = reinterpret_cast<uint32_t*>(smem + S::ql + (size_t)r * LD * 2) + lane * (HD / 64);
#pragma unroll
    for (int j = 0; j < HD / 64; j++) {
      dh[j] = hi[j];
      dl[j] = lo[j];
    }
    if (lane == 0) {
      row_scale[r] = up * scale;
      row_first[r] = t < n_tok ? (int)meta[t * 4 + 1] : 0;
      row_end[r] = t < n_tok ? (int)meta[t * 4 + 1] + (int)meta[t * 4 + 0] : 0;
    }
  }

  float o[NT][4];
#pragma unroll
  for (int i = 0; i < NT; i++)
#pragma unroll
    for (int e = 0; e < 4; e++) o[i][e] = 0.0f;
  float m0 = kNegInit, m1 = kNegInit, l0 = 0.0f, l1 = 0.0f;  // rows 16 rg + g and + 8; l over this warp's half of the positions
  const unsigned gr = lane >> 2, tc = lane & 3u, ra = 16u * rg + gr, rb = ra + 8u;

  for (int t0 = t_begin; t0 < t_end; t0 += CH_BN) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();  // the raw rows are there; the previous tile's operands are used up
    {
      const unsigned p = tid & (CH_BN - 1u);
      for (unsigned pr = tid >> 6; pr < NB / 2; pr += CH_THREADS / CH_BN) {
        Pair40 d;
        const uint32_t* wk = reinterpret_cast<const uint32_t*>(smem + S::raw + (size_t)p * RP) + 9u * pr;
        uint32_t w[9];
#pragma unroll
        for (int i = 0; i < 9; i++) w[i] = wk[i];
        decode_pair(w, d);
        uint4* kd = reinterpret_cast<uint4*>(smem + S::k + (size_t)p * LD * 2 + pr * 128u);
#pragma unroll
        for (int b = 0; b < 2; b++) {
          dk[(2u * pr + b) * CH_BN + p] = __half2float(d.d[b]);
#pragma unroll
          for (int i = 0; i < 4; i++)
            kd[4 * b + i] = make_uint4(pack_h2(d.v[b][4 * i]), pack_h2(d.v[b][4 * i + 1]), pack_h2(d.v[b][4 * i + 2]), pack_h2(d.v[b][4 * i + 3]));
        }
        const uint32_t* wv = reinterpret_cast<const uint32_t*>(smem + S::raw + (size_t)(CH_BN + p) * RP) + 9u * pr;
#pragma unroll
        for (int i = 0; i < 9; i++) w[i] = wv[i];
        decode_pair(w, d);
        uint4* hd4 = reinterpret_cast<uint4*>(smem + S::vh + (size_t)p * LD * 2 + pr * 128u);
        uint4* ld4 = reinterpret_cast<uint4*>(smem + S::vl + (size_t)p * LD * 2 + pr * 128u);
#pragma unroll
        for (int b = 0; b < 2; b++) {
          const __half2 dd = __half2half2(d.d[b]);
#pragma unroll
          for (int i = 0; i < 4; i++) {
            uint32_t hh[4], ll[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
              const __half2 x = __hmul2(d.v[b][4 * i + e], dd);
              hh[e] = pack_h2(x);
              ll[e] = pack_h2(__hfma2(d.v[b][4 * i + e], dd, __hneg2(x)));
            }
            hd4[4 * b + i] = make_uint4(hh[0], hh[1], hh[2], hh[3]);
            ld4[4 * b + i] = make_uint4(ll[0], ll[1], ll[2], ll[3]);
          }
        }
      }
    }
    __syncthreads();
    if (t0 + CH_BN < t_end) fetch(t0 + CH_BN);  // flies while this tile is multiplied

    // ---- scores of rows 16 rg .. +16 and positions 32 h .. +32 of the tile
    float s[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int e = 0; e < 4; e++) s[i][e] = 0.0f;
    const uint32_t qa = sb + ((16u * rg + (lane & 15u)) * LD + (lane >> 4) * 8u) * 2u;
    const uint32_t ka = sb + S::k + ((32u * h + (lane & 7u)) * LD + (lane >> 3) * 8u) * 2u;
#pragma unroll 2
    for (unsigned b = 0; b < NB; b++) {
      uint32_t ah0[4], ah1[4], al0[4], al1[4], kb[4][4];
      ldsm4(qa + S::qh + b * 64u, ah0);
      ldsm4(qa + S::qh + b * 64u + 32u, ah1);
      ldsm4(qa + S::ql + b * 64u, al0);
      ldsm4(qa + S::ql + b * 64u + 32u, al1);
#pragma unroll
      for (int i = 0; i < 4; i++) ldsm4(ka + (unsigned)i * 8u * LD * 2u + b * 64u, kb[i]);
      float c[4][4];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) c[i][e] = 0.0f;
#pragma unroll
      for (int i = 0; i < 4; i++) mma16816(c[i], ah0, kb[i][0], kb[i][1]);
#pragma unroll
      for (int i = 0; i < 4; i++) mma16816(c[i], ah1, kb[i][2], kb[i][3]);
#pragma unroll
      for (int i = 0; i < 4; i++) mma16816(c[i], al0, kb[i][0], kb[i][1]);
#pragma unroll
      for (int i = 0; i < 4; i++) mma16816(c[i], al1, kb[i][2], kb[i][3]);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const float2 d = *reinterpret_cast<const float2*>(dk + b * CH_BN + 32u * h + 8u * i + 2u * tc);
        s[i][0] = fmaf(c[i][0], d.x, s[i][0]);
        s[i][1] = fmaf(c[i][1], d.y, s[i][1]);
        s[i][2] = fmaf(c[i][2], d.x, s[i][2]);
        s[i][3] = fmaf(c[i][3], d.y, s[i][3]);
      }
    }
    const float sa = row_scale[ra], sbk = row_scale[rb];
    const int fa = row_first[ra], ea = row_end[ra], fb = row_first[rb], eb = row_end[rb];
    float xa = kNegInit, xb = kNegInit;
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int pos = t0 + (int)(32u * h + 8u * i + 2u * tc) + e;
        s[i][e] = pos >= fa && pos < ea ? s[i][e] * sa : -INFINITY;
        s[i][2 + e] = pos >= fb && pos < eb ? s[i][2 + e] * sbk : -INFINITY;
        xa = fmaxf(xa, s[i][e]);
        xb = fmaxf(xb, s[i][2 + e]);
      }
#pragma unroll
    for (int off = 1; off <= 2; off <<= 1) {
      xa = fmaxf(xa, __shfl_xor_sync(0xffffffffu, xa, off));
      xb = fmaxf(xb, __shfl_xor_sync(0xffffffffu, xb, off));
    }
    if (tc == 0) {
      red[h * CH_BM + ra] = xa;
      red[h * CH_BM + rb] = xb;
    }
    __syncthreads();
    const float na = fmaxf(m0, fmaxf(red[ra], red[CH_BM + ra])), nb = fmaxf(m1, fmaxf(red[rb], red[CH_BM + rb]));
    const float alpha_a = __expf(m0 - na), alpha_b = __expf(m1 - nb);
    m0 = na;
    m1 = nb;
    float suma = 0.0f, sumb = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      // a masked score is -infinity: its probability is 0 whatever the maximum
      const float p0 = __expf(s[i][0] - na), p1 = __expf(s[i][1] - na), p2 = __expf(s[i][2] - nb), p3 = __expf(s[i][3] - nb);
      suma += p0 + p1;
      sumb += p2 + p3;
      // 2^8 keeps the low terms of small probabilities out of the denormals; taken off with the sum
      const __half2 ha = __floats2half2_rn(p0 * 256.0f, p1 * 256.0f), hb = __floats2half2_rn(p2 * 256.0f, p3 * 256.0f);
      const float2 fa2 = __half22float2(ha), fb2 = __half22float2(hb);
      const unsigned col = 32u * h + 8u * i + 2u * tc;
      *reinterpret_cast<uint32_t*>(smem + S::ph + (ra * LP + col) * 2u) = pack_h2(ha);
      *reinterpret_cast<uint32_t*>(smem + S::ph + (rb * LP + col) * 2u) = pack_h2(hb);
      *reinterpret_cast<uint32_t*>(smem + S::pl + (ra * LP + col) * 2u) = pack_h2(__floats2half2_rn(p0 * 256.0f - fa2.x, p1 * 256.0f - fa2.y));
      *reinterpret_cast<uint32_t*>(smem + S::pl + (rb * LP + col) * 2u) = pack_h2(__floats2half2_rn(p2 * 256.0f - fb2.x, p3 * 256.0f - fb2.y));
    }
    l0 = l0 * alpha_a + suma;
    l1 = l1 * alpha_b + sumb;
#pragma unroll
    for (int i = 0; i < NT; i++) {
      o[i][0] *= alpha_a;
      o[i][1] *= alpha_a;
      o[i][2] *= alpha_b;
      o[i][3] *= alpha_b;
    }
    __syncthreads();
    // ---- values: all 64 positions, dims of half h
    const uint32_t pa = sb + ((16u * rg + (lane & 15u)) * LP + (lane >> 4) * 8u) * 2u;
    const uint32_t va = sb + (((lane & 15u)) * LD + h * (HD / 2) + (lane >> 4) * 8u) * 2u;
#pragma unroll 1
    for (unsigned ks = 0; ks < CH_BN / 16; ks++) {
      uint32_t ph[4], pl[4];
      ldsm4(pa + S::ph + ks * 32u, ph);
      ldsm4(pa + S::pl + ks * 32u, pl);
#pragma unroll
      for (int i = 0; i < NT; i += 2) {
        uint32_t vh[4], vl[4];
        ldsm4t(va + S::vh + (ks * 16u * LD + 8u * i) * 2u, vh);
        ldsm4t(va + S::vl + (ks * 16u * LD + 8u * i) * 2u, vl);
        mma16816(o[i], ph, vh[0], vh[1]);
        mma16816(o[i + 1], ph, vh[2], vh[3]);
        mma16816(o[i], pl, vh[0], vh[1]);
        mma16816(o[i + 1], pl, vh[2], vh[3]);
        mma16816(o[i], ph, vl[0], vl[1]);
        mma16816(o[i + 1], ph, vl[2], vl[3]);
      }
    }
  }
  // ---- records: l of the two halves together, O of this warp's dims
#pragma unroll
  for (int off = 1; off <= 2; off <<= 1) {
    l0 += __shfl_xor_sync(0xffffffffu, l0, off);
    l1 += __shfl_xor_sync(0xffffffffu, l1, off);
  }
  __syncthreads();
  if (tc == 0) {
    red[(2u + h) * CH_BM + ra] = l0;
    red[(2u + h) * CH_BM + rb] = l1;
  }
  __syncthreads();
#pragma unroll
  for (int half = 0; half < 2; half++) {
    const unsigned r = half ? rb : ra, t = (row0 + r) / G, head = kvh * G + (row0 + r) % G;
    if (t >= n_tok) continue;
    float* rec = tmp + (((size_t)t * n_q + head) * n_splits + split) * (HD + 2);
    if (h == 0 && tc == 0) {
      rec[0] = half ? m1 : m0;
      rec[1] = red[2u * CH_BM + r] + red[3u * CH_BM + r];
    }
#pragma unroll
    for (int i = 0; i < NT; i++)
      *reinterpret_cast<float2*>(rec + 2 + h * (HD / 2) + 8 * i + 2 * tc) =
          make_float2(o[i][2 * half] * (1.0f / 256.0f), o[i][2 * half + 1] * (1.0f / 256.0f));
  }
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
int launch_chunk(ks_ctx* ctx, dim3 grid, unsigned n_tok, unsigned n_q, unsigned n_kv, float scale, const float* q, const uint8_t* K, const uint8_t* V,
                 const float* meta, float* tmp, unsigned n_splits) {
  constexpr size_t smem = ChunkSmem<HD>::total;
  static bool set[16] = {false};
  if (!set[ctx->device & 15]) {
    cudaError_t e = cudaFuncSetAttribute(sdpa_chunk_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return ks_fail(ctx, KS_ERR_CUDA, "sdpa_chunk: cannot set %zu B shared memory: %s", smem, cudaGetErrorString(e));
    set[ctx->device & 15] = true;
  }
  KS_LAUNCH(ctx, sdpa_chunk_kernel<HD>, grid, CH_THREADS, smem, n_tok, n_q, n_kv, scale, q, K, V, meta, tmp, n_splits);
  return ks_after_launch(ctx, "sdpa_chunk");
}
}  // namespace

// Context splits of a chunk: enough blocks for every SM, at least two tiles each.  `ctx_len` may exceed what the rows see.
int ks_sdpa_chunk_splits(const ks_ctx* ctx, int n_tok, size_t n_q, size_t n_kv, size_t ctx_len, int most) {
  const size_t blocks = ((size_t)n_tok * (n_q / n_kv) + CH_BM - 1) / CH_BM * n_kv;
  size_t s = ((size_t)ctx->sm_count + blocks - 1) / blocks;
  if (s > 1 && s * blocks > (size_t)ctx->sm_count + (size_t)ctx->sm_count / 8) s--;  // a nearly empty second wave costs more than fewer splits
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

// Rows of one slot: q [n_tok, n_q hd] f32, meta [n_tok][4] = (tlen, start, -, -) with both ends growing along the rows
// -> records in tmp [n_tok][n_q][n_splits][hd + 2].
int ks_launch_sdpa_chunk(ks_ctx* ctx, int n_tok, size_t n_q, size_t n_kv, size_t hd, float scale, const float* q, const uint8_t* K, const uint8_t* V,
                         const float* meta, float* tmp, int n_splits) {
  const dim3 grid((unsigned)(((size_t)n_tok * (n_q / n_kv) + CH_BM - 1) / CH_BM), (unsigned)n_kv, (unsigned)n_splits);
  return hd == 256 ? launch_chunk<256>(ctx, grid, (unsigned)n_tok, (unsigned)n_q, (unsigned)n_kv, scale, q, K, V, meta, tmp, (unsigned)n_splits)
                   : launch_chunk<128>(ctx, grid, (unsigned)n_tok, (unsigned)n_q, (unsigned)n_kv, scale, q, K, V, meta, tmp, (unsigned)n_splits);
}

// Records of n_tok rows -> the Q4_K form of the operand image (rows past n_tok as zeros).
int ks_launch_sdpa_merge_split(ks_ctx* ctx, int n_tok, ks_gemm_blocks b, size_t n_q, size_t hd, const float* tmp, int n_splits, void* xt) {
  const unsigned chunks = (unsigned)(n_q * hd / 8), threads = chunks < 512u ? (chunks + 31u) / 32u * 32u : 512u;
  KS_LAUNCH(ctx, sdpa_merge_split_kernel, b.np, threads, (size_t)n_q * n_splits * sizeof(float), (unsigned)n_tok, b.np, b.tbn, (unsigned)n_q, (unsigned)hd, tmp, (unsigned)n_splits, (__half*)xt);
  return ks_after_launch(ctx, "sdpa_merge_split");
}
