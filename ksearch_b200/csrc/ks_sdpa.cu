// Decode attention (one query token per slot) over a Q4_0 KV cache, split over
// the context.
//
// Stands in for the reference's two attention lowerings,
//   crates/ksearch_codegen/src/lower.rs:4897-5359  single-pass online softmax (short contexts)
//   crates/ksearch_codegen/src/lower.rs:5367-6088  16-partition pass + LSE merge (tlen >= 128)
// dispatched by Eng::sdpa_hybrid_kv (crates/ksearch_kernels/src/lib.rs:1157-1178).
//
// Layout.  K and V: [max_t, n_kv, hd] in Q4_0 (18-byte blocks of 32 values), per
// slot.  Splits are merged through `tmp` with the reference's (m, l, O[hd])
// record layout, stride hd+2, m initialised to -1e30.  Two kernels leave such
// records: sdpa_mma_kernel (tensor cores; caches that start on 4 bytes, further
// below) and, for the others, sdpa_part_kernel: one block per (split, kv head,
// slot), its warps take the positions of the split round-robin.  A warp serves
// up to four query heads of the KV head's group from one read of the K/V row:
// lane L owns the dims that live in bytes [ (L % LPB)*BPL, +BPL ) of Q4_0 block
// L / LPB (low nibbles = dims i, high nibbles = dims i+16), so a row is read
// once, 2 bytes at a time, and is never dequantised to memory.
#include <cstdlib>

#include "ks_internal.h"

namespace {

template <typename T>
__device__ __forceinline__ float ld_act(const T* p, size_t i);
template <>
__device__ __forceinline__ float ld_act<float>(const float* p, size_t i) { return p[i]; }
template <>
__device__ __forceinline__ float ld_act<__half>(const __half* p, size_t i) { return __half2float(p[i]); }
template <typename T>
__device__ __forceinline__ void st_act(T* p, size_t i, float v);
template <>
__device__ __forceinline__ void st_act<float>(float* p, size_t i, float v) { p[i] = v; }
template <>
__device__ __forceinline__ void st_act<__half>(__half* p, size_t i, float v) { p[i] = __float2half_rn(v); }

constexpr int kWarps = 4;
constexpr float kNegInit = -1.0e30f;

// This lane's DPL values of one Q4_0 row, dims (low nibbles) then dims + 16 (high nibbles), as plain nibbles (0..15 as floats),
// and the block's scale: the -8 offset and the scale are applied once per (row, head) by the caller.
template <int DPL>
__device__ __forceinline__ float load_row_raw(const uint8_t* row, int lane, float (&out)[DPL]) {
  constexpr int BPL = DPL / 2;
  constexpr int LPB = 16 / BPL;
  const uint8_t* blk = row + (lane / LPB) * KS_Q40_BLOCK_BYTES;
  const float d = __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short*>(blk)));
  const unsigned short* qs = reinterpret_cast<const unsigned short*>(blk + 2 + (lane % LPB) * BPL);
#pragma unroll
  for (int w = 0; w < BPL / 2; w++) {
    const unsigned v = qs[w];
    out[2 * w] = (float)(v & 0xF);
    out[2 * w + 1] = (float)((v >> 8) & 0xF);
    out[BPL + 2 * w] = (float)((v >> 4) & 0xF);
    out[BPL + 2 * w + 1] = (float)(v >> 12);
  }
  return d;
}
// Sum over the warp of G values per lane; every lane gets all G sums.  G == 4: the lanes first trade halves
// (each keeps two, then one, of the four values), so 10 shuffles do what 20 would.
template <int G>
__device__ __forceinline__ void warp_sum_g(float (&s)[G], int lane) {
  if (G == 4) {
    const bool hi = (lane & 16) != 0, h8 = (lane & 8) != 0;
    float k0 = hi ? s[2] : s[0], k1 = hi ? s[3] : s[1];
    const float t0 = hi ? s[0] : s[2], t1 = hi ? s[1] : s[3];
    k0 += __shfl_xor_sync(0xffffffffu, t0, 16);
    k1 += __shfl_xor_sync(0xffffffffu, t1, 16);
    float k = h8 ? k1 : k0;
    const float t = h8 ? k0 : k1;
    k += __shfl_xor_sync(0xffffffffu, t, 8);
    k += __shfl_xor_sync(0xffffffffu, k, 4);
    k += __shfl_xor_sync(0xffffffffu, k, 2);
    k += __shfl_xor_sync(0xffffffffu, k, 1);
#pragma unroll
    for (int g = 0; g < G; g++) s[g] = __shfl_sync(0xffffffffu, k, 8 * (g & 1) + 16 * (g >> 1));
  } else {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
      for (int g = 0; g < G; g++) s[g] += __shfl_xor_sync(0xffffffffu, s[g], off);
  }
}
// Dimension index (within the head) of this lane's j-th value.
template <int DPL>
__device__ __forceinline__ int lane_dim(int lane, int j) {
  constexpr int BPL = DPL / 2;
  constexpr int LPB = 16 / BPL;
  const int base = (lane / LPB) * 32 + (lane % LPB) * BPL;
  return j < BPL ? base + j : base + 16 + (j - BPL);
}

constexpr int kRing = 8;  // rows of one warp in flight (K and V each)

__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

// ASYNC: the rows of a warp travel through a ring of kRing shared-memory buffers filled by cp.async (8 bytes per
// lane), so kRing rows of K and V are in flight per warp while one is being multiplied; without it a warp waited
// out one full memory round trip per row.  Needs 8-byte aligned rows; the plain path takes the rest.
// G: query heads served by one block (at most 4: more would not leave registers for enough warps per SM); a KV head
// with a larger group is served by hpk / G blocks (blockIdx.y = kvh * (hpk / G) + group), each reading the rows itself.
template <int G, int DPL, typename T, bool ASYNC>
__global__ void __launch_bounds__(kWarps * 32)
sdpa_part_kernel(unsigned n_q, unsigned n_kv, float scale, const T* q, const uint8_t* K, const uint8_t* V,
                 size_t slot_stride, const float* meta, float* tmp, T* out, int n_splits) {
  ks_pdl_entry();
  constexpr int HD = DPL * 32;
  constexpr unsigned ROWB = (HD / 32) * KS_Q40_BLOCK_BYTES;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned hpk = n_q / n_kv, gpk = hpk / G;  // heads and blocks per KV head
  const int split = blockIdx.x, kvh = blockIdx.y / gpk, slot = blockIdx.z;
  const unsigned head0 = (unsigned)kvh * hpk + (blockIdx.y % gpk) * G;  // first query head of this block
  const unsigned tlen = (unsigned)meta[slot * 4 + 0];
  const unsigned start = (unsigned)meta[slot * 4 + 1];
  const unsigned chunk = (tlen + n_splits - 1) / n_splits;
  const unsigned p0 = split * chunk;
  const unsigned p1 = min(p0 + chunk, tlen);
  const size_t rowb = ROWB;
  const uint8_t* Ks = K + (size_t)slot * slot_stride;
  const uint8_t* Vs = V + (size_t)slot * slot_stride;
  __shared__ __align__(16) uint8_t ring[ASYNC ? kWarps * kRing * 2 * ROWB : 16];

  // qs8[g] = 8 * (sum of this lane's q values): the -8 of Q4_0 leaves the dot product as one term per (row, head);
  // c[g] gathers sum(e * d) the same way for V, and is taken off o at the end
  float qr[G][DPL], o[G][DPL], m[G], l[G], qs8[G], c[G];
#pragma unroll
  for (int g = 0; g < G; g++) {
    const size_t qb = ((size_t)slot * n_q + head0 + g) * HD;
    float sum = 0.0f;
#pragma unroll
    for (int j = 0; j < DPL; j++) {
      qr[g][j] = ld_act<T>(q, qb + lane_dim<DPL>(lane, j)) * scale;
      sum += qr[g][j];
      o[g][j] = 0.0f;
    }
    qs8[g] = 8.0f * sum;
    c[g] = 0.0f;
    m[g] = kNegInit;
    l[g] = 0.0f;
  }

  // one position: scores of the G heads against the K row, then the online-softmax update with the V row
  auto step = [&](const uint8_t* krow, const uint8_t* vrow) {
    float kv[DPL];
    const float dk = load_row_raw<DPL>(krow, lane, kv);
    float s[G];
#pragma unroll
    for (int g = 0; g < G; g++) {
      float a = -qs8[g];
#pragma unroll
      for (int j = 0; j < DPL; j++) a = fmaf(qr[g][j], kv[j], a);
      s[g] = a * dk;
    }
    warp_sum_g<G>(s, lane);
    const float dv = load_row_raw<DPL>(vrow, lane, kv);
#pragma unroll
    for (int g = 0; g < G; g++) {
      if (s[g] > m[g]) {  // a new maximum (the same in every lane): rescale what was gathered so far
        const float alpha = __expf(m[g] - s[g]);
        l[g] *= alpha;
        c[g] *= alpha;
#pragma unroll
        for (int j = 0; j < DPL; j++) o[g][j] *= alpha;
        m[g] = s[g];
      }
      const float e = __expf(s[g] - m[g]);
      l[g] += e;
      const float ed = e * dv;
      c[g] += ed;
#pragma unroll
      for (int j = 0; j < DPL; j++) o[g][j] = fmaf(ed, kv[j], o[g][j]);
    }
  };

  if (ASYNC) {
    uint8_t* my = ring + (size_t)warp * (kRing * 2 * ROWB);
    const uint32_t my_s = (uint32_t)__cvta_generic_to_shared(my);
    auto fetch = [&](unsigned n) {  // the warp's n-th position into buffer n % kRing (an empty group past the end)
      const unsigned t = p0 + (unsigned)warp + n * kWarps;
      if (t < p1 && lane < (int)(ROWB / 8u)) {
        const size_t row = ((size_t)(start + t) * n_kv + kvh) * rowb + (size_t)lane * 8u;
        const uint32_t dst = my_s + (n % kRing) * (2u * ROWB) + (uint32_t)lane * 8u;
        cp_async8(dst, Ks + row);
        cp_async8(dst + ROWB, Vs + row);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll 1
    for (unsigned n = 0; n < (unsigned)kRing; n++) fetch(n);
    unsigned n = 0;
#pragma unroll 1
    for (unsigned t = p0 + warp; t < p1; t += kWarps, n++) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 1) : "memory");
      __syncwarp();
      const uint8_t* buf = my + (size_t)(n % kRing) * (2u * ROWB);
      step(buf, buf + ROWB);
      __syncwarp();  // every lane is done with the buffer before it is refilled
      fetch(n + kRing);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    for (unsigned t = p0 + warp; t < p1; t += kWarps) {
      const size_t row = ((size_t)(start + t) * n_kv + kvh) * rowb;
      step(Ks + row, Vs + row);
    }
  }

#pragma unroll
  for (int g = 0; g < G; g++)
#pragma unroll
    for (int j = 0; j < DPL; j++) o[g][j] = fmaf(-8.0f, c[g], o[g][j]);

  // merge the warps of this block: warp w leaves (m, l, O) in shared memory, warp 0 folds them in order
  __shared__ float sm_ml[kWarps][G][2];
  __shared__ float sm_o[kWarps][G][HD];
  if (warp > 0) {
#pragma unroll
    for (int g = 0; g < G; g++) {
      if (lane == 0) {
        sm_ml[warp][g][0] = m[g];
        sm_ml[warp][g][1] = l[g];
      }
#pragma unroll
      for (int j = 0; j < DPL; j++) sm_o[warp][g][j * 32 + lane] = o[g][j];
    }
  }
  __syncthreads();
  if (warp != 0) return;
#pragma unroll
  for (int g = 0; g < G; g++) {
    for (int w = 1; w < kWarps; w++) {
      const float mp = sm_ml[w][g][0], lp = sm_ml[w][g][1];
      const float m2 = fmaxf(m[g], mp);
      const float alpha = __expf(m[g] - m2), beta = __expf(mp - m2);
      l[g] = l[g] * alpha + lp * beta;
      m[g] = m2;
#pragma unroll
      for (int j = 0; j < DPL; j++) o[g][j] = o[g][j] * alpha + sm_o[w][g][j * 32 + lane] * beta;
    }
    const unsigned head = head0 + g;
    if (n_splits == 1) {
      const float inv_l = 1.0f / l[g];
      const size_t ob = ((size_t)slot * n_q + head) * HD;
#pragma unroll
      for (int j = 0; j < DPL; j++) st_act<T>(out, ob + lane_dim<DPL>(lane, j), o[g][j] * inv_l);
    } else {
      float* rec = tmp + (((size_t)slot * n_q + head) * n_splits + split) * (HD + 2);
      if (lane == 0) {
        rec[0] = m[g];
        rec[1] = l[g];
      }
#pragma unroll
      for (int j = 0; j < DPL; j++) rec[2 + lane_dim<DPL>(lane, j)] = o[g][j];
    }
  }
}

// Slots of unequal contexts share their launch's splits by length: every slot gets as many chunks of one size as its context has, or the
// launch lasts as long as a share of its longest context (four slots of 1024, 4096, 16384 and 16384 positions in 32 splits each: 24.2
// us, dealt 20.9; with 4 KV heads 39.0 and 28.7; eight of 50, 100, .. 6400 with one 18.6 and 13.2).  Contexts that are short for the splits
// (chunks of 128 positions) or average four fifths of the longest keep the plain layout; finding that out costs up to half a microsecond in
// each of the two launches (eight of 8192 24.4 and 25.4, eight of 300 11.0 and 11.8, four of 16384 24.6 and 24.7).  Chunk u of the launch leaves
// its record at place u, one head behind the other.  Steps of a model pass no max_t and keep the plain layout, the only one that the merge
// into an operand image knows.  A whole warp calls; lane s speaks for slot s.
constexpr unsigned kDealSlots = 32;
constexpr unsigned kMinChunk = 128;  // positions of a split at least: a tile of 16 per warp
struct Deal {
  unsigned chunk, count;  // positions of a chunk (0: not dealt); this lane's slot: how many
};
// tlen: of this lane's slot, 0 beyond the last
__device__ __forceinline__ Deal deal_splits(unsigned tlen, unsigned n_slots, unsigned n_splits) {
  const unsigned lane = threadIdx.x & 31u, most = n_slots * n_splits;
  const unsigned sum = __reduce_add_sync(0xffffffffu, tlen), top = __reduce_max_sync(0xffffffffu, tlen);
  Deal d{0u, 0u};
  if (top <= kMinChunk * n_splits || (unsigned long long)top * n_slots * 4u <= (unsigned long long)sum * 5u) return d;
  // the size that fills the launch if every context divides by it, else one with a chunk to spare for every slot: that always fits
  // (reciprocals, and a step either way: four divisions one behind the other took longer than the rest)
#pragma unroll
  for (int again = 0; again < 2; again++) {
    d.chunk = max(kMinChunk, ((unsigned)__fdividef((float)sum, (float)(again ? most - n_slots : most)) + 16u) & ~15u);
    d.count = (unsigned)__fdividef((float)tlen, (float)d.chunk);
    d.count += d.count * d.chunk < tlen;
    d.count -= d.count > 0u && (d.count - 1u) * d.chunk >= tlen;
    d.count = lane < n_slots ? max(1u, d.count) : 0u;
    if (__reduce_add_sync(0xffffffffu, d.count) <= most) break;
  }
  return d;
}

// Merge the per-split records of one (slot, head): lower.rs:5897-6088.  A block takes 64 dims; four threads share a dim's splits
// (p = part, part + 4, ...) and their sums meet in a fixed order.  The O values are requested before the (m, l) pairs are looked
// at, so the two trips to memory are one.  Bound by that trip and the launch.
constexpr int kRedDims = 64, kRedParts = 4, kRedFly = 8;
// DEAL: the launch's splits may have been dealt among gridDim.x / n_q slots.
template <typename T, bool DEAL>
__global__ void __launch_bounds__(kRedDims * kRedParts) sdpa_reduce_kernel(unsigned hd, const float* tmp, T* out, int n_splits, unsigned n_q, const float* meta) {
  ks_pdl_entry();
  __shared__ float fac[KS_SDPA_MAX_SPLITS];
  __shared__ float part_sum[kRedDims * kRedParts];
  const size_t sh = blockIdx.x;  // slot * n_q + head
  const float* rec0 = tmp + sh * n_splits * (hd + 2);
  size_t stride = hd + 2;
  const int part = threadIdx.x / kRedDims, lane = threadIdx.x & 31;
  const unsigned d = blockIdx.y * kRedDims + threadIdx.x % kRedDims;
  float v[kRedFly];
  auto request = [&](int p0) {
#pragma unroll
    for (int k = 0; k < kRedFly; k++) {
      const int p = p0 + k * kRedParts;
      v[k] = p < n_splits ? rec0[p * stride + 2 + d] : 0.0f;
    }
  };
  request(part);
  if constexpr (DEAL) {  // what was asked for above is right unless the splits were dealt
    const unsigned n_slots = gridDim.x / n_q, slot = blockIdx.x / n_q;
    const Deal g = deal_splits((unsigned)lane < n_slots ? (unsigned)meta[lane * 4] : 0u, n_slots, (unsigned)n_splits);
    if (g.chunk) {
      rec0 = tmp + ((size_t)__reduce_add_sync(0xffffffffu, (unsigned)lane < slot ? g.count : 0u) * n_q + blockIdx.x % n_q) * (hd + 2);
      n_splits = (int)__shfl_sync(0xffffffffu, g.count, slot);
      stride *= n_q;
      request(part);
    }
  }
  if (threadIdx.x < 32) {  // exp(m - M) / L of every split; an empty one (l = 0) has no O and counts for nothing
    float m[KS_SDPA_MAX_SPLITS / 32], l[KS_SDPA_MAX_SPLITS / 32], M = kNegInit, L = 0.0f;
#pragma unroll
    for (int k = 0; k < KS_SDPA_MAX_SPLITS / 32; k++) {
      const int p = lane + 32 * k;
      m[k] = p < n_splits ? rec0[p * stride] : kNegInit;
      l[k] = p < n_splits ? rec0[p * stride + 1] : 0.0f;
      M = fmaxf(M, m[k]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
#pragma unroll
    for (int k = 0; k < KS_SDPA_MAX_SPLITS / 32; k++) {
      m[k] = l[k] != 0.0f ? __expf(m[k] - M) : 0.0f;
      L = fmaf(l[k], m[k], L);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
#pragma unroll
    for (int k = 0; k < KS_SDPA_MAX_SPLITS / 32; k++)
      if (lane + 32 * k < n_splits) fac[lane + 32 * k] = m[k] / L;
  }
  __syncthreads();
  float o = 0.0f;
  for (int p0 = part; p0 < n_splits; p0 += kRedFly * kRedParts) {
    if (p0 != part) request(p0);
#pragma unroll
    for (int k = 0; k < kRedFly; k++) {
      const int p = p0 + k * kRedParts;
      const float f = p < n_splits ? fac[p] : 0.0f;
      if (f != 0.0f) o = fmaf(v[k], f, o);
    }
  }
  part_sum[threadIdx.x] = o;
  __syncthreads();
  if (threadIdx.x < kRedDims) {
#pragma unroll
    for (int k = 1; k < kRedParts; k++) o += part_sum[k * kRedDims + threadIdx.x];
    st_act<T>(out, sh * hd + d, o);
  }
}

// ---- the tensor-core form ------------------------------------------------------------------------------------
// One block of eight warps per (split, group of up to four query heads of a KV head, slot).  Warps take tiles of 16 positions
// round-robin and never wait for one another before the end; a warp's next tile is on its way (cp.async) meanwhile.  Per tile:
//   scores   mma m16n8k16 with positions as rows and heads as columns.  A cached value is d (n - 8): the integers n - 8 come out
//            of the packed words by one LOP3 and one HADD2 / HFMA2 per two values, in the order the words hold them (the dims of
//            a k step are permuted alike in q); each query is split into two f16 terms, columns 0..3 and 4..7, so one
//            instruction takes both; the integer product of a 32-dim block is multiplied by its d in f32.  q is scaled by a
//            power of two per head, so nothing leaves the f16 range;
//   values   dims as rows, positions as k, and p d(position, block) as columns, again as two f16 terms.  2^k brings the largest
//            p d of the warp so far below 2^15; a tile with a larger d lowers k and rescales like a new maximum does.
// What is dropped is below 2^-21 of the largest product.  No shuffle per position: six per tile for the running maximum.
// About 700 warp instructions per 16 positions and four heads; the kernel this replaced (positions across threads, f32 FMAs)
// took about 2900.  Bound by latency: a few tiles per warp, then two dependent launches.
constexpr int kMmaWarps = 8;
constexpr int kMmaTile = 16;
constexpr int kMmaRing = 2;
static_assert(kMinChunk == kMmaWarps * kMmaTile, "one tile per warp");

template <int HD>
struct MmaSmem {
  static constexpr unsigned NB = HD / 32, ROWB = NB * KS_Q40_BLOCK_BYTES, TILE = 2 * kMmaTile * ROWB;
  static constexpr unsigned q_off = 0, p_off = q_off + NB * 32 * 16, st_off = p_off + kMmaWarps * kMmaTile * 16,
                            ring_off = (st_off + kMmaWarps * 4 * 8 + 32 + 127) & ~127u;
  static constexpr unsigned ring = kMmaWarps * kMmaRing * TILE, merge = kMmaWarps * 4 * HD * 4;
  static constexpr unsigned total = ring_off + (ring > merge ? ring : merge);
};
__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 bits_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ uint32_t low_nibbles(uint32_t w) {   // nibbles 0 of bytes 0 and 2 -> n - 8
  return h2_bits(__hadd2(bits_h2((w & 0x000F000Fu) | 0x64006400u), __float2half2_rn(-1032.0f)));
}
__device__ __forceinline__ uint32_t high_nibbles(uint32_t w) {  // nibbles 1 of bytes 0 and 2 (1024 + 16 n) -> n - 8
  return h2_bits(__hfma2(bits_h2((w & 0x00F000F0u) | 0x64006400u), __float2half2_rn(0.0625f), __float2half2_rn(-72.0f)));
}
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ float half_at(const unsigned char* p) { return __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short*>(p))); }

// CH: bytes per copy of a cached row: 16 (8 for rows of 72 bytes) where the cache is aligned for it, else 4.
// DEAL: splits go to the slots by the lengths of their contexts where those are unequal enough.
template <int HD, typename T, unsigned CH, bool DEAL>
__global__ void __launch_bounds__(kMmaWarps * 32, 2)
sdpa_mma_kernel(unsigned n_q, unsigned n_kv, unsigned gb, float scale, const T* q, const uint8_t* K, const uint8_t* V, size_t slot_stride,
                const float* meta, float* tmp, T* out, int n_splits) {
  ks_pdl_entry();
  using S = MmaSmem<HD>;
  constexpr unsigned NB = S::NB, ROWB = S::ROWB;
  extern __shared__ __align__(128) unsigned char smem[];
  const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, g = lane >> 2, t = lane & 3u;
  const unsigned hpk = n_q / n_kv, gpk = hpk / gb;  // heads and blocks per KV head
  const unsigned kvh = blockIdx.y / gpk, head0 = kvh * hpk + (blockIdx.y % gpk) * gb;
  unsigned split = blockIdx.x, slot = blockIdx.z, dealt = 0;
  unsigned tlen, start;
  if constexpr (DEAL) {
    const float4 m = lane < gridDim.z ? *reinterpret_cast<const float4*>(meta + lane * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    const Deal d = deal_splits((unsigned)m.x, gridDim.z, gridDim.x);
    dealt = d.chunk;
    if (dealt) {
      unsigned end = d.count;  // of the slot's chunks
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned x = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= (unsigned)o) end += x;
      }
      const unsigned at = blockIdx.z * gridDim.x + blockIdx.x;  // of the launch's splits
      const unsigned before = __ballot_sync(0xffffffffu, end <= at);  // slots whose chunks lie in front
      slot = __popc(before);
      if (slot >= gridDim.z) return;  // more blocks than chunks: the merge looks at none beyond them
      split = at - __shfl_sync(0xffffffffu, end - d.count, slot);
    }
    tlen = (unsigned)__shfl_sync(0xffffffffu, m.x, slot);
    start = (unsigned)__shfl_sync(0xffffffffu, m.y, slot);
  } else {
    tlen = (unsigned)meta[slot * 4 + 0];
    start = (unsigned)meta[slot * 4 + 1];
  }
  // a split never holds fewer than kMinChunk positions: on a short context the later splits are empty and their
  // blocks leave after writing an empty record, so a split count sized for the longest context costs little
  const unsigned chunk = dealt ? dealt : max((tlen + n_splits - 1) / n_splits, kMinChunk);
  const unsigned p0 = split * chunk, p1 = min(p0 + chunk, tlen);
  auto record = [&](unsigned head) {
    if (DEAL && dealt) return tmp + ((size_t)(blockIdx.z * gridDim.x + blockIdx.x) * n_q + head) * (HD + 2);
    return tmp + (((size_t)slot * n_q + head) * n_splits + split) * (HD + 2);
  };
  if (p0 >= p1 && n_splits > 1) {  // nothing to do: the empty record (m = -1e30, l = 0) is all the merge needs
    if (tid < gb) {
      float* rec = record(head0 + tid);
      rec[0] = kNegInit;
      rec[1] = 0.0f;
    }
    return;
  }
  const uint8_t* Ks = K + (size_t)slot * slot_stride + ((size_t)start * n_kv + kvh) * ROWB;
  const uint8_t* Vs = V + (size_t)slot * slot_stride + ((size_t)start * n_kv + kvh) * ROWB;
  const size_t rowstride = (size_t)n_kv * ROWB;
  unsigned char* ring = smem + S::ring_off + warp * (kMmaRing * S::TILE);
  const uint32_t ring_s = (uint32_t)__cvta_generic_to_shared(ring);
  const unsigned n_tiles = p1 > p0 ? (p1 - p0 + kMmaTile - 1) / kMmaTile : 0u;

  auto fetch = [&](unsigned i, unsigned stage) {  // this warp's i-th tile (an empty group past the end; rows past the split repeat its last)
    const unsigned tile = warp + i * kMmaWarps;
    if (tile < n_tiles) {
      constexpr unsigned PER = ROWB / CH;
      const unsigned first = p0 + tile * kMmaTile, last = p1 - 1u - first;
#pragma unroll
      for (unsigned k = 0; k < (kMmaTile * PER + 31u) / 32u; k++) {
        const unsigned c = lane + 32u * k, r = c / PER, o = (c - r * PER) * CH;
        if (c >= kMmaTile * PER) break;
        const size_t src = (size_t)(first + min(r, last)) * rowstride + o;
        const uint32_t dst = ring_s + stage * S::TILE + r * ROWB + o;
        if constexpr (CH == 16u) {
          cp_async16(dst, Ks + src);
          cp_async16(dst + kMmaTile * ROWB, Vs + src);
        } else if constexpr (CH == 8u) {
          cp_async8(dst, Ks + src);
          cp_async8(dst + kMmaTile * ROWB, Vs + src);
        } else {
          cp_async4(dst, Ks + src);
          cp_async4(dst + kMmaTile * ROWB, Vs + src);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(0, 0);

  // ---- q: per head a power-of-two scale, then the B fragments of every block in the order the lanes read them.  A thread reads the
  // eight values of its fragment once; their largest meet over the lanes of a block and, through shared memory, over the blocks.  (A warp
  // per head looking for the maximum first made two trips to memory and a loop of 1.4 to 2 us: one slot of 16384 positions 15.9 -> 14.4
  // us, eight of 300 13.1 -> 11.7, the four unequal ones above 24 -> 22.)
  float* qscale = reinterpret_cast<float*>(smem + S::st_off + kMmaWarps * 4 * 8);  // [0..4) down, [4..8) up
  float* bmax = reinterpret_cast<float*>(smem + S::st_off);                        // [NB][4] (the warps' (m, l) come here later)
  static_assert(NB <= (unsigned)kMmaWarps && NB * 16u <= kMmaWarps * 4 * 8, "a warp per block, and its four largest values fit");
  {
    const unsigned n = lane >> 2, lt = lane & 3u, h = n & 3u;
    const bool in = warp < NB && h < gb;
    float x[2][4], m = 0.0f;
#pragma unroll
    for (int half = 0; half < 2; half++)
#pragma unroll
      for (int k = 0; k < 4; k++) {
        x[half][k] = in ? ld_act<T>(q, ((size_t)slot * n_q + head0 + h) * HD + 32u * warp + 4u * lt + 16u * half + k) : 0.0f;
        m = fmaxf(m, fabsf(x[half][k]));
      }
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
    if (warp < NB && lt == 0 && n < 4u) bmax[warp * 4u + h] = m;
    __syncthreads();
    m = 0.0f;
#pragma unroll
    for (unsigned b = 0; b < NB; b++) m = fmaxf(m, bmax[b * 4u + h]);
    int e = 0;
    if (m > 0.0f && m < 3.0e38f) {
      e = (int)((__float_as_uint(m) >> 23) & 0xFFu) - 127 - 14;
      e = e < -100 ? -100 : e;
    }
    const float dn = __uint_as_float((unsigned)(127 - e) << 23);
    if (warp == 0 && lt == 0 && n < 4u) {
      qscale[h] = h < gb ? dn : 0.0f;
      qscale[4 + h] = h < gb ? __uint_as_float((unsigned)(127 + e) << 23) : 0.0f;
    }
    if (warp < NB) {
      uint32_t w[4];
#pragma unroll
      for (int half = 0; half < 2; half++)
#pragma unroll
        for (int k = 0; k < 2; k++) {
          const float x0 = x[half][k] * dn, x1 = x[half][k + 2] * dn;
          const __half2 hh = __floats2half2_rn(x0, x1);
          const float2 hf = __half22float2(hh);
          w[2 * half + k] = n < 4u ? h2_bits(hh) : h2_bits(__floats2half2_rn(x0 - hf.x, x1 - hf.y));
        }
      reinterpret_cast<uint4*>(smem + S::q_off)[tid] = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
  __syncthreads();
  const uint4* qf = reinterpret_cast<const uint4*>(smem + S::q_off) + lane;
  float* pw = reinterpret_cast<float*>(smem + S::p_off) + warp * (kMmaTile * 4);
  const unsigned ha = 2u * (t & 1u);                       // this lane's two heads (columns 2t, 2t + 1 and their other halves)
  const float sa = qscale[4 + ha] * scale, sb = qscale[5 + ha] * scale;
  const bool is_lo = g >= 4u;

  float o[HD / 16][4];
#pragma unroll
  for (int i = 0; i < HD / 16; i++)
#pragma unroll
    for (int e = 0; e < 4; e++) o[i][e] = 0.0f;
  float m0 = kNegInit, m1 = kNegInit, l0 = 0.0f, l1 = 0.0f;
  int kx = 29;  // values carry 2^kx
  unsigned stage = 0;
  for (unsigned i = 0; warp + i * kMmaWarps < n_tiles; i++) {
    fetch(i + 1, stage ^ 1u);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const unsigned char* kt = ring + stage * S::TILE;
    const unsigned char* vt = kt + kMmaTile * ROWB;
    // ---- scores: rows g and g + 8 of the tile, columns 2t, 2t + 1
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    const unsigned char* ra = kt + g * ROWB;
    const unsigned char* rb = ra + 8u * ROWB;
#pragma unroll 2
    for (unsigned pr = 0; pr < NB / 2; pr++) {  // two blocks, 36 bytes: [d0 | 16 bytes][d1 | 16 bytes]; the first one's bytes straddle words
      const uint32_t* wa = reinterpret_cast<const uint32_t*>(ra + 36u * pr) + t;
      const uint32_t* wb = reinterpret_cast<const uint32_t*>(rb + 36u * pr) + t;
      const uint32_t a[2] = {__funnelshift_r(wa[0], wa[1], 16), wa[5]}, b[2] = {__funnelshift_r(wb[0], wb[1], 16), wb[5]};
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const uint4 f = qf[(2u * pr + k) * 32u];
        float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        mma16816(c, low_nibbles(a[k]), low_nibbles(b[k]), low_nibbles(a[k] >> 8), low_nibbles(b[k] >> 8), f.x, f.y);
        mma16816(c, high_nibbles(a[k]), high_nibbles(b[k]), high_nibbles(a[k] >> 8), high_nibbles(b[k] >> 8), f.z, f.w);
        const float da = half_at(ra + 36u * pr + 18u * k), db = half_at(rb + 36u * pr + 18u * k);
        s[0] = fmaf(c[0], da, s[0]);
        s[1] = fmaf(c[1], da, s[1]);
        s[2] = fmaf(c[2], db, s[2]);
        s[3] = fmaf(c[3], db, s[3]);
      }
    }
#pragma unroll
    for (int e = 0; e < 4; e++) s[e] += __shfl_xor_sync(0xffffffffu, s[e], 2);  // the two f16 terms of q
    const unsigned pos = p0 + (warp + i * kMmaWarps) * kMmaTile + g;
    s[0] = pos < p1 ? s[0] * sa : -INFINITY;
    s[1] = pos < p1 ? s[1] * sb : -INFINITY;
    s[2] = pos + 8u < p1 ? s[2] * sa : -INFINITY;
    s[3] = pos + 8u < p1 ? s[3] * sb : -INFINITY;
    float x0 = fmaxf(s[0], s[2]), x1 = fmaxf(s[1], s[3]);
#pragma unroll
    for (int off = 4; off <= 16; off <<= 1) {
      x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, off));
      x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, off));
    }
    // ---- the tile's largest |d| of V: its exponent bounds 2^kx
    unsigned dmax = 0;
    for (unsigned c = lane; c < kMmaTile * NB; c += 32u)
      dmax = max(dmax, (unsigned)*reinterpret_cast<const unsigned short*>(vt + (c / NB) * ROWB + (c % NB) * KS_Q40_BLOCK_BYTES) & 0x7FFFu);
    dmax = __reduce_max_sync(0xffffffffu, dmax);
    const int k2 = min(kx, 29 - (int)(dmax >> 10));
    const float n0 = fmaxf(m0, x0), n1 = fmaxf(m1, x1);
    const float f0 = __expf(m0 - n0), f1 = __expf(m1 - n1);
    l0 *= f0;
    l1 *= f1;
    if (__any_sync(0xffffffffu, f0 != 1.0f || f1 != 1.0f) || k2 != kx) {
      const float r = __uint_as_float((unsigned)(127 + k2 - kx) << 23), a0 = f0 * r, a1 = f1 * r;
#pragma unroll
      for (int j = 0; j < HD / 16; j++) {
        o[j][0] *= a0;
        o[j][1] *= a1;
        o[j][2] *= a0;
        o[j][3] *= a1;
      }
    }
    m0 = n0;
    m1 = n1;
    kx = k2;
    const float e0 = __expf(s[0] - m0), e1 = __expf(s[1] - m1), e2 = __expf(s[2] - m0), e3 = __expf(s[3] - m1);
    l0 += e0 + e2;
    l1 += e1 + e3;
    if (t < 2u) {
      *reinterpret_cast<float2*>(pw + g * 4u + ha) = make_float2(e0, e1);
      *reinterpret_cast<float2*>(pw + (g + 8u) * 4u + ha) = make_float2(e2, e3);
    }
    __syncwarp();
    // ---- values: k = positions 2t, 2t + 1, 2t + 8, 2t + 9; column g = head g & 3, its first or second f16 term
    const float up = __uint_as_float((unsigned)(127 + kx) << 23);
    const float* pr = pw + 2u * t * 4u + (g & 3u);
    const float p[4] = {pr[0] * up, pr[4] * up, pr[32] * up, pr[36] * up};
    const unsigned char* v0 = vt + 2u * t * ROWB;
#pragma unroll
    for (unsigned b = 0; b < NB; b++) {
      const unsigned char* vb = v0 + b * KS_Q40_BLOCK_BYTES;
      const float y0 = p[0] * half_at(vb), y1 = p[1] * half_at(vb + ROWB), y2 = p[2] * half_at(vb + 8u * ROWB), y3 = p[3] * half_at(vb + 9u * ROWB);
      __half2 h01 = __floats2half2_rn(y0, y1), h23 = __floats2half2_rn(y2, y3);
      if (is_lo) {
        const float2 q01 = __half22float2(h01), q23 = __half22float2(h23);
        h01 = __floats2half2_rn(y0 - q01.x, y1 - q01.y);
        h23 = __floats2half2_rn(y2 - q23.x, y3 - q23.y);
      }
      // bytes 2g, 2g + 1 of the block (rows g and g + 8 of the product are dims 2g, 2g + 1; 16 more for the high nibbles)
      const unsigned char* by = vb + 2u + 2u * g;
      const uint32_t w0 = __byte_perm(*reinterpret_cast<const unsigned short*>(by), *reinterpret_cast<const unsigned short*>(by + ROWB), 0x5410);
      const uint32_t w8 = __byte_perm(*reinterpret_cast<const unsigned short*>(by + 8u * ROWB), *reinterpret_cast<const unsigned short*>(by + 9u * ROWB), 0x5410);
      mma16816(o[2 * b], low_nibbles(w0), low_nibbles(w0 >> 8), low_nibbles(w8), low_nibbles(w8 >> 8), h2_bits(h01), h2_bits(h23));
      mma16816(o[2 * b + 1], high_nibbles(w0), high_nibbles(w0 >> 8), high_nibbles(w8), high_nibbles(w8 >> 8), h2_bits(h01), h2_bits(h23));
    }
    __syncwarp();  // every lane is done with the stage and the probabilities
    stage ^= 1u;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
  for (int off = 4; off <= 16; off <<= 1) {
    l0 += __shfl_xor_sync(0xffffffffu, l0, off);
    l1 += __shfl_xor_sync(0xffffffffu, l1, off);
  }
  // ---- the warps' (m, l, O) meet in shared memory (the rings are free), threads fold one dim each in warp order
  __syncthreads();
  float* ml = reinterpret_cast<float*>(smem + S::st_off);           // [warp][head](m, l)
  float* mo = reinterpret_cast<float*>(smem + S::ring_off);         // [warp][head][HD]
  const float down = __uint_as_float((unsigned)(127 - kx) << 23);
#pragma unroll
  for (int j = 0; j < HD / 16; j++) {
#pragma unroll
    for (int e = 0; e < 4; e++) o[j][e] = (o[j][e] + __shfl_xor_sync(0xffffffffu, o[j][e], 2)) * down;
    if (t < 2u) {
      const unsigned d = 32u * (j >> 1) + 16u * (j & 1) + 2u * g;
      *reinterpret_cast<float2*>(mo + (warp * 4u + ha) * HD + d) = make_float2(o[j][0], o[j][2]);
      *reinterpret_cast<float2*>(mo + (warp * 4u + ha + 1u) * HD + d) = make_float2(o[j][1], o[j][3]);
    }
  }
  if (g == 0 && t < 2u) {
    ml[(warp * 4u + ha) * 2u] = m0;
    ml[(warp * 4u + ha) * 2u + 1u] = l0;
    ml[(warp * 4u + ha + 1u) * 2u] = m1;
    ml[(warp * 4u + ha + 1u) * 2u + 1u] = l1;
  }
  __syncthreads();
  float* fac = reinterpret_cast<float*>(smem + S::p_off);  // [warp][head] exp(m - M); behind them per head (M, L)
  if (warp == 0) {  // lane = (warp w, head h)
    const unsigned w = lane >> 2, h = lane & 3u;
    const float m = ml[(w * 4u + h) * 2u], l = ml[(w * 4u + h) * 2u + 1u];
    float M = m;
#pragma unroll
    for (int off = 4; off <= 16; off <<= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
    const float f = __expf(m - M);
    float L = l * f;
#pragma unroll
    for (int off = 4; off <= 16; off <<= 1) L += __shfl_xor_sync(0xffffffffu, L, off);
    fac[lane] = f;
    if (w == 0) {
      fac[32u + h] = M;
      fac[36u + h] = L;
    }
  }
  __syncthreads();
  for (unsigned i = tid; i < gb * HD; i += kMmaWarps * 32) {
    const unsigned h = i / HD, d = i - h * HD;
    float a = 0.0f;
#pragma unroll
    for (unsigned w = 0; w < kMmaWarps; w++) a = fmaf(mo[(w * 4u + h) * HD + d], fac[w * 4u + h], a);
    const unsigned head = head0 + h;
    if (n_splits == 1) {
      st_act<T>(out, ((size_t)slot * n_q + head) * HD + d, a / fac[36u + h]);
    } else {
      float* rec = record(head);
      if (d == 0) {
        rec[0] = fac[32u + h];
        rec[1] = fac[36u + h];
      }
      rec[2 + d] = a;
    }
  }
}

template <int HD, typename T, unsigned CH, bool DEAL>
int launch_mma(ks_ctx* ctx, unsigned hpk, dim3 grid, unsigned n_q, unsigned n_kv, float scale, const void* q, const uint8_t* K, const uint8_t* V,
               size_t slot_stride, const float* meta, float* tmp, void* out, int n_splits) {
  const unsigned gb = hpk % 4 == 0 ? 4u : hpk % 2 == 0 ? 2u : 1u;
  auto kern = sdpa_mma_kernel<HD, T, CH, DEAL>;
  constexpr size_t smem = MmaSmem<HD>::total;
  static bool set[16] = {false};
  if (!set[ctx->device & 15]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return ks_fail(ctx, KS_ERR_CUDA, "sdpa: cannot set %zu B shared memory: %s", smem, cudaGetErrorString(e));
    set[ctx->device & 15] = true;
  }
  grid.y *= hpk / gb;
  KS_LAUNCH(ctx, kern, grid, kMmaWarps * 32, smem, n_q, n_kv, gb, scale, (const T*)q, K, V, slot_stride, meta, tmp, (T*)out, n_splits);
  return ks_after_launch(ctx, "sdpa_mma");
}

template <int G, int DPL, typename T>
int launch_part(ks_ctx* ctx, dim3 grid, unsigned n_q, unsigned n_kv, float scale, const void* q, const uint8_t* K,
                const uint8_t* V, size_t slot_stride, const float* meta, float* tmp, void* out, int n_splits) {
  const bool aligned = (((uintptr_t)K | (uintptr_t)V | (uintptr_t)slot_stride) & 7u) == 0;
  if (aligned)
    KS_LAUNCH(ctx, (sdpa_part_kernel<G, DPL, T, true>), grid, kWarps * 32, 0, n_q, n_kv, scale, (const T*)q, K, V, slot_stride, meta,
              tmp, (T*)out, n_splits);
  else
    KS_LAUNCH(ctx, (sdpa_part_kernel<G, DPL, T, false>), grid, kWarps * 32, 0, n_q, n_kv, scale, (const T*)q, K, V, slot_stride,
              meta, tmp, (T*)out, n_splits);
  return ks_after_launch(ctx, "sdpa_part");
}

template <int DPL, typename T>
int launch_part_g(ks_ctx* ctx, int G, dim3 grid, unsigned n_q, unsigned n_kv, float scale, const void* q, const uint8_t* K,
                  const uint8_t* V, size_t slot_stride, const float* meta, float* tmp, void* out, int n_splits) {
  switch (G) {
    case 1: return launch_part<1, DPL, T>(ctx, grid, n_q, n_kv, scale, q, K, V, slot_stride, meta, tmp, out, n_splits);
    case 2: return launch_part<2, DPL, T>(ctx, grid, n_q, n_kv, scale, q, K, V, slot_stride, meta, tmp, out, n_splits);
    case 4: return launch_part<4, DPL, T>(ctx, grid, n_q, n_kv, scale, q, K, V, slot_stride, meta, tmp, out, n_splits);
    default:  // 8 and 16: four heads per block, G / 4 blocks per KV head
      grid.y *= (unsigned)(G / 4);
      return launch_part<4, DPL, T>(ctx, grid, n_q, n_kv, scale, q, K, V, slot_stride, meta, tmp, out, n_splits);
  }
}

}  // namespace

int ks_launch_sdpa(ks_ctx* ctx, size_t n_slots, size_t n_q, size_t n_kv, size_t hd, float scale, ks_dtype act,
                   const void* q, const uint8_t* K, const uint8_t* V, size_t slot_stride_bytes, const float* meta,
                   float* tmp, void* out, int n_splits, bool records_only, size_t max_t) {
  const int G = (int)(n_q / n_kv);
  if (G != 1 && G != 2 && G != 4 && G != 8 && G != 16)  // one set of groups, whichever kernel the operands' alignment leads to
    return ks_fail(ctx, KS_ERR_UNSUPPORTED, "sdpa: n_q/n_kv = %d not supported (1, 2, 4, 8, 16)", G);
  dim3 grid((unsigned)n_splits, (unsigned)n_kv, (unsigned)n_slots);
  int rc = 1;
  bool deal = false;
  static const bool per_row = getenv("KSEARCH_SDPA_PER_ROW") != nullptr;  // keep the per-row kernel (comparison runs)
  const uintptr_t at = (uintptr_t)K | (uintptr_t)V | (uintptr_t)slot_stride_bytes;
  if (!per_row && (hd == 256 || hd == 128) && at % 4 == 0) {  // a cache that starts on 2 bytes is left to the per-row kernel
    const bool wide = at % (hd == 256 ? 16 : 8) == 0;
    // (contexts that cannot be long for the splits need not be looked at)
    deal = max_t > (size_t)n_splits * kMinChunk && n_slots > 1 && n_slots <= kDealSlots && n_splits > 1 && n_slots * n_splits <= KS_SDPA_MAX_SPLITS && !records_only && ((uintptr_t)meta & 15) == 0;
#define KS_MMA_D(HD_, T_, CH_, D_) launch_mma<HD_, T_, CH_, D_>(ctx, (unsigned)G, grid, (unsigned)n_q, (unsigned)n_kv, scale, q, K, V, slot_stride_bytes, meta, tmp, out, n_splits)
#define KS_MMA(HD_, T_, CH_) (deal ? KS_MMA_D(HD_, T_, CH_, true) : KS_MMA_D(HD_, T_, CH_, false))
#define KS_MMA_CH(HD_, CH_) (act == KS_F32 ? KS_MMA(HD_, float, CH_) : KS_MMA(HD_, __half, CH_))
    if (hd == 256) rc = wide ? KS_MMA_CH(256, 16u) : KS_MMA_CH(256, 4u);
    else rc = wide ? KS_MMA_CH(128, 8u) : KS_MMA_CH(128, 4u);
#undef KS_MMA_CH
#undef KS_MMA
#undef KS_MMA_D
  }
  if (rc != 1) {
    // the tensor-core kernel took it
  } else if (hd == 256) {
    rc = act == KS_F32 ? launch_part_g<8, float>(ctx, G, grid, (unsigned)n_q, (unsigned)n_kv, scale, q, K, V, slot_stride_bytes, meta, tmp, out, n_splits)
                       : launch_part_g<8, __half>(ctx, G, grid, (unsigned)n_q, (unsigned)n_kv, scale, q, K, V, slot_stride_bytes, meta, tmp, out, n_splits);
  } else if (hd == 128) {
    rc = act == KS_F32 ? launch_part_g<4, float>(ctx, G, grid, (unsigned)n_q, (unsigned)n_kv, scale, q, K, V, slot_stride_bytes, meta, tmp, out, n_splits)
                       : launch_part_g<4, __half>(ctx, G, grid, (unsigned)n_q, (unsigned)n_kv, scale, q, K, V, slot_stride_bytes, meta, tmp, out, n_splits);
  } else {
    return ks_fail(ctx, KS_ERR_UNSUPPORTED, "sdpa: head_dim %zu not supported (128, 256)", hd);
  }
  if (rc || n_splits == 1 || records_only) return rc;
  const dim3 blocks((unsigned)(n_slots * n_q), (unsigned)hd / kRedDims);
#define KS_RED(T_, D_) KS_LAUNCH(ctx, (sdpa_reduce_kernel<T_, D_>), blocks, kRedDims * kRedParts, 0, (unsigned)hd, tmp, (T_*)out, n_splits, (unsigned)n_q, meta)
  if (act == KS_F32) {
    if (deal) KS_RED(float, true);
    else KS_RED(float, false);
  } else {
    if (deal) KS_RED(__half, true);
    else KS_RED(__half, false);
  }
#undef KS_RED
  return ks_after_launch(ctx, "sdpa_reduce");
}

extern "C" {

size_t ks_sdpa_tmp_floats(size_t n_slots, size_t n_q, size_t hd, int n_splits) {
  if (n_splits <= 1) return 0;
  return n_slots * n_q * (size_t)n_splits * (hd + 2);
}

int ks_sdpa_pick_splits(const ks_ctx* ctx, size_t n_slots, size_t n_kv, size_t max_t) {
  // about 256 blocks in all (two fit an SM; a block serves up to four query heads, so a slot has at least two per split), at
  // least 128 positions per split: measured best over 1..8 slots x 1024..16384 positions on B200
  (void)ctx;
  const size_t per_split = (n_slots ? n_slots : 1) * (n_kv > 2 ? n_kv : 2);
  size_t want = 256 / per_split;
  size_t by_len = (max_t + 127) / 128;
  size_t s = want < by_len ? want : by_len;
  if (s < 1) s = 1;
  if (s > KS_SDPA_MAX_SPLITS) s = KS_SDPA_MAX_SPLITS;
  return (int)s;
}

int ks_sdpa_decode(ks_ctx* ctx, size_t n_slots, size_t n_q, size_t n_kv, size_t hd, size_t max_t, ks_dtype kv_dtype,
                   float scale, ks_dtype act, const ks_buf* q, const ks_buf* K, const ks_buf* V, size_t kv_byte_off,
                   size_t slot_stride_bytes, const ks_buf* meta, ks_buf* tmp, ks_buf* out, int n_splits) {
  if (!ctx) return KS_ERR_INVALID;
  KS_REQUIRE(ctx, kv_dtype == KS_Q40, "sdpa: KV dtype %d not supported (Q40)", (int)kv_dtype);
  KS_REQUIRE(ctx, ks_is_act(act), "sdpa: activation dtype must be F32 or F16");
  KS_REQUIRE(ctx, n_slots > 0 && n_slots < 65536 && n_q > 0 && n_kv > 0 && n_kv < 65536, "sdpa: bad slot or head count");
  KS_REQUIRE(ctx, n_q % n_kv == 0, "sdpa: n_q=%zu is not a multiple of n_kv=%zu", n_q, n_kv);
  KS_REQUIRE(ctx, hd % 32 == 0, "sdpa hd must be multiple of 32");
  KS_REQUIRE(ctx, max_t > 0, "sdpa: max_t must be > 0");
  if (n_splits == 0) n_splits = ks_sdpa_pick_splits(ctx, n_slots, n_kv, max_t);
  KS_REQUIRE(ctx, n_splits >= 1 && n_splits <= KS_SDPA_MAX_SPLITS, "sdpa: n_splits=%d outside 1..%d", n_splits, KS_SDPA_MAX_SPLITS);
  const size_t ab = ks_act_bytes(act);
  const size_t rowb = hd / 32 * KS_Q40_BLOCK_BYTES;
  const size_t slot_bytes = max_t * n_kv * rowb;
  KS_REQUIRE(ctx, n_slots == 1 || slot_stride_bytes >= slot_bytes, "sdpa: slot stride smaller than one slot's cache");
  KS_REQUIRE(ctx, kv_byte_off % 2 == 0 && slot_stride_bytes % 2 == 0, "sdpa: odd KV offset or stride");
  const size_t kv_need = (n_slots - 1) * slot_stride_bytes + slot_bytes;
  KS_REQUIRE(ctx, ks_fits(K, kv_byte_off, kv_need) && ks_fits(V, kv_byte_off, kv_need), "sdpa: KV buffer too small for max_t=%zu", max_t);
  KS_REQUIRE(ctx, ks_fits(q, 0, n_slots * n_q * hd * ab) && ks_fits(out, 0, n_slots * n_q * hd * ab), "sdpa: q/out buffer too small");
  KS_REQUIRE(ctx, ks_fits(meta, 0, n_slots * 16), "sdpa: meta buffer too small (4 f32 per slot)");
  if (n_splits > 1)
    KS_REQUIRE(ctx, ks_fits(tmp, 0, ks_sdpa_tmp_floats(n_slots, n_q, hd, n_splits) * 4), "sdpa: tmp buffer too small for %d splits", n_splits);
  // (tlen, start) are device-resident and trusted to satisfy start + tlen <= max_t, as in the reference.
  return ks_launch_sdpa(ctx, n_slots, n_q, n_kv, hd, scale, act, q->dptr, (const uint8_t*)K->dptr + kv_byte_off,
                        (const uint8_t*)V->dptr + kv_byte_off, slot_stride_bytes, (const float*)meta->dptr,
                        n_splits > 1 ? (float*)tmp->dptr : nullptr, out->dptr, n_splits, false, max_t);
}

}  // extern "C"
