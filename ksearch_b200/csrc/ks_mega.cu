// One persistent kernel for all layers of a decode token (single slot; f32 inside whatever the model's activation dtype).
//
// The op order is forward_token's (crates/ksearch_gemma/src/gemma_prim.rs:923-1197) for dense,
// KV-owning layers; what changes is WHERE the boundaries between ops are.  On B200 a token is a
// chain of ~180 dependent steps, each a few hundred kilobytes to ten megabytes of weights, and a
// kernel boundary costs more than most of those steps take.  Here one block per SM stays resident
// for the whole token:
//   * the weight stream never stops: one warp copies the block's row groups of all phases, in the order they are
//     needed, into a ring in shared memory (cp.async.bulk, one mbarrier per row group); the next phases' groups are
//     already there while the block waits at a barrier.  Fifteen other warps multiply: an item is a row group's share
//     of the columns, so a group is split over as many warps as that evens out;
//   * phases (qkv | attention | o-proj | gate-up | down, per layer) are separated by a grid barrier
//     on one global counter; activations cross it through global memory (L2), read with ld.cg;
//     one hop has no barrier: q/k/v go to the attention blocks as 64-bit (value, tag) words written
//     with relaxed stores and polled by their consumers (a hop of ~1 us instead of ~2 us);
//   * the norms are applied while x is staged; their weights come through the ring as well, because the acquire that
//     ends a wait drops the SM's L1 and every later plain load of a constant would be a full round trip to L2 (for the
//     same reason nothing may be spilled: local memory lives in L1);
//   * for the same reason nothing on the critical path reads a descriptor from global memory: the
//     five phase shapes and the per-layer pointers are copied to shared memory once;
//   * attention: per-head RMS + RoPE + Q4_0 pack of the new K/V row, split-context online softmax
//     and, for long contexts, the merge of the splits (last arriving block) happen inside one phase; a few splits are merged
//     by whoever stages them.
// Bound by the chain: a layer of the E2B shape is 25.5 us (32.5 before the copying warp, with eight warps of 242 registers), its
// weights 3 us of HBM.  Microseconds at 100 positions, E2B, before / now: q|k|v 4.8 / 3.8, attention 10.9 / 5.1, o 4.1 / 5.1,
// gate|up 7.7 / 5.9, down 5.1 / 5.7; E4B at 4000 positions: 6.0 / 5.1, 25.4 / 12.3, 4.7 / 4.4, 16.4 / 10.2, 8.6 / 9.2.  A phase
// is 1 to 2 us of waiting (barrier and slower blocks), 0.8 to 2 of staging, the rest multiplication.  Fifteen warps instead of
// eight, row groups dealt one by one instead of in runs of eight (a block had up to 64 gate|up rows where 42 is the mean) and no
// register spilled are what they owe it to: arrays left undefined in some lanes stayed live around the phase loop and spilled.
// Every spin (barrier, tagged word, mbarrier) is bounded; on expiry the block raises the context's status word,
// drains its copies and leaves, and the other blocks time out the same way.
#include <cstring>
#include <utility>
#include <vector>

#include "ks_mv_common.cuh"

namespace {

enum { MG_MATVEC = 0, MG_GATE_UP = 1, MG_ATTN = 2 };
enum { PH_QKV = 0, PH_ATTN = 1, PH_OPROJ = 2, PH_GATEUP = 3, PH_DOWN = 4, PH_PER_LAYER = 5 };

constexpr unsigned MG_WARPS = 15, MG_THREADS = MG_WARPS * 32;  // that multiply; a sixteenth warp copies
constexpr unsigned MG_JOBS = 64;                               // row groups in the ring at a time, at most (a power of two)
constexpr unsigned MG_EMPTY = 1024;                            // arrivals that free one: its items' shares add up to this

struct MegaShape {          // one of the five phases of a layer; the same for every layer
  int type;
  int n_seg;                // matvec: 1 or 3 (q, k, v)
  unsigned rows[3];
  unsigned grp_start[4];    // first group of each segment, [n_seg] = total groups (0 for attention)
  unsigned cols, row_bytes, seg_blocks, n_cseg;
  unsigned mats, w0;        // matrices of a group (2: gate and up), MegaLayer::W index of the first segment's
};

struct MegaLayer {          // per-layer pointers, copied to shared memory when the kernel starts
  const uint8_t* W[7];      // wq, wk, wv, wo, wgate, wup, wdown (Q4_K)
  const float* norm[6];     // attn_norm, q_norm, k_norm, post_attn_norm, ffn_norm, post_ffw_norm
  uint8_t *kv_k, *kv_v;     // this slot's cache rows [max_seq, n_kv, hd] Q4_0
  size_t window;            // positions the layer attends to (0: all), gemma_prim.rs:1009-1016
};

struct MegaArgs {
  const void* tables;       // MegaShape[5] then MegaLayer[n_layers], 16-byte aligned; copied to shared memory at start
  unsigned tables_bytes;    // multiple of 16
  int n_layers;
  unsigned ring_bytes;
  unsigned x_off, ring_off; // shared memory: staging area for x (also the attention scratch), the ring
  unsigned n_q, n_kv, hd, n_splits;
  float eps, attn_scale;
  const float* rope;        // [max_seq, hd]
  const int* pos;           // [1]
  float *x_a, *x_b;         // residual stream: layers read x_a / write x_b at the FFN, the reverse at the next qkv
  float* yb;
  unsigned char* ox;        // merged attention output, written in the staged fixed-point layout
  float* ff;                // GeGLU output
  float* att_tmp;           // [n_q][n_splits] records
  float4* nsum;             // [grid] per-block sums of the last o-proj / down phase: (sum y^2, sum x*y*wp, sum (y*wp)^2, sum x^2)
  unsigned* att_cnt;        // [n_q] arrival counters of the attention blocks, per head
  unsigned* bar;            // [0] running barrier counter, [1] its value when the previous token ended
  unsigned* err;
  unsigned long long* qkv_t;  // q | k | v rows of the current layer as (tag << 32 | f32 bits) words: the q/k/v phase hands
                              // them to the attention blocks without a grid barrier, consumers poll for the tag
  unsigned poll_limit;      // polls of the barrier counter (or of a tagged word) before a wait gives up
  unsigned test_stall;      // test hook: the barrier before phase 1 waits for this many arrivals more than ever come
  long long* prof;          // [2][phases][8] SM clocks of the first and last block: start, staged, computed, released
                            // (attention rows: 4..7 = q/k/v ready, positions done, folded, arrived)
};

__device__ __forceinline__ uint32_t sm32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mb_init(uint32_t bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mb_expect(uint32_t bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mb_wait(uint32_t bar, unsigned parity) {
  for (unsigned i = 0; i < (1u << 21); i++) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void bulk_in(uint32_t dst, const void* src, unsigned bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ float4 ldcg4(const float* p, unsigned c) { return __ldcg(reinterpret_cast<const float4*>(p) + c); }
// A value and its tag in one 64-bit word: single-copy atomic, so a consumer that sees the tag sees the value; no fence.
__device__ __forceinline__ void tag_store(unsigned long long* p, float v, unsigned tag) {
  const unsigned long long w = ((unsigned long long)tag << 32) | (unsigned long long)__float_as_uint(v);
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ unsigned long long tag_load(const unsigned long long* p) {
  unsigned long long w;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
  return w;
}
// Tagged words p[i], i = at[0..N), per lane until every tag matches; false when the limit ran out.
template <int N>
__device__ __forceinline__ bool tag_wait(const unsigned long long* p, const int (&at)[N], unsigned tag, unsigned limit, float (&v)[N]) {
  for (unsigned it = 0; it < limit; it++) {
    unsigned long long w[N];
    unsigned bad = 0;
#pragma unroll
    for (int j = 0; j < N; j++) w[j] = tag_load(p + at[j]);
#pragma unroll
    for (int j = 0; j < N; j++) {
      bad |= (unsigned)(w[j] >> 32) ^ tag;
      v[j] = __uint_as_float((unsigned)w[j]);
    }
    if (bad == 0) return true;
  }
#pragma unroll
  for (int j = 0; j < N; j++) v[j] = 0.0f;
  return false;
}

// The thread's index, read anew: what is computed from it stays where it is used.  Hoisted out of the phase loop, the addresses and
// predicates of all phases together do not fit the registers, and a spilled one comes back from L2.
__device__ __forceinline__ unsigned mg_tid() {
  unsigned t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}
// The warps that multiply; the copying warp never joins them.
__device__ __forceinline__ void cta_sync() { asm volatile("bar.sync 1, %0;" ::"n"(MG_THREADS) : "memory"); }

// Grid-wide barrier on a monotonically increasing counter, in two halves so that loads which do not
// depend on other blocks can be issued in between.
// n_wsum: that many warps left partial norm sums in wsum; thread 0 folds them (fixed order) into nsum[block].
__device__ __forceinline__ void grid_arrive(unsigned* counter, const float4* wsum, unsigned n_wsum, float4* nsum) {
  const unsigned tid = mg_tid();
  cta_sync();  // every store of this block is issued
  if (tid == 0) {
    if (n_wsum) {
      float4 t = wsum[0];
      for (unsigned w = 1; w < n_wsum; w++) {
        const float4 u = wsum[w];
        t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
      }
      nsum[blockIdx.x] = t;
    }
    // release: everything this block wrote (ordered before by the barrier above) is visible to whoever
    // acquires the counter; nothing comes back, so the thread does not wait for a round trip
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
  }
}
// Returns false when the wait gave up.
// Lane 0 of four warps polls: their loads drift apart in time, so the arrival of the last block is
// seen sooner than one poller's round trip allows.  sflag: 0 = waiting, 1 = released, 2 = gave up.
// Two flag words alternate between consecutive barriers, so a word is cleared a whole phase after its last reader.
__device__ __forceinline__ bool grid_wait(unsigned* counter, unsigned target, unsigned* err, int* flags, int parity, unsigned limit) {
  const unsigned tid = mg_tid();
  int* sflag = flags + parity;
  if (tid == 0) flags[parity ^ 1] = 0;
  if ((tid & 31) == 0 && tid < 128) {
    volatile int* vf = sflag;
    int state = 0;
    for (unsigned i = 0; i < limit; i++) {  // a second or two of polling at most
      if ((int)(ld_acquire_u32(counter) - target) >= 0) {
        state = 1;
        break;
      }
      if (*vf == 1) {  // another poller saw it; take the acquire ourselves before reading what other blocks wrote
        if ((int)(ld_acquire_u32(counter) - target) >= 0) {
          state = 1;
          break;
        }
      }
    }
    if (state == 1) {
      *vf = 1;
    } else {
      atomicOr(err, 2u);
      *vf = 2;
    }
  }
  cta_sync();
  return *sflag == 1;
}

// ---- x as 24-bit block fixed point, weights x x as byte dot products ----------------------------
// Each 32-element sub-block of the staged vector shares a scale s; element i is the integer
// X_i = round(x_i / s), |X_i| <= 8e6, kept as three byte planes (X = l2*65536 + l1*256 + l0, l2
// signed).  Four neighbouring nibbles of a weight word, masked in place, are the other operand of a
// dp4a, so 4 weights cost 3 integer dot-product instructions instead of ~9 f32 instructions, and the
// shared-memory traffic for x drops from 4 bytes to 3/4 byte per weight.  Integer accumulation is
// exact; the only approximation is x to 24 bits of its sub-block's largest element (f32 has 24 bits
// per element), far inside the parity tolerance.
// Shared-memory layout: plane k (k = 0..2) at k * units * 80 bytes, unit u at u * 80 inside it (64
// used: words 0..7 = elements 0..31 of the low-nibble sub-block, 8..15 = the high-nibble one; the pad
// keeps the 8 lanes of a row on different banks), then units * 16 bytes of (sum_lo, sum_hi, s_lo, s_hi).
constexpr int MG_RL = 4, MG_LPR = 8;  // 8 lanes per row, 4 rows side by side
constexpr unsigned MG_XU = 80;  // bytes per unit and plane
__device__ __forceinline__ void fx_put_chunk(unsigned char* xs, unsigned units, unsigned c, float4 v) {
  const unsigned e = c << 2;
  const unsigned u = e >> 6, hi = (e >> 5) & 1u, l = e & 31u;
  float s = (v.x + v.y) + (v.z + v.w);
  float am = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
#pragma unroll
  for (int o = 1; o <= 4; o <<= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
  }
  const float inv = am > 0.0f ? __fdividef(8.0e6f, am) : 0.0f;
  const float sc = am > 0.0f ? am * (1.0f / 8.0e6f) : 1.0f;
  const int X0 = __float2int_rn(v.x * inv), X1 = __float2int_rn(v.y * inv), X2 = __float2int_rn(v.z * inv),
            X3 = __float2int_rn(v.w * inv);
  const unsigned wi = hi * 8u + (l >> 2);
  unsigned char* base = xs + (size_t)u * MG_XU + wi * 4u;
  const size_t plane = (size_t)units * MG_XU;
  *reinterpret_cast<uint32_t*>(base) = __byte_perm(__byte_perm(X0, X1, 0x0040), __byte_perm(X2, X3, 0x0040), 0x5410);
  *reinterpret_cast<uint32_t*>(base + plane) = __byte_perm(__byte_perm(X0, X1, 0x0051), __byte_perm(X2, X3, 0x0051), 0x5410);
  *reinterpret_cast<uint32_t*>(base + 2 * plane) = __byte_perm(__byte_perm(X0, X1, 0x0062), __byte_perm(X2, X3, 0x0062), 0x5410);
  if ((c & 7u) == 0) {
    float* mt = reinterpret_cast<float*>(xs + 3 * plane + (size_t)u * 16u);
    mt[hi] = s;
    mt[2 + hi] = sc;
  }
}
// The same layout written to GLOBAL memory by a producer: the warp holds the 32 consecutive elements
// e0 .. e0+31 of one sub-block, one per lane (e0 a multiple of 32).
__device__ __forceinline__ void fx_store_subblock(unsigned char* dst, unsigned units, unsigned e0, float val, int lane) {
  float s = val, am = fabsf(val);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
  }
  const float inv = am > 0.0f ? __fdividef(8.0e6f, am) : 0.0f;
  const float sc = am > 0.0f ? am * (1.0f / 8.0e6f) : 1.0f;
  const int X = __float2int_rn(val * inv);
  const unsigned u = e0 >> 6, hi = (e0 >> 5) & 1u;
  const size_t plane = (size_t)units * MG_XU;
  unsigned char* base = dst + (size_t)u * MG_XU + hi * 32u + (unsigned)lane;
  base[0] = (unsigned char)(X & 0xFF);
  base[plane] = (unsigned char)((X >> 8) & 0xFF);
  base[2 * plane] = (unsigned char)((X >> 16) & 0xFF);
  if (lane == 0) {
    float* mt = reinterpret_cast<float*>(dst + 3 * plane + (size_t)u * 16u);
    mt[hi] = s;
    mt[2 + hi] = sc;
  }
}
// Bring a vector a producer left in that layout into shared memory (units * 256 bytes; the pad words travel too).
__device__ __forceinline__ void fx_copy_in(unsigned char* xs, const unsigned char* src, unsigned units) {
  const unsigned tid = mg_tid();
  const unsigned n16 = units * 16u;  // 3 planes of 80 bytes + 16 bytes of sums and scales per unit
  for (unsigned base = 0; base < n16; base += 2u * MG_THREADS) {
    uint4 v[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const unsigned i = base + tid + k * MG_THREADS;
      v[k] = i < n16 ? __ldcg(reinterpret_cast<const uint4*>(src) + i) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const unsigned i = base + tid + k * MG_THREADS;
      if (i < n16) reinterpret_cast<uint4*>(xs)[i] = v[k];
    }
  }
}
__device__ __forceinline__ unsigned dp4a_uu(unsigned a, unsigned b, unsigned c) {
  unsigned d;
  asm("dp4a.u32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ int dp4a_us(unsigned a, unsigned b, int c) {  // a: unsigned bytes, b: signed bytes
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
template <int OFF>
__device__ __forceinline__ float4 lds_f4o(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4+%5];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a), "n"(OFF));
  return v;
}
// One weight word (8 nibbles: elements j..j+3 of the low and of the high sub-block) against the
// matching x words of the three planes.
__device__ __forceinline__ void fx_word(uint32_t w, unsigned xl0, unsigned xl1, unsigned xl2, unsigned xh0, unsigned xh1,
                                        unsigned xh2, unsigned (&alo)[2], int& alo2, unsigned (&ahi)[2], int& ahi2) {
  const unsigned lo = w & 0x0F0F0F0Fu, hi = (w >> 4) & 0x0F0F0F0Fu;
  alo[0] = dp4a_uu(lo, xl0, alo[0]);
  alo[1] = dp4a_uu(lo, xl1, alo[1]);
  alo2 = dp4a_us(lo, xl2, alo2);
  ahi[0] = dp4a_uu(hi, xh0, ahi[0]);
  ahi[1] = dp4a_uu(hi, xh1, ahi[1]);
  ahi2 = dp4a_us(hi, xh2, ahi2);
}
// Multiply-accumulate one item (column segment cs of the four rows at slot_addr, MATS matrices) against the fixed-point x.
template <int MATS>
__device__ __forceinline__ void mg_item_compute_fx(uint32_t slot_addr, unsigned row_bytes, uint32_t xs_s, unsigned units, unsigned seg_blocks,
                                                   unsigned cs, int cl, int rl, float (&yacc)[2]) {
  const int g = cl & 3;
  const unsigned seg_units = seg_blocks * 4, upl = seg_units / MG_LPR;
  const uint32_t plane = units * MG_XU;
  uint32_t waddr = slot_addr + (uint32_t)rl * row_bytes + (cs * seg_blocks + (uint32_t)(cl >> 2)) * KS_Q4K_BLOCK_BYTES + (uint32_t)g * 32u;
  uint32_t xaddr = xs_s + (cs * seg_units + (unsigned)cl) * MG_XU;
  uint32_t maddr = xs_s + 3u * plane + (cs * seg_units + (unsigned)cl) * 16u;
#pragma unroll 1
  for (unsigned it = 0; it < upl; it++) {
    unsigned alo[MATS][2], ahi[MATS][2];
    int alo2[MATS], ahi2[MATS];
#pragma unroll
    for (int r = 0; r < MATS; r++) {
      alo[r][0] = alo[r][1] = ahi[r][0] = ahi[r][1] = 0u;
      alo2[r] = ahi2[r] = 0;
    }
    // 16 words per plane: [0..7] low sub-block, [8..15] high sub-block.  Half of each at a time: with all 48 words of x in registers
    // the kernel spills, and what is spilled has to come back from L2 (shared memory leaves no L1, an acquire empties it).
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t xa = xaddr + 16u * h;
      const uint4 a0 = lds_u4o<0>(xa), a2 = lds_u4o<32>(xa), b0 = lds_u4o<0>(xa + plane), b2 = lds_u4o<32>(xa + plane),
                  c0 = lds_u4o<0>(xa + 2 * plane), c2 = lds_u4o<32>(xa + 2 * plane);
#pragma unroll
      for (int r = 0; r < MATS; r++) {
        const uint4 q = lds_u4o<16>(waddr + (uint32_t)(r * MG_RL) * row_bytes + 16u * h);
        fx_word(q.x, a0.x, b0.x, c0.x, a2.x, b2.x, c2.x, alo[r], alo2[r], ahi[r], ahi2[r]);
        fx_word(q.y, a0.y, b0.y, c0.y, a2.y, b2.y, c2.y, alo[r], alo2[r], ahi[r], ahi2[r]);
        fx_word(q.z, a0.z, b0.z, c0.z, a2.z, b2.z, c2.z, alo[r], alo2[r], ahi[r], ahi2[r]);
        fx_word(q.w, a0.w, b0.w, c0.w, a2.w, b2.w, c2.w, alo[r], alo2[r], ahi[r], ahi2[r]);
      }
    }
    const float4 mt = lds_f4o<0>(maddr);
#pragma unroll
    for (int r = 0; r < MATS; r++) {
      const uint4 hdr = lds_u4o<0>(waddr + (uint32_t)(r * MG_RL) * row_bytes - (uint32_t)g * 32u);
      const float flo = fmaf((float)alo2[r], 65536.0f, fmaf((float)alo[r][1], 256.0f, (float)alo[r][0])) * mt.z;
      const float fhi = fmaf((float)ahi2[r], 65536.0f, fmaf((float)ahi[r][1], 256.0f, (float)ahi[r][0])) * mt.w;
      yacc[r] = q4k_apply_scales(hdr, g, flo, fhi, mt.x, mt.y, yacc[r]);
    }
    waddr += (MG_LPR / 4) * KS_Q4K_BLOCK_BYTES;
    xaddr += MG_LPR * MG_XU;
    maddr += MG_LPR * 16u;
  }
}


// ---- staging of x (with the fused norm prologues), reads through L2 ---------------------------
constexpr int MG_XMAX = 4;  // plain staging keeps up to 4 chunks per thread in flight (7680 columns), loops beyond
// x' = x
__device__ __forceinline__ void mg_stage_plain(unsigned char* xs, unsigned cols, const float* x) {
  const unsigned tid = mg_tid();
  const unsigned units = cols >> 6, nchunk = cols >> 2;
  for (unsigned base = 0; base < nchunk; base += MG_XMAX * MG_THREADS) {
    float4 v[MG_XMAX];
#pragma unroll
    for (int k = 0; k < MG_XMAX; k++) {
      const unsigned c = base + tid + k * MG_THREADS;
      v[k] = c < nchunk ? ldcg4(x, c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int k = 0; k < MG_XMAX; k++) {
      const unsigned c = base + tid + k * MG_THREADS;
      if (c < nchunk) fx_put_chunk(xs, units, c, v[k]);
    }
  }
}
// x' = rms(x) * w  (the first layer)
template <int PC>
__device__ __forceinline__ void mg_stage_norm(unsigned char* xs, float* red, unsigned cols, const float* x, float eps, const float4* w) {
  const unsigned tid = mg_tid();
  const unsigned units = cols >> 6, nchunk = cols >> 2;
  float4 v[PC];
  float ss = 0.0f;
#pragma unroll
  for (int k = 0; k < PC; k++) {
    const unsigned c = tid + k * MG_THREADS;
    v[k] = c < nchunk ? ldcg4(x, c) : make_float4(0.f, 0.f, 0.f, 0.f);
    ss = fmaf(v[k].x, v[k].x, ss); ss = fmaf(v[k].y, v[k].y, ss);
    ss = fmaf(v[k].z, v[k].z, ss); ss = fmaf(v[k].w, v[k].w, ss);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((tid & 31) == 0) red[tid >> 5] = ss;
  cta_sync();
  ss = 0.0f;
#pragma unroll
  for (unsigned w = 0; w < MG_WARPS; w++) ss += red[w];
  const float inv2 = 1.0f / sqrtf(ss * (1.0f / (float)cols) + eps);
#pragma unroll
  for (int k = 0; k < PC; k++) {
    const unsigned c = tid + k * MG_THREADS;
    if (c < nchunk) {
      const float4 w4 = w[c];
      float4 r;
      r.x = __fmul_rn(__fmul_rn(v[k].x, inv2), w4.x);
      r.y = __fmul_rn(__fmul_rn(v[k].y, inv2), w4.y);
      r.z = __fmul_rn(__fmul_rn(v[k].z, inv2), w4.z);
      r.w = __fmul_rn(__fmul_rn(v[k].w, inv2), w4.w);
      fx_put_chunk(xs, units, c, r);
    }
  }
}

// r = x + rms(y) * wp (block 0 stores r to out_x); x' = rms(r) * w.  Without a block-wide reduction over the vector: the blocks that
// produced y left the four sums that both norms need (K:539 expands to  sum r^2 = sum x^2 + 2 inv sum x y wp + inv^2 sum (y wp)^2,
// r = x + inv y wp).  A lane folds a block's sums while the loads of x and y are on their way.
template <int PC>
__device__ __forceinline__ void mg_stage_addnorm(unsigned char* xs, float* red, unsigned cols, const float* x, const float* y, float* out_x,
                                                 float eps, const float4* w, const float4* wp, const float4* nsum, unsigned nblocks) {
  const unsigned tid = mg_tid();
  const unsigned units = cols >> 6, nchunk = cols >> 2;
  float4 v[PC], yv[PC];
#pragma unroll
  for (int k = 0; k < PC; k++) {
    const unsigned c = tid + k * MG_THREADS;
    yv[k] = c < nchunk ? ldcg4(y, c) : make_float4(0.f, 0.f, 0.f, 0.f);
    v[k] = c < nchunk ? ldcg4(x, c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const unsigned fold = (nblocks + 31u) / 32u;
  float4* sums = reinterpret_cast<float4*>(red);
  if ((tid >> 5) < fold) {
    float4 t = tid < nblocks ? __ldcg(nsum + tid) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      t.x += __shfl_xor_sync(0xffffffffu, t.x, o);
      t.y += __shfl_xor_sync(0xffffffffu, t.y, o);
      t.z += __shfl_xor_sync(0xffffffffu, t.z, o);
      t.w += __shfl_xor_sync(0xffffffffu, t.w, o);
    }
    if ((tid & 31) == 0) sums[tid >> 5] = t;
  }
  cta_sync();
  float4 t = sums[0];
#pragma unroll 1
  for (unsigned w = 1; w < fold; w++) {
    const float4 u = sums[w];
    t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
  }
  const float invn = 1.0f / (float)cols;
  const float inv = __frsqrt_rn(t.x * invn + eps);
  const float rr = fmaf(inv * inv, t.z, fmaf(2.0f * inv, t.y, t.w));
  const float inv2 = __frsqrt_rn(fmaxf(rr, 0.0f) * invn + eps);
#pragma unroll
  for (int k = 0; k < PC; k++) {
    const unsigned c = tid + k * MG_THREADS;
    if (c < nchunk) {
      const float4 p4 = wp[c], w4 = w[c];
      float4 r = v[k];
      r.x = __fadd_rn(r.x, __fmul_rn(__fmul_rn(yv[k].x, inv), p4.x));
      r.y = __fadd_rn(r.y, __fmul_rn(__fmul_rn(yv[k].y, inv), p4.y));
      r.z = __fadd_rn(r.z, __fmul_rn(__fmul_rn(yv[k].z, inv), p4.z));
      r.w = __fadd_rn(r.w, __fmul_rn(__fmul_rn(yv[k].w, inv), p4.w));
      if (blockIdx.x == 0) reinterpret_cast<float4*>(out_x)[c] = r;
      float4 q;
      q.x = __fmul_rn(__fmul_rn(r.x, inv2), w4.x);
      q.y = __fmul_rn(__fmul_rn(r.y, inv2), w4.y);
      q.z = __fmul_rn(__fmul_rn(r.z, inv2), w4.z);
      q.w = __fmul_rn(__fmul_rn(r.w, inv2), w4.w);
      fx_put_chunk(xs, units, c, q);
    }
  }
}

// ---- the row groups of a block -------------------------------------------------------------------
// Groups of four rows go to blocks round-robin (block c owns groups c, c + grid, ...); each is one job of the copying warp.  A
// phase's items are its groups x column segments, item i to warp i % MG_WARPS; the partial sums of a row's segments meet in
// shared memory (slot i).
constexpr int MG_MAX_P = 192;  // items of one block in one phase
__host__ __device__ __forceinline__ unsigned block_groups(const MegaShape& sh, unsigned block, unsigned grid) {
  const unsigned total = sh.type == MG_ATTN ? 0u : sh.grp_start[sh.n_seg];
  return total > block ? (total - block + grid - 1) / grid : 0u;
}
// global group index of this block's k-th group
__device__ __forceinline__ unsigned block_group_id(unsigned k) { return blockIdx.x + k * gridDim.x; }
// jobs in front of a phase's row groups: two vectors of norm weights
__host__ __device__ __forceinline__ unsigned norm_jobs(int kind) { return kind == PH_QKV || kind == PH_GATEUP ? 1u : 0u; }
__host__ __device__ __forceinline__ unsigned job_bytes(const MegaShape& sh, bool norm, unsigned hidden) {
  return norm ? 8u * hidden : sh.mats * MG_RL * sh.row_bytes;
}
// The ring: jobs lie one behind the other and leave in that order.  None wraps: one that does not fit behind the last starts over,
// and the bytes it passes by are its own until it leaves.  Where a job lies depends on the shape and the block, never on timing.
struct MegaRing {
  unsigned bytes, at, used;
  __host__ __device__ unsigned takes(unsigned room) const { return at + room > bytes ? bytes - at + room : room; }
  __host__ __device__ bool fits(unsigned taken) const { return used + taken <= bytes; }
  __host__ __device__ unsigned put(unsigned room, unsigned taken) {
    const unsigned place = at + room > bytes ? 0u : at;
    at = place + room;
    used += taken;
    return place;
  }
  __host__ __device__ void drop(unsigned taken) {
    used -= taken;
    if (used == 0) at = 0;  // start over, or a job of more than half the ring might never fit
  }
};
// arrivals of item cs of a job with C items
__device__ __forceinline__ unsigned empty_share(unsigned cs, unsigned C) { return cs == 0 ? MG_EMPTY - C + 1u : 1u; }

// ---- attention phase ------------------------------------------------------------------------------
constexpr float kNegInit = -1.0e30f;

__device__ __forceinline__ float mg_warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float mg_warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Q4_0 pack of 32 values held one per lane (render.rs:1021-1059); blk is 2-byte aligned.
__device__ __forceinline__ void mg_pack_q40(float v, uint8_t* blk, int lane) {
  const float amax = mg_warp_max(fabsf(v));
  const float scale = amax > 0.0f ? amax / 7.0f : 1.0f;
  const float inv = 1.0f / scale;
  int q = (int)roundf(__fmul_rn(v, inv)) + 8;
  q = q < 0 ? 0 : q > 15 ? 15 : q;
  const int qhi = __shfl_down_sync(0xffffffffu, q, 16);
  if (lane < 16) blk[2 + lane] = (uint8_t)(q | (qhi << 4));
  if (lane == 0) *reinterpret_cast<__half*>(blk) = __float2half_rn(scale);
}

// This lane's share of one Q4_0 row, still packed: DPL/4 16-bit words of nibbles and the scale.
template <int DPL>
struct RawRow {
  unsigned short q[DPL / 4];
  unsigned short d;
};
template <int DPL>
__device__ __forceinline__ void raw_load(const uint8_t* row, int lane, RawRow<DPL>& r) {
  constexpr int BPL = DPL / 2, LPB = 16 / BPL;
  const uint8_t* blk = row + (lane / LPB) * KS_Q40_BLOCK_BYTES;
  r.d = *reinterpret_cast<const unsigned short*>(blk);
  const unsigned short* qs = reinterpret_cast<const unsigned short*>(blk + 2 + (lane % LPB) * BPL);
#pragma unroll
  for (int w = 0; w < BPL / 2; w++) r.q[w] = qs[w];
}
// Its values n - 8, each times the power of two its nibble sits at (q comes divided by it, o is divided by it at the end): a mask
// and an OR make the float 2^23 + n 2^k, a subtraction the rest, all exact.  The block's scale is applied to the sums.
template <int DPL>
__device__ __forceinline__ constexpr float raw_unit(int j) {
  constexpr int BPL = DPL / 2;
  return (j < BPL ? 1.0f : 16.0f) * (j & 1 ? 256.0f : 1.0f);
}
template <int DPL>
__device__ __forceinline__ void raw_ints(const RawRow<DPL>& r, float (&out)[DPL]) {
  constexpr int BPL = DPL / 2;
#pragma unroll
  for (int j = 0; j < DPL; j++) {
    const unsigned v = r.q[(j % BPL) / 2], mask = 0xFu * (unsigned)raw_unit<DPL>(j);
    out[j] = __uint_as_float((v & mask) | 0x4B000000u) - (8388608.0f + 8.0f * raw_unit<DPL>(j));
  }
}
template <int DPL>
__device__ __forceinline__ float raw_scale(const RawRow<DPL>& r) { return __half2float(__ushort_as_half(r.d)); }
template <int DPL>
__device__ __forceinline__ int mg_lane_dim(int lane, int j) {
  constexpr int BPL = DPL / 2, LPB = 16 / BPL;
  const int base = (lane / LPB) * 32 + (lane % LPB) * BPL;
  return j < BPL ? base + j : base + 16 + (j - BPL);
}

__host__ __device__ constexpr unsigned mg_rec(unsigned hd) { return hd + 4u; }  // floats of a record: O[hd], m, l, two unused
constexpr int MG_MAX_SPLITS = 18;  // context splits per head (the final merge keeps one record per split in registers)
constexpr int MG_FLY = 4;  // positions of a warp in flight
// Up to MG_DIRECT splits are merged by every block while it stages the o-projection's input (mg_stage_merge): no block waits for
// another one's merge, and a block reads at most n_q x 4 records (2.0 us of staging instead of 0.8).  From the second batch of
// positions per warp on (4 x 60) the eighteen win.  A token at 200 / 300 / 500 / 1000 / 2000 positions, four splits: E2B 943 / 984 / 1024 /
// 1131 / 1334 us, E4B 1516 / 1565 / 1612 / 1738 / 2020; all eighteen: 984 / 990 / 993 / 1001 / 1055 and 1562 / 1568 / 1572 / 1581 / 1679 (eight,
// merged while staging: 964 / 967 / 994 / 1051 / 1156 and 1543 / 1546 / 1578 / 1645 / 1775).  E2B at 64..128: one split 1017, two 1003, four 998.
constexpr unsigned MG_DIRECT = 4, MG_SINGLE_TLEN = MG_FLY * MG_WARPS, MG_DIRECT_TLEN = 320;

// Shared memory the attention phase needs (it reuses the x staging area).
__host__ __device__ inline unsigned mg_att_bytes(unsigned hd) {
  return MG_WARPS * (hd + 2u) * 4u + hd * 4u + 2u * ((hd / 32u) * KS_Q40_BLOCK_BYTES + 16u) + 32u;
}

// Splits in use for a context of tlen positions: one block per head while its warps get by with a few rows each, a few that every
// block merges for itself, then all of them and a merge by the head's last block.
__host__ __device__ inline unsigned mg_active_splits(unsigned tlen, unsigned max_splits) {
  const unsigned ns = tlen <= MG_SINGLE_TLEN ? 1u : tlen <= MG_DIRECT_TLEN ? MG_DIRECT : max_splits;
  return ns < max_splits ? ns : max_splits;
}
// The positions a layer attends to: [first, pos].
__device__ __forceinline__ unsigned mg_first(const MegaLayer& L, unsigned pos) {
  const unsigned win = (unsigned)L.window;
  return win && pos + 1u > win ? pos + 1u - win : 0u;
}
// A run of bytes into L2, as far as whole 16-byte pieces of it go.
__device__ __forceinline__ void l2_prefetch(const void* p, size_t bytes) {
  const uintptr_t a = ((uintptr_t)p + 15u) & ~(uintptr_t)15u, e = ((uintptr_t)p + bytes) & ~(uintptr_t)15u;
  if (e > a) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((unsigned)(e - a)) : "memory");
}
// The weights of a token push everything else out of L2 (they are five times its size), so the cached rows a layer's attention
// reads are asked for a phase or more ahead; one thread per block, each split's rows once.
__device__ __forceinline__ void mg_prefetch_kv(const MegaArgs& a, const MegaLayer& L, unsigned pos) {
  const unsigned NSMAX = a.n_splits, first = mg_first(L, pos), tlen = pos + 1u - first;
  const unsigned NS = mg_active_splits(tlen, NSMAX), split = blockIdx.x % NSMAX, head = blockIdx.x / NSMAX;
  if (head == 0 && split < NS) {
    const unsigned chunk = (tlen + NS - 1) / NS, p0 = first + split * chunk, p1 = min(p0 + chunk, pos);
    const size_t row = (size_t)a.n_kv * (a.hd / 32u) * KS_Q40_BLOCK_BYTES;
    if (p0 < p1) {
      l2_prefetch(L.kv_k + p0 * row, (p1 - p0) * row);
      l2_prefetch(L.kv_v + p0 * row, (p1 - p0) * row);
    }
  }
  if (blockIdx.x >= gridDim.x - 2u) l2_prefetch(L.norm[gridDim.x - blockIdx.x], a.hd * 4u);  // the head norms
}

// One block per (query head, context split): the work of a short context is tiny, so it is spread
// as widely as the grid allows and every serial step stays short.
//   1. one warp polls for the head's q and leaves it roped, normed and scaled in shared memory; in the blocks of the split that
//      holds the newest position, four others pack the new K row and four the new V row to Q4_0 in shared memory
//      (lower.rs:4231-4702), block pairs (b, b+NB/2) per warp because RoPE pairs those halves; the block of the KV group's
//      first head stores them;
//   2. warps take the positions of the split round-robin, online softmax per warp;
//   3. the warps' (m, l, O) meet in shared memory, thread d folds dimension d;
//   4. the block leaves a (m, l, O[hd]) record; few records of a head are merged by their readers, more by the last block of
//      the head to arrive (lower.rs:5897-6088).
template <int DPL>
__device__ __forceinline__ void mg_attention(const MegaArgs& a, const MegaLayer& L, unsigned char* sm, int* sflag, long long* pf,
                                             unsigned tag, unsigned pos) {
  const unsigned tid = mg_tid();
  constexpr int HD = DPL * 32, HALF = HD / 2, NB = HD / 32;
  constexpr unsigned ROWB = NB * KS_Q40_BLOCK_BYTES;
  const int lane = tid & 31, warp = tid >> 5;
  const unsigned NSMAX = a.n_splits;
  if (blockIdx.x >= a.n_q * NSMAX) return;
  const unsigned head = blockIdx.x / NSMAX, split = blockIdx.x % NSMAX;
  const unsigned G = a.n_q / a.n_kv, kvh = head / G;
  const unsigned first = mg_first(L, pos), tlen = pos + 1u - first;
  const unsigned NS = mg_active_splits(tlen, NSMAX);
  if (split >= NS) return;
  const unsigned chunk = (tlen + NS - 1) / NS;
  const unsigned p0 = first + split * chunk, p1 = min(p0 + chunk, pos + 1u);
  const bool owner = pos >= p0 && pos < p1;  // the split that holds the newest position
  float* part = reinterpret_cast<float*>(sm);     // [MG_WARPS][HD + 2]
  float* sq = part + MG_WARPS * (HD + 2);         // the head's q
  uint8_t* skrow = reinterpret_cast<uint8_t*>(sq + HD);
  uint8_t* svrow = skrow + ROWB + 16u;
  const float* cs = a.rope + (size_t)pos * HD;
  const size_t rowstride = (size_t)a.n_kv * ROWB;
  uint8_t* Kc = L.kv_k + (size_t)kvh * ROWB;
  uint8_t* Vc = L.kv_v + (size_t)kvh * ROWB;
  // MG_FLY positions of this warp at a time (t, t + MG_WARPS, ...): K of the next ones is asked for as soon as the scores are
  // there, V once it is summed, and the first do not wait for q.  (One position at a time, its successor in flight: 640 ns a
  // position; 250 positions a block took 20 us.)
  constexpr int FLY = MG_FLY;
  RawRow<DPL> kn[FLY], vn[FLY];
  auto row_at = [&](unsigned t, int i) { return min(t + MG_WARPS * i, p1 - 1u); };  // past the split's end: loaded, not used
  auto load_rows = [&](unsigned t, RawRow<DPL>(&r)[FLY], const uint8_t* cache, const uint8_t* newest) {
#pragma unroll
    for (int i = 0; i < FLY; i++) {
      const unsigned p = row_at(t, i);
      raw_load<DPL>(p == pos ? newest : cache + (size_t)p * rowstride, lane, r[i]);
    }
  };
  unsigned t = p0 + warp;
  load_rows(t, kn, Kc, skrow);
  load_rows(t, vn, Vc, svrow);

  const int pb = (warp - 1) & 3;  // block pair of the K / V job
  const bool kjob = owner && warp >= 1 && warp < 5 && pb < NB / 2, vjob = owner && warp >= 5 && warp < 9 && pb < NB / 2;
  if (warp == 0) {
    float qv[DPL], qw[DPL], qc[DPL], qs[DPL];
    const float* qnw = L.norm[1];
#pragma unroll
    for (int j = 0; j < DPL; j++) {  // constants first: they are on their way while the tagged words are polled
      const int d = mg_lane_dim<DPL>(lane, j);
      qw[j] = qnw[d];
      qc[j] = cs[d & (HALF - 1)];
      qs[j] = cs[HALF + (d & (HALF - 1))];
    }
    // q (and, in the owner split, k / v) arrive as tagged words straight from the blocks that computed them
    int at[DPL];
#pragma unroll
    for (int j = 0; j < DPL; j++) at[j] = mg_lane_dim<DPL>(lane, j);
    const bool got = tag_wait<DPL>(a.qkv_t + (size_t)head * HD, at, tag, a.poll_limit, qv);
    if (!got) atomicOr(a.err, 2u);  // a tagged word never came: the values are zeros, the status word tells the host
    float ss = 0.0f;
#pragma unroll
    for (int j = 0; j < DPL; j++) ss = fmaf(qv[j], qv[j], ss);
    ss = mg_warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)HD + a.eps);
    // lanes 0..15 hold dims of the first half, lanes 16..31 their RoPE partners (dim + HD/2)
#pragma unroll
    for (int j = 0; j < DPL; j++) {
      const float u = __fmul_rn(__fmul_rn(qv[j], inv), qw[j]);
      const float pu = __shfl_xor_sync(0xffffffffu, u, 16);
      const float r = lane < 16 ? __fsub_rn(__fmul_rn(u, qc[j]), __fmul_rn(pu, qs[j]))
                                : __fadd_rn(__fmul_rn(pu, qs[j]), __fmul_rn(u, qc[j]));
      sq[mg_lane_dim<DPL>(lane, j)] = r * a.attn_scale;
    }
  } else if (kjob || vjob) {
    float rv[DPL], r_w0 = 0.f, r_w1 = 0.f, r_c = 0.f, r_s = 0.f;
    if (kjob) {
      const float* w = L.norm[2];
      r_w0 = w[32 * pb + lane];
      r_w1 = w[HALF + 32 * pb + lane];
      r_c = cs[32 * pb + lane];
      r_s = cs[HALF + 32 * pb + lane];
    }
    const unsigned long long* src = a.qkv_t + (size_t)a.n_q * HD + (kjob ? 0u : (size_t)a.n_kv * HD) + (size_t)kvh * HD;
    int at[DPL];
#pragma unroll
    for (int j = 0; j < DPL; j++) at[j] = lane + 32 * j;
    const bool got = tag_wait<DPL>(src, at, tag, a.poll_limit, rv);
    if (!got) atomicOr(a.err, 2u);
    float ss = 0.0f;
#pragma unroll
    for (int j = 0; j < DPL; j++) ss = fmaf(rv[j], rv[j], ss);
    ss = mg_warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)HD + a.eps);
    float x0 = 0.f, x1 = 0.f;  // this lane's element of block pb and of block pb + NB/2
#pragma unroll
    for (int j = 0; j < DPL / 2; j++)
      if (j == pb) {
        x0 = rv[j];
        x1 = rv[j + DPL / 2];
      }
    float lo, hi;
    if (kjob) {
      const float u = __fmul_rn(__fmul_rn(x0, inv), r_w0), vv = __fmul_rn(__fmul_rn(x1, inv), r_w1);
      lo = __fsub_rn(__fmul_rn(u, r_c), __fmul_rn(vv, r_s));
      hi = __fadd_rn(__fmul_rn(u, r_s), __fmul_rn(vv, r_c));
    } else {
      lo = __fmul_rn(x0, inv);
      hi = __fmul_rn(x1, inv);
    }
    uint8_t* dst = kjob ? skrow : svrow;
    // values pass through f16 before packing (render.rs:1046)
    mg_pack_q40(__half2float(__float2half_rn(lo)), dst + pb * KS_Q40_BLOCK_BYTES, lane);
    mg_pack_q40(__half2float(__float2half_rn(hi)), dst + (pb + NB / 2) * KS_Q40_BLOCK_BYTES, lane);
  }
  cta_sync();
  float qr[DPL];
#pragma unroll
  for (int j = 0; j < DPL; j++) qr[j] = sq[mg_lane_dim<DPL>(lane, j)] * (1.0f / raw_unit<DPL>(j));
  if (owner) {
    if (head == kvh * G) {
      const unsigned n16 = ROWB / 2;
      if (tid < n16)
        reinterpret_cast<unsigned short*>(Kc + (size_t)pos * rowstride)[tid] = reinterpret_cast<const unsigned short*>(skrow)[tid];
      else if (tid < 2 * n16)
        reinterpret_cast<unsigned short*>(Vc + (size_t)pos * rowstride)[tid - n16] =
            reinterpret_cast<const unsigned short*>(svrow)[tid - n16];
    }
  }
  if (pf) pf[4] = clock64();

  float o[DPL], m = kNegInit, l = 0.0f;
#pragma unroll
  for (int j = 0; j < DPL; j++) o[j] = 0.0f;
  if (owner && t < p1) {  // the row packed above
#pragma unroll
    for (int i = 0; i < FLY; i++)
      if (row_at(t, i) == pos) {
        raw_load<DPL>(skrow, lane, kn[i]);
        raw_load<DPL>(svrow, lane, vn[i]);
      }
  }
#pragma unroll 1
  for (; t < p1; t += MG_WARPS * FLY) {
    float kv[DPL], sc[FLY], m2 = m;
#pragma unroll
    for (int i = 0; i < FLY; i++) {
      raw_ints<DPL>(kn[i], kv);
      sc[i] = 0.0f;
#pragma unroll
      for (int j = 0; j < DPL; j++) sc[i] = fmaf(qr[j], kv[j], sc[i]);
      sc[i] *= raw_scale<DPL>(kn[i]);
    }
    const bool more = t + MG_WARPS * FLY < p1;
    if (more) load_rows(t + MG_WARPS * FLY, kn, Kc, skrow);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
      for (int i = 0; i < FLY; i++) sc[i] += __shfl_xor_sync(0xffffffffu, sc[i], off);
#pragma unroll
    for (int i = 0; i < FLY; i++) {
      sc[i] = t + MG_WARPS * i < p1 ? sc[i] : -INFINITY;
      m2 = fmaxf(m2, sc[i]);
    }
    const float alpha = __expf(m - m2);
    l *= alpha;
    m = m2;
#pragma unroll
    for (int j = 0; j < DPL; j++) o[j] *= alpha;
#pragma unroll
    for (int i = 0; i < FLY; i++) {
      if (t + MG_WARPS * i >= p1) break;
      const float e = __expf(sc[i] - m2);
      l += e;
      raw_ints<DPL>(vn[i], kv);
      const float ed = e * raw_scale<DPL>(vn[i]);
#pragma unroll
      for (int j = 0; j < DPL; j++) o[j] = fmaf(ed, kv[j], o[j]);
    }
    if (more) load_rows(t + MG_WARPS * FLY, vn, Vc, svrow);
  }
  {
    float* dst = part + warp * (HD + 2);
    if (lane == 0) {
      dst[0] = m;
      dst[1] = l;
    }
#pragma unroll
    for (int j = 0; j < DPL; j++) dst[2 + j * 32 + lane] = o[j] * (1.0f / raw_unit<DPL>(j));
  }
  cta_sync();
  if (pf) pf[5] = clock64();
  // thread d folds head dimension d over the warps; it sits in slot j * 32 + lane of the warps' layout
  const int d = tid;
  int dslot;
  {
    constexpr int BPL = DPL / 2, LPB = 16 / BPL;
    const int within = d & 31, hh = within >> 4, w16 = within & 15;
    dslot = (hh * BPL + (w16 % BPL)) * 32 + ((d >> 5) * LPB + w16 / BPL);
  }
  float M = kNegInit, Lsum = 0.0f, O = 0.0f;
  if (d < HD) {
    float mw[MG_WARPS];
#pragma unroll
    for (unsigned w = 0; w < MG_WARPS; w++) {
      mw[w] = part[w * (HD + 2)];
      M = fmaxf(M, mw[w]);
    }
#pragma unroll
    for (unsigned w = 0; w < MG_WARPS; w++) {
      const float f = __expf(mw[w] - M);
      Lsum = fmaf(part[w * (HD + 2) + 1], f, Lsum);
      O = fmaf(part[w * (HD + 2) + 2 + dslot], f, O);
    }
  }
  if (pf) pf[6] = clock64();
  const unsigned ounits = (a.n_q * HD) >> 6;
  if (NS == 1) {  // one split: this block's result is final
    if (d < HD) fx_store_subblock(a.ox, ounits, head * HD + (d & ~31), O / Lsum, lane);
    return;
  }
  float* rec = a.att_tmp + ((size_t)head * NSMAX + split) * mg_rec(HD);
  if (d < HD) {
    rec[d] = O;  // records are kept in dimension order
    if (d == 0) {
      rec[HD] = M;
      rec[HD + 1] = Lsum;
    }
  }
  if (NS <= MG_DIRECT) return;  // merged by whoever reads them, behind the grid barrier
  __threadfence();
  cta_sync();
  if (tid == 0) *sflag = (atomicAdd(a.att_cnt + head, 1u) == NS - 1) ? 1 : 0;
  cta_sync();
  if (pf) pf[7] = clock64();
  if (*sflag) {
    // last block of this head to arrive: merge the head's records, every load first
    __threadfence();
    if (d < HD) {
      const float* rec0 = a.att_tmp + (size_t)head * NSMAX * mg_rec(HD);
      float mp[MG_MAX_SPLITS], lp[MG_MAX_SPLITS], ov[MG_MAX_SPLITS];
#pragma unroll
      for (int p = 0; p < MG_MAX_SPLITS; p++) {
        if ((unsigned)p < NS) {
          const float* r = rec0 + (size_t)p * mg_rec(HD);
          const float2 u = __ldcg(reinterpret_cast<const float2*>(r + HD));
          mp[p] = u.x;
          lp[p] = u.y;
          ov[p] = __ldcg(r + d);
        } else {
          mp[p] = kNegInit;
          lp[p] = 0.0f;
          ov[p] = 0.0f;
        }
      }
      float MM = kNegInit;
#pragma unroll
      for (int p = 0; p < MG_MAX_SPLITS; p++) MM = fmaxf(MM, mp[p]);
      float LL = 0.0f, OO = 0.0f;
#pragma unroll
      for (int p = 0; p < MG_MAX_SPLITS; p++) {
        const float f = __expf(mp[p] - MM);
        LL = fmaf(lp[p], f, LL);
        OO = fmaf(ov[p], f, OO);
      }
      fx_store_subblock(a.ox, ounits, head * HD + (d & ~31), OO / LL, lane);
    }
    if (tid == 0) a.att_cnt[head] = 0u;
  }
}

// The o-projection's input out of the records of at most MG_DIRECT splits: each thread merges four neighbouring dims of a head at
// a time, every load first.
__device__ __forceinline__ void mg_stage_merge(unsigned char* xs, const MegaArgs& a, unsigned NS, unsigned cols) {
  const unsigned tid = mg_tid();
  const unsigned units = cols >> 6, nchunk = cols >> 2, rec_len = mg_rec(a.hd);
  for (unsigned c = tid; c < nchunk; c += MG_THREADS) {  // (whole warps: nchunk is a multiple of 128)
    const unsigned head = (c << 2) / a.hd, d = (c << 2) - head * a.hd;
    const float* rec = a.att_tmp + (size_t)head * a.n_splits * rec_len;
    float2 ml[MG_DIRECT];
    float4 o[MG_DIRECT];
#pragma unroll
    for (unsigned s = 0; s < MG_DIRECT; s++) {
      const float* r = rec + s * rec_len;
      ml[s] = s < NS ? __ldcg(reinterpret_cast<const float2*>(r + a.hd)) : make_float2(kNegInit, 0.0f);
      o[s] = s < NS ? __ldcg(reinterpret_cast<const float4*>(r + d)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    float M = kNegInit, Ls = 0.0f;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (unsigned s = 0; s < MG_DIRECT; s++) M = fmaxf(M, ml[s].x);
#pragma unroll
    for (unsigned s = 0; s < MG_DIRECT; s++) {
      const float f = __expf(ml[s].x - M);
      Ls = fmaf(ml[s].y, f, Ls);
      v.x = fmaf(o[s].x, f, v.x);
      v.y = fmaf(o[s].y, f, v.y);
      v.z = fmaf(o[s].z, f, v.z);
      v.w = fmaf(o[s].w, f, v.w);
    }
    const float inv = 1.0f / Ls;
    v.x *= inv; v.y *= inv; v.z *= inv; v.w *= inv;
    fx_put_chunk(xs, units, c, v);
  }
}

// ---- the kernel -------------------------------------------------------------------------------------
// Shared memory: what has a fixed size first, so that its addresses are constants; then the tables, x (and the attention
// scratch) and the ring.
constexpr unsigned SM_BAR = 0, SM_RED = SM_BAR + 2u * MG_JOBS * 8u,    // per job: its rows are there; its items are done
                   SM_WSUM = SM_RED + 256u, SM_PSUM = SM_WSUM + MG_WARPS * 16u,
                   SM_FLAG = SM_PSUM + MG_MAX_P * 32u,                 // 4 flag words, the copying warp's stop word, 8 words of group counts
                   SM_JOB = SM_FLAG + 64u,                             // a job's place in the ring; bytes it takes there
                   SM_TAB = SM_JOB + 2u * MG_JOBS * 4u;
constexpr unsigned SM_LAYERS = SM_TAB + ((PH_PER_LAYER * (unsigned)sizeof(MegaShape) + 15u) & ~15u);
static_assert(SM_TAB % 16u == 0 && SM_PSUM % 16u == 0, "vector access");

// One thread copies the row groups of the whole token in the order they are multiplied, as far ahead as the ring has room.
__device__ __forceinline__ void mg_copy_jobs(const MegaArgs& a, const MegaShape* shapes, const MegaLayer* layers, const unsigned* ngrp, uint32_t ring_s,
                                             uint32_t full, uint32_t empty, unsigned* joff, unsigned* jbytes, volatile int* stop, unsigned H, unsigned pos) {
  unsigned head = 0, tail = 0;
  MegaRing ring{a.ring_bytes, 0u, 0u};
  for (int layer = 0; layer < a.n_layers; layer++) {
    const MegaLayer& L = layers[layer];
    mg_prefetch_kv(a, L, pos);
    for (int kind = 0; kind < PH_PER_LAYER; kind++) {
      const MegaShape& sh = shapes[kind];
      const unsigned n = ngrp[kind], row_bytes = sh.row_bytes, mats = sh.mats;
      // in front of a phase that stages a norm: its weights, those of the norm inside the residual update behind them
      const unsigned norms = norm_jobs(kind);
      for (unsigned kk = 0; kk < n + norms; kk++) {
        const bool norm = kk < norms;
        const unsigned k = kk - norms, g = norm ? 0u : block_group_id(k);
        unsigned seg = 0;
        if (sh.n_seg > 1 && g >= sh.grp_start[1]) seg = 1;
        if (sh.n_seg > 2 && g >= sh.grp_start[2]) seg = 2;
        const unsigned row0 = (g - sh.grp_start[seg]) * MG_RL, valid = min((unsigned)MG_RL, sh.rows[seg] - row0);
        const unsigned room = job_bytes(sh, norm, H);
        unsigned taken = ring.takes(room);
        while (head - tail >= MG_JOBS || !ring.fits(taken)) {
          const uint32_t bar = empty + (tail & (MG_JOBS - 1u)) * 8u;
          const unsigned parity = (tail / MG_JOBS) & 1u;
          bool ok = false;
          for (unsigned i = 0; i < (1u << 22) && !ok && !*stop; i++) {
            unsigned r;
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(r)
                : "r"(bar), "r"(parity)
                : "memory");
            ok = r != 0;
          }
          if (!ok) {
            if (!*stop) atomicOr(a.err, 1u);
            goto out;
          }
          ring.drop(jbytes[tail & (MG_JOBS - 1u)]);
          tail++;
          if (ring.used == 0) taken = room;
        }
        const unsigned b = head & (MG_JOBS - 1u), at = ring.put(room, taken);
        joff[b] = at;
        jbytes[b] = taken;
        mb_expect(full + b * 8u, norm ? room : mats * valid * row_bytes);  // (its arrival publishes joff)
        if (norm) {
          bulk_in(ring_s + at, kind == PH_QKV ? L.norm[0] : L.norm[4], 4u * H, full + b * 8u);
          // (the first layer has no residual update in front of it: any weights)
          bulk_in(ring_s + at + 4u * H, kind == PH_QKV ? layers[max(layer - 1, 0)].norm[5] : L.norm[3], 4u * H, full + b * 8u);
        }
        for (unsigned m = 0; m < mats && !norm; m++)
          bulk_in(ring_s + at + m * MG_RL * row_bytes, L.W[sh.w0 + seg + m] + (size_t)row0 * row_bytes, valid * row_bytes, full + b * 8u);
        head++;
      }
    }
  }
out:
  // copies still in flight must land before this block's shared memory goes away (bounded)
  for (unsigned j = tail; j < head; j++) mb_wait(full + (j & (MG_JOBS - 1u)) * 8u, (j / MG_JOBS) & 1u);
}

template <int DPL, int PC>
__global__ void __launch_bounds__(MG_THREADS + 32, 1) mega_kernel(const MegaArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const uint32_t ring_s = sm32(smem) + a.ring_off, full = sm32(smem) + SM_BAR, empty = full + MG_JOBS * 8u, xs_s = sm32(smem) + a.x_off;
  unsigned char* xs = smem + a.x_off;
  float* red = reinterpret_cast<float*>(smem + SM_RED);
  float4* wsum = reinterpret_cast<float4*>(smem + SM_WSUM);
  float* psum = reinterpret_cast<float*>(smem + SM_PSUM);
  int* sflag = reinterpret_cast<int*>(smem + SM_FLAG);
  volatile int* stop = sflag + 4;
  unsigned* ngrp = reinterpret_cast<unsigned*>(smem + SM_FLAG + 32u);  // this block's group count per phase kind
  unsigned* joff = reinterpret_cast<unsigned*>(smem + SM_JOB);
  const MegaShape* shapes = reinterpret_cast<const MegaShape*>(smem + SM_TAB);
  const MegaLayer* layers = reinterpret_cast<const MegaLayer*>(smem + SM_LAYERS);
  const unsigned bar_base = a.bar[1];
  const int n_phases = a.n_layers * PH_PER_LAYER;
  // tag of this token's words: position and layer; a slot reset clears the words, so a replayed position never
  // meets its own old tags
  const unsigned pos = (unsigned)a.pos[0], tag_base = ((pos + 1u) << 8) + 1u;

  for (unsigned i = threadIdx.x; i < a.tables_bytes / 16u; i += blockDim.x)
    reinterpret_cast<uint4*>(smem + SM_TAB)[i] = reinterpret_cast<const uint4*>(a.tables)[i];
  if (threadIdx.x < MG_JOBS) {
    mb_init(full + threadIdx.x * 8u, 1);
    mb_init(empty + threadIdx.x * 8u, MG_EMPTY);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (threadIdx.x == 0) {
    sflag[2] = sflag[3] = 0;  // barrier flag words ([0] belongs to the attention phase)
    *stop = 0;
  }
  __syncthreads();
  if (threadIdx.x < PH_PER_LAYER) ngrp[threadIdx.x] = block_groups(shapes[threadIdx.x], blockIdx.x, gridDim.x);
  __syncthreads();
  const unsigned hidden = shapes[PH_QKV].cols;
  if (threadIdx.x >= MG_THREADS) {
    if (threadIdx.x == MG_THREADS) mg_copy_jobs(a, shapes, layers, ngrp, ring_s, full, empty, joff, joff + MG_JOBS, stop, hidden, pos);
    return;
  }

  bool dead = false;  // this warp gave up (a copy never landed): it keeps the block-level steps only
  unsigned job0 = 0;  // jobs of the phases before this one
  long long* prof = nullptr;
  if (threadIdx.x == 0 && (blockIdx.x == 0 || blockIdx.x == gridDim.x - 1))
    prof = a.prof + (size_t)(blockIdx.x == 0 ? 0 : 1) * n_phases * 8;
  int p = 0, layer = 0, kind = 0;
  for (; p < n_phases; p++) {
    unsigned H = hidden;
    asm volatile("" : "+r"(H));
    const unsigned tid = mg_tid();
    const int lane = (int)(tid & 31u), warp = (int)(tid >> 5), cl = lane % MG_LPR, rl = lane / MG_LPR;
    const MegaLayer& L = layers[layer];
    // No barrier in front of attention: its inputs are tagged words.  Every block still ARRIVES after every phase,
    // so the targets of the barriers that remain are unchanged; the flag word this wait would have cleared is
    // cleared all the same.
    if (p > 0 && kind == PH_ATTN) {
      if (tid == 0) sflag[2 + ((p & 1) ^ 1)] = 0;
    } else if (p > 0) {
      if (!grid_wait(a.bar, bar_base + (unsigned)p * gridDim.x + (p == 2 ? a.test_stall : 0u), a.err, sflag + 2, p & 1, a.poll_limit)) break;
      if (prof) prof[(p - 1) * 8 + 3] = clock64();
    }
    if (prof) prof[p * 8 + 0] = clock64();
    unsigned n_wsum = 0;
    if (kind == PH_ATTN) {
      mg_attention<DPL>(a, L, xs, sflag, prof ? prof + p * 8 : nullptr, tag_base + (unsigned)layer, pos);
    } else {
      const MegaShape& sh = shapes[kind];
      // o-proj and down feed a residual-add + norm: their rows also leave the sums that norm needs
      const bool sums = kind == PH_OPROJ || kind == PH_DOWN;
      // Thread f finishes row (f & 3) of this block's group (f >> 2): it adds the column segments'
      // partial sums in order, applies the epilogue and stores the row.
      const unsigned n_g = ngrp[kind], C = sh.n_cseg;
      unsigned frow = 0;
      int fseg = 0;
      bool fin = false;
      float xr = 0.0f, wpr = 0.0f;
      if ((tid >> 2) < n_g) {
        const unsigned g = block_group_id(tid >> 2);
        if (sh.n_seg > 1 && g >= sh.grp_start[1]) fseg = 1;
        if (sh.n_seg > 2 && g >= sh.grp_start[2]) fseg = 2;
        frow = (g - sh.grp_start[fseg]) * MG_RL + (tid & 3u);
        fin = frow < sh.rows[fseg];
        if (fin && sums) {  // in flight while x is staged
          xr = __ldcg((kind == PH_OPROJ ? a.x_a : a.x_b) + frow);
          wpr = (kind == PH_OPROJ ? L.norm[3] : L.norm[5])[frow];
        }
      }
      unsigned ik = (unsigned)warp / C, ics = (unsigned)warp - ik * C;  // this warp's first item
      const unsigned dk = MG_WARPS / C, dcs = MG_WARPS - dk * C;        // from one to the next
      // input and prologue of this phase
      const unsigned ns_att = mg_active_splits(pos + 1u - mg_first(L, pos), a.n_splits);
      const unsigned nb = job0 & (MG_JOBS - 1u);
      if (norm_jobs(kind)) {
        if (!dead && !mb_wait(full + nb * 8u, (job0 / MG_JOBS) & 1u)) {
          dead = true;
          if (lane == 0) atomicOr(a.err, 1u);
        }
        const float4* w = reinterpret_cast<const float4*>(smem + a.ring_off + (dead ? 0u : joff[nb]));
        if (layer == 0 && kind == PH_QKV)
          mg_stage_norm<PC>(xs, red, H, a.x_a, a.eps, w);
        else
          mg_stage_addnorm<PC>(xs, red, H, kind == PH_QKV ? a.x_b : a.x_a, a.yb, kind == PH_QKV ? a.x_a : a.x_b, a.eps, w, w + H / 4u, a.nsum, gridDim.x);
      } else if (kind == PH_DOWN)
        mg_stage_plain(xs, sh.cols, a.ff);
      else if (ns_att > 1u && ns_att <= MG_DIRECT)
        mg_stage_merge(xs, a, ns_att, sh.cols);
      else
        fx_copy_in(xs, a.ox, sh.cols >> 6);
      cta_sync();
      if (norm_jobs(kind)) {
        if (tid == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(empty + nb * 8u), "n"(MG_EMPTY) : "memory");
        job0++;
      }
      if (prof) prof[p * 8 + 1] = clock64();
      const unsigned units = sh.cols >> 6;
      for (unsigned i = (unsigned)warp; ik < n_g && !dead; i += MG_WARPS) {
        const unsigned cs = ics, job = job0 + ik, b = job & (MG_JOBS - 1u);
        ik += dk;
        ics += dcs;
        if (ics >= C) {
          ics -= C;
          ik++;
        }
        if (!mb_wait(full + b * 8u, (job / MG_JOBS) & 1u)) {
          dead = true;
          if (lane == 0) atomicOr(a.err, 1u);
          break;
        }
        const uint32_t slot = ring_s + joff[b];
        float yacc[2] = {0.0f, 0.0f};
        if (kind == PH_GATEUP)
          mg_item_compute_fx<2>(slot, sh.row_bytes, xs_s, units, sh.seg_blocks, cs, cl, rl, yacc);
        else
          mg_item_compute_fx<1>(slot, sh.row_bytes, xs_s, units, sh.seg_blocks, cs, cl, rl, yacc);
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(empty + b * 8u), "r"(empty_share(cs, C)) : "memory");
        float v0 = yacc[0], v1 = yacc[1];
#pragma unroll
        for (int o = MG_LPR / 2; o > 0; o >>= 1) {
          v0 += __shfl_xor_sync(0xffffffffu, v0, o);
          v1 += __shfl_xor_sync(0xffffffffu, v1, o);
        }
        if (cl == 0) {
          psum[i * 8u + (unsigned)rl] = v0;
          if (kind == PH_GATEUP) psum[i * 8u + 4u + (unsigned)rl] = v1;
        }
      }
      job0 += n_g;
      cta_sync();  // the partial sums of every item of this block are in shared memory
      float ns0 = 0.0f, ns1 = 0.0f, ns2 = 0.0f, ns3 = 0.0f;
      if (fin) {
        const float* ps = psum + (size_t)(tid >> 2) * C * 8u + (tid & 3u);
        float v0 = 0.0f, v1 = 0.0f;
        for (unsigned cs = 0; cs < C; cs++) {
          v0 += ps[cs * 8u];
          if (kind == PH_GATEUP) v1 += ps[cs * 8u + 4u];
        }
        if (kind == PH_QKV) {  // handed to the attention blocks as tagged words (no barrier follows this phase)
          const size_t at = fseg == 0 ? 0u : fseg == 1 ? (size_t)a.n_q * a.hd : (size_t)(a.n_q + a.n_kv) * a.hd;
          tag_store(a.qkv_t + at + frow, v0, tag_base + (unsigned)layer);
        } else if (kind == PH_GATEUP) {
          a.ff[frow] = gelu_mul(v0, v1);
        } else {
          a.yb[frow] = v0;
          const float t = v0 * wpr;
          ns0 = v0 * v0;
          ns1 = xr * t;
          ns2 = t * t;
          ns3 = xr * xr;
        }
      }
      if (sums) {
        n_wsum = n_g ? (n_g * MG_RL + 31u) / 32u : 1u;
        if ((unsigned)warp < n_wsum) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            ns0 += __shfl_xor_sync(0xffffffffu, ns0, o);
            ns1 += __shfl_xor_sync(0xffffffffu, ns1, o);
            ns2 += __shfl_xor_sync(0xffffffffu, ns2, o);
            ns3 += __shfl_xor_sync(0xffffffffu, ns3, o);
          }
          if (lane == 0) wsum[warp] = make_float4(ns0, ns1, ns2, ns3);
        }
      }
    }
    if (prof) prof[p * 8 + 2] = clock64();
    if (p + 1 == n_phases) {  // the end of the kernel orders the last phase before whatever follows
      p++;
      break;
    }
    grid_arrive(a.bar, wsum, n_wsum, a.nsum);
    if (++kind == PH_PER_LAYER) {
      kind = 0;
      layer++;
    }
  }
  if (p == n_phases && blockIdx.x == 0 && threadIdx.x == 0) a.bar[1] = bar_base + (unsigned)(n_phases - 1) * gridDim.x;
  if (p < n_phases || dead) *stop = 1;  // the copying warp need not wait for the rest to be used
}

}  // namespace

// ---- host side --------------------------------------------------------------------------------------
struct ks_mega {
  MegaArgs args{};
  void* d_tables = nullptr;
  unsigned* d_sync = nullptr;  // words 0..1 barrier (a 128-byte line of its own: every block polls it), 64..111 per-head
                               // attention arrival counters, from byte 512: per-block norm sums
  long long* d_prof = nullptr;
  unsigned long long* d_qkv = nullptr;  // tagged q | k | v words
  size_t qkv_words = 0;
  unsigned char* d_fx = nullptr;  // merged attention output in the staged layout, GeGLU output
  float* d_att = nullptr;         // records of the attention splits
  unsigned grid = 0;
  size_t smem = 0;
  int dpl = 0, pc = 2;  // pc: 4-element chunks of the hidden vector per thread (480 threads)
  float* residual = nullptr;  // buffer that holds the residual stream when the kernel ends
};

namespace {
template <int DPL, int PC>
int mega_launch_t(ks_ctx* ctx, ks_mega* mg) {
  auto kern = mega_kernel<DPL, PC>;
  static size_t smem_set[16] = {0};
  if (mg->smem > smem_set[ctx->device & 15]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mg->smem);
    if (e != cudaSuccess) return ks_fail(ctx, KS_ERR_CUDA, "decode kernel: cannot set %zu B shared memory: %s", mg->smem, cudaGetErrorString(e));
    smem_set[ctx->device & 15] = mg->smem;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(mg->grid);
  cfg.blockDim = dim3(MG_THREADS + 32);
  cfg.dynamicSmemBytes = mg->smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;  // every block resident: the grid barrier needs it
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, mg->args);
  if (e != cudaSuccess) return ks_fail(ctx, KS_ERR_CUDA, "decode kernel launch failed: %s", cudaGetErrorString(e));
  return ks_after_launch(ctx, "decode_layers");
}
}  // namespace

int ks_mega_launch(ks_ctx* ctx, ks_mega* mg) {
  if (mg->dpl == 4) return mg->pc == 1 ? mega_launch_t<4, 1>(ctx, mg) : mg->pc == 2 ? mega_launch_t<4, 2>(ctx, mg) : mega_launch_t<4, 3>(ctx, mg);
  if (mg->dpl == 8) return mg->pc == 1 ? mega_launch_t<8, 1>(ctx, mg) : mg->pc == 2 ? mega_launch_t<8, 2>(ctx, mg) : mega_launch_t<8, 3>(ctx, mg);
  return ks_fail(ctx, KS_ERR_UNSUPPORTED, "decode kernel: head size not supported");
}

float* ks_mega_residual(const ks_mega* mg) { return mg->residual; }

// Zero the barrier words and arrival counters (stream-ordered).  They only leave their rest state when
// a bounded wait gave up; a slot reset puts the kernel back in working order.
int ks_mega_reset(ks_ctx* ctx, ks_mega* mg) {
  cudaError_t e = cudaMemsetAsync(mg->d_sync, 0, 512, ctx->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(mg->d_qkv, 0, mg->qkv_words * sizeof(unsigned long long), ctx->stream);  // no stale tags
  if (e != cudaSuccess) return ks_fail(ctx, KS_ERR_CUDA, "decode kernel: reset failed: %s", cudaGetErrorString(e));
  return KS_OK;
}
const long long* ks_mega_prof(const ks_mega* mg) { return mg->d_prof; }

// Test knobs (the next launch sees them; graphs captured before must be dropped by the caller):
// 0 = polls before a barrier wait gives up, 1 = make the first barrier of a token wait for `value`
// arrivals that never come (exercises the give-up path; 0 switches it off).  2 and 3 belong to the
// dataflow kernel (attention split point, stamps on or off) and are accepted without effect.
int ks_mega_set(ks_mega* mg, int what, unsigned value) {
  if (what == 0) mg->args.poll_limit = value ? value : 1u;
  else if (what == 1) mg->args.test_stall = value;
  else if (what != 2 && what != 3) return KS_ERR_INVALID;
  return KS_OK;
}

void ks_mega_destroy(ks_mega* mg) {
  if (!mg) return;
  if (mg->d_tables) cudaFree(mg->d_tables);
  if (mg->d_sync) cudaFree(mg->d_sync);
  if (mg->d_qkv) cudaFree(mg->d_qkv);
  if (mg->d_prof) cudaFree(mg->d_prof);
  if (mg->d_fx) cudaFree(mg->d_fx);
  if (mg->d_att) cudaFree(mg->d_att);
  delete mg;
}

namespace {
struct MegaPlan {
  MegaShape sh[PH_PER_LAYER];
  unsigned grid, n_splits, tables_bytes, x_off, ring_off, ring_bytes;
};
// Phases, splits and shared memory for a model on a chip of `sms` SMs; false: the kernel does not take the shape.
bool mega_plan(unsigned sms, unsigned smem, const ks_mega_desc& d, MegaPlan& p) {
  const unsigned H = d.hidden, F = d.ffn, hd = d.hd, nq = d.n_q, nkv = d.n_kv;
  const unsigned qn = nq * hd, kvn = nkv * hd;
  auto even_blocks = [](unsigned cols) { return cols && cols % 512 == 0; };
  if (!even_blocks(H) || !even_blocks(F) || !even_blocks(qn)) return false;
  if (H > 16u * 256u) return false;  // the fused norms hold the vector in registers
  if (nkv < 1 || nq < nkv || nq % nkv || !(hd == 128 || hd == 256)) return false;
  // one block per (query head, split)
  p.n_splits = sms / nq;
  if (p.n_splits > (unsigned)MG_MAX_SPLITS) p.n_splits = MG_MAX_SPLITS;
  if (p.n_splits < 1 || nq > 48) return false;
  if (d.n_layers < 1 || d.n_layers > 128) return false;

  p.tables_bytes = (unsigned)((SM_LAYERS - SM_TAB + d.n_layers * sizeof(MegaLayer) + 15u) & ~15u);
  unsigned maxcols = H > F ? H : F;
  if (qn > maxcols) maxcols = qn;
  unsigned x_bytes = (maxcols / 64u) * (3u * MG_XU + 16u);
  const unsigned att = mg_att_bytes(hd);
  if (att > x_bytes) x_bytes = att;
  p.x_off = (SM_TAB + p.tables_bytes + 127u) & ~127u;
  p.ring_off = (p.x_off + x_bytes + 127u) & ~127u;
  unsigned most_job = 4u * (maxcols > 2u * H ? maxcols : 2u * H) / 256u * KS_Q4K_BLOCK_BYTES;  // (gate and up rows are one job)
  if (most_job < 8u * H) most_job = 8u * H;
  if (p.ring_off + most_job + 128u > smem) return false;
  p.ring_bytes = (smem - p.ring_off) & ~127u;
  // Blocks per column segment.  A block's items (its groups x column segments) are shared by its warps, so more segments shorten
  // the longest warp until the per-item overhead (measured: a little more than one unit's worth of time) wins; segments hold an
  // even number of blocks (8 lanes per row).
  const unsigned grid = p.grid = sms;
  if (grid > MG_THREADS) return false;  // a thread folds the norm sums of a block
  auto pick_seg = [&](unsigned cols, unsigned mats, unsigned total_groups) {
    const unsigned nb = cols / 256u, n_g = (total_groups + grid - 1) / grid;
    unsigned best = 0;
    float best_cost = 0.f;
    for (unsigned C = 1; C <= nb && C < MG_EMPTY; C++) {
      if (nb % C) continue;
      const unsigned sb = nb / C;
      if (sb % 2 || n_g * C > (unsigned)MG_MAX_P) continue;
      const float cost = (float)((n_g * C + MG_WARPS - 1u) / MG_WARPS) * ((float)(sb * mats) * 0.5f + 1.2f);
      if (!best || cost < best_cost) {
        best = sb;
        best_cost = cost;
      }
    }
    return best;
  };
  const unsigned g_qkv = (qn + 3) / 4 + 2 * ((kvn + 3) / 4), g_h = (H + 3) / 4, g_f = (F + 3) / 4;
  const unsigned most_g = MG_THREADS / MG_RL * grid;  // a block finishes a row per thread
  if (g_qkv > most_g || g_f > most_g || g_h > most_g) return false;
  const unsigned sb_h = pick_seg(H, 1, g_qkv), sb_q = pick_seg(qn, 1, g_h), sb_f = pick_seg(F, 1, g_h), sb_h2 = pick_seg(H, 2, g_f);
  if (!sb_h || !sb_h2 || !sb_q || !sb_f) return false;
  MegaShape* sh = p.sh;
  for (int k = 0; k < PH_PER_LAYER; k++) {
    sh[k] = MegaShape{};
    sh[k].mats = 1;
  }
  sh[PH_OPROJ].w0 = 3;
  sh[PH_DOWN].w0 = 6;
  auto set_rows = [](MegaShape& p, unsigned cols, unsigned sb) {
    p.cols = cols;
    p.row_bytes = cols / 256u * KS_Q4K_BLOCK_BYTES;
    p.seg_blocks = sb;
    p.n_cseg = cols / 256u / sb;
    unsigned g0 = 0;
    for (int s = 0; s < p.n_seg; s++) {
      p.grp_start[s] = g0;
      g0 += (p.rows[s] + 3u) / 4u;
    }
    p.grp_start[p.n_seg] = g0;
  };
  sh[PH_QKV].type = MG_MATVEC; sh[PH_QKV].n_seg = 3;
  sh[PH_QKV].rows[0] = qn; sh[PH_QKV].rows[1] = kvn; sh[PH_QKV].rows[2] = kvn;
  set_rows(sh[PH_QKV], H, sb_h);
  sh[PH_ATTN].type = MG_ATTN; sh[PH_ATTN].n_seg = 1; sh[PH_ATTN].n_cseg = 1;
  sh[PH_OPROJ].type = MG_MATVEC; sh[PH_OPROJ].n_seg = 1; sh[PH_OPROJ].rows[0] = H;
  set_rows(sh[PH_OPROJ], qn, sb_q);
  sh[PH_GATEUP].type = MG_GATE_UP; sh[PH_GATEUP].n_seg = 1; sh[PH_GATEUP].rows[0] = F; sh[PH_GATEUP].mats = 2; sh[PH_GATEUP].w0 = 4;
  set_rows(sh[PH_GATEUP], H, sb_h2);
  sh[PH_DOWN].type = MG_MATVEC; sh[PH_DOWN].n_seg = 1; sh[PH_DOWN].rows[0] = H;
  set_rows(sh[PH_DOWN], F, sb_f);
  return true;
}
}  // namespace

// The places block `block`'s jobs take in its ring during a token, in order: out[3 j] = place, [3 j + 1] = bytes, [3 j + 2] = the first
// job still there (`max_jobs` of them at most).  Returns their number, 0 where the kernel does not take the shape.  Host only.
extern "C" int ks_debug_decode_ring(int hidden, int ffn, int n_q, int n_kv, int hd, int n_layers, int sm_count, size_t smem_optin, int block,
                                    unsigned* ring_bytes, unsigned* out, int max_jobs) {
  ks_mega_desc d{};
  d.n_layers = n_layers;
  d.hidden = (unsigned)hidden; d.ffn = (unsigned)ffn; d.n_q = (unsigned)n_q; d.n_kv = (unsigned)n_kv; d.hd = (unsigned)hd;
  MegaPlan p;
  if (hidden < 1 || ffn < 1 || n_q < 1 || n_kv < 1 || hd < 1 || block < 0 || block >= sm_count || !mega_plan((unsigned)sm_count, (unsigned)smem_optin, d, p)) return 0;
  if (ring_bytes) *ring_bytes = p.ring_bytes;
  MegaRing ring{p.ring_bytes, 0u, 0u};
  unsigned taken[MG_JOBS], head = 0, tail = 0;
  for (int layer = 0; layer < n_layers; layer++)
    for (int kind = 0; kind < PH_PER_LAYER; kind++) {
      const unsigned norms = norm_jobs(kind), n = block_groups(p.sh[kind], (unsigned)block, p.grid) + norms;
      for (unsigned k = 0; k < n; k++, head++) {
        const unsigned room = job_bytes(p.sh[kind], k < norms, d.hidden);
        unsigned t = ring.takes(room);
        for (; head - tail >= MG_JOBS || !ring.fits(t); tail++) {
          ring.drop(taken[tail & (MG_JOBS - 1u)]);
          if (ring.used == 0) t = room;
        }
        const unsigned at = ring.put(room, t);
        taken[head & (MG_JOBS - 1u)] = t;
        if (out && head < (unsigned)max_jobs) {
          out[3 * head] = at;
          out[3 * head + 1] = room;
          out[3 * head + 2] = tail;
        }
      }
    }
  return (int)head;
}

// Returns KS_OK and *out == nullptr when the shape is outside what the kernel covers (the caller keeps
// the launch-per-op path), a negative code on a CUDA failure.
int ks_mega_create(ks_ctx* ctx, const ks_mega_desc* d, const ks_mega_layer* layers, ks_mega** out) {
  *out = nullptr;
  MegaPlan p;
  if (!mega_plan((unsigned)ctx->sm_count, (unsigned)ctx->smem_optin, *d, p)) return KS_OK;
  const unsigned H = d->hidden, F = d->ffn, hd = d->hd, nq = d->n_q, nkv = d->n_kv, qn = nq * hd, kvn = nkv * hd, n_splits = p.n_splits;
  std::vector<unsigned char> tab(p.tables_bytes, 0);
  memcpy(tab.data(), p.sh, sizeof(p.sh));
  MegaLayer* ly = reinterpret_cast<MegaLayer*>(tab.data() + (SM_LAYERS - SM_TAB));
  for (int l = 0; l < d->n_layers; l++) {
    const ks_mega_layer& L = layers[l];
    MegaLayer& o = ly[l];
    o.W[0] = (const uint8_t*)L.wq; o.W[1] = (const uint8_t*)L.wk; o.W[2] = (const uint8_t*)L.wv; o.W[3] = (const uint8_t*)L.wo;
    o.W[4] = (const uint8_t*)L.wgate; o.W[5] = (const uint8_t*)L.wup; o.W[6] = (const uint8_t*)L.wdown;
    o.norm[0] = (const float*)L.attn_norm; o.norm[1] = (const float*)L.q_norm; o.norm[2] = (const float*)L.k_norm;
    o.norm[3] = (const float*)L.post_attn_norm; o.norm[4] = (const float*)L.ffn_norm; o.norm[5] = (const float*)L.post_ffw_norm;
    o.window = (size_t)L.window;
    o.kv_k = L.kv_k; o.kv_v = L.kv_v;
  }

  ks_mega* mg = new ks_mega();
  cudaSetDevice(ctx->device);
  const size_t n_phases = (size_t)d->n_layers * PH_PER_LAYER;
  if (cudaMalloc(&mg->d_tables, p.tables_bytes) != cudaSuccess || cudaMalloc((void**)&mg->d_sync, 512 + 16 * (size_t)ctx->sm_count) != cudaSuccess ||
      cudaMalloc((void**)&mg->d_prof, n_phases * 16 * sizeof(long long)) != cudaSuccess ||
      cudaMalloc((void**)&mg->d_fx, (size_t)qn / 64 * 256 + F * sizeof(float)) != cudaSuccess ||
      cudaMalloc((void**)&mg->d_att, (size_t)nq * n_splits * mg_rec(hd) * sizeof(float)) != cudaSuccess ||
      cudaMalloc((void**)&mg->d_qkv, ((size_t)qn + 2 * (size_t)kvn) * sizeof(unsigned long long)) != cudaSuccess) {
    ks_mega_destroy(mg);
    return ks_fail(ctx, KS_ERR_OOM, "decode kernel: cannot allocate its tables");
  }
  cudaError_t e = cudaMemcpyAsync(mg->d_tables, tab.data(), p.tables_bytes, cudaMemcpyHostToDevice, ctx->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(mg->d_sync, 0, 512 + 16 * (size_t)ctx->sm_count, ctx->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(mg->d_fx, 0, (size_t)qn / 64 * 256 + F * sizeof(float), ctx->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(mg->d_prof, 0, n_phases * 16 * sizeof(long long), ctx->stream);
  mg->qkv_words = (size_t)qn + 2 * (size_t)kvn;
  if (e == cudaSuccess) e = cudaMemsetAsync(mg->d_qkv, 0, mg->qkv_words * sizeof(unsigned long long), ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);  // tab is a local
  if (e != cudaSuccess) {
    ks_mega_destroy(mg);
    return ks_fail(ctx, KS_ERR_CUDA, "decode kernel: table upload failed: %s", cudaGetErrorString(e));
  }
  MegaArgs& a = mg->args;
  a.tables = mg->d_tables;
  a.tables_bytes = p.tables_bytes;
  a.n_layers = d->n_layers;
  a.ring_bytes = p.ring_bytes;
  a.x_off = p.x_off;
  a.ring_off = p.ring_off;
  a.n_q = nq; a.n_kv = nkv; a.hd = hd; a.n_splits = n_splits;
  a.eps = d->eps; a.attn_scale = d->attn_scale;
  a.rope = d->rope; a.pos = d->pos;
  a.x_a = d->x_a; a.x_b = d->x_b;
  a.yb = d->yb;
  a.ox = mg->d_fx;
  a.ff = reinterpret_cast<float*>(mg->d_fx + (size_t)qn / 64 * 256);
  a.att_tmp = mg->d_att;
  a.bar = mg->d_sync;
  a.qkv_t = mg->d_qkv;
  a.att_cnt = mg->d_sync + 64;
  a.nsum = reinterpret_cast<float4*>(mg->d_sync + 128);
  a.err = (unsigned*)ctx->ws + KS_WS_ERR_WORD;
  a.poll_limit = 1u << 21;
  a.test_stall = 0;
  a.prof = mg->d_prof;
  mg->grid = p.grid;
  mg->smem = p.ring_off + p.ring_bytes;
  mg->dpl = (int)(hd / 32);
  mg->pc = (int)((H / 4u + MG_THREADS - 1u) / MG_THREADS);
  mg->residual = d->x_b;
  *out = mg;
  return KS_OK;
}
