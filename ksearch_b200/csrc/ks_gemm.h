// Between ks_gemm.cu (images, epilogues, dispatch), ks_gemm_q4k.cu (the Q4_K kernel) and ks_gemm_skinny.cu (up to 8 token rows).
#pragma once
#include "ks_gemm_common.cuh"

constexpr int KS_GEMM_SKINNY = 8;  // token rows of the kernel in ks_gemm_skinny.cu (the columns of one mma)

struct ks_gemm_job {
  int n_seg;
  const uint8_t* W[3];
  size_t rows[3];
  float* y[3];               // partial `slot` of matrix i: y[i] + slot * part_stride[i], [token][row] with row stride ldy[i]
  size_t ldy[3], part_stride[3];
  unsigned cols, n_tok, np;
  const __half* xt;
  ks_gemm_map map;
};
// `tbn`: token rows of a block; more than 64 take row tiles in pairs.  `plain`: undivided sums need no second launch.  `cost`:
// the estimate the map was chosen by, in us.
ks_gemm_map ks_gemm_q4k_map(const ks_ctx* ctx, const size_t* rows, int n_seg, unsigned cols, unsigned np, unsigned tbn, bool plain,
                            double* cost = nullptr);
int ks_launch_gemm_q4k(ks_ctx* ctx, const ks_gemm_job& job);
unsigned ks_gemm_skinny_splits(const ks_ctx* ctx, size_t rows, unsigned cols);  // column shares; 0: not covered
int ks_launch_gemm_skinny(ks_ctx* ctx, const ks_gemm_job& job);
bool ks_gemm_q6k_skinny_covers(const ks_ctx* ctx, size_t rows, unsigned cols);
int ks_launch_gemm_q6k_skinny(ks_ctx* ctx, const ks_gemm_job& job);
