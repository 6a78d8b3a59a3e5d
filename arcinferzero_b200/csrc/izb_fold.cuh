// Host interface of the folded GEMM (csrc/izb_gemm_fold.cu) for csrc/izb_gemm_tc.cu, which owns scratch, the cut of K and the dispatch.
#pragma once
#include "izb_common.cuh"

struct FoldParams {
  unsigned char* img;     // operand images: per token tile and superblock [lo, hi][4 stages of 64][tt rows][128 B], rows 128-byte swizzled
  unsigned char* fine;    // ... [4 stages of 64][tt rows][128 B], swizzled alike: the third term, of the rows that have one
  unsigned char* tail;    // ... [tt rows][16] fp16 min-term factors, [tt] f32 row scales s, [tt] bytes: kinds of the rows
  const float* asc;       // the activations' scales [K / 32][lda], read again for rows whose kind is wide
  int lda;
  int tt;                 // token rows of a tile (a multiple of 16, at most 128)
  int n_mtiles;           // token tiles
  int M;                  // rows to store
  int N, K;               // per matrix
  int mat;                // matrix of the stack
  int n_split;            // parts the K range of every tile is cut into
  float* part;            // n_split > 1: [n_split][M][N] partial sums, stored instead of C
  uint32_t* part_bad;     // n_split > 1: set when a wait gave up (split_reduce_kernel then stores nothing); the pre-pass clears it; may be null
  float* C;
  int ldc, c_off;
  uint32_t* err;
  uint32_t spin_limit;    // polls after which a wait gives up
  int pdl;                // programmatic dependent launch (csrc/izb_gemm_tc.cu: tc_pdl)
  int skip_stage;         // diagnostics: the unit of the activation ring that its producer leaves out (-1: none)
};

// weights it takes
static inline bool izb_fold_takes(const izb_weight* w) { return w->type == IZB_Q4_K || (w->type == IZB_K16 && w->has_min); }
int izb_fold_tile_rows(int device, int M, int N);
// scratch for n_mtiles * tt rows
size_t izb_fold_img_bytes(int rows, int K);
size_t izb_fold_fine_bytes(int rows, int K);
size_t izb_fold_tail_bytes(int rows, int K);
// pre-pass over rows already quantised (rows past `rows` count as zeros), or with the quantiser in it
int izb_fold_prepare(const izb_weight* w, const int8_t* aq, const float* asc, int lda, int rows, const FoldParams& p, cudaStream_t st);
int izb_fold_quant_prepare(const izb_weight* w, const float* x, int ldx, int M, int Mp, int8_t* aq, float* asc, const FoldParams& p, cudaStream_t st);
// Do the kernels that quantise and prepare `rows` rows at once take one row per warp (blocks of 8 rows) instead of four?
bool izb_one_row_per_warp(int rows, int K);
int izb_fold_gemm(const izb_weight* w, const FoldParams& p, int grid, cudaStream_t st);
