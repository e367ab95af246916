// FP32 contraction of a row-major tensor read in place ("view" kernels).
//
// A tensor X is seen as A x I x B (element (a, i, b) at (a I + i) B + b) and
// contracted over (a, b):
//   out[i, c] = sum_{a, b} X[a, i, b] K[(a, b), c],
// where K's rows are Khatri-Rao rows formed on the fly (the MTTKRP), or the
// columns of a matrix (the n-mode product, batched). No unfolding of X is
// ever written.
//
// The contracted columns come in runs: the S rows of one "inner" factor (the
// fastest contracted mode unless it is too short), scaled column-wise by the
// product of one row of each other contracted factor. A step is one chunk of
// columns inside a run, so its addresses are uniform over the CTA.
#pragma once
#include "mttkrp.cuh"

namespace tsr {

constexpr int kViewOuterMax = kMaxModes - 2;

struct ViewArgs {
  const float* X;
  int64_t rows;        // I
  int64_t row_stride;  // elements between rows i and i + 1
  int64_t k_stride;    // elements between columns of a run
  uint32_t S;          // columns per run
  int kc;              // columns per chunk (a multiple of 4, at most 32)
  uint32_t chunks;     // chunks per run
  int64_t steps;       // chunks over all runs
  int64_t steps_per_split;
  int R;               // output columns
  int map;             // how a tile is loaded (ViewMap)
  const float* inner;  // K[(o, s), c] = inner[s * inner_s + c * inner_c] * (outer products)
  int64_t inner_s, inner_c;
  int inner_vec;       // 16-byte loads along c (R a multiple of 4, aligned)
  // the other contracted modes, the last varying fastest with the run number
  int n_outer;
  uint32_t size[kViewOuterMax];
  int64_t stride[kViewOuterMax];
  const float* f[kViewOuterMax];
  // out[split * out_split + i * out_row + c * out_col] (+ batch strides)
  float* out;
  int64_t out_split, out_row, out_col;
  int64_t batch, x_batch, out_batch;
};

// Tile load patterns: VEC reads 16 bytes along a run (everything a multiple of
// 4 floats), ALONG one float per lane along a run, ACROSS 8 rows x 4 columns
// per warp (the row index is the tensor's contiguous direction), STRIDED the
// same where neither direction is contiguous.
enum ViewMap { VIEW_VEC = 0, VIEW_ALONG = 1, VIEW_ACROSS = 2, VIEW_STRIDED = 3 };

struct ViewPlan {
  int bn = 32;  // output columns per CTA
  int bm = 128;  // output rows per CTA
  int splits = 1;
  int64_t steps_per_split = 0;
};

// The geometry of one mode's contraction (rows, strides, runs, chunks, outer
// modes) and its inner mode; element-type independent. cut >= 0: only `cut_len`
// indices of the contracted mode `cut` (X and its factor start at the first).
void describe_view(int ndim, const int64_t* shape, int mode, ViewArgs* g, int* inner,
                   int cut = -1, int64_t cut_len = 0);
// The MTTKRP of X (row-major, `shape`) for `mode`, R columns; `reserve`: SMs
// the plan leaves to other kernels.
ViewPlan plan_view(const tsr_ctx* ctx, int ndim, const int64_t* shape, int mode, int R,
                   int reserve);
// Microseconds of an MTTKRP of a rows x cols unfolding: its padded FMAs (a tile
// is at least 32 rows and 16 columns, and costs its fixed part) at the measured
// rate. Good to about a third.
double view_estimate_us(int64_t rows, int64_t cols, int R);
// Partial sums [splits][I_mode][R] (f: one factor per mode; f[mode] unused).
int launch_view(tsr_ctx* ctx, cudaStream_t s, const float* X, int ndim, const int64_t* shape,
                int mode, const float* const* f, int R, const ViewPlan& plan, float* partials);
// Y[a, j, b] = sum_i mat[j, i] X[a, i, b] for X seen as A x I x B, mat J x I.
int launch_view_matrix(tsr_ctx* ctx, cudaStream_t s, const float* X, int64_t A, int64_t I,
                       int64_t B, const float* mat, int64_t J, float* Y);
void init_view_attributes();

// One translation unit per column-tile width.
template <int BN>
int launch_view_bn(tsr_ctx* ctx, cudaStream_t s, const ViewArgs& g, int bm, dim3 grid);
template <int BN>
int view_ctas_per_sm(int bm);  // resident CTAs per SM; raises the shared-memory limits

}  // namespace tsr
