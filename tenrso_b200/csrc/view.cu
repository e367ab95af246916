// Planning and launch of the view kernels (see view.cuh): the FP32 MTTKRP of
// every dense entry point but the allocation-free one, and the n-mode products.
#include "view.cuh"

#include <algorithm>
#include <cstring>

namespace tsr {

namespace {

constexpr int kWidths[] = {16, 24, 32, 48, 64};
constexpr int kRows[] = {32, 48, 64, 96, 128};
constexpr int64_t VIEW_MIN_RUN = 16;
int g_ctas[5][5];  // resident CTAs per SM, filled by init_view_attributes

int width_index(int bn) {
  for (int i = 0; i < 5; ++i)
    if (kWidths[i] == bn) return i;
  return 4;
}
int rows_index(int bm) {
  for (int i = 0; i < 5; ++i)
    if (kRows[i] == bm) return i;
  return 4;
}

int dispatch(tsr_ctx* ctx, cudaStream_t s, const ViewArgs& g, int bn, int bm, dim3 grid) {
  switch (bn) {
    case 16: return launch_view_bn<16>(ctx, s, g, bm, grid);
    case 24: return launch_view_bn<24>(ctx, s, g, bm, grid);
    case 32: return launch_view_bn<32>(ctx, s, g, bm, grid);
    case 48: return launch_view_bn<48>(ctx, s, g, bm, grid);
    default: return launch_view_bn<64>(ctx, s, g, bm, grid);
  }
}

// The narrowest tile that holds R (or an equal share of R beyond 64), and the
// tile height with the least padded work: a tile of m rows costs about m + 16
// (its FMAs, and the share of K's tile and of the barriers).
void choose_tile(int64_t rows, int R, int* bn, int* bm) {
  const int64_t nt = ceil_div(R, 64), share = ceil_div(R, nt);
  *bn = 64;
  for (int w : kWidths)
    if (w >= share) {
      *bn = w;
      break;
    }
  int64_t best = INT64_MAX;
  for (int i = 4; i >= 0; --i) {
    const int64_t cost = ceil_div(rows, kRows[i]) * (kRows[i] + 16);
    if (cost < best) {
      best = cost;
      *bm = kRows[i];
    }
  }
}

// Tile of a product that is not split over its contraction: the least work of
// the busiest SM (its tiles, each padded by the fixed part of a step), weighted
// by how well the warps it holds cover latency (w / (w + 4): 8 warps reach two
// thirds, 16 four fifths of the rate of a full SM). A tile that is turned
// through shared memory on its way out is at most 32 columns wide: then four
// CTAs share an SM and one's stores overlap another's loads, which short
// contractions are made of. us at widths 64 / 32: 16 x 1000000 to 64 193 / 156,
// 64 x 256 x 256 to 64 33 / 31, 256 x 64 x 64 to 256 35 / 31, 30 x 30 x 4000
// to 64 37 / 29; no size measured wants the wider ones.
void choose_tile_unsplit(const tsr_ctx* ctx, int64_t rows, int64_t R, int64_t batch, bool turned,
                         int* bn, int* bm) {
  double best = 0.0;
  for (int wi = 0; wi < (turned ? 3 : 5); ++wi)
    for (int ri = 0; ri < 5; ++ri) {
      const int w = kWidths[wi], m = kRows[ri];
      const int64_t tiles = ceil_div(rows, m) * ceil_div(R, w) * batch;
      const int64_t per_sm = ceil_div(tiles, ctx->sm_count);
      const double warps = (double)std::min<int64_t>(g_ctas[wi][ri], per_sm) * (w / 8);
      const double cost = (double)per_sm * (m + 16) * (w + 8) * (warps + 4) / warps;
      if (best == 0.0 || cost < best) {
        best = cost;
        *bn = w;
        *bm = m;
      }
    }
}

}  // namespace

// Which contracted mode is the inner one, and the strides of all of them. The
// inner mode is the fastest contracted one, where a chunk is contiguous in
// memory (or, for the last mode's MTTKRP, its rows are); one shorter than half a
// chunk would leave most of each step empty, so then it is the longest one.
void describe_view(int ndim, const int64_t* shape, int mode, ViewArgs* g, int* inner, int cut,
                   int64_t cut_len) {
  int64_t stride[kMaxModes], size[kMaxModes], st = 1;
  for (int m = ndim - 1; m >= 0; --m) {
    stride[m] = st;
    st *= shape[m];
    size[m] = m == cut ? cut_len : shape[m];
  }
  int in = mode == ndim - 1 ? ndim - 2 : ndim - 1;
  if (size[in] < VIEW_MIN_RUN)
    for (int m = ndim - 1; m >= 0; --m)
      if (m != mode && size[m] > size[in]) in = m;
  *inner = in;
  g->rows = shape[mode];
  g->row_stride = stride[mode];
  g->k_stride = stride[in];
  g->S = (uint32_t)size[in];
  int64_t runs = 1;
  for (int m = 0; m < ndim; ++m) {
    if (m == mode || m == in) continue;
    g->size[g->n_outer] = (uint32_t)size[m];
    g->stride[g->n_outer] = stride[m];
    ++g->n_outer;
    runs *= size[m];
  }
  // equal chunks of at most 32 columns
  g->chunks = (uint32_t)ceil_div(g->S, 32);
  g->kc = (int)round_up(ceil_div(g->S, g->chunks), 4);
  g->chunks = (uint32_t)ceil_div(g->S, g->kc);
  g->steps = runs * g->chunks;
}

namespace {
int tile_map(const ViewArgs& g) {
  if (g.k_stride != 1) return g.row_stride == 1 ? VIEW_ACROSS : VIEW_STRIDED;
  bool vec = ((uintptr_t)g.X & 15) == 0 && g.S % 4 == 0 && g.row_stride % 4 == 0 &&
             g.x_batch % 4 == 0;
  for (int p = 0; p < g.n_outer; ++p) vec = vec && g.stride[p] % 4 == 0;
  return vec ? VIEW_VEC : VIEW_ALONG;
}

}  // namespace

double view_estimate_us(int64_t rows, int64_t cols, int R) {
  int bn = 0, bm = 0;
  choose_tile(rows, R, &bn, &bm);
  const double tile = (double)(bm + 16) * (bn + 8);
  return 2.0 * (double)(ceil_div(rows, bm) * ceil_div(R, bn)) * tile * (double)cols / 33e6;
}

void init_view_attributes() {
  for (int i = 0; i < 5; ++i) {
    g_ctas[0][i] = view_ctas_per_sm<16>(kRows[i]);
    g_ctas[1][i] = view_ctas_per_sm<24>(kRows[i]);
    g_ctas[2][i] = view_ctas_per_sm<32>(kRows[i]);
    g_ctas[3][i] = view_ctas_per_sm<48>(kRows[i]);
    g_ctas[4][i] = view_ctas_per_sm<64>(kRows[i]);
  }
}

ViewPlan plan_view(const tsr_ctx* ctx, int ndim, const int64_t* shape, int mode, int R,
                   int reserve) {
  ViewPlan p;
  ViewArgs g;
  std::memset(&g, 0, sizeof(g));
  int inner;
  choose_tile(shape[mode], R, &p.bn, &p.bm);
  describe_view(ndim, shape, mode, &g, &inner);
  const int per_sm = std::max(1, g_ctas[width_index(p.bn)][rows_index(p.bm)]);
  const int64_t tiles = ceil_div(g.rows, p.bm) * ceil_div(R, p.bn);
  const int64_t slots = (int64_t)std::max(1, ctx->sm_count - reserve) * per_sm;
  // one wave of resident CTAs, but no more splits than SMs where a split would
  // be left with fewer than four steps
  const int64_t few = std::max<int64_t>(ceil_div(g.steps, 4), ctx->sm_count - reserve);
  const int64_t want = std::max<int64_t>(
      1, std::min<int64_t>({slots / tiles, std::min(few, g.steps), (int64_t)65535}));
  p.steps_per_split = ceil_div(g.steps, want);
  p.splits = (int)ceil_div(g.steps, p.steps_per_split);
  return p;
}

int launch_view(tsr_ctx* ctx, cudaStream_t s, const float* X, int ndim, const int64_t* shape,
                int mode, const float* const* f, int R, const ViewPlan& plan, float* partials) {
  ViewArgs g;
  std::memset(&g, 0, sizeof(g));
  int inner;
  describe_view(ndim, shape, mode, &g, &inner);
  int64_t cols = 1;
  for (int m = 0; m < ndim; ++m)
    if (m != mode) cols *= shape[m];
  if (cols >= (int64_t)UINT32_MAX) return fail(TSR_E_UNSUPPORTED, "unfolding too wide");
  g.X = X;
  g.steps_per_split = plan.steps_per_split;
  g.R = R;
  g.inner = f[inner];
  g.inner_s = R;
  g.inner_c = 1;
  g.inner_vec = R % 4 == 0 && ((uintptr_t)f[inner] & 15) == 0;
  for (int m = 0, p = 0; m < ndim; ++m)
    if (m != mode && m != inner) g.f[p++] = f[m];
  g.out = partials;
  g.out_split = g.rows * R;
  g.out_row = R;
  g.out_col = 1;
  g.map = tile_map(g);
  dim3 grid((unsigned)ceil_div(g.rows, plan.bm), (unsigned)plan.splits,
            (unsigned)ceil_div(R, plan.bn));
  if (grid.z > 65535) return fail(TSR_E_UNSUPPORTED, "MTTKRP grid too large");
  return dispatch(ctx, s, g, plan.bn, plan.bm, grid);
}

int launch_view_matrix(tsr_ctx* ctx, cudaStream_t s, const float* X, int64_t A, int64_t I,
                       int64_t B, const float* mat, int64_t J, float* Y) {
  if (ceil_div(B > 1 ? J : A, 64) > 65535)
    return fail(TSR_E_UNSUPPORTED, "output too tall for one launch");
  if (I > (int64_t)UINT32_MAX - 64) return fail(TSR_E_UNSUPPORTED, "contracted mode too long");
  if (I == 0) {  // an empty sum
    TSR_CUDA(cudaMemsetAsync(Y, 0, sizeof(float) * A * J * B, s));
    return TSR_OK;
  }
  ViewArgs g;
  std::memset(&g, 0, sizeof(g));
  g.X = X;
  g.S = (uint32_t)I;
  g.chunks = (uint32_t)ceil_div(I, 32);
  g.kc = (int)round_up(ceil_div(I, g.chunks), 4);
  g.chunks = (uint32_t)ceil_div(I, g.kc);
  g.steps = g.steps_per_split = g.chunks;
  g.inner_s = 1;
  g.inner_c = I;
  if (B > 1) {  // per a: rows b, columns i at stride B; Y's contiguous direction is b
    g.rows = B;
    g.row_stride = 1;
    g.k_stride = B;
    g.out_row = 1;
    g.out_col = B;
    g.batch = A;
    g.x_batch = I * B;
    g.out_batch = J * B;
  } else {  // the last mode: rows a of I columns
    g.rows = A;
    g.row_stride = I;
    g.k_stride = 1;
    g.out_row = J;
    g.out_col = 1;
    g.batch = 1;
  }
  g.map = tile_map(g);
  for (int64_t j0 = 0, cols; j0 < J; j0 += cols) {
    int bn, bm;
    choose_tile_unsplit(ctx, g.rows, J - j0, g.batch, B > 1, &bn, &bm);
    cols = std::min<int64_t>(J - j0, (int64_t)65535 * bn);  // one launch's column tiles
    g.R = (int)cols;
    g.inner = mat + j0 * I;
    g.out = Y + j0 * g.out_col;
    const dim3 grid((unsigned)ceil_div(g.rows, bm),
                    (unsigned)std::min<int64_t>(g.batch, 65535), (unsigned)ceil_div(g.R, bn));
    TSR_TRY(dispatch(ctx, s, g, bn, bm, grid));
  }
  return TSR_OK;
}

}  // namespace tsr
