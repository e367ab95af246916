// The f64 instantiation of the drop-in: tenrso_kernels::mttkrp<f64>
// (crates/tenrso-kernels/src/mttkrp.rs:74-146) and tenrso_decomp::cp_als<f64>
// (crates/tenrso-decomp/src/cp/core.rs:59-182) with every value in FP64.
//
// MTTKRP: the FP64 form of the view kernels (view.cuh): X read in place, the
// contracted columns in runs of one inner factor, scaled by the product of one
// row of each other factor. A CTA owns 64 rows x up to 32 columns of M and a
// range of chunks (split-K); the splits meet in M with FP64 atomics.
//
// CP-ALS: the same device state, inverse and fit kernels as the fp32 sweep
// (als.cu), with an FP64 solve (U = M G^-1, the new Gram and, for the last
// mode, <M, U> and ||Xhat||^2) and FP64 factors; the ridge of
// solve_least_squares is f64's eps * rank * 10 (helpers.rs:477-490).
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <limits>
#include <vector>

#include "als.cuh"
#include "dense.cuh"

namespace tsr {

namespace {

struct M64Args {
  ViewArgs v;  // geometry only
  const double* X;
  const double* inner;
  const double* f[kViewOuterMax];
  const int* done;  // CP-ALS: set once the run has stopped (null: standalone)
  double* M;        // I x R, zeroed by the caller
};

constexpr int kF64Look = 8;
constexpr int64_t kF64Columns = (int64_t)1 << 31;  // of one launch's unfolding
constexpr int F64_BM = 64, F64_K = 32, F64_P = F64_K + 1;

template <int BN>
constexpr size_t f64_smem() {
  return sizeof(double) * 2 * (F64_BM * F64_P + F64_K * BN);
}

__device__ __forceinline__ void f64_cp8(double* dst, const double* src, bool ok) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = ok ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n)
               : "memory");
}

// 4 x 4 outputs per thread (rows ty + 16 i, columns tx + (BN/4) q): eight 8-byte
// words read from shared memory per 16 FMAs, which for a warp are about eight
// wavefronts against eight cycles of FP64 issue. At 120x100x80 rank 24, 13-21 us
// per mode where the FMAs need 1.4: too few chunks per CTA to hide the loads. The
// former kernel divided a 64-bit index per element and multiplied 64 columns
// whatever the rank: 36 us.
template <int BN>
__global__ void __launch_bounds__(4 * BN) mttkrp_f64_kernel(const __grid_constant__ M64Args g) {
  constexpr int TX = BN / 4, NT = 4 * BN, NW = NT / 32;
  extern __shared__ __align__(16) double sm64[];
  double* As = sm64;                          // [2][F64_BM][F64_P]
  double* Bs = sm64 + 2 * F64_BM * F64_P;     // [2][F64_K][BN]
  if (g.done) {
    // the inverse on the other stream may be setting the flag right now: one
    // thread looks, so that the CTA stays or leaves as a whole (a CTA that
    // stays only writes M, which the solve, after the join, then ignores)
    const int stop = threadIdx.x == 0 ? *(volatile const int*)g.done : 0;
    if (__syncthreads_or(stop)) return;
  }
  const ViewArgs& v = g.v;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int tx = tid % TX, ty = tid / TX;
  const int64_t i0 = (int64_t)blockIdx.x * F64_BM;
  const int n0 = blockIdx.z * BN, R = v.R;
  const int rows_here = (int)min((int64_t)F64_BM, v.rows - i0);
  const int64_t g0 = (int64_t)blockIdx.y * v.steps_per_split;
  const int nsteps = (int)min(v.steps_per_split, v.steps - g0);
  const int bc = tid % BN, bk = tid / BN;  // K's tile: column bc, rows bk, bk + 4, ..
  const int c = n0 + bc;
  for (int e = rows_here * F64_P + tid; e < F64_BM * F64_P; e += NT)
    As[e] = As[F64_BM * F64_P + e] = 0.0;

  const double* X = g.X + i0 * v.row_stride;
  uint32_t o = (uint32_t)g0 / v.chunks, s0 = ((uint32_t)g0 - o * v.chunks) * v.kc;
  const double* run = X;
  double wt = 1.0, braw[F64_K / 4];
  bool new_run = true;
  int valid = 0;
  auto load = [&](int buf) {
    if (new_run) {
      run = X;
      wt = 1.0;
      uint32_t q = o;
      for (int p = v.n_outer - 1; p >= 0; --p) {
        const uint32_t t = p > 0 ? q / v.size[p] : 0, i = q - t * v.size[p];
        run += i * v.stride[p];
        if (c < R) wt *= __ldg(g.f[p] + (int64_t)i * R + c);
        q = t;
      }
      new_run = false;
    }
    valid = (int)min((uint32_t)v.kc, v.S - s0);
    double* dst = As + buf * F64_BM * F64_P;
    if (v.k_stride == 1) {  // lanes along the run
      const bool in = lane < valid;
      const double* src = in ? run + s0 + lane + w * v.row_stride : g.X;
      const int64_t inc = in ? NW * v.row_stride : 0;
      if (lane < v.kc)
        for (int m = w; m < rows_here; m += NW) {
          f64_cp8(dst + m * F64_P + lane, src, in);
          src += inc;
        }
    } else {  // lanes along the rows
      for (int k = w; k < v.kc; k += NW) {
        const bool in = k < valid;
        const double* src = in ? run + (s0 + k) * v.k_stride + lane * v.row_stride : g.X;
        for (int m = lane; m < rows_here; m += 32) {
          f64_cp8(dst + m * F64_P + k, src, in);
          if (in) src += 32 * v.row_stride;
        }
      }
    }
    const double* ks = g.inner + (int64_t)(s0 + bk) * R + c;
#pragma unroll
    for (int t = 0; t < F64_K / 4; ++t) {
      braw[t] = c < R && bk + 4 * t < valid ? __ldg(ks) : 0.0;
      ks += 4 * R;
    }
  };
  auto store_b = [&](int buf) {
#pragma unroll
    for (int t = 0; t < F64_K / 4; ++t)
      Bs[(buf * F64_K + bk + 4 * t) * BN + bc] = bk + 4 * t < valid ? braw[t] * wt : 0.0;
  };
  double acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[i][q] = 0.0;
  load(0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  store_b(0);
  for (int s = 0; s < nsteps; ++s) {
    const int buf = s & 1;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (s + 1 < nsteps) {
      s0 += v.kc;
      if (s0 >= v.S) {
        s0 = 0;
        ++o;
        new_run = true;
      }
      load(buf ^ 1);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const double* a = As + buf * F64_BM * F64_P + ty * F64_P;
    const double* b = Bs + buf * F64_K * BN + tx;
#pragma unroll 4
    for (int k = 0; k < v.kc; ++k) {
      double av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = a[i * 16 * F64_P + k];
#pragma unroll
      for (int q = 0; q < 4; ++q) bv[q] = b[k * BN + TX * q];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[i][q] = fma(av[i], bv[q], acc[i][q]);
    }
    if (s + 1 < nsteps) store_b(buf ^ 1);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = ty + 16 * i;
    if (m >= rows_here) continue;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int cc = n0 + tx + TX * q;
      if (cc < R) atomicAdd(g.M + (i0 + m) * R + cc, acc[i][q]);
    }
  }
}

// Upper triangle of the Gram of rows r0.. of a (rows x R) FP64 block held in
// shared memory (Us, nr rows), accumulated into registers.
template <int RB>
__device__ __forceinline__ void gram_rows(const double* Us, int nr, int R,
                                          double (&acc)[RB][RB]) {
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  for (int i = 0; i < nr; ++i) {
    double x[RB], y[RB];
#pragma unroll
    for (int a = 0; a < RB; ++a) x[a] = ty + 16 * a < R ? Us[i * R + ty + 16 * a] : 0.0;
#pragma unroll
    for (int b = 0; b < RB; ++b) y[b] = tx + 16 * b < R ? Us[i * R + tx + 16 * b] : 0.0;
#pragma unroll
    for (int a = 0; a < RB; ++a)
#pragma unroll
      for (int b = 0; b < RB; ++b) acc[a][b] = fma(x[a], y[b], acc[a][b]);
  }
}

// U (rows x R, FP64) = M G^-1 with G^-1 from the inverse kernel (b.ginv);
// gram += U^T U (upper, FP64 atomics); for the last mode <M, U> and
// ||Xhat||^2 = sum(H o U^T U) into the state, and the fit marked pending.
// With M null the kernel only accumulates the Gram of U (initial Grams).
template <int RB>
__global__ void __launch_bounds__(256)
solve_f64_kernel(AlsBuffers b, int ndim, int R, int64_t rows, const double* __restrict__ M,
                 double* __restrict__ U, double* __restrict__ gram, int last, int rpc) {
  extern __shared__ __align__(16) double sm[];
  __shared__ double red[16];
  AlsState* st = b.state;
  if (M && st->done) return;
  double* Gi = sm;                    // R x R (solve only)
  double* Us = sm + (M ? R * R : 0);  // rpc x R
  double* Ms = Us + rpc * R;          // rpc x R (solve only)
  if (M)
    for (int e = threadIdx.x; e < R * R; e += blockDim.x) Gi[e] = b.ginv[e];
  double acc[RB][RB];
#pragma unroll
  for (int a = 0; a < RB; ++a)
#pragma unroll
    for (int c = 0; c < RB; ++c) acc[a][c] = 0.0;
  double ip = 0.0;
  for (int64_t r0 = (int64_t)blockIdx.x * rpc; r0 < rows; r0 += (int64_t)gridDim.x * rpc) {
    const int nr = (int)(rows - r0 < rpc ? rows - r0 : rpc);
    __syncthreads();
    if (M) {
      for (int e = threadIdx.x; e < nr * R; e += blockDim.x) Ms[e] = M[r0 * R + e];
      __syncthreads();
    }
    for (int e = threadIdx.x; e < nr * R; e += blockDim.x) {
      const int64_t g = r0 * R + e;
      double u;
      if (M) {
        const int i = e / R, c = e % R;
        const double* m = Ms + i * R;
        u = 0.0;
        for (int k = 0; k < R; ++k) u = fma(m[k], Gi[k * R + c], u);
        U[g] = u;
        if (last) ip += m[c] * u;
      } else {
        u = U[g];
      }
      Us[e] = u;
    }
    __syncthreads();
    gram_rows<RB>(Us, nr, R, acc);
  }
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  double xs = 0.0;
  const double* H = b.hadam + (int64_t)(ndim - 1) * R * R;
#pragma unroll
  for (int a = 0; a < RB; ++a)
#pragma unroll
    for (int c = 0; c < RB; ++c) {
      const int i = ty + 16 * a, j = tx + 16 * c;
      if (i < R && j < R && j >= i) {
        atomicAdd(gram + i * R + j, acc[a][c]);
        if (last) xs += (i == j ? 1.0 : 2.0) * H[i * R + j] * acc[a][c];
      }
    }
  if (!last || !M) return;
  for (int o = 16; o > 0; o >>= 1) {
    ip += __shfl_down_sync(0xffffffffu, ip, o);
    xs += __shfl_down_sync(0xffffffffu, xs, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[threadIdx.x >> 5] = ip;
    red[8 + (threadIdx.x >> 5)] = xs;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0, x = 0.0;
    for (int w = 0; w < 8; ++w) {
      s += red[w];
      x += red[8 + w];
    }
    atomicAdd(&st->inner, s);
    atomicAdd(&st->xhat_sq, x);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) st->fit_pending = 1;
}

__global__ void norm_sq_f64_kernel(const double* __restrict__ X, int64_t n, double* out) {
  double s = 0.0;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x) {
    const double v = X[e];
    s = fma(v, v, s);
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}

unsigned f64_grid(const tsr_ctx* ctx, int64_t n) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, 256), ctx->sm_count * 8));
}

template <int BN>
void go_f64(cudaStream_t s, const M64Args& g, dim3 grid) {
  mttkrp_f64_kernel<BN><<<grid, 4 * BN, f64_smem<BN>(), s>>>(g);
}

// Rows [c0, c0 + len) of mode `cut` of the contraction, added into M.
int launch_mttkrp_f64_part(tsr_ctx* ctx, const double* X, int ndim, const int64_t* shape,
                           const double* const* U, int R, int mode, int cut, int64_t c0,
                           int64_t len, double* M, const int* done) {
  cudaStream_t s = ctx->stream;
  M64Args g;
  std::memset(&g, 0, sizeof(g));
  int64_t st = 1;  // elements between indices of `cut`
  for (int m = cut + 1; m < ndim; ++m) st *= shape[m];
  int inner;
  describe_view(ndim, shape, mode, &g.v, &inner, cut, len);
  g.v.R = R;
  g.X = X + c0 * st;
  g.M = M;
  g.done = done;
  auto rows_of = [&](int m) { return U[m] + (m == cut ? c0 * R : 0); };
  g.inner = rows_of(inner);
  for (int m = 0, p = 0; m < ndim; ++m)
    if (m != mode && m != inner) g.f[p++] = rows_of(m);
  const int64_t share = ceil_div(R, ceil_div(R, 32));
  const int bn = share <= 8 ? 8 : share <= 16 ? 16 : share <= 24 ? 24 : 32;
  const int64_t tiles = ceil_div(g.v.rows, F64_BM) * ceil_div(R, bn);
  // about three CTAs per SM, at least two chunks each
  const int64_t want = std::max<int64_t>(
      1, std::min<int64_t>({3 * (int64_t)ctx->sm_count / tiles, ceil_div(g.v.steps, 2),
                            (int64_t)65535}));
  g.v.steps_per_split = ceil_div(g.v.steps, want);
  dim3 grid((unsigned)ceil_div(g.v.rows, F64_BM),
            (unsigned)ceil_div(g.v.steps, g.v.steps_per_split), (unsigned)ceil_div(R, bn));
  if (grid.z > 65535u) return fail(TSR_E_UNSUPPORTED, "f64 MTTKRP grid too large");
  switch (bn) {
    case 8: go_f64<8>(s, g, grid); break;
    case 16: go_f64<16>(s, g, grid); break;
    case 24: go_f64<24>(s, g, grid); break;
    default: go_f64<32>(s, g, grid); break;
  }
  ctx->launches++;
  TSR_CUDA(cudaGetLastError());
  return TSR_OK;
}

int launch_mttkrp_f64(tsr_ctx* ctx, const double* X, int ndim, const int64_t* shape,
                      const double* const* U, int R, int mode, double* M,
                      const int* done = nullptr) {
  int64_t J = 1;
  for (int m = 0; m < ndim; ++m)
    if (m != mode) J *= shape[m];
  TSR_CUDA(cudaMemsetAsync(M, 0, sizeof(double) * shape[mode] * R, ctx->stream));
  if (shape[mode] == 0 || R == 0 || J == 0) return TSR_OK;
  // The kernel counts runs, chunks and a run's columns in 32 bits: a wider
  // unfolding is taken in pieces of its longest contracted mode, whose sums meet
  // in M as the splits do.
  int cut = mode == 0 ? 1 : 0;
  for (int m = 0; m < ndim; ++m)
    if (m != mode && shape[m] > shape[cut]) cut = m;
  const int64_t part = std::max<int64_t>(1, kF64Columns / (J / shape[cut]));
  for (int64_t c0 = 0; c0 < shape[cut]; c0 += part)
    TSR_TRY(launch_mttkrp_f64_part(ctx, X, ndim, shape, U, R, mode, cut, c0,
                                   std::min(part, shape[cut] - c0), M, done));
  return TSR_OK;
}

int launch_solve_f64(tsr_ctx* ctx, const AlsBuffers& b, int ndim, int R, int64_t rows,
                     const double* M, double* U, double* gram, bool last) {
  // 4 rows per step where that still leaves few CTAs (the serial FP64 dot
  // products set the pace), 16 for tall factors
  const int rpc = rows <= 8 * (int64_t)ctx->sm_count ? 4 : 16;
  const unsigned grid = (unsigned)std::max<int64_t>(
      1, std::min<int64_t>(ceil_div(rows, rpc), 2 * (int64_t)ctx->sm_count));
  const size_t smem = sizeof(double) * ((M ? (size_t)R * R + rpc * (size_t)R : 0) +
                                        rpc * (size_t)R);
  const int lst = last ? 1 : 0;
#define TSR_S64(RB) \
  solve_f64_kernel<RB><<<grid, 256, smem, ctx->stream>>>(b, ndim, R, rows, M, U, gram, lst, rpc)
  switch ((R + 15) / 16) {
    case 1: TSR_S64(1); break;
    case 2: TSR_S64(2); break;
    case 3: TSR_S64(3); break;
    case 4: TSR_S64(4); break;
    case 5: TSR_S64(5); break;
    case 6: TSR_S64(6); break;
    default: TSR_S64(7); break;
  }
#undef TSR_S64
  ctx->launches++;
  TSR_CUDA(cudaGetLastError());
  return TSR_OK;
}

// Host seeded U(0,1) doubles of the library's stream (InitStrategy::Random).
void seeded_uniform_f64(uint64_t seed, uint64_t stream, int64_t n, double* out) {
  auto mix = [](uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
  };
  const uint64_t golden = 0x9E3779B97F4A7C15ull;
  const uint64_t key = mix(seed * 0x100000001B3ull + stream * 0x2545F4914F6CDD1Dull + golden);
  for (int64_t i = 0; i < n; ++i)
    out[i] = (double)(mix(key + (uint64_t)i * golden) >> 11) * (1.0 / 9007199254740992.0);
}

}  // namespace

void init_f64_attributes() {
  const int big = (int)(sizeof(double) * (kMaxRank * kMaxRank + 32 * kMaxRank));
  cudaFuncSetAttribute(mttkrp_f64_kernel<24>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)f64_smem<24>());
  cudaFuncSetAttribute(mttkrp_f64_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)f64_smem<32>());
  cudaFuncSetAttribute(solve_f64_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(solve_f64_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(solve_f64_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(solve_f64_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(solve_f64_kernel<5>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(solve_f64_kernel<6>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
  cudaFuncSetAttribute(solve_f64_kernel<7>, cudaFuncAttributeMaxDynamicSharedMemorySize, big);
}

// Gives a call's larger device copies back when it ends: an FP64 tensor may be
// most of the GPU, and the context would keep it until it is destroyed. Slots
// that an earlier call had already grown, and small ones (kept, so that repeated
// small calls allocate nothing), stay.
struct ReturnSlots {
  static constexpr size_t kKeep = (size_t)64 << 20;
  static constexpr int kSlots[4] = {SLOT_TENSOR, SLOT_FACTORS, SLOT_OUT, SLOT_PARTIALS};
  tsr_ctx* ctx;
  size_t before[4];
  explicit ReturnSlots(tsr_ctx* c) : ctx(c) {
    for (int i = 0; i < 4; ++i) before[i] = c->slots[kSlots[i]].bytes;
  }
  ~ReturnSlots() {
    for (int i = 0; i < 4; ++i) {
      Buffer& b = ctx->slots[kSlots[i]];
      if (b.bytes <= before[i] || b.bytes <= kKeep) continue;
      cudaStreamSynchronize(ctx->aux);
      cudaStreamSynchronize(ctx->stream);
      cudaFree(b.ptr);
      b.ptr = nullptr;
      b.bytes = 0;
    }
  }
};

// cp_als<f64> on device data (dX row-major FP64; factors FP64 in d_out).
int cp_als_f64_device(tsr_ctx* ctx, const double* dX, int ndim, const int64_t* shape,
                      int64_t rank, int max_iters, double tol, double time_limit_s,
                      double* d_out, tsr_cp_info* info) {
  const auto t_start = std::chrono::steady_clock::now();
  const int R = (int)rank;
  cudaStream_t s = ctx->stream;
  int64_t rmax = 0, n = numel(ndim, shape);
  const double* U[kMaxModes];
  int64_t off = 0;
  for (int m = 0; m < ndim; ++m) {
    U[m] = d_out + off;
    off += shape[m] * R;
    rmax = std::max<int64_t>(rmax, shape[m]);
  }
  const int hist_n = std::max(max_iters, 1);
  void *gp, *mp, *stp;
  TSR_TRY(slot_get(ctx, SLOT_GRAMS, sizeof(double) * (size_t)(2 * ndim + 1) * R * R, &gp));
  TSR_TRY(slot_get(ctx, SLOT_PARTIALS, sizeof(double) * (size_t)rmax * R, &mp));
  TSR_TRY(slot_get(ctx, SLOT_STATE, 256 + sizeof(double) * hist_n, &stp));
  double *grams = (double*)gp, *Mbuf = (double*)mp;
  AlsBuffers b;
  b.grams = grams;
  b.hadam = grams + (size_t)ndim * R * R;
  b.ginv = b.hadam + (size_t)ndim * R * R;
  b.state = (AlsState*)stp;
  b.history = (double*)((char*)stp + 256);
  TSR_CUDA(cudaMemsetAsync(stp, 0, 256 + sizeof(double) * hist_n, s));
  TSR_CUDA(cudaMemsetAsync(grams, 0, sizeof(double) * (2 * ndim + 1) * R * R, s));
  norm_sq_f64_kernel<<<f64_grid(ctx, n), 256, 0, s>>>(dX, n, &b.state->xnorm_sq);
  ctx->launches++;
  for (int m = 0; m < ndim; ++m)
    TSR_TRY(launch_solve_f64(ctx, b, ndim, R, shape[m], nullptr, const_cast<double*>(U[m]),
                             grams + (size_t)m * R * R, false));
  const float ridge = (float)(std::numeric_limits<double>::epsilon() * (double)(R * 10));
  bool by_time = false;
  for (int iter = 0; iter < max_iters; ++iter) {
    if (time_limit_s >= 0.0) {  // core.rs:104-110
      const double el =
          std::chrono::duration<double>(std::chrono::steady_clock::now() - t_start).count();
      if (el > time_limit_s) {
        by_time = true;
        break;
      }
    }
    for (int m = 0; m < ndim; ++m) {
      const bool last = m == ndim - 1;
      // the inverse runs beside the MTTKRP, as in the fp32 sweep
      TSR_CUDA(cudaEventRecord(ctx->ev[0], s));
      TSR_CUDA(cudaStreamWaitEvent(ctx->aux, ctx->ev[0], 0));
      TSR_TRY(launch_chol(ctx, ctx->aux, b, ndim, m, R, ridge, last, tol));
      TSR_CUDA(cudaEventRecord(ctx->ev[1], ctx->aux));
      TSR_TRY(launch_mttkrp_f64(ctx, dX, ndim, shape, U, R, m, Mbuf, &b.state->done));
      TSR_CUDA(cudaStreamWaitEvent(s, ctx->ev[1], 0));
      TSR_TRY(launch_solve_f64(ctx, b, ndim, R, shape[m], Mbuf, const_cast<double*>(U[m]),
                               grams + (size_t)m * R * R, last));
    }
    // the next sweep's first inverse forms this sweep's fit and decides whether
    // to stop; every kernel after a stop returns at once, so the host looks
    // only every kF64Look sweeps (and each sweep under a time limit)
    if (time_limit_s < 0.0 && (iter + 1) % kF64Look != 0) continue;
    TSR_TRY(launch_fit(ctx, s, b, ndim, R, tol));
    AlsState hs;
    TSR_CUDA(cudaMemcpyAsync(&hs, b.state, sizeof(hs), cudaMemcpyDeviceToHost, s));
    TSR_CUDA(cudaStreamSynchronize(s));
    if (hs.status & DS_NOT_SPD)
      return fail(TSR_E_NOT_SPD,
                  "Linear algebra error: Gram matrix is not positive definite (ridge %g also "
                  "failed)",
                  (double)ridge);
    if (hs.done) break;
  }
  if (max_iters > 0) TSR_TRY(launch_fit(ctx, s, b, ndim, R, tol));
  AlsState hs;
  TSR_CUDA(cudaMemcpyAsync(&hs, b.state, sizeof(hs), cudaMemcpyDeviceToHost, s));
  TSR_CUDA(cudaStreamSynchronize(s));
  if (hs.status & DS_NOT_SPD)
    return fail(TSR_E_NOT_SPD,
                "Linear algebra error: Gram matrix is not positive definite (ridge %g also "
                "failed)",
                (double)ridge);
  if (info) {
    info->fit = hs.fit;
    // core.rs:116-124: the time check comes before the sweep is counted
    info->iters = hs.iter;
    info->reason = by_time    ? TSR_REASON_TIME_LIMIT
                   : hs.done ? hs.reason
                             : TSR_REASON_MAX_ITERATIONS;
    info->oscillation_count = hs.osc;
    info->oscillated = hs.osc > 0;
    info->final_fit_change = hs.final_change;
    info->ridge_used = hs.ridge_used;
    if (info->fit_history && hs.iter > 0)
      TSR_CUDA(cudaMemcpy(info->fit_history, b.history, sizeof(double) * hs.iter,
                          cudaMemcpyDeviceToHost));
  }
  return TSR_OK;
}

}  // namespace tsr

using namespace tsr;

extern "C" {

int tsr_mttkrp_f64(tsr_ctx* ctx, const double* tensor, int ndim, const int64_t* shape,
                   const double* const* factors, int n_factors, const int64_t* factor_rows,
                   const int64_t* factor_cols, int mode, double* out) {
  if (!tensor || !shape || !factors || !factor_rows || !factor_cols || !out)
    return fail(TSR_E_INVALID_ARG, "null argument");
  TSR_TRY(validate_mttkrp(ndim, shape, n_factors, factor_rows, factor_cols, mode));
  TSR_TRY(check_sizes(ndim, shape, factor_cols[0]));
  TSR_TRY(check_ctx(ctx));
  const ReturnSlots give_back(ctx);
  const int R = (int)factor_cols[0];
  const int64_t n = numel(ndim, shape);
  int64_t ftotal = 0;
  for (int m = 0; m < ndim; ++m) ftotal += shape[m] * R;
  void *xp, *fp, *mp;
  TSR_TRY(slot_get(ctx, SLOT_TENSOR, sizeof(double) * std::max<int64_t>(n, 1), &xp));
  TSR_TRY(slot_get(ctx, SLOT_FACTORS, sizeof(double) * std::max<int64_t>(ftotal, 1), &fp));
  TSR_TRY(slot_get(ctx, SLOT_OUT, sizeof(double) * std::max<int64_t>(shape[mode] * R, 1), &mp));
  double *dX = (double*)xp, *dF = (double*)fp, *dM = (double*)mp;
  TSR_CUDA(cudaMemcpyAsync(dX, tensor, sizeof(double) * n, cudaMemcpyHostToDevice, ctx->stream));
  const double* U[kMaxModes];
  int64_t off = 0;
  for (int m = 0; m < ndim; ++m) {
    TSR_CUDA(cudaMemcpyAsync(dF + off, factors[m], sizeof(double) * shape[m] * R,
                             cudaMemcpyHostToDevice, ctx->stream));
    U[m] = dF + off;
    off += shape[m] * R;
  }
  TSR_TRY(launch_mttkrp_f64(ctx, dX, ndim, shape, U, R, mode, dM));
  TSR_CUDA(cudaMemcpyAsync(out, dM, sizeof(double) * shape[mode] * R, cudaMemcpyDeviceToHost,
                           ctx->stream));
  TSR_CUDA(cudaStreamSynchronize(ctx->stream));
  return TSR_OK;
}

int tsr_cp_als_f64(tsr_ctx* ctx, const double* tensor, int ndim, const int64_t* shape,
                   int64_t rank, int max_iters, double tol, const double* init_factors,
                   uint64_t seed, double time_limit_s, double* out_factors, tsr_cp_info* info) {
  if (!shape || !tensor || !out_factors) return fail(TSR_E_INVALID_ARG, "null argument");
  // core.rs:82-94 (as the f32 entry point)
  if (rank == 0) return fail(TSR_E_INVALID_RANK, "Invalid rank: %lld", (long long)rank);
  for (int d = 0; d < ndim; ++d)
    if (rank > shape[d]) return fail(TSR_E_INVALID_RANK, "Invalid rank: %lld", (long long)rank);
  if (!(tol >= 0.0 && tol < 1.0)) return fail(TSR_E_INVALID_TOL, "Invalid tolerance: %g", tol);
  TSR_TRY(check_sizes(ndim, shape, rank));
  if (ndim > kMaxModes)
    return fail(TSR_E_UNSUPPORTED, "tensor rank %d exceeds the supported %d", ndim, kMaxModes);
  if (rank > kMaxRank)
    return fail(TSR_E_UNSUPPORTED, "rank %lld exceeds the supported %d", (long long)rank,
                kMaxRank);
  if (ndim < 2 && max_iters > 0)
    return fail(TSR_E_SHAPE, "Shape mismatch: Need at least 2 factor matrices for MTTKRP");
  TSR_TRY(check_ctx(ctx));
  const int64_t n = numel(ndim, shape);
  int64_t ftotal = 0;
  for (int m = 0; m < ndim; ++m) ftotal += shape[m] * rank;
  std::vector<double> init_buf;
  const double* init = init_factors;
  if (!init) {  // InitStrategy::Random from the library's seeded stream, in FP64
    init_buf.resize(ftotal);
    int64_t off = 0;
    for (int m = 0; m < ndim; ++m) {
      seeded_uniform_f64(seed, 200 + m, shape[m] * rank, init_buf.data() + off);
      off += shape[m] * rank;
    }
    init = init_buf.data();
  }
  const ReturnSlots give_back(ctx);
  void *xp, *fp;
  TSR_TRY(slot_get(ctx, SLOT_TENSOR, sizeof(double) * std::max<int64_t>(n, 1), &xp));
  TSR_TRY(slot_get(ctx, SLOT_FACTORS, sizeof(double) * std::max<int64_t>(ftotal, 1), &fp));
  double *dX = (double*)xp, *dF = (double*)fp;
  TSR_CUDA(cudaMemcpyAsync(dX, tensor, sizeof(double) * n, cudaMemcpyHostToDevice, ctx->stream));
  TSR_CUDA(cudaMemcpyAsync(dF, init, sizeof(double) * ftotal, cudaMemcpyHostToDevice,
                           ctx->stream));
  TSR_TRY(cp_als_f64_device(ctx, dX, ndim, shape, rank, max_iters, tol, time_limit_s, dF, info));
  TSR_CUDA(cudaMemcpyAsync(out_factors, dF, sizeof(double) * ftotal, cudaMemcpyDeviceToHost,
                           ctx->stream));
  TSR_CUDA(cudaStreamSynchronize(ctx->stream));
  return TSR_OK;
}

}  // extern "C"
