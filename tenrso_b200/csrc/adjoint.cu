// CP reconstruction, its adjoint, and the loss/gradient of a CP model.
//
//   tenrso_kernels::cp_reconstruct                  crates/tenrso-kernels/src/outer.rs:223-274
//     Xhat = sum_r w_r U_0[:, r] o U_1[:, r] o ... o U_{N-1}[:, r]
//   CpReconstructionGrad::compute_factor_gradients  crates/tenrso-ad/src/grad.rs:81-120
//     dL/dU_n = unfold(G, n) . KR_{m != n}(U_m) . diag(w),  G = dL/dXhat
//   that is, the MTTKRP of G; the Khatri-Rao rows are formed on the fly by the
//   MTTKRP kernels and never stored (grad.rs:128-150 materialises them).
//
// The loss/gradient entry evaluates  L = ||X - [[U]]||^2 + reg * sum_n ||U_n||^2
// and all dL/dU_n without forming Xhat, from the Gram identities
//   ||Xhat||^2   = sum_{r,s} prod_n (U_n^T U_n)[r, s]
//   <X, Xhat>    = sum_{i,r} MTTKRP(X, 0)[i, r] U_0[i, r]
//   dL/dU_n      = 2 (U_n H_n - MTTKRP(X, n)) + 2 reg U_n,  H_n = *_{m != n} U_m^T U_m
// with the Grams, H_n, the loss and the U_n H_n product in FP64.
#include <cstring>

#include "als.cuh"
#include "dense.cuh"

// A dense tensor prepared for repeated MTTKRPs: FP32 reads the tensor in
// place, BF16x3 keeps what its kernels read (halves in X's own layout, or
// unfoldings) in HBM. The tensor itself stays the caller's and must not change
// while the object is in use.
struct tsr_dense {
  int ndim = 0;
  int64_t shape[tsr::kMaxModes] = {};
  int precision = 0;
  int device = 0;
  const float* dX = nullptr;
  void* owned[2 * tsr::kMaxModes + 2] = {};
  tsr::ModeOperand ops[tsr::kMaxModes];
  double* d_scalars = nullptr;  // [0] ||X||^2, [1] <X, Xhat>, [2] loss, [3] scratch
  // BF16x3 tensors of 3 or more modes whose trailing-two-modes view
  // (prod of the leading modes, I_{N-2}, I_{N-1}) suits the two-sided
  // contraction or the single-layout 3-way MTTKRP: X's bf16 halves in its own
  // layout (owned[2N], owned[2N+1])
  bool d3_on = false;
  bool d3_three = false;  // the view suits the single-layout 3-way MTTKRP
  bool d3_two = false;    // the view suits the two-sided contraction
  tsr::Dense3 d3{};
  // Tensors of 3 or more modes without that copy: T and P contracted in FP32
  // from X seen as an A x C matrix (A the leading modes' product, C = I_{N-2}
  // I_{N-1})
  bool v2_on = false;
  int64_t v2_shape[2] = {0, 0};
};

namespace tsr {

namespace {

constexpr int RC_THREADS = 256;
constexpr int RC_TILE = 128;  // output tile: 128 rows x 128 columns, 8 x 8 per thread
constexpr int RC_CHUNK = 32;  // rank columns staged in shared memory per pass

// The row-major output seen as a P x Lc matrix: rows run over modes
// [0, split), columns over the trailing modes [split, N) (the last fastest),
// so element (p, c) sits at p * Lc + c. Both operands of the tile product are
// Khatri-Rao rows built from the factors inside the kernel.
struct ReconArgs {
  FactorTable ft;
  int ndim;
  int split;
  int R;
  int64_t P, Lc;
  int64_t col_tiles;
  const float* w;    // weights (R) or null for all ones
  const float* X;    // residual mode: the target tensor
  float* out;        // Xhat, or alpha * (Xhat - X)
  float alpha;
  double* sq_err;    // residual mode: sum of (Xhat - X)^2 added here
};

__device__ __forceinline__ void rc_fma2(uint64_t& d, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// Stages ranks r0 .. r0 + RC_CHUNK - 1 of the KR row `idx` over modes [m0, m1)
// into column `at` of dst (rank-major), ranks [rb, rb + RC_CHUNK / 2) of it;
// zero past R and for rows outside the tensor (ok false).
__device__ __forceinline__ void rc_stage(const ReconArgs& a, int m0, int m1, int64_t idx, bool ok,
                                         const float* scale, int r0, int rb, float* dst, int at) {
  constexpr int H = RC_CHUNK / 2;
  float v[H];
#pragma unroll
  for (int r = 0; r < H; ++r) {
    const int rr = r0 + rb + r;
    v[r] = ok && rr < a.R ? (scale ? __ldg(scale + rr) : 1.f) : 0.f;
  }
  for (int m = m1 - 1; m >= m0; --m) {
    const int64_t n = a.ft.rows[m], q = m > m0 ? idx / n : 0;
    const float* row = a.ft.ptr[m] + (ok ? (idx - q * n) * a.R : 0) + r0 + rb;
    idx = q;
#pragma unroll
    for (int r = 0; r < H; ++r)
      if (r0 + rb + r < a.R) v[r] *= __ldg(row + r);
  }
#pragma unroll
  for (int r = 0; r < H; ++r) dst[(rb + r) * RC_TILE + at] = v[r];
}

// A CTA owns 128 rows and walks column tiles, so the row operand is staged
// once (per 32 ranks). A thread owns rows ty 4 + {0..3} (+ 64) and columns
// tx + 16 j: the column operand is stored permuted so that one 128-bit word
// holds four of them, and a warp's stores cover whole 64-byte runs whatever
// the alignment. Packed fp32 FMAs over column pairs. Bound: 137 MB written
// (21 us at HBM rate) and 0.82e9 FMAs (23 us) at 121x95x63x47 rank 24.
template <bool RESIDUAL>
__global__ void __launch_bounds__(RC_THREADS, 2)
reconstruct_kernel(const __grid_constant__ ReconArgs a) {
  __shared__ __align__(16) float Ws[RC_CHUNK * RC_TILE];
  __shared__ __align__(16) float Vs[RC_CHUNK * RC_TILE];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int si = threadIdx.x & (RC_TILE - 1), sh = (threadIdx.x / RC_TILE) * (RC_CHUNK / 2);
  const int64_t p0 = (int64_t)blockIdx.y * RC_TILE;
  const int64_t ps = p0 + si;
  // column si of a tile sits at word (si % 16) of half si / 64, element (si / 16) % 4
  const int vat = (si >> 6) * 64 + (si & 15) * 4 + ((si >> 4) & 3);
  double sq = 0.0;
  for (int64_t ct = blockIdx.x; ct < a.col_tiles; ct += gridDim.x) {
    const int64_t c0 = ct * RC_TILE, cs = c0 + si;
    uint64_t acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0;
    for (int r0 = 0; r0 < a.R; r0 += RC_CHUNK) {
      __syncthreads();
      if (a.R > RC_CHUNK || ct == blockIdx.x)
        rc_stage(a, 0, a.split, ps, ps < a.P, a.w, r0, sh, Ws, si);
      rc_stage(a, a.split, a.ndim, cs, cs < a.Lc, nullptr, r0, sh, Vs, vat);
      __syncthreads();
      const int rn = a.R - r0 < RC_CHUNK ? a.R - r0 : RC_CHUNK;
#pragma unroll 2
      for (int r = 0; r < rn; ++r) {
        const float4 w0 = *reinterpret_cast<const float4*>(Ws + r * RC_TILE + ty * 4);
        const float4 w1 = *reinterpret_cast<const float4*>(Ws + r * RC_TILE + 64 + ty * 4);
        const ulonglong2 v0 = *reinterpret_cast<const ulonglong2*>(Vs + r * RC_TILE + tx * 4);
        const ulonglong2 v1 = *reinterpret_cast<const ulonglong2*>(Vs + r * RC_TILE + 64 + tx * 4);
        const float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          uint64_t d;
          asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(wv[i]));
          rc_fma2(acc[i][0], d, v0.x);
          rc_fma2(acc[i][1], d, v0.y);
          rc_fma2(acc[i][2], d, v1.x);
          rc_fma2(acc[i][3], d, v1.y);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int64_t p = p0 + ty * 4 + (i & 3) + (i >> 2) * 64;
      if (p >= a.P) continue;
      const int64_t base = p * a.Lc + c0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int c = tx + 16 * j;
        if (c0 + c >= a.Lc) continue;
        const uint64_t u = acc[i][j >> 1];
        float v = __uint_as_float((uint32_t)((j & 1) ? u >> 32 : u));
        if (RESIDUAL) {
          const float d = v - __ldg(a.X + base + c);
          sq += (double)d * d;
          v = a.alpha * d;
        }
        __stcs(a.out + base + c, v);
      }
    }
  }
  if (RESIDUAL) {
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(a.sq_err, sq);
  }
}

__device__ __forceinline__ double sym_at(const double* g, int R, int a, int c) {
  return a <= c ? g[a * R + c] : g[c * R + a];
}

// Gradient rows of one mode in Gram form:
//   out[i, :] = 2 (U[i, :] H - M[i, :] + reg U[i, :]),  H = *_{m != mode} Gram_m
// where M is the sum of the split MTTKRP partials. Mode 0 also accumulates
// <M, U> (= <X, Xhat>) into scal[1]. Shared (FP64): H (R x R), M (rows x R),
// and the per-group partial sums: `groups` threads share one element of M and
// each sums a strided subset of the splits with 8 loads in flight.
__device__ __forceinline__ void gram_grad_block(
    const double* __restrict__ grams, int ndim, int mode, const float* __restrict__ partials,
    int splits, int64_t rows, int R, int rows_per_cta, const float* __restrict__ U, double reg,
    float* __restrict__ out, double* scal, int64_t blk, double* sh) {
  const int RR = R * R;
  double* H = sh;
  double* Ms = sh + RR;
  for (int e = threadIdx.x; e < RR; e += blockDim.x) {
    const int a = e / R, c = e % R;
    double h = 1.0;
    for (int m = 0; m < ndim; ++m)
      if (m != mode) h *= sym_at(grams + (int64_t)m * RR, R, a, c);
    H[e] = h;
  }
  const int64_t r0 = blk * rows_per_cta;
  const int nr = (int)(rows - r0 < rows_per_cta ? rows - r0 : rows_per_cta);
  const int64_t pstride = rows * R;
  const int ne = nr * R;
  const int full = rows_per_cta * R;
  const int groups = full >= (int)blockDim.x ? 1 : (int)blockDim.x / full;
  double* red = Ms + full;  // [groups][ne]
  for (int t = threadIdx.x; t < ne * groups; t += blockDim.x) {
    const int e = t % ne, g = t / ne;
    const float* p = partials + r0 * R + e;
    double s = 0.0;
    int q = g;
    for (; q + 7 * groups < splits; q += 8 * groups) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = __ldg(p + (int64_t)(q + u * groups) * pstride);
#pragma unroll
      for (int u = 0; u < 8; ++u) s += (double)v[u];
    }
    for (; q < splits; q += groups) s += (double)__ldg(p + (int64_t)q * pstride);
    red[g * ne + e] = s;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < ne; e += blockDim.x) {
    double s = 0.0;
    for (int g = 0; g < groups; ++g) s += red[g * ne + e];
    Ms[e] = s;
  }
  __syncthreads();
  double ip = 0.0;
  for (int e = threadIdx.x; e < ne; e += blockDim.x) {
    const int i = e / R, c = e % R;
    const float* urow = U + (r0 + i) * R;
    double s0 = 0.0, s1 = 0.0;
    int k = 0;
    for (; k + 2 <= R; k += 2) {
      s0 += (double)__ldg(urow + k) * H[k * R + c];
      s1 += (double)__ldg(urow + k + 1) * H[(k + 1) * R + c];
    }
    if (k < R) s0 += (double)__ldg(urow + k) * H[k * R + c];
    const double u = (double)__ldg(urow + c);
    out[(r0 + i) * R + c] = (float)(2.0 * ((s0 + s1) - Ms[e] + reg * u));
    ip += Ms[e] * u;
  }
  if (mode == 0) {
    for (int o = 16; o > 0; o >>= 1) ip += __shfl_down_sync(0xffffffffu, ip, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(scal + 1, ip);
  }
}

__global__ void __launch_bounds__(256)
gram_grad_kernel(const double* __restrict__ grams, int ndim, int mode,
                 const float* __restrict__ partials, int splits, int64_t rows, int R,
                 int rows_per_cta, const float* __restrict__ U, double reg,
                 float* __restrict__ out, double* scal) {
  extern __shared__ double sh[];
  gram_grad_block(grams, ndim, mode, partials, splits, rows, R, rows_per_cta, U, reg, out, scal,
                  blockIdx.x, sh);
}

// sum_{r,s} prod_n Gram_n[r, s] + reg sum_n tr(Gram_n) over one CTA of
// `blockDim.x` threads (a multiple of 32), valid in thread 0
__device__ __forceinline__ double gram_loss_part(const double* __restrict__ grams, int ndim, int R,
                                                 double reg) {
  const int RR = R * R;
  double s = 0.0;
  for (int e = threadIdx.x; e < RR; e += blockDim.x) {
    const int a = e / R, c = e % R;
    double h = 1.0, tr = 0.0;
    for (int m = 0; m < ndim; ++m) {
      const double g = sym_at(grams + (int64_t)m * RR, R, a, c);
      h *= g;
      if (a == c) tr += g;
    }
    s += h + reg * tr;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  __shared__ double ws[32];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += ws[w];
  return t;
}

// loss = ||X||^2 - 2 <X, Xhat> + sum_{r,s} prod_n Gram_n[r, s] + reg sum_n tr(Gram_n)
__global__ void gram_loss_kernel(const double* __restrict__ grams, int ndim, int R, double reg,
                                 double* scal) {
  const double t = gram_loss_part(grams, ndim, R, reg);
  if (threadIdx.x == 0) scal[2] = scal[0] - 2.0 * scal[1] + t;
}

// MTTKRPs from a partial contraction. A side holds S (rows a over nlead
// modes, row-major, fewer than 2^31 rows) with
//   S[a, r] = sum over the other modes of X[a, ...] prod_{other p} U_p[., r],
// and the mode-m MTTKRP of one of its modes is
//   M_m[i, r] = sum_{a : a_m = i} S[a, r] prod_{p in side, p != m} U_p[a_p, r].
// The leading modes 0..N-3 come from T (S over the leading modes, the
// trailing two contracted), the trailing two from P (S over (I_{N-2},
// I_{N-1}), the leading modes contracted). One launch for every requested
// mode: block b is row i of mode n (the modes' rows stacked in `out`), lane r
// of a group of R threads, the groups split the side's other indices; FP64
// sums, fp32 output.
struct TSideC {
  const float* S;
  int nlead;
  int arows;
  int size[kMaxModes];
  int stride[kMaxModes];
  const float* U[kMaxModes];
};

struct TContract {
  TSideC side[2];
  int R, nmodes;
  int side_of[kMaxModes];  // output mode -> side
  int pos[kMaxModes];      // output mode -> its index within the side
  int row0[kMaxModes + 1];
  float* out[kMaxModes];  // per mode: I_m x R
  const float* w;         // column scale (R), or null
};

// Thread (g, r)'s share of M_m[i, r]: groups g < groups split the side's
// other indices (FP64).
__device__ __forceinline__ double t_contract_part(const TSideC& sd, int m, int i, int R, int g,
                                                  int groups, int r) {
  double s = 0.0;
  if (g >= groups) return s;
  if (sd.nlead == 2) {
    // the other mode's index is the loop index: four independent loads per step
    const int o = 1 - m;
    const int cnt = sd.size[o], so = sd.stride[o];
    const float* Sp = sd.S + (int64_t)i * sd.stride[m] * R + r;
    const float* Uo = sd.U[o] + r;
    int q = g;
    for (; q + 3 * groups < cnt; q += 4 * groups) {
      float sv[4], wv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        sv[u] = __ldg(Sp + (int64_t)(q + u * groups) * so * R);
        wv[u] = __ldg(Uo + (int64_t)(q + u * groups) * R);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) s += (double)sv[u] * (double)wv[u];
    }
    for (; q < cnt; q += groups)
      s += (double)__ldg(Sp + (int64_t)q * so * R) * (double)__ldg(Uo + (int64_t)q * R);
    return s;
  }
  const int count = sd.arows / sd.size[m];
  for (int q = g; q < count; q += groups) {
    int rem = q, a = i * sd.stride[m];
    double w = 1.0;
    for (int p = sd.nlead - 1; p >= 0; --p) {
      if (p == m) continue;
      const int ip = rem % sd.size[p];
      rem /= sd.size[p];
      a += ip * sd.stride[p];
      w *= (double)__ldg(sd.U[p] + (int64_t)ip * R + r);
    }
    s += (double)__ldg(sd.S + (int64_t)a * R + r) * w;
  }
  return s;
}

__global__ void __launch_bounds__(256) t_contract_kernel(const __grid_constant__ TContract c) {
  __shared__ double part[256];
  const int b = blockIdx.x;
  int n = 0;
  while (n + 1 < c.nmodes && b >= c.row0[n + 1]) ++n;
  const int R = c.R;
  const int groups = blockDim.x / R;
  part[threadIdx.x] = t_contract_part(c.side[c.side_of[n]], c.pos[n], b - c.row0[n], R,
                                      threadIdx.x / R, groups, threadIdx.x % R);
  __syncthreads();
  if (threadIdx.x < R) {
    double t = 0.0;
    for (int q = 0; q < groups; ++q) t += part[q * R + threadIdx.x];
    if (c.w) t *= (double)__ldg(c.w + threadIdx.x);
    c.out[n][(int64_t)(b - c.row0[n]) * R + threadIdx.x] = (float)t;
  }
}

// The same contraction with the gradient row formed in place (R <= 32): block
// b is row i of mode n; with M_n[i, :] reduced in shared memory,
//   grad[i, c] = 2 (sum_k U_n[i, k] H_n[k, c] - M_n[i, c] + reg U_n[i, c]),
// H_n = *_{m != n} Gram_m formed by the block (FP64, the Grams stay in L1).
// Mode-0 rows add <M_0, U_0> (= <X, Xhat>) into scal[1]; the extra last
// block writes the Gram part of the loss into scal[3].
struct GradArgs {
  const double* grams;
  int ndim;
  double reg;
  float* G[kMaxModes];
  double* scal;
};

__global__ void __launch_bounds__(256)
t_contract_grad_kernel(const __grid_constant__ TContract c, const __grid_constant__ GradArgs ga) {
  __shared__ double part[256];
  __shared__ double H[32 * 32];
  __shared__ double Mrow[32];
  // programmatic launch: T, P and, through the earlier kernels' own waits,
  // the Grams are complete once the predecessor is
  grid_dep_wait();
  const int b = blockIdx.x;
  const int R = c.R;
  if (b >= c.row0[c.nmodes]) {
    const double t = gram_loss_part(ga.grams, ga.ndim, R, ga.reg);
    if (threadIdx.x == 0) ga.scal[3] = t;
    return;
  }
  int n = 0;
  while (n + 1 < c.nmodes && b >= c.row0[n + 1]) ++n;
  const TSideC& sd = c.side[c.side_of[n]];
  const int m = c.pos[n], i = b - c.row0[n];
  const int groups = blockDim.x / R;
  part[threadIdx.x] = t_contract_part(sd, m, i, R, threadIdx.x / R, groups, threadIdx.x % R);
  const int RR = R * R;
  for (int e = threadIdx.x; e < RR; e += blockDim.x) {
    const int a = e / R, cc = e % R;
    double h = 1.0;
    for (int q = 0; q < ga.ndim; ++q)
      if (q != n) h *= sym_at(ga.grams + (int64_t)q * RR, R, a, cc);
    H[e] = h;
  }
  __syncthreads();
  if (threadIdx.x < R) {
    double t = 0.0;
    for (int q = 0; q < groups; ++q) t += part[q * R + threadIdx.x];
    Mrow[threadIdx.x] = t;
  }
  __syncthreads();
  if (threadIdx.x < 32) {  // R <= 32: one warp
    const int cc = threadIdx.x;
    double ip = 0.0;
    if (cc < R) {
      const float* urow = sd.U[m] + (int64_t)i * R;
      double s0 = 0.0, s1 = 0.0;
      int k = 0;
      for (; k + 2 <= R; k += 2) {
        s0 += (double)__ldg(urow + k) * H[k * R + cc];
        s1 += (double)__ldg(urow + k + 1) * H[(k + 1) * R + cc];
      }
      if (k < R) s0 += (double)__ldg(urow + k) * H[k * R + cc];
      const double u = (double)__ldg(urow + cc);
      ga.G[n][(int64_t)i * R + cc] = (float)(2.0 * ((s0 + s1) - Mrow[cc] + ga.reg * u));
      ip = Mrow[cc] * u;
    }
    if (n == 0) {
      for (int o = 16; o > 0; o >>= 1) ip += __shfl_down_sync(0xffffffffu, ip, o);
      if (cc == 0) atomicAdd(ga.scal + 1, ip);
    }
  }
}

// side k of c over modes m0 .. m1-1 of the tensor, the partial contraction S
void set_side(TContract& c, int k, const float* S, const int64_t* shape, int m0, int m1,
              const float* const* U) {
  TSideC& sd = c.side[k];
  sd.S = S;
  sd.nlead = m1 - m0;
  int st = 1;
  for (int p = m1 - 1; p >= m0; --p) {
    sd.size[p - m0] = (int)shape[p];
    sd.stride[p - m0] = st;
    sd.U[p - m0] = U[p];
    st *= (int)shape[p];
  }
  sd.arows = st;
}

int64_t prod_range(const int64_t* shape, int m0, int m1) {
  int64_t p = 1;
  for (int m = m0; m < m1; ++m) p *= shape[m];
  return p;
}

// T (A x R) = X KR(trailing two) and P (C x R) = X^T KR(leading modes) of X
// seen as A x C (N >= 3 modes, row-major), read in place.
int contract_sides(tsr_ctx* ctx, const float* dX, int N, const int64_t* shape,
                   const float* const* U, int R, float* T, float* P) {
  const int64_t A = prod_range(shape, 0, N - 2), C = shape[N - 2] * shape[N - 1];
  // T is the mode-0 MTTKRP of X seen as (A, I_{N-2}, I_{N-1}), P the last
  // mode's of X seen as (I_0, .., I_{N-3}, C)
  const int64_t tshape[3] = {A, shape[N - 2], shape[N - 1]};
  const float* tf[3] = {nullptr, U[N - 2], U[N - 1]};
  int64_t pshape[kMaxModes];
  const float* pf[kMaxModes];
  for (int m = 0; m < N - 2; ++m) {
    pshape[m] = shape[m];
    pf[m] = U[m];
  }
  pshape[N - 2] = C;
  pf[N - 2] = nullptr;
  for (int v = 0; v < 2; ++v) {
    const int nd = v == 0 ? 3 : N - 1, mode = v == 0 ? 0 : N - 2;
    const int64_t* sh = v == 0 ? tshape : pshape;
    const int64_t rows = v == 0 ? A : C;
    const ViewPlan plan = plan_view(ctx, nd, sh, mode, R, 0);
    float* dst = v == 0 ? T : P;
    float* out = dst;
    if (plan.splits > 1) {
      void* p;
      TSR_TRY(slot_get(ctx, SLOT_PARTIALS, sizeof(float) * (size_t)plan.splits * rows * R, &p));
      out = (float*)p;
    }
    TSR_TRY(launch_view(ctx, ctx->stream, dX, nd, sh, mode, v == 0 ? tf : pf, R, plan, out));
    if (plan.splits > 1)
      TSR_TRY(launch_mttkrp_reduce(ctx, out, plan.splits, rows * R, dst));
  }
  return TSR_OK;
}

// Microseconds of the longest block of the contraction of T and P: each row of
// each mode is one block, whose threads walk the other indices of its side,
// about 0.25 us per step of the 256 threads. A short mode beside a long one has
// few blocks of very many steps.
double contract_estimate_us(int N, const int64_t* shape, int R) {
  const int64_t A = prod_range(shape, 0, N - 2), C = shape[N - 2] * shape[N - 1];
  double steps = 0.0;
  for (int m = 0; m < N; ++m)
    if (m >= N - 2 || N > 3)  // (a side of one mode is its own result)
      steps = std::max(steps, (double)((m < N - 2 ? A : C) / shape[m]) * R / 256.0);
  return 0.25 * steps;
}

// Whether T and P (two passes over X, both no larger than X) and their
// contraction pay against one FP32 pass per mode with its launches and gaps
// (16 us, so that near-ties stay with two passes). Measured, us, per mode / two passes:
// 100 x 2 x 200000 rank 32 1945 / 11709, 30 x 30 x 4000 rank 16 64 / 101,
// 40 x 3000 x 2 x 2 x 40 rank 16 1340 / 5016; and the other way 128^3 rank 32
// 59 / 50, 100 x 2 x 20000 rank 4 145 / 113, 64 x 64 x 2 x 20000 rank 64
// 17523 / 3849, 10^6 rank 16 163 / 97, 3000 x 2 x 2 x 2 x 40 x 40 rank 32
// 7552 / 1584.
bool sides_pay(int N, const int64_t* shape, int R) {
  const int64_t A = prod_range(shape, 0, N - 2), C = shape[N - 2] * shape[N - 1];
  if (A < R || C < R) return false;
  double passes = 16.0 * (N - 2);
  for (int m = 0; m < N; ++m) passes += view_estimate_us(shape[m], A * C / shape[m], R);
  passes -= view_estimate_us(A, C, R) + view_estimate_us(C, A, R);
  return contract_estimate_us(N, shape, R) <= passes;
}

// The same choice for a prepared BF16x3 tensor without a copy in X's own
// layout, whose alternative is one tensor-core pass over each mode's bf16
// unfolding: about 25 us, the 4 bytes per element, and the Khatri-Rao rows (0.2
// ns per column, 0.8 from four modes on). T and P go through memory three times
// and may not take much more of it than X. Measured, us, tensor cores / two
// passes: 301 x 223 x 187 rank 32 156 / 126, 401 x 399 x 397 rank 16 302 / 257,
// 97 x 83 x 61 x 45 rank 32 1000 / 186; and 401 x 399 x 397 rank 32 327 / 384,
// 501 x 499 x 497 rank 8 400 / 479, 33 x 41 x 20001 rank 32 365 / 718,
// 5 x 3001 x 1001 rank 32 649 / 772.
bool sides_pay_prepared(int N, const int64_t* shape, int R) {
  const int64_t A = prod_range(shape, 0, N - 2), C = shape[N - 2] * shape[N - 1];
  const int64_t n = A * C;
  if ((A + C) * R > std::max<int64_t>(2 * n, (int64_t)1 << 26)) return false;
  const double two = view_estimate_us(A, C, R) + view_estimate_us(C, A, R) +
                     contract_estimate_us(N, shape, R) + 12.0 * (double)((A + C) * R) / 6.4e6;
  double tc = 0.0;
  for (int m = 0; m < N; ++m)
    tc += 25.0 + (double)(n / shape[m]) * (N == 3 ? 0.2e-3 : 0.8e-3) + 0.62e-6 * (double)n;
  return 1.1 * two <= tc;
}

// The four loss scalars and the status word in one read-back into pinned
// memory and one synchronization.
int read_scalars(tsr_ctx* ctx, const double* d_scalars, double (&sc)[4]) {
  void* rb;
  TSR_TRY(readback_get(ctx, sizeof(sc) + 16, &rb));
  uint8_t* b = (uint8_t*)rb;
  TSR_CUDA(cudaMemcpyAsync(b, d_scalars, sizeof(sc), cudaMemcpyDeviceToHost, ctx->stream));
  TSR_CUDA(cudaMemcpyAsync(b + sizeof(sc), ctx->d_status, sizeof(unsigned),
                           cudaMemcpyDeviceToHost, ctx->stream));
  TSR_CUDA(cudaStreamSynchronize(ctx->stream));
  std::memcpy(sc, b, sizeof(sc));
  unsigned st;
  std::memcpy(&st, b + sizeof(sc), sizeof(st));
  if (st) TSR_TRY(reset_status(ctx));
  if (st & DS_TIMEOUT) return fail(TSR_E_TIMEOUT, "device wait timed out in the MTTKRP kernel");
  return TSR_OK;
}

// Shared validation of tenrso's cp_reconstruct (outer.rs:231-255).
int validate_reconstruct(int n_factors, const int64_t* fcols, int64_t n_weights, bool has_w) {
  if (n_factors <= 0)
    return fail(TSR_E_SHAPE, "Need at least one factor matrix for CP reconstruction");
  const int64_t R = fcols[0];
  for (int i = 0; i < n_factors; ++i)
    if (fcols[i] != R)
      return fail(TSR_E_RANK_MISMATCH, "Factor %d has %lld columns, expected %lld", i,
                  (long long)fcols[i], (long long)R);
  if (has_w && n_weights != R)
    return fail(TSR_E_SHAPE, "Weights length %lld must match rank %lld", (long long)n_weights,
                (long long)R);
  if (n_factors > kMaxModes)
    return fail(TSR_E_UNSUPPORTED, "tensor rank %d exceeds the supported %d", n_factors,
                kMaxModes);
  return TSR_OK;
}

}  // namespace

void init_adjoint_attributes() {
  cudaFuncSetAttribute(gram_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
}

// Xhat (or alpha * (Xhat - X) with sum of squares) on the context's stream.
int launch_reconstruct(tsr_ctx* ctx, const FactorTable& ft, int ndim, int R, const float* w,
                       const float* X, float alpha, double* sq_err, float* out) {
  ReconArgs a;
  std::memset(&a, 0, sizeof(a));
  a.ft = ft;
  a.ndim = ndim;
  a.R = R;
  a.w = w;
  a.X = X;
  a.out = out;
  a.alpha = alpha;
  a.sq_err = sq_err;
  int64_t shape[kMaxModes];
  for (int m = 0; m < ndim; ++m) shape[m] = ft.rows[m];
  // the row / column split whose 128 x 128 tiles hold the least padding (ties:
  // the most columns), rows within the grid's y extent
  int64_t best = INT64_MAX;
  for (int split = 0; split < ndim; ++split) {
    const int64_t p = prod_range(shape, 0, split), l = prod_range(shape, split, ndim);
    if (p == 0 || l == 0) return TSR_OK;
    const int64_t rt = ceil_div(p, RC_TILE);
    const int64_t tiles = rt * ceil_div(l, RC_TILE);
    if (rt <= 65535 && tiles < best) {
      best = tiles;
      a.split = split;
      a.P = p;
      a.Lc = l;
    }
  }
  a.col_tiles = ceil_div(a.Lc, RC_TILE);
  const int64_t row_tiles = ceil_div(a.P, RC_TILE);
  // about four CTAs per resident slot: enough to even out the last wave, few
  // enough that a CTA's rows are staged once for several column tiles
  const int64_t gx = std::min<int64_t>(
      a.col_tiles, std::max<int64_t>(1, ceil_div(8 * (int64_t)ctx->sm_count, row_tiles)));
  const dim3 grid((unsigned)gx, (unsigned)row_tiles);
  if (X) reconstruct_kernel<true><<<grid, RC_THREADS, 0, ctx->stream>>>(a);
  else reconstruct_kernel<false><<<grid, RC_THREADS, 0, ctx->stream>>>(a);
  ctx->launches++;
  TSR_CUDA(cudaGetLastError());
  return TSR_OK;
}

namespace {

// dL/dU_n for every mode of a device gradient tensor G (grad.rs:81-120).
int reconstruction_grad_device(tsr_ctx* ctx, const float* dG, int ndim, const int64_t* shape,
                               const FactorTable& ft, int R, const float* dw, int precision,
                               float* const* d_out) {
  // Three or more modes: two FP32 passes over G (T and P) and a small
  // contraction of each instead of one pass per mode, where that pays.
  // 121x95x63x47 rank 24: 4 FP32 passes 390 us, this 190. A BF16x3 request
  // takes it too: G comes new with every call, so each of its N passes would
  // first write a bf16 unfolding.
  const int64_t total = numel(ndim, shape);
  if (ndim >= 3 && R >= 1 && R <= 256 && total > 0) {
    const int64_t A = prod_range(shape, 0, ndim - 2), C = shape[ndim - 2] * shape[ndim - 1];
    if (sides_pay(ndim, shape, R) && A <= ((int64_t)1 << 30) && C < INT32_MAX) {
      void* tp;
      TSR_TRY(slot_get(ctx, SLOT_MISC1, sizeof(float) * (A + C) * R, &tp));
      float *T = (float*)tp, *P = T + A * R;
      TSR_TRY(contract_sides(ctx, dG, ndim, shape, ft.ptr, R, T, P));
      TContract c{};
      set_side(c, 0, T, shape, 0, ndim - 2, ft.ptr);
      set_side(c, 1, P, shape, ndim - 2, ndim, ft.ptr);
      c.R = R;
      c.nmodes = ndim;
      c.w = dw;
      for (int m = 0; m < ndim; ++m) {
        c.side_of[m] = m < ndim - 2 ? 0 : 1;
        c.pos[m] = m < ndim - 2 ? m : m - (ndim - 2);
        c.row0[m + 1] = c.row0[m] + (int)shape[m];
        c.out[m] = d_out[m];
      }
      t_contract_kernel<<<(unsigned)c.row0[ndim], 256, 0, ctx->stream>>>(c);
      ctx->launches++;
      TSR_CUDA(cudaGetLastError());
      return TSR_OK;
    }
  }
  for (int n = 0; n < ndim; ++n) {
    if (shape[n] == 0) continue;
    if (numel(ndim, shape) == 0 || R == 0) {
      TSR_CUDA(cudaMemsetAsync(d_out[n], 0, sizeof(float) * shape[n] * R, ctx->stream));
      continue;
    }
    // the precision a single MTTKRP of G would run in
    const int prec = mttkrp_precision(ctx, ndim, shape, n, R, precision);
    ModeOperand op;
    TSR_TRY(prepare_mode(ctx, dG, ndim, shape, n, prec, 0, &op));
    float* partials;
    int splits;
    TSR_TRY(run_mttkrp_partials(ctx, op, ft, R, prec, &partials, &splits));
    TSR_TRY(launch_mttkrp_reduce_scaled(ctx, partials, splits, shape[n], R, dw, d_out[n]));
  }
  return TSR_OK;
}

int validate_grad(int g_ndim, const int64_t* shape, int n_factors, const int64_t* frows,
                  const int64_t* fcols) {
  // grad.rs:84-91
  if (g_ndim != n_factors)
    return fail(TSR_E_SHAPE, "Gradient rank %d doesn't match number of factors %d", g_ndim,
                n_factors);
  // grad.rs:137-139: the Khatri-Rao product of the other factors needs one
  if (n_factors < 2)
    return fail(TSR_E_NEED_2_FACTORS, "Need at least one factor for Khatri-Rao product");
  return validate_mttkrp(g_ndim, shape, n_factors, frows, fcols, 0);
}

}  // namespace

}  // namespace tsr

using namespace tsr;

extern "C" {

int tsr_cp_reconstruct_f32(tsr_ctx* ctx, const float* const* factors, int n_factors,
                           const int64_t* factor_rows, const int64_t* factor_cols,
                           const float* weights, int64_t n_weights, float* out) {
  if (n_factors > 0 && (!factors || !factor_rows || !factor_cols))
    return fail(TSR_E_INVALID_ARG, "null argument");
  TSR_TRY(validate_reconstruct(n_factors, factor_cols, n_weights, weights != nullptr));
  if (!out) return fail(TSR_E_INVALID_ARG, "null argument");
  TSR_TRY(check_ctx(ctx));
  const int64_t R = factor_cols[0];
  const int64_t total = numel(n_factors, factor_rows);
  if (total == 0) return TSR_OK;
  if (R == 0) {
    std::memset(out, 0, sizeof(float) * total);
    return TSR_OK;
  }
  FactorTable ft{};
  TSR_TRY(upload_factors(ctx, n_factors, factor_rows, factors, R, &ft));
  const float* dw = nullptr;
  if (weights) {
    void* p;
    TSR_TRY(slot_get(ctx, SLOT_MISC0, sizeof(float) * R, &p));
    TSR_CUDA(cudaMemcpyAsync(p, weights, sizeof(float) * R, cudaMemcpyHostToDevice, ctx->stream));
    dw = (const float*)p;
  }
  void* dout;
  TSR_TRY(slot_get(ctx, SLOT_OUT, sizeof(float) * total, &dout));
  TSR_TRY(launch_reconstruct(ctx, ft, n_factors, (int)R, dw, nullptr, 0.f, nullptr,
                             (float*)dout));
  TSR_CUDA(cudaMemcpyAsync(out, dout, sizeof(float) * total, cudaMemcpyDeviceToHost,
                           ctx->stream));
  TSR_CUDA(cudaStreamSynchronize(ctx->stream));
  return TSR_OK;
}

int tsr_cp_reconstruct_dev_f32(tsr_ctx* ctx, const float* const* d_factors, int ndim,
                               const int64_t* shape, int64_t rank, const float* d_weights,
                               float* d_out) {
  if (!d_factors || !shape || !d_out) return fail(TSR_E_INVALID_ARG, "null argument");
  std::vector<int64_t> cols(ndim > 0 ? ndim : 1, rank);
  TSR_TRY(validate_reconstruct(ndim, cols.data(), rank, false));
  TSR_TRY(check_ctx(ctx));
  const int64_t total = numel(ndim, shape);
  if (total == 0) return TSR_OK;
  if (rank == 0) {
    TSR_CUDA(cudaMemsetAsync(d_out, 0, sizeof(float) * total, ctx->stream));
    return TSR_OK;
  }
  FactorTable ft{};
  for (int m = 0; m < ndim; ++m) {
    ft.ptr[m] = d_factors[m];
    ft.rows[m] = shape[m];
  }
  return launch_reconstruct(ctx, ft, ndim, (int)rank, d_weights, nullptr, 0.f, nullptr, d_out);
}

int tsr_cp_residual_dev_f32(tsr_ctx* ctx, const float* d_tensor, int ndim, const int64_t* shape,
                            const float* const* d_factors, int64_t rank, const float* d_weights,
                            float alpha, float* d_out, double* sq_err) {
  if (!d_tensor || !d_factors || !shape || !d_out) return fail(TSR_E_INVALID_ARG, "null argument");
  std::vector<int64_t> cols(ndim > 0 ? ndim : 1, rank);
  TSR_TRY(validate_reconstruct(ndim, cols.data(), rank, false));
  if (rank <= 0) return fail(TSR_E_INVALID_RANK, "Invalid rank: %lld", (long long)rank);
  TSR_TRY(check_ctx(ctx));
  void* p;
  TSR_TRY(slot_get(ctx, SLOT_MISC2, sizeof(double), &p));
  TSR_CUDA(cudaMemsetAsync(p, 0, sizeof(double), ctx->stream));
  FactorTable ft{};
  for (int m = 0; m < ndim; ++m) {
    ft.ptr[m] = d_factors[m];
    ft.rows[m] = shape[m];
  }
  TSR_TRY(launch_reconstruct(ctx, ft, ndim, (int)rank, d_weights, d_tensor, alpha, (double*)p,
                             d_out));
  if (sq_err) {
    TSR_CUDA(cudaMemcpyAsync(sq_err, p, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    TSR_CUDA(cudaStreamSynchronize(ctx->stream));
  }
  return TSR_OK;
}

int tsr_cp_reconstruction_grad_f32(tsr_ctx* ctx, const float* grad_output, int grad_ndim,
                                   const int64_t* shape, const float* const* factors,
                                   int n_factors, const int64_t* factor_rows,
                                   const int64_t* factor_cols, const float* weights,
                                   int64_t n_weights, int precision, float* const* out_grads) {
  if (!shape || !grad_output || !out_grads || (n_factors > 0 && (!factors || !factor_rows ||
                                                                  !factor_cols)))
    return fail(TSR_E_INVALID_ARG, "null argument");
  TSR_TRY(validate_grad(grad_ndim, shape, n_factors, factor_rows, factor_cols));
  const int64_t R = factor_cols[0];
  if (weights && n_weights != R)
    return fail(TSR_E_SHAPE, "Weights length %lld must match rank %lld", (long long)n_weights,
                (long long)R);
  TSR_TRY(check_precision(precision));
  TSR_TRY(check_ctx(ctx));
  float* dG;
  TSR_TRY(upload_tensor(ctx, grad_output, grad_ndim, shape, nullptr, &dG));
  FactorTable ft{};
  TSR_TRY(upload_factors(ctx, n_factors, shape, factors, R, &ft));
  const float* dw = nullptr;
  if (weights && R > 0) {
    void* p;
    TSR_TRY(slot_get(ctx, SLOT_MISC0, sizeof(float) * R, &p));
    TSR_CUDA(cudaMemcpyAsync(p, weights, sizeof(float) * R, cudaMemcpyHostToDevice, ctx->stream));
    dw = (const float*)p;
  }
  int64_t total = 0;
  for (int m = 0; m < n_factors; ++m) total += shape[m] * R;
  void* dout;
  TSR_TRY(slot_get(ctx, SLOT_OUT, sizeof(float) * (total > 0 ? total : 1), &dout));
  std::vector<float*> outs(n_factors);
  int64_t off = 0;
  for (int m = 0; m < n_factors; ++m) {
    outs[m] = (float*)dout + off;
    off += shape[m] * R;
  }
  TSR_TRY(reconstruction_grad_device(ctx, dG, grad_ndim, shape, ft, (int)R, dw, precision,
                                     outs.data()));
  for (int m = 0; m < n_factors; ++m)
    if (shape[m] * R > 0)
      TSR_CUDA(cudaMemcpyAsync(out_grads[m], outs[m], sizeof(float) * shape[m] * R,
                               cudaMemcpyDeviceToHost, ctx->stream));
  TSR_CUDA(cudaStreamSynchronize(ctx->stream));
  return TSR_OK;
}

int tsr_cp_reconstruction_grad_dev_f32(tsr_ctx* ctx, const float* d_grad_output, int ndim,
                                       const int64_t* shape, const float* const* d_factors,
                                       int64_t rank, const float* d_weights, int precision,
                                       float* const* d_out_grads) {
  if (!shape || !d_grad_output || !d_factors || !d_out_grads)
    return fail(TSR_E_INVALID_ARG, "null argument");
  std::vector<int64_t> cols(ndim > 0 ? ndim : 1, rank);
  TSR_TRY(validate_grad(ndim, shape, ndim, shape, cols.data()));
  TSR_TRY(check_precision(precision));
  TSR_TRY(check_ctx(ctx));
  FactorTable ft{};
  for (int m = 0; m < ndim; ++m) {
    ft.ptr[m] = d_factors[m];
    ft.rows[m] = shape[m];
  }
  return reconstruction_grad_device(ctx, d_grad_output, ndim, shape, ft, (int)rank, d_weights,
                                    precision, d_out_grads);
}

int tsr_dense_create_dev_f32(tsr_ctx* ctx, const float* d_tensor, int ndim, const int64_t* shape,
                             int precision, tsr_dense** out) {
  if (!d_tensor || !shape || !out) return fail(TSR_E_INVALID_ARG, "null argument");
  *out = nullptr;
  if (ndim < 2) return fail(TSR_E_NEED_2_FACTORS, "Need at least 2 factor matrices for MTTKRP");
  if (ndim > kMaxModes)
    return fail(TSR_E_UNSUPPORTED, "tensor rank %d exceeds the supported %d", ndim, kMaxModes);
  for (int m = 0; m < ndim; ++m)
    if (shape[m] <= 0) return fail(TSR_E_SHAPE, "mode %d has size %lld", m, (long long)shape[m]);
  TSR_TRY(check_precision(precision));
  TSR_TRY(check_ctx(ctx));
  tsr_dense* d = new tsr_dense();
  d->ndim = ndim;
  d->precision = precision;
  d->device = ctx->device;
  d->dX = d_tensor;
  for (int m = 0; m < ndim; ++m) d->shape[m] = shape[m];
  auto cleanup = [&](int rc) {
    tsr_dense_destroy(d);
    return rc;
  };
  for (int m = 0; m < ndim; ++m) {
    size_t ab, bb;
    mode_operand_bytes(make_unfolding(ndim, shape, m), precision, &ab, &bb);
    if (ab && cudaMalloc(&d->owned[2 * m], ab) != cudaSuccess)
      return cleanup(fail(TSR_E_CUDA, "cudaMalloc of %zu bytes failed", ab));
    if (bb && cudaMalloc(&d->owned[2 * m + 1], bb) != cudaSuccess)
      return cleanup(fail(TSR_E_CUDA, "cudaMalloc of %zu bytes failed", bb));
    int rc = prepare_mode_into(ctx, d_tensor, ndim, shape, m, precision, d->owned[2 * m],
                               d->owned[2 * m + 1], &d->ops[m]);
    if (rc != TSR_OK) return cleanup(rc);
  }
  if (cudaMalloc(&d->d_scalars, 4 * sizeof(double)) != cudaSuccess)
    return cleanup(fail(TSR_E_CUDA, "cudaMalloc of the loss scalars failed"));
  // BF16x3, 3+ modes: the trailing-two-modes view (with 3 modes the leading
  // side is mode 0 alone)
  const int64_t vshape[3] = {prod_range(shape, 0, ndim - 2), shape[ndim - 2], shape[ndim - 1]};
  d->d3_three = dense3_supported(3, vshape, 1);
  d->d3_two = twosided_supported(vshape[0], vshape[1] * vshape[2], 1);
  if (precision == TSR_PREC_BF16X3 && ndim >= 3 && (d->d3_three || d->d3_two) &&
      vshape[0] <= ((int64_t)1 << 30) &&
      ((uintptr_t)d_tensor & 15) == 0) {
    const int64_t n = numel(ndim, shape);
    void *hp, *lp;
    if (cudaMalloc(&hp, sizeof(__nv_bfloat16) * n) != cudaSuccess)
      return cleanup(fail(TSR_E_CUDA, "cudaMalloc of the bf16 halves failed"));
    d->owned[2 * kMaxModes] = hp;
    if (cudaMalloc(&lp, sizeof(__nv_bfloat16) * n) != cudaSuccess)
      return cleanup(fail(TSR_E_CUDA, "cudaMalloc of the bf16 halves failed"));
    d->owned[2 * kMaxModes + 1] = lp;
    int rc = launch_split_bf16(ctx, ctx->stream, d_tensor, n, (__nv_bfloat16*)hp,
                               (__nv_bfloat16*)lp, d->d_scalars + 3);
    if (rc != TSR_OK) return cleanup(rc);
    d->d3_on = true;
    d->d3.I = vshape[0];
    d->d3.J = vshape[1];
    d->d3.K = vshape[2];
    d->d3.hi = (const __nv_bfloat16*)hp;
    d->d3.lo = (const __nv_bfloat16*)lp;
  }
  // (a BF16x3 tensor whose view does not suit the two-sided kernel too, see
  // sides_pay_prepared)
  if (!d->d3_on && ndim >= 3 && vshape[0] <= ((int64_t)1 << 30) &&
      vshape[1] * vshape[2] < INT32_MAX) {
    const int64_t v2[2] = {vshape[0], vshape[1] * vshape[2]};
    d->v2_on = true;
    d->v2_shape[0] = v2[0];
    d->v2_shape[1] = v2[1];
  }
  cudaError_t e = cudaMemsetAsync(d->d_scalars, 0, 4 * sizeof(double), ctx->stream);
  if (e != cudaSuccess) return cleanup(fail(TSR_E_CUDA, "%s", cudaGetErrorString(e)));
  int rc = launch_norm_sq(ctx, ctx->stream, d_tensor, numel(ndim, shape), d->d_scalars);
  if (rc != TSR_OK) return cleanup(rc);
  e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) return cleanup(fail(TSR_E_CUDA, "%s", cudaGetErrorString(e)));
  *out = d;
  return TSR_OK;
}

int tsr_dense_destroy(tsr_dense* d) {
  if (!d) return TSR_OK;
  int prev = 0;
  cudaGetDevice(&prev);
  cudaSetDevice(d->device);
  for (void* p : d->owned)
    if (p) cudaFree(p);
  if (d->d_scalars) cudaFree(d->d_scalars);
  cudaSetDevice(prev);
  delete d;
  return TSR_OK;
}

int tsr_cp_loss_grad_dev_f32(tsr_ctx* ctx, const tsr_dense* X, const float* const* d_factors,
                             int64_t rank, double reg, float* const* d_grads, double* loss) {
  if (!X || !d_factors || !d_grads) return fail(TSR_E_INVALID_ARG, "null argument");
  if (rank <= 0) return fail(TSR_E_INVALID_RANK, "Invalid rank: %lld", (long long)rank);
  if (rank > kMaxRank)
    return fail(TSR_E_UNSUPPORTED, "rank %lld exceeds the supported %d", (long long)rank,
                kMaxRank);
  TSR_TRY(check_ctx(ctx));
  if (ctx->device != X->device)
    return fail(TSR_E_INVALID_ARG, "tensor prepared on device %d, context on device %d",
                X->device, ctx->device);
  const int N = X->ndim, R = (int)rank, RR = R * R;
  FactorTable ft{};
  for (int m = 0; m < N; ++m) {
    ft.ptr[m] = d_factors[m];
    ft.rows[m] = X->shape[m];
  }
  void* gp;
  TSR_TRY(slot_get(ctx, SLOT_GRAMS, sizeof(double) * N * RR, &gp));
  double* grams = (double*)gp;
  TSR_CUDA(cudaMemsetAsync(X->d_scalars + 1, 0, 2 * sizeof(double), ctx->stream));
  TSR_CUDA(cudaMemsetAsync(grams, 0, sizeof(double) * N * RR, ctx->stream));
  TSR_TRY(launch_gram_all(ctx, ctx->stream, N, d_factors, X->shape, R, grams));
  auto grad_of = [&](int n, const float* partials, int splits) -> int {
    const int64_t rows = X->shape[n];
    const int rpc =
        (int)std::max<int64_t>(1, std::min<int64_t>(16, ceil_div(rows, 2 * ctx->sm_count)));
    const int full = rpc * R;
    const int groups = full >= 256 ? 1 : 256 / full;
    const size_t smem = sizeof(double) * ((size_t)RR + full + (size_t)groups * full);
    if (smem > 200 * 1024)
      return fail(TSR_E_UNSUPPORTED, "rank %d too large for the gradient kernel", R);
    gram_grad_kernel<<<(unsigned)ceil_div(rows, rpc), 256, smem, ctx->stream>>>(
        grams, N, n, partials, splits, rows, R, rpc, d_factors[n], reg, d_grads[n],
        X->d_scalars);
    ctx->launches++;
    TSR_CUDA(cudaGetLastError());
    return TSR_OK;
  };
  auto finish = [&]() -> int {
    gram_loss_kernel<<<1, 256, 0, ctx->stream>>>(grams, N, R, reg, X->d_scalars);
    ctx->launches++;
    TSR_CUDA(cudaGetLastError());
    if (loss) {
      double sc[4];
      TSR_TRY(read_scalars(ctx, X->d_scalars, sc));
      *loss = sc[2];
    }
    return TSR_OK;
  };
  // From T (A x R: the leading modes, the trailing two contracted) and P
  // (C x R: the trailing two, the leading contracted): every mode's MTTKRP
  // and gradient rows and the Gram part of the loss in one programmatic
  // launch (R <= 32), then the loss when requested.
  auto contract_grad = [&](const float* T, const float* P) -> int {
    int total_rows = 0;
    for (int p = 0; p < N; ++p) total_rows += (int)X->shape[p];
    TContract c{};
    set_side(c, 0, T, X->shape, 0, N - 2, d_factors);
    set_side(c, 1, P, X->shape, N - 2, N, d_factors);
    c.R = R;
    c.nmodes = N;
    c.row0[0] = 0;
    for (int p = 0; p < N; ++p) {
      c.side_of[p] = p < N - 2 ? 0 : 1;
      c.pos[p] = p < N - 2 ? p : p - (N - 2);
      c.row0[p + 1] = c.row0[p] + (int)X->shape[p];
    }
    GradArgs g{};
    g.grams = grams;
    g.ndim = N;
    g.reg = reg;
    g.scal = X->d_scalars;
    for (int m = 0; m < N; ++m) g.G[m] = d_grads[m];
    TSR_CUDA(launch_pdl(t_contract_grad_kernel, dim3((unsigned)total_rows + 1), dim3(256), 0,
                        ctx->stream, c, g));
    ctx->launches++;
    TSR_CUDA(cudaGetLastError());
    if (loss) {
      double sc[4];
      TSR_TRY(read_scalars(ctx, X->d_scalars, sc));
      *loss = sc[0] - 2.0 * sc[1] + sc[3];
    }
    return TSR_OK;
  };
  if (X->d3_on && X->d3_two && twosided_supported(X->d3.I, X->d3.J * X->d3.K, R)) {
    // one read of X's bf16 halves: T = X_(lead) KR(trailing two) and
    // P = X_(lead)^T KR(leading) from the two-sided contraction, then every
    // mode's MTTKRP from T (modes 0..N-3) or P (modes N-2, N-1)
    const int64_t A = X->d3.I, C = X->d3.J * X->d3.K;
    const int64_t Ap = twosided_pad(A), Cp = twosided_pad(C);
    void *tp, *ip;
    // B images of V = KR(leading factors) and W = KR(trailing two), rows
    // formed on the fly
    const size_t vb = bimage_bytes(Ap, 32), wb = bimage_bytes(Cp, 32);
    TSR_TRY(slot_get(ctx, SLOT_D3_IMG, vb + wb, &ip));
    KRImages ki{};
    ki.n = 2;
    ki.R = R;
    ki.n_pad = 32;
    for (int w = 0; w < 2; ++w) {
      KRImage& im = ki.im[w];
      const int m0 = w == 0 ? 0 : N - 2, m1 = w == 0 ? N - 2 : N;
      im.nf = m1 - m0;
      for (int f = 0; f < im.nf; ++f) {
        im.U[f] = d_factors[m0 + f];
        im.size[f] = X->shape[m0 + f];
      }
      im.L = w == 0 ? A : C;
      im.chunks = (int)((w == 0 ? vb : wb) / 16);
      im.img = (uint8_t*)ip + (w == 0 ? 0 : vb);
    }
    // T and P (accumulated into by the two-sided kernel) are zeroed by the
    // same launch, whole float4s (the slot is padded to them)
    const int64_t tp_n4 = ceil_div((A + C) * R, 4);
    TSR_TRY(slot_get(ctx, SLOT_MISC0, sizeof(float) * 4 * tp_n4, &tp));
    ki.zero = (float*)tp;
    ki.zero_n4 = tp_n4;
    // programmatic launches from here to the end of the evaluation: each
    // kernel's launch and prologue overlap its predecessor, whose writes it
    // awaits before reading them
    TSR_TRY(launch_kr_images(ctx, ctx->stream, ki, true));
    TwoSided ts;
    ts.hi = X->d3.hi;
    ts.lo = X->d3.lo;
    ts.A = A;
    ts.C = C;
    ts.R = R;
    ts.vimg = (const uint8_t*)ip;
    ts.wimg = (const uint8_t*)ip + vb;
    ts.T = (float*)tp;
    ts.P = (float*)tp + A * R;
    TSR_TRY(launch_twosided(ctx, ctx->stream, ts));
    return contract_grad(ts.T, ts.P);
  }
  if (X->v2_on && R <= 32 &&
      (X->precision == TSR_PREC_FP32 || sides_pay_prepared(N, X->shape, R))) {
    // FP32: T = X KR(trailing two) and P = X^T KR(leading), both read from X
    // in place: two passes over X's bytes instead of one per mode, and half
    // the FLOPs of N MTTKRPs
    const int64_t A = X->v2_shape[0], C = X->v2_shape[1];
    void* tp;
    TSR_TRY(slot_get(ctx, SLOT_MISC0, sizeof(float) * (A + C) * R, &tp));
    float* T = (float*)tp;
    float* P = T + A * R;
    TSR_TRY(contract_sides(ctx, X->dX, N, X->shape, d_factors, R, T, P));
    return contract_grad(T, P);
  }
  if (X->d3_on && X->d3_three && R <= 64) {
    // three single-layout passes over X's bf16 halves instead of one MTTKRP
    // per mode: the view (A = prod of the leading modes, I_{N-2}, I_{N-1})
    Dense3 d = X->d3;
    d.R = R;
    d.n_pad = dense3_n_pad(R);
    const int64_t A = d.I;
    // Khatri-Rao of the leading factors (forward order): the view's U0
    void *kp, *kq, *tp, *mp, *ip;
    TSR_TRY(slot_get(ctx, SLOT_MISC1, sizeof(float) * A * R, &kp));
    TSR_TRY(slot_get(ctx, SLOT_MISC3, sizeof(float) * A * R, &kq));
    const float* kr = d_factors[0];
    int64_t krows = X->shape[0];
    float* bufs[2] = {(float*)kp, (float*)kq};
    for (int p = 1; p < N - 2; ++p) {
      float* dst = bufs[p & 1];
      TSR_TRY(launch_khatri_rao(ctx, kr, krows, d_factors[p], X->shape[p], R, dst));
      kr = dst;
      krows *= X->shape[p];
    }
    const size_t img1 = bimage_bytes(d.J, d.n_pad), img2 = bimage_bytes(d.K, d.n_pad);
    TSR_TRY(slot_get(ctx, SLOT_D3_IMG, img1 + img2, &ip));
    d.bimg[0] = nullptr;
    d.bimg[1] = (uint8_t*)ip;
    d.bimg[2] = (uint8_t*)ip + img1;
    TSR_TRY(launch_bimage(ctx, ctx->stream, d_factors[N - 2], d.J, R, d.n_pad, d.bimg[1]));
    TSR_TRY(launch_bimage(ctx, ctx->stream, d_factors[N - 1], d.K, R, d.n_pad, d.bimg[2]));
    FactorTable vt{};
    vt.ptr[0] = kr;
    vt.rows[0] = A;
    vt.ptr[1] = d_factors[N - 2];
    vt.rows[1] = d.J;
    vt.ptr[2] = d_factors[N - 1];
    vt.rows[2] = d.K;
    size_t pmax = 0;
    for (int v = 0; v < 3; ++v) {
      const SplitPlan pl = plan_mttkrp3(ctx, d, v);
      pmax = std::max(pmax, (size_t)pl.splits * dense3_rows(d, v) * R);
    }
    void* pp;
    TSR_TRY(slot_get(ctx, SLOT_PARTIALS, sizeof(float) * pmax, &pp));
    float* partials = (float*)pp;
    // T = the view's mode-0 MTTKRP (A x R), then the leading modes from it
    TSR_TRY(slot_get(ctx, SLOT_MISC0, sizeof(float) * A * R, &tp));
    {
      const SplitPlan pl = plan_mttkrp3(ctx, d, 0);
      TSR_TRY(launch_mttkrp3(ctx, ctx->stream, d, 0, vt, pl, partials, true));
      TSR_TRY(launch_mttkrp_reduce(ctx, partials, pl.splits, A * R, (float*)tp));
    }
    int lead_rows = 0;
    for (int p = 0; p < N - 2; ++p) lead_rows += (int)X->shape[p];
    TSR_TRY(slot_get(ctx, SLOT_MISC2, sizeof(float) * lead_rows * R, &mp));
    TContract c{};
    set_side(c, 0, (const float*)tp, X->shape, 0, N - 2, d_factors);
    c.R = R;
    c.nmodes = N - 2;
    c.row0[0] = 0;
    for (int p = 0; p < N - 2; ++p) {
      c.side_of[p] = 0;
      c.pos[p] = p;
      c.row0[p + 1] = c.row0[p] + (int)X->shape[p];
    }
    for (int p = 0; p < N - 2; ++p) c.out[p] = (float*)mp + (int64_t)c.row0[p] * R;
    t_contract_kernel<<<(unsigned)lead_rows, 256, 0, ctx->stream>>>(c);
    ctx->launches++;
    TSR_CUDA(cudaGetLastError());
    for (int m = 0; m < N - 2; ++m)
      TSR_TRY(grad_of(m, (const float*)mp + (int64_t)c.row0[m] * R, 1));
    // the trailing two modes straight from the view's modes 1 and 2
    for (int v = 1; v <= 2; ++v) {
      const SplitPlan pl = plan_mttkrp3(ctx, d, v);
      TSR_TRY(launch_mttkrp3(ctx, ctx->stream, d, v, vt, pl, partials, true));
      TSR_TRY(grad_of(N - 3 + v, partials, pl.splits));
    }
    return finish();
  }
  for (int n = 0; n < N; ++n) {
    float* partials;
    int splits;
    TSR_TRY(run_mttkrp_partials(ctx, X->ops[n], ft, R, X->precision, &partials, &splits));
    TSR_TRY(grad_of(n, partials, splits));
  }
  return finish();
}

}  // extern "C"
