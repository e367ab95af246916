// CP factor initialisation: tenrso_decomp's initialize_factors
// (crates/tenrso-decomp/src/cp/helpers.rs:192-377) for every InitStrategy.
//
//   Random        U(0,1) per entry (helpers.rs:215-222)
//   RandomNormal  N(0,1) per entry (helpers.rs:223-231)
//   Svd           the leading left singular vectors of each unfolding X_(n),
//                 N(0, 0.01) columns past the unfolding's rank (:232-263)
//   Nnsvd         per component r the dominant sign part of (u_r, v_r),
//                 scaled by sqrt(s_r * |u_part| |v_part|) (:264-317)
//   LeverageScore u_r sqrt(s_r) sqrt(I_n * lev_i), lev the normalised row
//                 leverage scores of the leading singular vectors (:318-373)
//
// Random draws come from the library's seeded SplitMix64 stream (tenrso's
// thread_rng cannot be seeded): U(0,1) on stream 200 + n, N(0,1) on stream
// 400 + n (Box-Muller over streams 400 + n and 400 + n + 0x5151), the
// N(0, 0.01) padding columns on stream 500 + n.
//
// The singular vectors on the device: the FP64 Gram G = X_(n) X_(n)^T
// (I_n x I_n; the order of the unfolding's columns does not enter G), then its
// leading eigenpairs by tridiagonalisation (modes of up to 160 rows with
// separated leading eigenvalues), else a cyclic Jacobi eigensolver on G in
// round-robin order (I_n / 2 disjoint rotations per round, each round three
// launches: rotation angles, row update, column update with the eigenvector
// update), sweeps until the off-diagonal mass is below 1e-26 of the
// diagonal's. s_r = sqrt(lambda_r).
// v_r (needed by Nnsvd, only through the norms of its positive and negative
// parts) is X_(n)^T u_r / s_r, formed and reduced on the fly. SVD signs are
// arbitrary; each u_r is oriented so that its entry of largest magnitude is
// positive (Nnsvd's result does not depend on the sign).
#include <algorithm>
#include <cmath>
#include <numeric>
#include <vector>

#include "dense.cuh"

namespace tsr {

namespace {

// ---- host generators --------------------------------------------------------

uint64_t mix64h(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

double uniform_at(uint64_t seed, uint64_t stream, int64_t i) {
  const uint64_t golden = 0x9E3779B97F4A7C15ull;
  const uint64_t key = mix64h(seed * 0x100000001B3ull + stream * 0x2545F4914F6CDD1Dull + golden);
  return (double)(mix64h(key + (uint64_t)i * golden) >> 11) * (1.0 / 9007199254740992.0);
}

// N(0, sigma^2) doubles, identical to tenrso_b200.synth.normal(seed, stream) * sigma.
void seeded_normal(uint64_t seed, uint64_t stream, int64_t n, double sigma, double* out) {
  const double two_pi = 6.283185307179586;
  for (int64_t i = 0; i < n; ++i) {
    const double u1 = 1.0 - uniform_at(seed, stream, i);
    const double u2 = uniform_at(seed, stream + 0x5151, i);
    out[i] = sigma * std::sqrt(-2.0 * std::log(u1)) * std::cos(two_pi * u2);
  }
}

// ---- Gram of an unfolding ---------------------------------------------------

// G[i, i'] = sum_{a, b} X[a, i, b] X[a, i', b], X viewed as A x I x B
// (A = prod of the modes before n, B = prod after), in FP64 (the products of
// fp32 values are exact). 64 x 64 output tiles of the upper triangle, 4 x 4
// per 256-thread CTA, the columns split over blockIdx.y into partial Grams:
// with one CTA per tile and no split, a 160 x 12288 unfolding occupied 25 of
// 148 SMs. Bound: shared-memory reads (two operand words per four FMAs).
constexpr int GR_T = 64, GR_K = 32;

__global__ void __launch_bounds__(256) unfold_gram_kernel(const float* __restrict__ X, int64_t A,
                                                          int64_t I, int64_t B,
                                                          int64_t j_per_split,
                                                          double* __restrict__ parts) {
  __shared__ double xs[2][GR_K][GR_T + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  // tile pair (ti <= tk) of the upper triangle
  const int nt = (int)((I + GR_T - 1) / GR_T);
  int ti = 0, rest = blockIdx.x;
  while (rest >= nt - ti) rest -= nt - ti++;
  const int tk = ti + rest;
  const int64_t i0 = (int64_t)ti * GR_T, k0 = (int64_t)tk * GR_T;
  const int64_t jb = blockIdx.y * j_per_split, je = min(A * B, jb + j_per_split);
  const int nop = ti == tk ? 1 : 2;
  double acc[4][4];
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[p][q] = 0.0;
  for (int64_t j0 = jb; j0 < je; j0 += GR_K) {
    __syncthreads();
    if (B > 1) {  // lanes along the columns: one (a, b) per thread and step
      const int c = threadIdx.x & 31;
      const int64_t j = j0 + c, a = j / B;
      const float* src = X + a * I * B + (j - a * B);
      for (int w = 0; w < nop; ++w)
#pragma unroll
        for (int q = 0; q < GR_T / 8; ++q) {
          const int r = (threadIdx.x >> 5) + 8 * q;
          const int64_t row = (w ? k0 : i0) + r;
          xs[w][c][r] = row < I && j < je ? (double)__ldg(src + row * B) : 0.0;
        }
    } else {  // the last mode: lanes along the rows
      const int r = threadIdx.x & 63;
      for (int w = 0; w < nop; ++w)
#pragma unroll
        for (int q = 0; q < GR_K / 4; ++q) {
          const int c = (threadIdx.x >> 6) + 4 * q;
          const int64_t row = (w ? k0 : i0) + r, j = j0 + c;
          xs[w][c][r] = row < I && j < je ? (double)__ldg(X + j * I + row) : 0.0;
        }
    }
    __syncthreads();
    const double(*ys)[GR_T + 1] = xs[nop - 1];
#pragma unroll 4
    for (int c = 0; c < GR_K; ++c) {
      double x[4], y[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) x[p] = xs[0][c][ty + 16 * p];
#pragma unroll
      for (int q = 0; q < 4; ++q) y[q] = ys[c][tx + 16 * q];
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[p][q] = fma(x[p], y[q], acc[p][q]);
    }
  }
  double* G = parts + (int64_t)blockIdx.y * I * I;
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int64_t i = i0 + ty + 16 * p, k = k0 + tx + 16 * q;
      if (i < I && k < I) G[i * I + k] = acc[p][q];
    }
}

// G = the sum of the partial Grams, mirrored from the tiles of the upper
// triangle. Eight threads share an element, each summing every eighth split.
__global__ void __launch_bounds__(256) gram_reduce_kernel(const double* __restrict__ parts,
                                                          int splits, int64_t I,
                                                          double* __restrict__ G) {
  const int64_t e = (int64_t)blockIdx.x * 32 + (threadIdx.x >> 3);
  const int g = threadIdx.x & 7;
  double t = 0.0;
  if (e < I * I) {
    const int64_t i = e / I, k = e - i * I;
    const double* p = parts + (i / GR_T <= k / GR_T ? e : k * I + i);
    for (int q = g; q < splits; q += 8) t += __ldg(p + q * I * I);
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (g == 0 && e < I * I) G[e] = t;
}

// ---- leading eigenpairs by tridiagonalisation ------------------------------------
//
// Householder reduction of G to a tridiagonal T, the leading eigenvalues of T
// by bisection on Sturm counts, each eigenvector of T from its twisted
// factorisation (T - lambda I = L D L^T from the top and U D U^T from the
// bottom, joined at the row with the smallest |gamma|), and the reflections
// applied back. All FP64. Each eigenvector comes out by itself, to about eps |T|
// / gap, so the host takes this path only where the leading eigenvalues are
// separated by more than kTriGap of the largest, and the Jacobi solver below
// otherwise (repeated or zero eigenvalues, non-finite tensors) and beyond
// kTriRows rows. Off-diagonal of U^T U as returned in FP32, largest of eight
// matrices of 40 rows: 3.3e-8 at gaps of 1.2e-8, 7e-9 at 1.1e-7, 2e-9 at 2e-7,
// where rounding exact vectors to FP32 alone leaves about 2e-8.
// About 4/3 I^3 operations in two launches for all modes together, against
// some ten Jacobi sweeps of 6 I^3 in three launches per round each. 160 rows are
// what one CTA holds: 50 doubles of the matrix in each of 512 threads, of 128
// registers at most.
constexpr int kTriRows = 160;
constexpr double kTriGap = 1e-7;

struct TriMode {
  const double* G;  // I x I
  int I, k;         // rows, leading pairs wanted
  double* d;        // I diagonal, then I off-diagonal, then I reflection scales
  double* V;        // I x I: reflection j in row j, columns j + 1 ..
  double* lam;      // min(k + 1, I) leading eigenvalues
  double* U;        // I x k eigenvectors
};
struct TriArgs {
  TriMode m[kMaxModes];
};

// One CTA per mode, the matrix in registers: warp w holds rows w + 16 a, lane l
// columns l + 32 b. Four barriers per column; the reflection and the sums over
// warps are formed by the CB warps that own a column block (every warp forming
// them for itself made the kernel instruction-bound, 553 us at 160 rows).
template <int RA, int CB>
__global__ void __launch_bounds__(512, 1) tridiag_kernel(const __grid_constant__ TriArgs g) {
  constexpr int W = 32 * CB > 16 * RA ? 32 * CB : 16 * RA;
  __shared__ double xr[2][W];  // the current row of the matrix, the next one
  __shared__ double vs[W], pb[W];
  __shared__ double part[16][32 * CB];
  __shared__ double dotp[CB], scal[1];
  const TriMode& M = g.m[blockIdx.x];
  const int I = M.I, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double a[RA][CB];
#pragma unroll
  for (int ra = 0; ra < RA; ++ra)
#pragma unroll
    for (int cb = 0; cb < CB; ++cb) {
      const int row = w + 16 * ra, col = lane + 32 * cb;
      a[ra][cb] = row < I && col < I ? M.G[(int64_t)row * I + col] : 0.0;
    }
  for (int i = threadIdx.x; i < W; i += 512) vs[i] = pb[i] = xr[0][i] = xr[1][i] = 0.0;
  __syncthreads();
  if (w == 0)
#pragma unroll
    for (int cb = 0; cb < CB; ++cb) xr[0][lane + 32 * cb] = a[0][cb];
  __syncthreads();
  int buf = 0;
  for (int j = 0; j < I; ++j, buf ^= 1) {
    if (threadIdx.x == 0) M.d[j] = xr[buf][j];
    if (j == I - 1) break;
    if (w < CB) {
      // the reflection of x = row j past the diagonal: alpha = -+|x|,
      // tau = 1 + |x0| / |x|, v = (1, x_i / (x0 - alpha))
      const double x0 = xr[buf][j + 1];
      double ss = 0.0;
#pragma unroll
      for (int cb = 0; cb < CB; ++cb) {
        const double x = xr[buf][lane + 32 * cb];
        if (lane + 32 * cb > j + 1) ss = fma(x, x, ss);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      double alpha = x0, tau = 0.0, inv = 0.0;
      if (ss > 0.0) {  // the same in every warp
        const double n2 = fma(x0, x0, ss), rn = rsqrt(n2), nrm = n2 * rn;
        alpha = x0 >= 0.0 ? -nrm : nrm;
        tau = fma(fabs(x0), rn, 1.0);
        inv = 1.0 / (x0 - alpha);
      }
      const int col = threadIdx.x;
      const double v = col == j + 1 ? 1.0 : col > j + 1 ? xr[buf][col] * inv : 0.0;
      vs[col] = v;
      if (tau != 0.0 && col > j && col < I) M.V[(int64_t)j * I + col] = v;
      if (threadIdx.x == 0) {
        scal[0] = tau;
        M.d[I + j] = alpha;
        M.d[2 * I + j] = tau;
      }
    }
    __syncthreads();
    const double tau = scal[0];
    if (tau == 0.0) {  // nothing to reflect: only publish the next row
#pragma unroll
      for (int ra = 0; ra < RA; ++ra)
        if (w + 16 * ra == j + 1)
#pragma unroll
          for (int cb = 0; cb < CB; ++cb) xr[buf ^ 1][lane + 32 * cb] = a[ra][cb];
      __syncthreads();
      continue;
    }
    // p = tau A v, rows and columns past j
    double acc[CB];
#pragma unroll
    for (int cb = 0; cb < CB; ++cb) acc[cb] = 0.0;
#pragma unroll
    for (int ra = 0; ra < RA; ++ra)
      if (16 * ra + 15 > j) {
        const double vr = vs[w + 16 * ra];
#pragma unroll
        for (int cb = 0; cb < CB; ++cb) acc[cb] = fma(a[ra][cb], vr, acc[cb]);
      }
#pragma unroll
    for (int cb = 0; cb < CB; ++cb) part[w][lane + 32 * cb] = acc[cb];
    __syncthreads();
    if (w < CB) {
      const int col = threadIdx.x;
      double p0 = 0.0, p1 = 0.0;
#pragma unroll
      for (int q = 0; q < 16; q += 2) {
        p0 += part[q][col];
        p1 += part[q + 1][col];
      }
      const double p = col > j ? (p0 + p1) * tau : 0.0;
      pb[col] = p;
      double dp = p * vs[col];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) dp += __shfl_xor_sync(0xffffffffu, dp, o);
      if (lane == 0) dotp[w] = dp;
    }
    __syncthreads();
    // A -= v w^T + w v^T, w = p - (tau / 2 p.v) v
    double K = 0.0;
#pragma unroll
    for (int cb = 0; cb < CB; ++cb) K += dotp[cb];
    K *= -0.5 * tau;
    double vl[CB], wl[CB];
#pragma unroll
    for (int cb = 0; cb < CB; ++cb) {
      vl[cb] = vs[lane + 32 * cb];
      wl[cb] = fma(K, vl[cb], pb[lane + 32 * cb]);
    }
#pragma unroll
    for (int ra = 0; ra < RA; ++ra)
      if (16 * ra + 15 > j) {
        const int row = w + 16 * ra;
        const double vr = -vs[row], wr = fma(K, vr, -pb[row]);
#pragma unroll
        for (int cb = 0; cb < CB; ++cb) a[ra][cb] = fma(wr, vl[cb], fma(vr, wl[cb], a[ra][cb]));
        if (row == j + 1)
#pragma unroll
          for (int cb = 0; cb < CB; ++cb) xr[buf ^ 1][lane + 32 * cb] = a[ra][cb];
      }
    __syncthreads();
  }
}

// One CTA per wanted eigenvalue and mode (blockIdx.x = r counts them from the
// largest; r = k gives only the next eigenvalue, for the separation test).
// Each bisection round tests 256 points at once (8 bits); bound by the serial
// recurrences over I, a division per row.
__global__ void __launch_bounds__(256) tri_eigen_kernel(const __grid_constant__ TriArgs g) {
  __shared__ double d[kTriRows], e[kTriRows], e2[kTriRows];
  __shared__ double dp[kTriRows], dm[kTriRows], z[kTriRows];
  __shared__ double lim[2];
  __shared__ int below;
  const TriMode& M = g.m[blockIdx.y];
  const int I = M.I, r = blockIdx.x, t = threadIdx.x;
  if (r > M.k || r >= I) return;
  for (int i = t; i < I; i += 256) {
    d[i] = M.d[i];
    e[i] = i < I - 1 ? M.d[I + i] : 0.0;
    e2[i] = e[i] * e[i];
  }
  __syncthreads();
  if (t < 32) {  // Gershgorin bounds
    double lo = INFINITY, hi = -INFINITY;
    for (int i = t; i < I; i += 32) {
      const double rad = fabs(e[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0);
      lo = fmin(lo, d[i] - rad);
      hi = fmax(hi, d[i] + rad);
    }
    for (int o = 16; o > 0; o >>= 1) {
      lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (t == 0) {
      const double m = fmax(fabs(lo), fabs(hi)) * 4e-16 + 1e-300;
      lim[0] = lo - m;
      lim[1] = hi + m;
    }
  }
  __syncthreads();
  // pivots smaller than this are replaced: they stand for a zero pivot
  const double piv = fmax(fabs(lim[0]), fabs(lim[1])) * 4.9e-32 + 1e-300;
  for (int round = 0; round < 7; ++round) {
    const double lo = lim[0], hi = lim[1];
    const double x = lo + (hi - lo) * ((t + 1) * (1.0 / 257.0));
    int above = 0;  // eigenvalues > x: positive pivots of T - x I
    double q = 1.0;
    for (int i = 0; i < I; ++i) {
      q = d[i] - x - (i > 0 ? e2[i - 1] / q : 0.0);
      if (fabs(q) < piv) q = -piv;
      above += q > 0.0;
    }
    // the points with more than r eigenvalues above them are a prefix
    const int n = __syncthreads_count(above > r);
    if (t == n - 1) lim[0] = x;
    if (t == n) lim[1] = x;
    __syncthreads();
  }
  const double lam = 0.5 * (lim[0] + lim[1]);
  if (t == 0) M.lam[r] = lam;
  if (r >= M.k) return;
  if (t == 0) {
    double q = 1.0;
    for (int i = 0; i < I; ++i) {
      q = d[i] - lam - (i > 0 ? e2[i - 1] / q : 0.0);
      if (fabs(q) < piv) q = -piv;
      dp[i] = q;
    }
  } else if (t == 32) {
    double q = 1.0;
    for (int i = I - 1; i >= 0; --i) {
      q = d[i] - lam - (i < I - 1 ? e2[i] / q : 0.0);
      if (fabs(q) < piv) q = -piv;
      dm[i] = q;
    }
  }
  __syncthreads();
  if (t < 32) {
    double best = INFINITY;
    int at = 0;
    for (int i = t; i < I; i += 32) {
      const double gm = fabs(dp[i] + dm[i] - (d[i] - lam));
      if (gm < best) {
        best = gm;
        at = i;
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, at, o);
      if (ob < best || (ob == best && oi < at)) {
        best = ob;
        at = oi;
      }
    }
    if (t == 0) below = at;
  }
  __syncthreads();
  const int at = below;
  for (int i = t; i < I; i += 256)  // step ratios away from the twist
    z[i] = i < at ? -e[i] / dp[i] : i > at ? -e[i - 1] / dm[i] : 1.0;
  __syncthreads();
  if (t == 0) {
    double q = 1.0;
    for (int i = at - 1; i >= 0; --i) z[i] = q *= z[i];
  } else if (t == 32) {
    double q = 1.0;
    for (int i = at + 1; i < I; ++i) z[i] = q *= z[i];
  }
  __syncthreads();
  if (t >= 32) return;
  // normalise, then u = H_0 H_1 .. H_{I-3} z; the next reflection is loaded
  // while the current one is applied
  constexpr int N = kTriRows / 32;
  double u[N], ss = 0.0;
#pragma unroll
  for (int q = 0; q < N; ++q) {
    u[q] = t + 32 * q < I ? z[t + 32 * q] : 0.0;
    ss = fma(u[q], u[q], ss);
  }
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const double sc = 1.0 / sqrt(ss);
#pragma unroll
  for (int q = 0; q < N; ++q) u[q] *= sc;
  double v[N], tau = 0.0;
  auto fetch = [&](int j) {
    tau = j >= 0 ? M.d[2 * I + j] : 0.0;
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const int col = t + 32 * q;
      v[q] = j >= 0 && col > j && col < I ? M.V[(int64_t)j * I + col] : 0.0;
    }
  };
  fetch(I - 3);
  for (int j = I - 3; j >= 0; --j) {
    double cv[N], s = 0.0;
    const double ct = tau;
#pragma unroll
    for (int q = 0; q < N; ++q) cv[q] = v[q];
    fetch(j - 1);
    if (ct == 0.0) continue;  // no reflection was stored
#pragma unroll
    for (int q = 0; q < N; ++q) s = fma(cv[q], u[q], s);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    s *= -ct;
#pragma unroll
    for (int q = 0; q < N; ++q) u[q] = fma(s, cv[q], u[q]);
  }
#pragma unroll
  for (int q = 0; q < N; ++q)
    if (t + 32 * q < I) M.U[(int64_t)(t + 32 * q) * M.k + r] = u[q];
}

// ---- cyclic Jacobi (round-robin pairs) ------------------------------------------

// Angles of this round's rotations: zero A[p][q] for each pair (p < q).
__global__ void jacobi_angles_kernel(const double* __restrict__ Am, int m,
                                     const int2* __restrict__ pairs, int npairs,
                                     double2* __restrict__ cs) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npairs) return;
  const int p = pairs[t].x, q = pairs[t].y;
  const double apq = Am[(int64_t)p * m + q], app = Am[(int64_t)p * m + p],
               aqq = Am[(int64_t)q * m + q];
  double c = 1.0, s = 0.0;
  if (fabs(apq) > 1e-300 && fabs(apq) > 1e-18 * sqrt(fabs(app * aqq))) {
    const double th = (aqq - app) / (2.0 * apq);
    double tn;
    if (fabs(th) > 1e150)
      tn = 0.5 / th;
    else
      tn = (th >= 0.0 ? 1.0 : -1.0) / (fabs(th) + sqrt(th * th + 1.0));
    c = 1.0 / sqrt(tn * tn + 1.0);
    s = tn * c;
  }
  cs[t] = make_double2(c, s);
}

// Rows p, q of A become c A_p - s A_q and s A_p + c A_q.
__global__ void jacobi_rows_kernel(double* __restrict__ Am, int m, const int2* __restrict__ pairs,
                                   int npairs, const double2* __restrict__ cs) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)npairs * m) return;
  const int i = (int)(t / m), k = (int)(t % m);
  const int p = pairs[i].x, q = pairs[i].y;
  const double c = cs[i].x, s = cs[i].y;
  const double ap = Am[(int64_t)p * m + k], aq = Am[(int64_t)q * m + k];
  Am[(int64_t)p * m + k] = c * ap - s * aq;
  Am[(int64_t)q * m + k] = s * ap + c * aq;
}

// Columns p, q of A and of V likewise.
__global__ void jacobi_cols_kernel(double* __restrict__ Am, double* __restrict__ V, int m,
                                   const int2* __restrict__ pairs, int npairs,
                                   const double2* __restrict__ cs) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)npairs * m) return;
  const int i = (int)(t % npairs), k = (int)(t / npairs);
  const int p = pairs[i].x, q = pairs[i].y;
  const double c = cs[i].x, s = cs[i].y;
  double* ar = Am + (int64_t)k * m;
  const double ap = ar[p], aq = ar[q];
  ar[p] = c * ap - s * aq;
  ar[q] = s * ap + c * aq;
  double* vr = V + (int64_t)k * m;
  const double vp = vr[p], vq = vr[q];
  vr[p] = c * vp - s * vq;
  vr[q] = s * vp + c * vq;
}

// out[0] = sum of squared off-diagonal entries, out[1] = sum of squared
// diagonal entries (out zeroed by the caller).
__global__ void jacobi_offdiag_kernel(const double* __restrict__ Am, int m, double* out) {
  double off = 0.0, dia = 0.0;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < (int64_t)m * m;
       e += (int64_t)gridDim.x * blockDim.x) {
    const double v = Am[e];
    if (e / m == e % m)
      dia += v * v;
    else
      off += v * v;
  }
  for (int o = 16; o > 0; o >>= 1) {
    off += __shfl_down_sync(0xffffffffu, off, o);
    dia += __shfl_down_sync(0xffffffffu, dia, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(out, off);
    atomicAdd(out + 1, dia);
  }
}

// ---- factors from the singular vectors -------------------------------------------

// U[i, r] = +-V[i, col[r]] for r < k (the sign that makes the largest-|.|
// entry positive), one CTA per column; also writes the oriented column into
// Uo (I x k, FP64) for the later kernels.
__global__ void orient_kernel(const double* __restrict__ V, int m, int I,
                              const int* __restrict__ col, double* __restrict__ Uo, int k,
                              double* __restrict__ upn) {
  const int r = blockIdx.x;
  __shared__ double best_v[32];
  __shared__ int best_i[32];
  double bv = -1.0;
  int bi = 0x7fffffff;
  for (int i = threadIdx.x; i < I; i += blockDim.x) {
    const double a = fabs(V[(int64_t)i * m + col[r]]);
    if (a > bv || (a == bv && i < bi)) {
      bv = a;
      bi = i;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double ov = __shfl_down_sync(0xffffffffu, bv, o);
    const int oi = __shfl_down_sync(0xffffffffu, bi, o);
    if (ov > bv || (ov == bv && oi < bi)) {
      bv = ov;
      bi = oi;
    }
  }
  if ((threadIdx.x & 31) == 0) {
    best_v[threadIdx.x >> 5] = bv;
    best_i[threadIdx.x >> 5] = bi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
      if (best_v[w] > best_v[0] || (best_v[w] == best_v[0] && best_i[w] < best_i[0])) {
        best_v[0] = best_v[w];
        best_i[0] = best_i[w];
      }
  }
  __syncthreads();
  const double sg = V[(int64_t)best_i[0] * m + col[r]] < 0.0 ? -1.0 : 1.0;
  double up = 0.0, un = 0.0;
  for (int i = threadIdx.x; i < I; i += blockDim.x) {
    const double u = sg * V[(int64_t)i * m + col[r]];
    Uo[(int64_t)i * k + r] = u;
    if (u > 0.0) up += u * u;
    if (u < 0.0) un += u * u;
  }
  // norms^2 of the column's positive and negative parts (Nnsvd)
  __syncthreads();
  for (int o = 16; o > 0; o >>= 1) {
    up += __shfl_down_sync(0xffffffffu, up, o);
    un += __shfl_down_sync(0xffffffffu, un, o);
  }
  if ((threadIdx.x & 31) == 0) {
    best_v[threadIdx.x >> 5] = up;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += best_v[w];
    upn[2 * r] = t;
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) best_v[threadIdx.x >> 5] = un;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += best_v[w];
    upn[2 * r + 1] = t;
  }
}

// Norms^2 of the positive and negative parts of v_r = X_(n)^T u_r / s_r:
// one thread per unfolding column j (a, b), all k components; pn[2r] and
// pn[2r+1] accumulate (zeroed by the caller). Uo is I x k, sv the s_r.
__global__ void __launch_bounds__(256) vnorm_kernel(const float* __restrict__ X, int64_t A,
                                                    int64_t I, int64_t B,
                                                    const double* __restrict__ Uo, int k,
                                                    const double* __restrict__ sv,
                                                    double* __restrict__ pn) {
  extern __shared__ double us[];  // chunk of Uo rows: 64 x k
  const int64_t J = A * B;
  for (int r0 = 0; r0 < k; r0 += 16) {
    const int nr = min(16, k - r0);
    double pos[16], neg[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) pos[q] = neg[q] = 0.0;
    for (int64_t j0 = (int64_t)blockIdx.x * blockDim.x; j0 < J;
         j0 += (int64_t)gridDim.x * blockDim.x) {
      const int64_t j = j0 + threadIdx.x;
      const bool ok = j < J;
      const int64_t a = ok ? j / B : 0, b = ok ? j % B : 0;
      double w[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) w[q] = 0.0;
      for (int64_t i0 = 0; i0 < I; i0 += 64) {
        const int ni = (int)(I - i0 < 64 ? I - i0 : 64);
        __syncthreads();
        for (int e = threadIdx.x; e < ni * 16; e += blockDim.x) {
          const int ii = e / 16, q = e % 16;
          us[e] = q < nr ? Uo[(i0 + ii) * k + r0 + q] : 0.0;
        }
        __syncthreads();
        if (ok)
          for (int ii = 0; ii < ni; ++ii) {
            const double x = (double)__ldg(X + (a * I + i0 + ii) * B + b);
#pragma unroll
            for (int q = 0; q < 16; ++q) w[q] = fma(x, us[ii * 16 + q], w[q]);
          }
      }
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const double s = q < nr ? sv[r0 + q] : 0.0;
        const double v = (ok && s > 0.0) ? w[q] / s : 0.0;
        if (v > 0.0) pos[q] += v * v;
        if (v < 0.0) neg[q] += v * v;
      }
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      double p = pos[q], n = neg[q];
      for (int o = 16; o > 0; o >>= 1) {
        p += __shfl_down_sync(0xffffffffu, p, o);
        n += __shfl_down_sync(0xffffffffu, n, o);
      }
      if ((threadIdx.x & 31) == 0 && q < nr) {
        atomicAdd(pn + 2 * (r0 + q), p);
        atomicAdd(pn + 2 * (r0 + q) + 1, n);
      }
    }
  }
}

// The strategy's factor from the oriented singular vectors (one CTA; I x R
// outputs, FP64 arithmetic, fp32 result). pad holds the N(0, 0.01) draws for
// the columns k..R-1 (I x (R - k)).
__global__ void svd_factor_kernel(int strategy, const double* __restrict__ Uo, int I, int k,
                                  int R, const double* __restrict__ sv,
                                  const double* __restrict__ pn, const double* __restrict__ upn,
                                  const double* __restrict__ pad, float* __restrict__ out) {
  extern __shared__ double lev[];  // I leverage scores (LeverageScore only)
  __shared__ double red[32];
  if (strategy == TSR_INIT_LEVERAGE_SCORE) {
    // helpers.rs:331-349: lev_i = sum_{j<k} u_ij^2 / k, normalised by its sum
    // when that exceeds fp32 epsilon
    double part = 0.0;
    for (int i = threadIdx.x; i < I; i += blockDim.x) {
      double sc = 0.0;
      for (int j = 0; j < k; ++j) sc += Uo[(int64_t)i * k + j] * Uo[(int64_t)i * k + j];
      lev[i] = k > 0 ? sc / k : 0.0;
      part += lev[i];
    }
    for (int o = 16; o > 0; o >>= 1) part += __shfl_down_sync(0xffffffffu, part, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = part;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
      red[0] = t;
    }
    __syncthreads();
    const double total = red[0];
    if (total > 1.1920928955078125e-07)
      for (int i = threadIdx.x; i < I; i += blockDim.x) lev[i] /= total;
    __syncthreads();
  }
  for (int64_t e = threadIdx.x; e < (int64_t)I * R; e += blockDim.x) {
    const int i = (int)(e / R), r = (int)(e % R);
    double v;
    if (r < k) {
      const double u = Uo[(int64_t)i * k + r];
      if (strategy == TSR_INIT_SVD) {
        v = u;
      } else if (strategy == TSR_INIT_NNSVD) {
        // |u_pos| |v_pos| against |u_neg| |v_neg| (helpers.rs:277-300)
        const double pos_prod = sqrt(upn[2 * r]) * sqrt(pn[2 * r]);
        const double neg_prod = sqrt(upn[2 * r + 1]) * sqrt(pn[2 * r + 1]);
        if (pos_prod >= neg_prod)
          v = (u > 0.0 ? u : 0.0) * sqrt(sv[r] * pos_prod);
        else
          v = (u < 0.0 ? -u : 0.0) * sqrt(sv[r] * neg_prod);
      } else {  // LeverageScore
        v = u * sqrt(sv[r]) * sqrt(lev[i] * (double)I);
      }
    } else {
      const double z = pad[(int64_t)i * (R - k) + (r - k)];
      if (strategy == TSR_INIT_SVD)
        v = z;
      else if (strategy == TSR_INIT_NNSVD)
        v = fabs(z);
      else
        v = z * lev[i];
    }
    out[(int64_t)i * R + r] = (float)v;
  }
}

// Device scratch of one call: carved from a context slot reserved up front,
// allocated only past it (the Jacobi solver's matrices).
struct DevBuf {
  std::vector<void*> ptrs;
  uint8_t* base = nullptr;
  size_t left = 0;
  int reserve(tsr_ctx* ctx, size_t bytes) {
    void* p;
    TSR_TRY(slot_get(ctx, SLOT_MISC0, bytes, &p));
    base = (uint8_t*)p;
    left = bytes;
    return TSR_OK;
  }
  static size_t room(size_t bytes) { return (bytes + 255) & ~(size_t)255; }
  template <class T>
  int get(T** p, size_t n) {
    const size_t bytes = room(std::max<size_t>(n, 1) * sizeof(T));
    if (bytes <= left) {
      *p = (T*)base;
      base += bytes;
      left -= bytes;
      return TSR_OK;
    }
    void* q = nullptr;
    cudaError_t e = cudaMalloc(&q, std::max<size_t>(n, 1) * sizeof(T));
    if (e != cudaSuccess)
      return fail(TSR_E_CUDA, "cudaMalloc (%zu bytes): %s", n * sizeof(T), cudaGetErrorString(e));
    ptrs.push_back(q);
    *p = (T*)q;
    return TSR_OK;
  }
  ~DevBuf() {
    for (void* q : ptrs) cudaFree(q);
  }
};

constexpr int kMaxSvdRows = 1024;  // Jacobi on I_n x I_n: cubic in I_n

// Leading eigenpairs of G (I x I, device, overwritten): eigenvalues
// descending into lam (host, all I), eigenvector matrix V (device, m x m row
// major, column c = eigenvector of A's diagonal entry c) and the column of
// each rank position in order.
int jacobi_eigen(tsr_ctx* ctx, cudaStream_t s, DevBuf& buf, double* G, int I, double** Vout,
                 int* m_out, std::vector<double>* lam, std::vector<int>* order) {
  const int m = I + (I & 1);
  double *Am, *V, *off;
  TSR_TRY(buf.get(&Am, (size_t)m * m));
  TSR_TRY(buf.get(&V, (size_t)m * m));
  TSR_TRY(buf.get(&off, 2));
  TSR_CUDA(cudaMemsetAsync(Am, 0, sizeof(double) * m * m, s));
  TSR_CUDA(cudaMemcpy2DAsync(Am, sizeof(double) * m, G, sizeof(double) * I, sizeof(double) * I,
                             I, cudaMemcpyDeviceToDevice, s));
  std::vector<double> eye((size_t)m * m, 0.0);
  for (int i = 0; i < m; ++i) eye[(size_t)i * m + i] = 1.0;
  TSR_CUDA(cudaMemcpyAsync(V, eye.data(), sizeof(double) * m * m, cudaMemcpyHostToDevice, s));
  // round-robin pairing: player 0 fixed, the others rotate
  const int np = m / 2, rounds = m - 1;
  std::vector<int2> tab((size_t)rounds * np);
  std::vector<int> pl(m);
  std::iota(pl.begin(), pl.end(), 0);
  for (int r = 0; r < rounds; ++r) {
    for (int i = 0; i < np; ++i) {
      const int a = pl[i], b = pl[m - 1 - i];
      tab[(size_t)r * np + i] = make_int2(std::min(a, b), std::max(a, b));
    }
    std::rotate(pl.begin() + 1, pl.end() - 1, pl.end());
  }
  int2* pairs;
  double2* cs;
  TSR_TRY(buf.get(&pairs, tab.size()));
  TSR_TRY(buf.get(&cs, np));
  TSR_CUDA(cudaMemcpyAsync(pairs, tab.data(), sizeof(int2) * tab.size(), cudaMemcpyHostToDevice,
                           s));
  const unsigned g_rot = (unsigned)ceil_div(np, 128);
  const unsigned g_upd = (unsigned)ceil_div((int64_t)np * m, 256);
  for (int sweep = 0; sweep < 40; ++sweep) {
    double h[2];
    TSR_CUDA(cudaMemsetAsync(off, 0, 2 * sizeof(double), s));
    jacobi_offdiag_kernel<<<(unsigned)std::min<int64_t>(ceil_div((int64_t)m * m, 256), 1024), 256,
                            0, s>>>(Am, m, off);
    ctx->launches++;
    TSR_CUDA(cudaMemcpyAsync(h, off, sizeof(h), cudaMemcpyDeviceToHost, s));
    TSR_CUDA(cudaStreamSynchronize(s));
    if (!(h[0] > 1e-26 * h[1])) break;  // also stops on a zero matrix
    for (int r = 0; r < rounds; ++r) {
      const int2* pr = pairs + (size_t)r * np;
      jacobi_angles_kernel<<<g_rot, 128, 0, s>>>(Am, m, pr, np, cs);
      jacobi_rows_kernel<<<g_upd, 256, 0, s>>>(Am, m, pr, np, cs);
      jacobi_cols_kernel<<<g_upd, 256, 0, s>>>(Am, V, m, pr, np, cs);
      ctx->launches += 3;
    }
    TSR_CUDA(cudaGetLastError());
  }
  // eigenvalues: the diagonal (the padding index, if any, holds 0 and is dropped)
  std::vector<double> diag((size_t)m * m);
  TSR_CUDA(cudaMemcpy(diag.data(), Am, sizeof(double) * m * m, cudaMemcpyDeviceToHost));
  lam->assign(I, 0.0);
  for (int i = 0; i < I; ++i) (*lam)[i] = diag[(size_t)i * m + i];
  order->resize(I);
  std::iota(order->begin(), order->end(), 0);
  std::stable_sort(order->begin(), order->end(),
                   [&](int a, int b) { return (*lam)[a] > (*lam)[b]; });
  *Vout = V;
  *m_out = m;
  return TSR_OK;
}

}  // namespace

// The Gram of X's mode-n unfolding (A x I x B) into G.
static int launch_unfold_gram(tsr_ctx* ctx, cudaStream_t s, const float* X, int64_t A, int64_t I,
                              int64_t B, double* G) {
  const int64_t J = A * B, nt = ceil_div(I, GR_T), tiles = nt * (nt + 1) / 2;
  if (J == 0) {
    TSR_CUDA(cudaMemsetAsync(G, 0, sizeof(double) * I * I, s));
    return TSR_OK;
  }
  // about four CTAs per SM, at least two chunks each
  int64_t splits = std::max<int64_t>(1, 4 * (int64_t)ctx->sm_count / tiles);
  splits = std::min<int64_t>({splits, ceil_div(J, 2 * GR_K), 65535});
  const int64_t per = round_up(ceil_div(J, splits), GR_K);
  splits = ceil_div(J, per);
  void* pp;
  TSR_TRY(slot_get(ctx, SLOT_PARTIALS, sizeof(double) * (size_t)(splits * I * I), &pp));
  double* parts = (double*)pp;
  unfold_gram_kernel<<<dim3((unsigned)tiles, (unsigned)splits), 256, 0, s>>>(X, A, I, B, per,
                                                                             parts);
  gram_reduce_kernel<<<(unsigned)ceil_div(I * I, 32), 256, 0, s>>>(parts, (int)splits, I, G);
  ctx->launches += 2;
  TSR_CUDA(cudaGetLastError());
  return TSR_OK;
}

static int launch_tri(tsr_ctx* ctx, cudaStream_t s, const TriArgs& t, int n, int rows, int k) {
  switch ((rows + 31) / 32) {
    case 1: tridiag_kernel<2, 1><<<n, 512, 0, s>>>(t); break;
    case 2: tridiag_kernel<4, 2><<<n, 512, 0, s>>>(t); break;
    case 3: tridiag_kernel<6, 3><<<n, 512, 0, s>>>(t); break;
    case 4: tridiag_kernel<8, 4><<<n, 512, 0, s>>>(t); break;
    default: tridiag_kernel<10, 5><<<n, 512, 0, s>>>(t); break;
  }
  tri_eigen_kernel<<<dim3((unsigned)k + 1, (unsigned)n), 256, 0, s>>>(t);
  ctx->launches += 2;
  TSR_CUDA(cudaGetLastError());
  return TSR_OK;
}

int init_factors_device(tsr_ctx* ctx, const float* dX, int ndim, const int64_t* shape, int R,
                        int strategy, uint64_t seed, float* d_out) {
  cudaStream_t s = ctx->stream;
  if (strategy == TSR_INIT_RANDOM || strategy == TSR_INIT_RANDOM_NORMAL) {
    int64_t off = 0;
    for (int mode = 0; mode < ndim; ++mode) {
      const int64_t I = shape[mode];
      std::vector<float> h((size_t)(I * R));
      if (strategy == TSR_INIT_RANDOM) {
        seeded_uniform(seed, 200 + mode, I * R, h.data());
      } else {
        std::vector<double> z((size_t)(I * R));
        seeded_normal(seed, 400 + mode, I * R, 1.0, z.data());
        for (size_t e = 0; e < z.size(); ++e) h[e] = (float)z[e];
      }
      TSR_CUDA(cudaMemcpyAsync(d_out + off, h.data(), sizeof(float) * I * R,
                               cudaMemcpyHostToDevice, s));
      TSR_CUDA(cudaStreamSynchronize(s));
      off += I * R;
    }
    return TSR_OK;
  }
  // mode n of X as A x I x B, its thin SVD's leading components
  struct Mode {
    int64_t A = 1, I = 0, B = 1;
    int k = 0, m = 0;
    double *G = nullptr, *V = nullptr;  // Gram; eigenvectors (row stride m)
    std::vector<double> lam;
    std::vector<int> order;
    bool ready = false;
  };
  std::vector<Mode> ms(ndim);
  DevBuf buf;
  size_t bytes = 0;
  for (int mode = 0; mode < ndim; ++mode) {
    const size_t I = (size_t)std::min<int64_t>(shape[mode], kMaxSvdRows), r = (size_t)R;
    // Gram, reflections, vectors, their oriented copy, padding columns, vectors of I or R
    bytes += sizeof(double) * (2 * I * I + 2 * I * std::min(I, r) + I * r + 3 * I + 7 * r) +
             16 * 256;
  }
  TSR_TRY(buf.reserve(ctx, bytes));
  TriArgs tri{};
  int tri_mode[kMaxModes], n_tri = 0, tri_rows = 0, tri_k = 0;
  size_t lam_off[kMaxModes], lam_n = 0;
  for (int mode = 0; mode < ndim; ++mode) {
    Mode& q = ms[mode];
    q.I = shape[mode];
    if (q.I > kMaxSvdRows)
      return fail(TSR_E_UNSUPPORTED,
                  "SVD-based initialisation supports mode sizes up to %d (mode %d has %lld)",
                  kMaxSvdRows, mode, (long long)q.I);
    for (int m = 0; m < mode; ++m) q.A *= shape[m];
    for (int m = mode + 1; m < ndim; ++m) q.B *= shape[m];
    // the thin SVD of the I x J unfolding has min(I, J) components
    q.k = (int)std::min<int64_t>(R, std::min<int64_t>(q.I, q.A * q.B));
    if (q.I == 0) continue;
    TSR_TRY(buf.get(&q.G, (size_t)(q.I * q.I)));
    TSR_TRY(launch_unfold_gram(ctx, s, dX, q.A, q.I, q.B, q.G));
    if (q.I <= kTriRows && q.k > 0) {
      TriMode& t = tri.m[n_tri];
      t.G = q.G;
      t.I = (int)q.I;
      t.k = q.k;
      TSR_TRY(buf.get(&t.d, (size_t)(3 * q.I)));
      TSR_TRY(buf.get(&t.V, (size_t)(q.I * q.I)));
      TSR_TRY(buf.get(&t.U, (size_t)(q.I * q.k)));
      lam_off[n_tri] = lam_n;
      lam_n += (size_t)std::min<int64_t>(q.k + 1, q.I);
      tri_rows = std::max(tri_rows, t.I);
      tri_k = std::max(tri_k, t.k);
      tri_mode[n_tri++] = mode;
    }
  }
  if (n_tri > 0) {
    double* lam;
    TSR_TRY(buf.get(&lam, lam_n));
    for (int t = 0; t < n_tri; ++t) tri.m[t].lam = lam + lam_off[t];
    TSR_TRY(launch_tri(ctx, s, tri, n_tri, tri_rows, tri_k));
    std::vector<double> h(lam_n);
    TSR_CUDA(cudaMemcpyAsync(h.data(), lam, sizeof(double) * lam_n, cudaMemcpyDeviceToHost, s));
    TSR_CUDA(cudaStreamSynchronize(s));
    for (int t = 0; t < n_tri; ++t) {
      Mode& q = ms[tri_mode[t]];
      const double* l = h.data() + lam_off[t];
      const int n = (int)std::min<int64_t>(q.k + 1, q.I);
      bool apart = std::isfinite(l[0]) && l[0] > 0.0;
      for (int i = 0; i + 1 < n; ++i) apart = apart && l[i] - l[i + 1] > kTriGap * l[0];
      if (!apart) continue;
      q.ready = true;
      q.V = tri.m[t].U;
      q.m = q.k;
      q.lam.assign(l, l + q.k);
      q.order.resize(q.k);
      std::iota(q.order.begin(), q.order.end(), 0);
    }
  }
  int64_t off = 0;
  for (int mode = 0; mode < ndim; ++mode) {
    Mode& q = ms[mode];
    const int64_t I = q.I;
    const int k = q.k;
    float* out = d_out + off;
    off += I * R;
    if (I > 0 && !q.ready)
      TSR_TRY(jacobi_eigen(ctx, s, buf, q.G, (int)I, &q.V, &q.m, &q.lam, &q.order));
    std::vector<int> col(std::max(k, 1));
    std::vector<double> sv(std::max(k, 1));
    for (int r = 0; r < k; ++r) {
      col[r] = q.order[r];
      sv[r] = std::sqrt(std::max(q.lam[q.order[r]], 0.0));
    }
    int* dcol;
    double *dsv, *Uo, *pn, *upn, *dpad;
    TSR_TRY(buf.get(&dcol, col.size()));
    TSR_TRY(buf.get(&dsv, sv.size()));
    TSR_TRY(buf.get(&Uo, (size_t)I * std::max(k, 1)));
    TSR_TRY(buf.get(&pn, 2 * (size_t)std::max(k, 1)));
    TSR_TRY(buf.get(&upn, 2 * (size_t)std::max(k, 1)));
    TSR_TRY(buf.get(&dpad, (size_t)I * std::max(R - k, 1)));
    TSR_CUDA(cudaMemcpyAsync(dcol, col.data(), sizeof(int) * col.size(), cudaMemcpyHostToDevice, s));
    TSR_CUDA(cudaMemcpyAsync(dsv, sv.data(), sizeof(double) * sv.size(), cudaMemcpyHostToDevice, s));
    TSR_CUDA(cudaMemsetAsync(pn, 0, sizeof(double) * 2 * std::max(k, 1), s));
    std::vector<double> pad((size_t)I * std::max(R - k, 1), 0.0);
    if (R > k) {
      seeded_normal(seed, 500 + mode, I * (R - k), 0.01, pad.data());
      TSR_CUDA(cudaMemcpyAsync(dpad, pad.data(), sizeof(double) * pad.size(),
                               cudaMemcpyHostToDevice, s));
    }
    if (k > 0) {
      orient_kernel<<<k, 256, 0, s>>>(q.V, q.m, (int)I, dcol, Uo, k, upn);
      ctx->launches++;
      if (strategy == TSR_INIT_NNSVD) {
        const unsigned g = (unsigned)std::max<int64_t>(
            1, std::min<int64_t>(ceil_div(q.A * q.B, 256), 4 * (int64_t)ctx->sm_count));
        vnorm_kernel<<<g, 256, sizeof(double) * 64 * 16, s>>>(dX, q.A, I, q.B, Uo, k, dsv, pn);
        ctx->launches++;
      }
    }
    const size_t lev_bytes = strategy == TSR_INIT_LEVERAGE_SCORE ? sizeof(double) * I : 0;
    svd_factor_kernel<<<1, 1024, lev_bytes, s>>>(strategy, Uo, (int)I, k, R, dsv, pn, upn, dpad,
                                                  out);
    ctx->launches++;
    TSR_CUDA(cudaGetLastError());
    TSR_CUDA(cudaStreamSynchronize(s));
  }
  return TSR_OK;
}

void init_init_attributes() {
  cudaFuncSetAttribute(svd_factor_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)(sizeof(double) * kMaxSvdRows));
}

}  // namespace tsr

using namespace tsr;

extern "C" {

int tsr_cp_init_dev_f32(tsr_ctx* ctx, const float* d_tensor, int ndim, const int64_t* shape,
                        int64_t rank, int strategy, uint64_t seed, float* d_out_factors) {
  if (!shape || !d_out_factors) return fail(TSR_E_INVALID_ARG, "null argument");
  if (ndim < 1 || ndim > kMaxModes)
    return fail(TSR_E_UNSUPPORTED, "tensor rank %d outside 1..%d", ndim, kMaxModes);
  TSR_TRY(check_sizes(ndim, shape, rank));
  if (rank == 0) return fail(TSR_E_INVALID_RANK, "Invalid rank: 0");
  if (strategy < TSR_INIT_RANDOM || strategy > TSR_INIT_LEVERAGE_SCORE)
    return fail(TSR_E_INVALID_ARG, "unknown initialisation strategy %d", strategy);
  if (strategy >= TSR_INIT_SVD && !d_tensor) return fail(TSR_E_INVALID_ARG, "null argument");
  TSR_TRY(check_ctx(ctx));
  return init_factors_device(ctx, d_tensor, ndim, shape, (int)rank, strategy, seed,
                             d_out_factors);
}

int tsr_cp_init_f32(tsr_ctx* ctx, const float* tensor, int ndim, const int64_t* shape,
                    int64_t rank, int strategy, uint64_t seed, float* out_factors) {
  if (!shape || !out_factors || !tensor) return fail(TSR_E_INVALID_ARG, "null argument");
  if (ndim < 1 || ndim > kMaxModes)
    return fail(TSR_E_UNSUPPORTED, "tensor rank %d outside 1..%d", ndim, kMaxModes);
  TSR_TRY(check_sizes(ndim, shape, rank));
  if (rank == 0) return fail(TSR_E_INVALID_RANK, "Invalid rank: 0");
  if (strategy < TSR_INIT_RANDOM || strategy > TSR_INIT_LEVERAGE_SCORE)
    return fail(TSR_E_INVALID_ARG, "unknown initialisation strategy %d", strategy);
  TSR_TRY(check_ctx(ctx));
  int64_t ftotal = 0;
  for (int m = 0; m < ndim; ++m) ftotal += shape[m] * rank;
  float* dX = nullptr;
  if (strategy >= TSR_INIT_SVD) TSR_TRY(upload_tensor(ctx, tensor, ndim, shape, nullptr, &dX));
  void* df;
  TSR_TRY(slot_get(ctx, SLOT_OUT, sizeof(float) * ftotal, &df));
  TSR_TRY(init_factors_device(ctx, dX, ndim, shape, (int)rank, strategy, seed, (float*)df));
  TSR_CUDA(cudaMemcpyAsync(out_factors, df, sizeof(float) * ftotal, cudaMemcpyDeviceToHost,
                           ctx->stream));
  TSR_CUDA(cudaStreamSynchronize(ctx->stream));
  return TSR_OK;
}

}  // extern "C"
