// Batched CP-ALS: many independent 3-way instances of uneven shape and rank
// in one persistent launch. Each instance runs tenrso's cp_als loop
// (crates/tenrso-decomp/src/cp/core.rs:59-182) from its own injected factors:
// the same mode order, Gram-Hadamard solve with the reference's ridge
// fallback (cp/helpers.rs:455-495), fit (helpers.rs:513-530) and
// convergence / oscillation rules (core.rs:142-166).
//
// Design:
//  - one CTA owns one instance at a time and keeps its three factors (fp32)
//    and their Grams (FP64) in shared memory for all of its sweeps, so the
//    instance's tensor stays hot in L2 across sweeps; CTAs take instances
//    from a queue in decreasing order of work (largest first);
//  - a sweep reads the tensor twice, both times with coalesced 128-bit loads
//    straight from global memory into register accumulators:
//      pass 1: V = X x_2 B (positions (i, k), loop over j), then
//              M_0[i, r] = sum_k V[i, k, r] C[k, r]   (mode-0 MTTKRP)
//      pass 2: U = X x_1 A_new (positions (j, k), loop over i), then
//              M_1[j, r] = sum_k U[j, k, r] C[k, r]   (mode-1 MTTKRP)
//              M_2[k, r] = sum_j U[j, k, r] B_new[j, r] (mode-2 MTTKRP, after
//              the mode-1 solve; U is kept in a per-CTA global scratch)
//    which equals the reference's three MTTKRPs (mttkrp.rs:74-146) up to the
//    fp32 summation order;
//  - the R x R FP64 Gram-Hadamard inverse is one warp's Gauss-Jordan;
//  - the tensor is stored with its last mode padded to a multiple of 4
//    (zeros), so every fiber starts 16-byte aligned.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <limits>
#include <string>

#include "als.cuh"
#include "dense.cuh"

namespace tsr {
namespace {

constexpr int kBatchMaxR = 16;
// Rows of M that so many items (float4s of the last mode) meet in are worth a
// resident CTA: the staging rows of add_rows against shared-memory atomics. us,
// two 256-thread CTAs with atomics / one with the staging rows, instances of
// 102 KB, rank 16, last mode 16: 4095 / 5549, 32: 6976 / 7758, 48: 11033 /
// 10208, 64: 14465 / 11663, 128: 34477 / 19055.
constexpr int kCrowded = 12;
constexpr size_t kBatchMaxSmem = 200 * 1024;
// Shared memory of an SM, and what a CTA takes of it beside its dynamic part
// (1 KB, and the kernel's static arrays).
constexpr size_t kSmSmem = 228 * 1024, kBatchOwnSmem = 1024 + 512;

struct BatchInst {
  int n0, n1, n2, n2p;  // mode sizes; n2p = n2 rounded up to a multiple of 4
  int R, rq;            // rank and ceil(R / 4)
  int64_t x_off;        // floats into the padded tensor store (multiple of 4)
  int64_t f_off;        // floats into the packed factors (A | B | C, row stride R)
};

struct BatchState {
  double xnorm_sq, fit, prev_fit, final_change;
  int iter, osc, reason, done;
  unsigned status;
  int ridge_used;
  int pad[2];
};

struct BatchArgs {
  const BatchInst* inst;
  const int* order;  // instance ids, largest work first
  int n_inst;
  const float* X;
  float* F;
  BatchState* st;
  double* hist;      // [n_inst][hist_stride]
  int hist_stride;
  float* uscratch;   // per CTA: n1 * n2p * 16 floats for the largest instance
  int64_t uscratch_floats;
  int* counter;
  int sweeps;
  int stage_off;     // bytes into the dynamic shared memory (0: no room, see add_rows)
  int ring_off;      // the same, see stream_rows
  double tol;
  float ridge_eps;   // f32 epsilon * R * 10 is formed per instance
};

// ---------------------------------------------------------------------------
// shared-memory layout of one instance (Rp = 4 * rq)
struct InstSmem {
  float* A;   // n0 x Rp
  float* B;   // n1 x Rp
  float* C;   // n2p x Rp (rows >= n2 are zero)
  float* Ct;  // Rp x n2p: C transposed, for conflict-free float4 reads of four C rows
  float* M;   // max(n0, n1, n2p) x Rp
  double* GA;  // 16 x 16 each (FP64 Grams)
  double* GB;
  double* GC;
  double* H;   // 16 x 16 Hadamard (identity padded)
  double* Hi;  // 16 x 16 inverse
  double* red;  // block-reduction scratch [32]
};

__device__ __forceinline__ InstSmem carve(unsigned char* base, const BatchInst& in) {
  InstSmem s;
  double* d = reinterpret_cast<double*>(base);
  s.GA = d;
  s.GB = d + 256;
  s.GC = d + 512;
  s.H = d + 768;
  s.Hi = d + 1024;
  s.red = d + 1280;
  float* f = reinterpret_cast<float*>(d + 1312);
  const int Rp = 4 * in.rq;
  s.A = f;
  s.B = s.A + in.n0 * Rp;
  s.C = s.B + in.n1 * Rp;
  s.Ct = s.C + in.n2p * Rp;
  s.M = s.Ct + in.n2p * Rp;
  return s;
}

__host__ __device__ inline size_t inst_smem_bytes(int n0, int n1, int n2p, int rq) {
  const int Rp = 4 * rq;
  const int mx = n0 > n1 ? (n0 > n2p ? n0 : n2p) : (n1 > n2p ? n1 : n2p);
  return sizeof(double) * 1312 + sizeof(float) * (size_t)(n0 + n1 + 2 * n2p + mx) * Rp;
}

// Block sum of one double per thread (all threads call it).
template <int NT>
__device__ double block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < NT / 32; ++w) t += red[w];
  return t;
}

// G = U^T U over `rows` rows (FP64), Rp x Rp stored in a 16 x 16 block.
template <int NT>
__device__ void gram16(const float* U, int rows, int Rp, double* G) {
  for (int e = threadIdx.x; e < 256; e += NT) {
    const int a = e >> 4, b = e & 15;
    double s = 0.0;
    if (a < Rp && b < Rp)
      for (int i = 0; i < rows; ++i) s += (double)U[i * Rp + a] * (double)U[i * Rp + b];
    G[e] = s;
  }
}

// U_out = M . (G1 * G2)^-1 with the reference's ridge fallback; updates G_out
// = U_out^T U_out. Returns false (uniformly) when no ridge makes it SPD.
template <int NT>
__device__ bool solve_mode(const InstSmem& s, const float* M, int rows, int R, int Rp,
                           const double* G1, const double* G2, float* U, double* G_out,
                           float ridge_eps, int* ridge_used) {
  __shared__ int ok_flag;
  __shared__ double diag_mean;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int e = threadIdx.x; e < 256; e += NT) {
    const int a = e >> 4, b = e & 15;
    s.H[e] = (a < R && b < R) ? G1[e] * G2[e] : (a == b ? 1.0 : 0.0);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double d = 0.0;
    for (int a = 0; a < R; ++a) d += fabs(s.H[a * 17]);
    diag_mean = d / R;
  }
  __syncthreads();
  // attempts: plain, + eps R 10, + eps R 10 * mean diagonal (as the dense path)
  for (int attempt = 0; attempt < 3; ++attempt) {
    if (warp == 0) {
      const double ridge = attempt == 0 ? 0.0
                           : attempt == 1 ? (double)ridge_eps
                                          : (double)ridge_eps * fmax(diag_mean, 1.0);
      double v[8];
      const int c = lane & 15, r0 = lane >> 4;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int r = r0 + 2 * q;
        v[q] = s.H[r * 16 + c] + ((r == c && r < R) ? ridge : 0.0);
      }
      const bool ok = warp_gj16(v, lane);
#pragma unroll
      for (int q = 0; q < 8; ++q) s.Hi[(r0 + 2 * q) * 16 + c] = v[q];
      if (lane == 0) ok_flag = ok ? 1 : 0;
    }
    __syncthreads();
    if (ok_flag) {
      if (attempt > 0 && threadIdx.x == 0) *ridge_used = attempt;
      break;
    }
    __syncthreads();
  }
  if (!ok_flag) return false;
  for (int e = threadIdx.x; e < rows * Rp; e += NT) {
    const int i = e / Rp, c = e - (e / Rp) * Rp;
    double acc = 0.0;
    if (c < R)
      for (int k = 0; k < R; ++k) acc += (double)M[i * Rp + k] * s.Hi[k * 16 + c];
    U[e] = (float)acc;
  }
  __syncthreads();
  gram16<NT>(U, rows, Rp, G_out);
  __syncthreads();
  return true;
}

// acc[p] += x[p] * W for the four k of x (W: one shared-memory factor row, Rp
// floats), as packed fp32 FMAs over column pairs: the same products and sums
// as scalar FMAs at half the issue slots.
__device__ __forceinline__ void fma2(uint64_t& d, float x, uint64_t b) {
  uint64_t xx;
  asm("mov.b64 %0, {%1, %1};" : "=l"(xx) : "f"(x));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(xx), "l"(b));
}
template <int RQ>
__device__ __forceinline__ void fma_row4(uint64_t (&acc)[4][2 * RQ], const float4 x,
                                         const float* W) {
  const ulonglong2* w2 = reinterpret_cast<const ulonglong2*>(W);
#pragma unroll
  for (int rq = 0; rq < RQ; ++rq) {
    const ulonglong2 b = w2[rq];
    fma2(acc[0][2 * rq], x.x, b.x);
    fma2(acc[0][2 * rq + 1], x.x, b.y);
    fma2(acc[1][2 * rq], x.y, b.x);
    fma2(acc[1][2 * rq + 1], x.y, b.y);
    fma2(acc[2][2 * rq], x.z, b.x);
    fma2(acc[2][2 * rq + 1], x.z, b.y);
    fma2(acc[3][2 * rq], x.w, b.x);
    fma2(acc[3][2 * rq + 1], x.w, b.y);
  }
}
template <int RQ>
__device__ __forceinline__ float acc_at(const uint64_t (&acc)[4][2 * RQ], int p, int r) {
  const uint64_t v = acc[p][r >> 1];
  return __uint_as_float((uint32_t)((r & 1) ? v >> 32 : v));
}

// acc += sum over q of x_q W[q], q = j0, j0 + split, .. below n, x_q the float4
// at xp + q * stride. With `ring` (kRing float4s of shared memory per thread,
// NT apart; its own slots, so no barrier) the loads run kRing - 2 ahead by
// cp.async; without it four at a time through registers, all of them consumed
// before the next four start, so a warp waits out a load latency per four rows.
// Sums and order are the same. 512 instances of 16..96 on 512 threads, 9.0 ms
// through registers, 7.7 through the ring; fewer than 24 rows per item do not
// pay for the ring's start (300 instances of 8..40: 0.60 ms against 0.64).
constexpr int kRing = 8;
template <int NT, int RQ>
__device__ __forceinline__ void stream_rows(uint64_t (&acc)[4][2 * RQ], const float4* xp,
                                            size_t stride, int j0, int n, int split,
                                            const float* W, uint32_t ring) {
  constexpr int Rp = 4 * RQ;
  if (!ring || n < 24 * split) {
    int j = j0;
    for (; j + 3 * split < n; j += 4 * split) {
      float4 xs[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) xs[u] = __ldg(xp + (size_t)(j + u * split) * stride);
#pragma unroll
      for (int u = 0; u < 4; ++u) fma_row4<RQ>(acc, xs[u], W + (j + u * split) * Rp);
    }
    for (; j < n; j += split) fma_row4<RQ>(acc, __ldg(xp + (size_t)j * stride), W + j * Rp);
    return;
  }
  const int count = j0 < n ? (n - j0 + split - 1) / split : 0;
  const int pairs = count / 2;
  const float4* src = xp + (size_t)j0 * stride;
  const float* w = W + j0 * Rp;
  const size_t step = (size_t)split * stride;
  int next = 0;  // first pair not yet requested
  auto request = [&]() {
    if (next < pairs) {
      const uint32_t at = ring + (uint32_t)(next % (kRing / 2)) * (2 * NT * 16);
      asm volatile(
          "cp.async.cg.shared.global [%0], [%1], 16;\n\t"
          "cp.async.cg.shared.global [%2], [%3], 16;" ::"r"(at),
          "l"(src), "r"(at + NT * 16), "l"(src + step)
          : "memory");
      src += 2 * step;
    }
    ++next;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int u = 0; u < kRing / 2 - 1; ++u) request();
  for (int q = 0; q < pairs; ++q) {
    // the slots requested here held the pair of the previous turn, whose FMAs
    // have their values
    request();
    asm volatile("cp.async.wait_group %0;" ::"n"(kRing / 2 - 1) : "memory");
    const uint32_t at = ring + (uint32_t)(q % (kRing / 2)) * (2 * NT * 16);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      float4 x;
      asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                   : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w)
                   : "r"(at + u * (NT * 16))
                   : "memory");
      fma_row4<RQ>(acc, x, w);
      w += split * Rp;
    }
  }
  if (count & 1) fma_row4<RQ>(acc, __ldg(src), w);
  // nothing in flight into the ring when its next use begins
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Adds the items' contributions to their rows of M: v[r] of item t0 + thread
// belongs to row (t / nkq) % rows. All threads of the CTA call it for the same
// t0. With `stage` (Rp rows of NT + 1 floats of shared memory) the items meet
// there and one thread sums each row's run of nkq; without it (instances that
// leave it no room, see plan_smem) they add with shared-memory atomics, which a
// warp's lanes on one row serialise: at 96^3 rank 16 that took most of a pass.
template <int NT, int Rp>
__device__ __forceinline__ void add_rows(const float (&v)[Rp], int t0, int items, int nkq,
                                         int rows, bool split, int R, float* M, float* stage) {
  const int t = t0 + threadIdx.x;
  if (!stage) {
    if (t < items)
#pragma unroll
      for (int r = 0; r < Rp; ++r)
        if (r < R) atomicAdd(M + ((t / nkq) % rows) * Rp + r, v[r]);
    return;
  }
  const int n = min(NT, items - t0);
  __syncthreads();  // the previous batch of items has been summed
#pragma unroll
  for (int r = 0; r < Rp; ++r) stage[r * (NT + 1) + threadIdx.x] = v[r];
  __syncthreads();
  const int s0 = t0 / nkq, ns = (t0 + n - 1) / nkq - s0 + 1;
  for (int e = threadIdx.x; e < ns * Rp; e += NT) {
    const int r = e % Rp, sg = s0 + e / Rp;
    const int x0 = max(sg * nkq - t0, 0), x1 = min((sg + 1) * nkq - t0, n);
    const float* p = stage + r * (NT + 1);
    float s4[4] = {0.f, 0.f, 0.f, 0.f};  // four short chains: less latency and rounding
    int x = x0;
    for (; x + 3 < x1; x += 4)
#pragma unroll
      for (int u = 0; u < 4; ++u) s4[u] += p[x + u];
    for (; x < x1; ++x) s4[0] += p[x];
    const float sum = (s4[0] + s4[1]) + (s4[2] + s4[3]);
    if (r < R) {
      float* m = M + (sg % rows) * Rp + r;
      if (split) atomicAdd(m, sum);  // other groups of items share the row
      else *m += sum;
    }
  }
}

// Ct = C^T (Rp x n2p), the whole CTA; ends with a barrier.
__device__ __forceinline__ void transpose_c(const InstSmem& s, int n2p, int Rp, int nt) {
  for (int e = threadIdx.x; e < n2p * Rp; e += nt) {
    const int k = e / Rp, r = e - k * Rp;
    s.Ct[r * n2p + k] = s.C[e];
  }
  __syncthreads();
}

// pass 1: M[i, r] += sum_k (sum_j X[i, j, k] B[j, r]) C[k, r]
template <int NT, int RQ>
__device__ void pass_v(const float4* __restrict__ X4, int n0, int n1, int nkq, const float* B,
                       const float* Ct, float* M, int R, float* stage, uint32_t ring) {
  constexpr int Rp = 4 * RQ;
  const int nq = n0 * nkq;
  const int split = nq >= NT ? 1 : min(n1, NT / nq);
  const int items = nq * split;
  for (int t0 = 0; t0 < items; t0 += NT) {
    const int t = t0 + threadIdx.x;
    float v[Rp];
#pragma unroll
    for (int r = 0; r < Rp; ++r) v[r] = 0.f;
    if (t < items) {
      const int g = t / nq, q = t - g * nq;
      const int i = q / nkq, kq = q - i * nkq;
      uint64_t acc[4][2 * RQ];
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int r = 0; r < 2 * RQ; ++r) acc[p][r] = 0;
      stream_rows<NT, RQ>(acc, X4 + (size_t)i * n1 * nkq + kq, nkq, g, n1, split, B, ring);
      // C rows 4kq .. 4kq+3 at column r: one float4 of Ct (lanes read
      // consecutive float4s; the rows of C would all map to one bank)
      const float4* Ct4 = reinterpret_cast<const float4*>(Ct);
#pragma unroll
      for (int r = 0; r < Rp; ++r) {
        const float4 c = Ct4[r * nkq + kq];
        v[r] = fmaf(acc_at<RQ>(acc, 0, r), c.x, 0.f);
        v[r] = fmaf(acc_at<RQ>(acc, 1, r), c.y, v[r]);
        v[r] = fmaf(acc_at<RQ>(acc, 2, r), c.z, v[r]);
        v[r] = fmaf(acc_at<RQ>(acc, 3, r), c.w, v[r]);
      }
    }
    add_rows<NT, Rp>(v, t0, items, nkq, n0, split > 1, R, M, stage);
  }
}

// pass 2: U[j, k, r] = sum_i X[i, j, k] A[i, r] (to the global scratch) and
// M[j, r] += sum_k U[j, k, r] C[k, r]
template <int NT, int RQ>
__device__ void pass_u(const float4* __restrict__ X4, int n0, int n1, int nkq, const float* A,
                       const float* Ct, float* M, float* U, int R, float* stage,
                       uint32_t ring) {
  constexpr int Rp = 4 * RQ;
  const int nq = n1 * nkq;
  const int split = nq >= NT ? 1 : min(n0, NT / nq);
  const int items = nq * split;
  for (int t0 = 0; t0 < items; t0 += NT) {
    const int t = t0 + threadIdx.x;
    float v[Rp];
#pragma unroll
    for (int r = 0; r < Rp; ++r) v[r] = 0.f;
    if (t < items) {
      const int g = t / nq, q = t - g * nq;
      const int j = q / nkq, kq = q - j * nkq;
      uint64_t acc[4][2 * RQ];
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int r = 0; r < 2 * RQ; ++r) acc[p][r] = 0;
      stream_rows<NT, RQ>(acc, X4 + (size_t)j * nkq + kq, (size_t)n1 * nkq, g, n0, split, A, ring);
      const float4* Ct4 = reinterpret_cast<const float4*>(Ct);
#pragma unroll
      for (int r = 0; r < Rp; ++r) {
        const float4 c = Ct4[r * nkq + kq];
        v[r] = fmaf(acc_at<RQ>(acc, 0, r), c.x, 0.f);
        v[r] = fmaf(acc_at<RQ>(acc, 1, r), c.y, v[r]);
        v[r] = fmaf(acc_at<RQ>(acc, 2, r), c.z, v[r]);
        v[r] = fmaf(acc_at<RQ>(acc, 3, r), c.w, v[r]);
      }
      // U rows (j, 4kq + p), Rp floats each
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        float4* u4 = reinterpret_cast<float4*>(U + ((size_t)j * (4 * nkq) + 4 * kq + p) * Rp);
#pragma unroll
        for (int rq = 0; rq < RQ; ++rq) {
          const float4 uv =
              make_float4(acc_at<RQ>(acc, p, 4 * rq), acc_at<RQ>(acc, p, 4 * rq + 1),
                          acc_at<RQ>(acc, p, 4 * rq + 2), acc_at<RQ>(acc, p, 4 * rq + 3));
          if (split == 1)
            u4[rq] = uv;
          else
            atomicAdd(u4 + rq, uv);
        }
      }
    }
    add_rows<NT, Rp>(v, t0, items, nkq, n1, split > 1, R, M, stage);
  }
}

template <int NT, int RQ>
__device__ void run_instance(const BatchArgs& a, int id, unsigned char* smem_raw) {
  constexpr int Rp = 4 * RQ;
  const BatchInst in = a.inst[id];
  const InstSmem s = carve(smem_raw, in);
  const int n0 = in.n0, n1 = in.n1, n2 = in.n2, n2p = in.n2p, R = in.R, nkq = n2p / 4;
  const float4* X4 = reinterpret_cast<const float4*>(a.X + in.x_off);
  float* F = a.F + in.f_off;
  float* U = a.uscratch + (size_t)blockIdx.x * a.uscratch_floats;
  float* stage = a.stage_off ? reinterpret_cast<float*>(smem_raw + a.stage_off) : nullptr;
  const uint32_t ring =
      a.ring_off ? (uint32_t)__cvta_generic_to_shared(smem_raw + a.ring_off) + threadIdx.x * 16 : 0;
  __shared__ BatchState st;
  __shared__ int ridge_used;
  if (threadIdx.x == 0) {
    st = a.st[id];
    ridge_used = st.ridge_used;
  }
  // factors into shared memory, rank padded to Rp (zeros), C rows padded to n2p
  for (int e = threadIdx.x; e < n0 * Rp; e += NT) {
    const int i = e / Rp, r = e - i * Rp;
    s.A[e] = r < R ? F[(size_t)i * R + r] : 0.f;
  }
  for (int e = threadIdx.x; e < n1 * Rp; e += NT) {
    const int i = e / Rp, r = e - i * Rp;
    s.B[e] = r < R ? F[(size_t)(n0 + i) * R + r] : 0.f;
  }
  for (int e = threadIdx.x; e < n2p * Rp; e += NT) {
    const int i = e / Rp, r = e - i * Rp;
    s.C[e] = (r < R && i < n2) ? F[(size_t)(n0 + n1 + i) * R + r] : 0.f;
  }
  __syncthreads();
  transpose_c(s, n2p, Rp, NT);
  gram16<NT>(s.A, n0, Rp, s.GA);
  gram16<NT>(s.B, n1, Rp, s.GB);
  gram16<NT>(s.C, n2p, Rp, s.GC);
  __syncthreads();
  const float ridge_eps = a.ridge_eps * (float)R;
  for (int sweep = 0; sweep < a.sweeps; ++sweep) {
    if (st.done) break;  // uniform: written by thread 0 before a barrier
    // ---- mode 0
    for (int e = threadIdx.x; e < n0 * Rp; e += NT) s.M[e] = 0.f;
    __syncthreads();
    pass_v<NT, RQ>(X4, n0, n1, nkq, s.B, s.Ct, s.M, R, stage, ring);
    __syncthreads();
    bool ok = solve_mode<NT>(s, s.M, n0, R, Rp, s.GB, s.GC, s.A, s.GA, ridge_eps, &ridge_used);
    // ---- mode 1
    if (ok) {
      for (int e = threadIdx.x; e < n1 * Rp; e += NT) s.M[e] = 0.f;
      const int nq = n1 * nkq;
      if (nq < NT && n0 > 1) {  // split passes add partial U rows atomically
        float4* u4 = reinterpret_cast<float4*>(U);
        const int n4 = n1 * n2p * Rp / 4;
        for (int e = threadIdx.x; e < n4; e += NT) u4[e] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      __syncthreads();
      pass_u<NT, RQ>(X4, n0, n1, nkq, s.A, s.Ct, s.M, U, R, stage, ring);
      __syncthreads();
      ok = solve_mode<NT>(s, s.M, n1, R, Rp, s.GA, s.GC, s.B, s.GB, ridge_eps, &ridge_used);
    }
    // ---- mode 2: M_2[k, r] = sum_j U[j, k, r] B[j, r] (float4 over r)
    if (ok) {
      const float4* U4 = reinterpret_cast<const float4*>(U);
      const float4* B4 = reinterpret_cast<const float4*>(s.B);
      for (int e = threadIdx.x; e < n2p * RQ; e += NT) {
        const int k = e / RQ, rq = e - k * RQ;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k < n2) {
#pragma unroll 8
          for (int j = 0; j < n1; ++j) {
            const float4 u = U4[((size_t)j * n2p + k) * RQ + rq];
            const float4 b = B4[j * RQ + rq];
            v.x = fmaf(u.x, b.x, v.x);
            v.y = fmaf(u.y, b.y, v.y);
            v.z = fmaf(u.z, b.z, v.z);
            v.w = fmaf(u.w, b.w, v.w);
          }
        }
        reinterpret_cast<float4*>(s.M)[e] = v;
      }
      __syncthreads();
      ok = solve_mode<NT>(s, s.M, n2p, R, Rp, s.GA, s.GB, s.C, s.GC, ridge_eps, &ridge_used);
      transpose_c(s, n2p, Rp, NT);  // the next sweep's passes read the new C through Ct
    }
    if (!ok) {
      if (threadIdx.x == 0) {
        st.status |= DS_NOT_SPD;
        st.done = 1;
      }
      __syncthreads();
      break;
    }
    // ---- fit (helpers.rs:513-530) and the rules of core.rs:142-166
    double inner = 0.0;
    for (int e = threadIdx.x; e < n2 * Rp; e += NT)
      inner += (double)s.M[e] * (double)s.C[e];
    inner = block_sum<NT>(inner, s.red);
    double rn = 0.0;
    for (int e = threadIdx.x; e < 256; e += NT) rn += s.GA[e] * s.GB[e] * s.GC[e];
    rn = block_sum<NT>(rn, s.red);
    if (threadIdx.x == 0) {
      const double xn = st.xnorm_sq;
      const double err = sqrt(fmax(xn + rn - 2.0 * inner, 0.0));
      double fit = 1.0 - err / sqrt(xn);
      fit = fmin(fmax(fit, 0.0), 1.0);
      const int iter = st.iter;
      st.fit = fit;
      if (iter < a.hist_stride) a.hist[(size_t)id * a.hist_stride + iter] = fit;
      if (iter > 0 && fit < st.prev_fit) st.osc += 1;
      const double change = fabs(fit - st.prev_fit);
      st.final_change = change;
      st.iter = iter + 1;
      if (iter > 0 && change < a.tol) {
        st.reason = TSR_REASON_FIT_TOLERANCE;
        st.done = 1;
      } else if (st.osc > 5 && iter > 10) {
        st.reason = TSR_REASON_OSCILLATION;
        st.done = 1;
      } else {
        st.prev_fit = fit;
      }
    }
    __syncthreads();
  }
  // factors back to global (unpadded) and the state
  for (int e = threadIdx.x; e < n0 * R; e += NT) F[e] = s.A[(e / R) * Rp + e % R];
  for (int e = threadIdx.x; e < n1 * R; e += NT) F[(size_t)n0 * R + e] = s.B[(e / R) * Rp + e % R];
  for (int e = threadIdx.x; e < n2 * R; e += NT)
    F[(size_t)(n0 + n1) * R + e] = s.C[(e / R) * Rp + e % R];
  if (threadIdx.x == 0) {
    st.ridge_used = ridge_used;
    a.st[id] = st;
  }
  __syncthreads();
}

template <int NT>
__global__ void __launch_bounds__(NT, 512 / NT) batched_als_kernel(BatchArgs a) {
  extern __shared__ __align__(16) unsigned char bsmem[];
  __shared__ int s_w;
  for (;;) {
    if (threadIdx.x == 0) s_w = atomicAdd(a.counter, 1);
    __syncthreads();
    const int w = s_w;
    __syncthreads();
    if (w >= a.n_inst) return;
    const int id = a.order[w];
    switch (a.inst[id].rq) {
      case 1: run_instance<NT, 1>(a, id, bsmem); break;
      case 2: run_instance<NT, 2>(a, id, bsmem); break;
      case 3: run_instance<NT, 3>(a, id, bsmem); break;
      default: run_instance<NT, 4>(a, id, bsmem); break;
    }
  }
}

// ||X||^2 of every instance (FP64), one CTA per instance.
__global__ void batch_norms_kernel(const BatchInst* inst, const float* X, BatchState* st) {
  const BatchInst in = inst[blockIdx.x];
  const float4* x4 = reinterpret_cast<const float4*>(X + in.x_off);
  const int64_t n4 = (int64_t)in.n0 * in.n1 * in.n2p / 4;
  double s = 0.0;
  for (int64_t e = threadIdx.x; e < n4; e += blockDim.x) {
    const float4 v = __ldg(x4 + e);
    s += (double)v.x * v.x + (double)v.y * v.y + (double)v.z * v.z + (double)v.w * v.w;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  __shared__ double red[32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
    st[blockIdx.x].xnorm_sq = t;
  }
}

// Fresh run state (keeping ||X||^2).
__global__ void batch_reset_kernel(BatchState* st, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double xn = st[i].xnorm_sq;
  BatchState z;
  memset(&z, 0, sizeof(z));
  z.xnorm_sq = xn;
  st[i] = z;
}

}  // namespace

void init_batched_attributes() {
  cudaFuncSetAttribute(batched_als_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)kBatchMaxSmem);
  cudaFuncSetAttribute(batched_als_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)kBatchMaxSmem);
  cudaFuncSetAttribute(batched_als_kernel<512>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)kBatchMaxSmem);
}

}  // namespace tsr

// ---------------------------------------------------------------------------
struct tsr_batch {
  int device = 0;
  int n_inst = 0;
  std::vector<tsr::BatchInst> inst;
  std::vector<int> order;
  int64_t x_floats = 0, f_floats = 0;
  size_t smem = 0;
  int rq = 1;   // the largest padded rank, in fours
  int nkq = 1;  // the longest last mode, in fours
  int64_t uscratch_floats = 0;
  tsr::BatchInst* d_inst = nullptr;
  int* d_order = nullptr;
  float* d_X = nullptr;
  tsr::BatchState* d_st = nullptr;
  int* d_counter = nullptr;  // one work counter per launch of a run
  int n_counters = 0;
  float* d_uscratch = nullptr;
  int uscratch_ctas = 0;
  double* d_hist = nullptr;
  int hist_stride = 0;
  // launch configuration (autotuned or set): threads per CTA, sweeps per launch
  int threads = 256;
  int sweeps_per_launch = 0;  // 0 = all of max_iters in one launch
  int ctas_per_sm = 2;
  // captured run graph and its key
  cudaGraphExec_t exec = nullptr;
  std::vector<uint8_t> key;
  int64_t graph_launches = 0;
};

namespace tsr {
namespace {

// Dynamic shared memory of a launch: the largest instance, then (where they
// fit) the staging rows of add_rows and the load ring of stream_rows.
struct SmemPlan {
  int held;  // CTAs that one SM holds
  int stage_off = 0, ring_off = 0;
  size_t bytes;
};

SmemPlan plan_smem(const tsr_batch* bt, int threads, int ctas_per_sm) {
  SmemPlan p;
  p.bytes = bt->smem;
  p.held = std::max(
      1, std::min(std::max(1, ctas_per_sm), (int)(kSmSmem / (bt->smem + kBatchOwnSmem))));
  auto most = [&]() { return std::min(kBatchMaxSmem, kSmSmem / p.held - kBatchOwnSmem); };
  const size_t stage = sizeof(float) * 4 * bt->rq * (threads + 1);
  if (bt->nkq >= kCrowded)
    while (p.held > 1 && bt->smem + stage > most()) --p.held;
  if (bt->smem + stage > most()) return p;
  p.stage_off = (int)bt->smem;
  p.bytes = bt->smem + stage;
  const size_t at = (p.bytes + 15) / 16 * 16, ring = (size_t)16 * kRing * threads;
  if (at + ring <= most()) {  // 16-byte slots; never at the price of a CTA
    p.ring_off = (int)at;
    p.bytes = at + ring;
  }
  return p;
}

// The configuration a new batch starts with (tsr_batch_autotune times them
// all): one 512-thread CTA per SM, or two of 256. A sweep of an instance of
// w = n0 n1 n2p (rank padded to 4) takes about 20 us (the solves) + 24 us per
// 1e6 of w on 512 threads, + 33 us on 256; two CTAs on an SM slow each other's
// passes by a third. (Rates from before the load ring of stream_rows, which took
// a fifth off each: of seven batches measured since, from one instance of 64^3
// to 512 of 16..96, the choice was the faster one in each.) The makespan is that of the largest instance or of the
// whole batch spread over the slots. Measured: 512 instances of 16..96, 7.6 ms
// (512 x 1) against 9.2; 300 instances of 8..40, 0.91 against 0.61. Where the SM
// holds one CTA of 256 only, it is 512: 296 instances of 4 x 5900 x 8 rank 4,
// 12.4 ms against 13.5, of 350 x 16 x 350 rank 16, 13.6 against 24.8.
void initial_config(const tsr_ctx* ctx, const tsr_batch* bt, int* threads, int* ctas_per_sm) {
  double wmax = 0.0, wsum = 0.0;
  for (const BatchInst& in : bt->inst) {
    const double w = 1e-6 * in.n0 * in.n1 * in.n2p * 4 * in.rq;
    wmax = std::max(wmax, w);
    wsum += w;
  }
  const double n = (double)bt->n_inst, sms = ctx->sm_count;
  const double one = std::max(20 + 24 * wmax, (20 * n + 24 * wsum) / sms);
  const double two = std::max(20 + 33 * wmax, (20 * n + 44 * wsum) / (2 * sms));
  const bool wide = one <= two || plan_smem(bt, 256, 2).held < 2;
  *threads = wide ? 512 : 256;
  *ctas_per_sm = wide ? 1 : 2;
}

int batch_validate(int n_inst, const int64_t* shapes, const int64_t* ranks) {
  if (n_inst <= 0) return fail(TSR_E_INVALID_ARG, "empty batch");
  for (int b = 0; b < n_inst; ++b) {
    const int64_t* sh = shapes + 3 * b;
    for (int m = 0; m < 3; ++m)
      if (sh[m] <= 0)
        return fail(TSR_E_SHAPE, "instance %d: mode %d has size %lld", b, m, (long long)sh[m]);
    const int64_t R = ranks[b];
    // core.rs:82-90
    if (R == 0 || R > std::min(sh[0], std::min(sh[1], sh[2])))
      return fail(TSR_E_INVALID_RANK, "instance %d: Invalid rank: %lld", b, (long long)R);
    if (R > kBatchMaxR)
      return fail(TSR_E_UNSUPPORTED, "instance %d: batched CP-ALS supports rank <= %d (got %lld)",
                  b, kBatchMaxR, (long long)R);
    if (sh[0] * sh[1] * ((sh[2] + 3) / 4 * 4) >= (int64_t)INT32_MAX)
      return fail(TSR_E_UNSUPPORTED, "instance %d is too large for the batched kernel", b);
  }
  return TSR_OK;
}

template <class T>
int dmalloc(T** p, size_t n) {
  cudaError_t e = cudaMalloc((void**)p, std::max<size_t>(n, 1) * sizeof(T));
  if (e != cudaSuccess) {
    *p = nullptr;
    return fail(TSR_E_CUDA, "cudaMalloc (%zu bytes): %s", n * sizeof(T), cudaGetErrorString(e));
  }
  return TSR_OK;
}

int ctas_for(const tsr_ctx* ctx, const tsr_batch* bt) {
  return std::max(1, std::min(bt->n_inst, ctx->sm_count * std::max(1, bt->ctas_per_sm)));
}

int ensure_run_buffers(tsr_ctx* ctx, tsr_batch* bt, int max_iters, int launches) {
  const int ctas = ctas_for(ctx, bt);
  if (bt->uscratch_ctas < ctas) {
    if (bt->d_uscratch) cudaFree(bt->d_uscratch);
    bt->d_uscratch = nullptr;
    bt->uscratch_ctas = 0;
    TSR_TRY(dmalloc(&bt->d_uscratch, (size_t)ctas * bt->uscratch_floats));
    bt->uscratch_ctas = ctas;
  }
  if (bt->n_counters < launches) {
    if (bt->d_counter) cudaFree(bt->d_counter);
    bt->d_counter = nullptr;
    bt->n_counters = 0;
    TSR_TRY(dmalloc(&bt->d_counter, launches));
    bt->n_counters = launches;
  }
  const int hs = std::max(max_iters, 1);
  if (bt->hist_stride < hs) {
    if (bt->d_hist) cudaFree(bt->d_hist);
    bt->d_hist = nullptr;
    bt->hist_stride = 0;
    TSR_TRY(dmalloc(&bt->d_hist, (size_t)bt->n_inst * hs));
    bt->hist_stride = hs;
  }
  return TSR_OK;
}

int sweeps_per_launch(const tsr_batch* bt, int max_iters) {
  return bt->sweeps_per_launch > 0 ? std::min(bt->sweeps_per_launch, max_iters) : max_iters;
}

// One whole run on the context's stream: reset the run state, then
// ceil(max_iters / S) persistent launches of S sweeps each (S = sweeps per
// launch), each taking instances from its own zeroed work counter.
int enqueue_run(tsr_ctx* ctx, tsr_batch* bt, int max_iters, double tol, float* dF) {
  const int S = sweeps_per_launch(bt, max_iters);
  const int launches = (max_iters + S - 1) / S;
  batch_reset_kernel<<<(bt->n_inst + 255) / 256, 256, 0, ctx->stream>>>(bt->d_st, bt->n_inst);
  ctx->launches++;
  TSR_CUDA(cudaGetLastError());
  TSR_CUDA(cudaMemsetAsync(bt->d_counter, 0, sizeof(int) * launches, ctx->stream));
  const int ctas = ctas_for(ctx, bt);
  for (int l = 0; l < launches; ++l) {
    BatchArgs a;
    a.inst = bt->d_inst;
    a.order = bt->d_order;
    a.n_inst = bt->n_inst;
    a.X = bt->d_X;
    a.F = dF;
    a.st = bt->d_st;
    a.hist = bt->d_hist;
    a.hist_stride = bt->hist_stride;
    a.uscratch = bt->d_uscratch;
    a.uscratch_floats = bt->uscratch_floats;
    a.counter = bt->d_counter + l;
    a.sweeps = std::min(S, max_iters - l * S);
    a.tol = tol;
    a.ridge_eps = std::numeric_limits<float>::epsilon() * 10.0f;
    const SmemPlan p = plan_smem(bt, bt->threads, bt->ctas_per_sm);
    a.stage_off = p.stage_off;
    a.ring_off = p.ring_off;
    const size_t smem = p.bytes;
    switch (bt->threads) {
      case 128: batched_als_kernel<128><<<ctas, 128, smem, ctx->stream>>>(a); break;
      case 512: batched_als_kernel<512><<<ctas, 512, smem, ctx->stream>>>(a); break;
      default: batched_als_kernel<256><<<ctas, 256, smem, ctx->stream>>>(a); break;
    }
    ctx->launches++;
    TSR_CUDA(cudaGetLastError());
  }
  return TSR_OK;
}

struct RunKey {
  int max_iters;
  double tol;
  const float* dF;
  int threads, spl, ctas_per_sm;
  cudaStream_t stream;
};

// Captured (once per key) and replayed run graph.
int run_graph(tsr_ctx* ctx, tsr_batch* bt, int max_iters, double tol, float* dF) {
  const int S = sweeps_per_launch(bt, max_iters);
  const int launches = (max_iters + S - 1) / S;
  TSR_TRY(ensure_run_buffers(ctx, bt, max_iters, launches));
  RunKey k;
  std::memset(&k, 0, sizeof(k));
  k.max_iters = max_iters;
  k.tol = tol;
  k.dF = dF;
  k.threads = bt->threads;
  k.spl = S;
  k.ctas_per_sm = bt->ctas_per_sm;
  k.stream = ctx->stream;
  std::vector<uint8_t> key((const uint8_t*)&k, (const uint8_t*)&k + sizeof(k));
  if (!bt->exec || key != bt->key) {
    if (bt->exec) {
      cudaGraphExecDestroy(bt->exec);
      bt->exec = nullptr;
    }
    cudaGraph_t g;
    const int64_t before = ctx->launches;
    TSR_CUDA(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    const int rc = enqueue_run(ctx, bt, max_iters, tol, dF);
    cudaError_t ce = cudaStreamEndCapture(ctx->stream, &g);
    if (rc != TSR_OK) return rc;
    TSR_CUDA(ce);
    bt->graph_launches = ctx->launches - before;
    ctx->launches = before;
    cudaError_t ie = cudaGraphInstantiate(&bt->exec, g, 0);
    cudaGraphDestroy(g);
    TSR_CUDA(ie);
    bt->key = key;
  }
  TSR_CUDA(cudaGraphLaunch(bt->exec, ctx->stream));
  ctx->launches += bt->graph_launches;
  return TSR_OK;
}

int read_infos(tsr_ctx* ctx, tsr_batch* bt, tsr_cp_info* infos) {
  std::vector<BatchState> hs(bt->n_inst);
  TSR_CUDA(cudaMemcpyAsync(hs.data(), bt->d_st, sizeof(BatchState) * bt->n_inst,
                           cudaMemcpyDeviceToHost, ctx->stream));
  std::vector<double> hist;
  bool want_hist = false;
  for (int b = 0; b < bt->n_inst && infos; ++b) want_hist |= infos[b].fit_history != nullptr;
  if (want_hist) {
    hist.resize((size_t)bt->n_inst * bt->hist_stride);
    TSR_CUDA(cudaMemcpyAsync(hist.data(), bt->d_hist, sizeof(double) * hist.size(),
                             cudaMemcpyDeviceToHost, ctx->stream));
  }
  TSR_CUDA(cudaStreamSynchronize(ctx->stream));
  int bad = -1;
  for (int b = 0; b < bt->n_inst; ++b) {
    if ((hs[b].status & DS_NOT_SPD) && bad < 0) bad = b;
    if (!infos) continue;
    tsr_cp_info& I = infos[b];
    I.fit = hs[b].fit;
    I.iters = hs[b].iter;
    I.reason = hs[b].done ? hs[b].reason : TSR_REASON_MAX_ITERATIONS;
    I.oscillation_count = hs[b].osc;
    I.oscillated = hs[b].osc > 0;
    I.final_fit_change = hs[b].final_change;
    I.ridge_used = hs[b].ridge_used;
    if (I.fit_history && hs[b].iter > 0)
      std::memcpy(I.fit_history, hist.data() + (size_t)b * bt->hist_stride,
                  sizeof(double) * std::min(hs[b].iter, bt->hist_stride));
  }
  if (bad >= 0)
    return fail(TSR_E_NOT_SPD,
                "instance %d: Linear algebra error: Gram matrix is not positive definite", bad);
  return TSR_OK;
}

}  // namespace
}  // namespace tsr

using namespace tsr;

extern "C" {

int tsr_batch_create_f32(tsr_ctx* ctx, int n_inst, const int64_t* shapes, const int64_t* ranks,
                         const float* const* tensors, tsr_batch** out) {
  if (!shapes || !ranks || !tensors || !out) return fail(TSR_E_INVALID_ARG, "null argument");
  *out = nullptr;
  TSR_TRY(batch_validate(n_inst, shapes, ranks));
  for (int b = 0; b < n_inst; ++b)
    if (!tensors[b]) return fail(TSR_E_INVALID_ARG, "instance %d: null tensor", b);
  TSR_TRY(check_ctx(ctx));
  tsr_batch* bt = new tsr_batch();
  bt->device = ctx->device;
  bt->n_inst = n_inst;
  bt->inst.resize(n_inst);
  std::vector<double> work(n_inst);
  for (int b = 0; b < n_inst; ++b) {
    BatchInst& in = bt->inst[b];
    in.n0 = (int)shapes[3 * b];
    in.n1 = (int)shapes[3 * b + 1];
    in.n2 = (int)shapes[3 * b + 2];
    in.n2p = (in.n2 + 3) / 4 * 4;
    in.R = (int)ranks[b];
    in.rq = (in.R + 3) / 4;
    in.x_off = bt->x_floats;
    bt->x_floats += (int64_t)in.n0 * in.n1 * in.n2p;
    in.f_off = bt->f_floats;
    bt->f_floats += (int64_t)(in.n0 + in.n1 + in.n2) * in.R;
    bt->rq = std::max(bt->rq, in.rq);
    bt->nkq = std::max(bt->nkq, in.n2p / 4);
    bt->smem = std::max(bt->smem, inst_smem_bytes(in.n0, in.n1, in.n2p, in.rq));
    bt->uscratch_floats =
        std::max<int64_t>(bt->uscratch_floats, (int64_t)in.n1 * in.n2p * 4 * in.rq);
    work[b] = (double)in.n0 * in.n1 * in.n2p * (4 * in.rq + 4);
  }
  bt->uscratch_floats = (bt->uscratch_floats + 3) / 4 * 4;
  initial_config(ctx, bt, &bt->threads, &bt->ctas_per_sm);
  auto cleanup = [&](int rc) {
    tsr_batch_destroy(bt);
    return rc;
  };
  if (bt->smem > kBatchMaxSmem)
    return cleanup(fail(TSR_E_UNSUPPORTED, "batch instances too large for shared memory"));
  bt->order.resize(n_inst);
  for (int b = 0; b < n_inst; ++b) bt->order[b] = b;
  std::stable_sort(bt->order.begin(), bt->order.end(),
                   [&](int x, int y) { return work[x] > work[y]; });
  int rc = dmalloc(&bt->d_inst, n_inst);
  if (rc == TSR_OK) rc = dmalloc(&bt->d_order, n_inst);
  if (rc == TSR_OK) rc = dmalloc(&bt->d_X, bt->x_floats);
  if (rc == TSR_OK) rc = dmalloc(&bt->d_st, n_inst);
  if (rc != TSR_OK) return cleanup(rc);
  // pack every tensor with its last mode padded to a multiple of 4 (zeros)
  std::vector<float> stage((size_t)bt->x_floats, 0.f);
  for (int b = 0; b < n_inst; ++b) {
    const BatchInst& in = bt->inst[b];
    for (int64_t f = 0; f < (int64_t)in.n0 * in.n1; ++f)
      std::memcpy(stage.data() + in.x_off + f * in.n2p, tensors[b] + f * in.n2,
                  sizeof(float) * in.n2);
  }
  cudaError_t e = cudaMemcpyAsync(bt->d_X, stage.data(), sizeof(float) * stage.size(),
                                  cudaMemcpyHostToDevice, ctx->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(bt->d_inst, bt->inst.data(), sizeof(BatchInst) * n_inst,
                        cudaMemcpyHostToDevice, ctx->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(bt->d_order, bt->order.data(), sizeof(int) * n_inst,
                        cudaMemcpyHostToDevice, ctx->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(bt->d_st, 0, sizeof(BatchState) * n_inst, ctx->stream);
  if (e != cudaSuccess) return cleanup(fail(TSR_E_CUDA, "%s", cudaGetErrorString(e)));
  batch_norms_kernel<<<n_inst, 256, 0, ctx->stream>>>(bt->d_inst, bt->d_X, bt->d_st);
  ctx->launches++;
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) return cleanup(fail(TSR_E_CUDA, "%s", cudaGetErrorString(e)));
  init_kernel_attributes();
  *out = bt;
  return TSR_OK;
}

int tsr_batch_destroy(tsr_batch* bt) {
  if (!bt) return TSR_OK;
  int prev = 0;
  cudaGetDevice(&prev);
  cudaSetDevice(bt->device);
  if (bt->exec) cudaGraphExecDestroy(bt->exec);
  cudaFree(bt->d_inst);
  cudaFree(bt->d_order);
  cudaFree(bt->d_X);
  cudaFree(bt->d_st);
  cudaFree(bt->d_counter);
  cudaFree(bt->d_uscratch);
  cudaFree(bt->d_hist);
  cudaSetDevice(prev);
  delete bt;
  return TSR_OK;
}

int tsr_batch_factor_layout(const tsr_batch* bt, int64_t* total_floats, int64_t* offsets) {
  if (!bt) return fail(TSR_E_INVALID_ARG, "null batch");
  if (total_floats) *total_floats = bt->f_floats;
  if (offsets)
    for (int b = 0; b < bt->n_inst; ++b) offsets[b] = bt->inst[b].f_off;
  return TSR_OK;
}

int tsr_batch_set_config(tsr_batch* bt, int threads, int sweeps_per_launch, int ctas_per_sm) {
  if (!bt) return fail(TSR_E_INVALID_ARG, "null batch");
  if (threads != 128 && threads != 256 && threads != 512)
    return fail(TSR_E_INVALID_ARG, "threads per instance must be 128, 256 or 512");
  if (sweeps_per_launch < 0 || ctas_per_sm < 1 || ctas_per_sm > 4)
    return fail(TSR_E_INVALID_ARG, "invalid sweeps per launch or CTAs per SM");
  bt->threads = threads;
  bt->sweeps_per_launch = sweeps_per_launch;
  bt->ctas_per_sm = ctas_per_sm;
  return TSR_OK;
}

int tsr_batch_get_config(const tsr_batch* bt, int* threads, int* sweeps_per_launch,
                         int* ctas_per_sm) {
  if (!bt) return fail(TSR_E_INVALID_ARG, "null batch");
  if (threads) *threads = bt->threads;
  if (sweeps_per_launch) *sweeps_per_launch = bt->sweeps_per_launch;
  if (ctas_per_sm) *ctas_per_sm = bt->ctas_per_sm;
  return TSR_OK;
}

int tsr_cp_als_batched_dev_f32(tsr_ctx* ctx, tsr_batch* bt, int max_iters, double tol,
                               const float* d_init, float* d_out, tsr_cp_info* infos) {
  if (!bt || !d_init || !d_out) return fail(TSR_E_INVALID_ARG, "null argument");
  if (!(tol >= 0.0 && tol < 1.0)) return fail(TSR_E_INVALID_TOL, "Invalid tolerance: %g", tol);
  if (max_iters < 0) return fail(TSR_E_INVALID_ARG, "max_iters must be >= 0");
  TSR_TRY(check_ctx(ctx));
  if (ctx->device != bt->device)
    return fail(TSR_E_INVALID_ARG, "batch created on device %d, context on device %d",
                bt->device, ctx->device);
  if (d_init != d_out)
    TSR_CUDA(cudaMemcpyAsync(d_out, d_init, sizeof(float) * bt->f_floats,
                             cudaMemcpyDeviceToDevice, ctx->stream));
  if (max_iters > 0) TSR_TRY(run_graph(ctx, bt, max_iters, tol, d_out));
  if (infos) TSR_TRY(read_infos(ctx, bt, infos));
  return TSR_OK;
}

int tsr_cp_als_batched_f32(tsr_ctx* ctx, tsr_batch* bt, int max_iters, double tol,
                           const float* init, uint64_t seed, float* out, tsr_cp_info* infos) {
  if (!bt || !out) return fail(TSR_E_INVALID_ARG, "null argument");
  if (!(tol >= 0.0 && tol < 1.0)) return fail(TSR_E_INVALID_TOL, "Invalid tolerance: %g", tol);
  TSR_TRY(check_ctx(ctx));
  std::vector<float> init_buf;
  const float* h_init = init;
  if (!h_init) {  // InitStrategy::Random per instance from the library's seeded stream
    init_buf.resize(bt->f_floats);
    for (int b = 0; b < bt->n_inst; ++b) {
      const BatchInst& in = bt->inst[b];
      const int64_t ns[3] = {in.n0, in.n1, in.n2};
      int64_t off = in.f_off;
      for (int m = 0; m < 3; ++m) {
        seeded_uniform(seed + (uint64_t)b, 200 + m, ns[m] * in.R, init_buf.data() + off);
        off += ns[m] * in.R;
      }
    }
    h_init = init_buf.data();
  }
  void* dF;
  TSR_TRY(slot_get(ctx, SLOT_OUT, sizeof(float) * bt->f_floats, &dF));
  TSR_CUDA(cudaMemcpyAsync(dF, h_init, sizeof(float) * bt->f_floats, cudaMemcpyHostToDevice,
                           ctx->stream));
  TSR_TRY(tsr_cp_als_batched_dev_f32(ctx, bt, max_iters, tol, (const float*)dF, (float*)dF,
                                     nullptr));
  TSR_CUDA(cudaMemcpyAsync(out, dF, sizeof(float) * bt->f_floats, cudaMemcpyDeviceToHost,
                           ctx->stream));
  return read_infos(ctx, bt, infos);
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Autotuner: times each launch configuration on the batch itself and keeps
// the fastest; results are cached in a small JSON file, one entry per line:
//   "<device>|<batch signature>": {"threads": T, "sweeps_per_launch": S,
//                                  "ctas_per_sm": C, "ms": t},
namespace {

std::string batch_signature(const tsr_batch* bt, int max_iters) {
  uint64_t h = 1469598103934665603ull;  // FNV-1a over the instance shapes and ranks
  auto mix = [&](uint64_t v) {
    for (int i = 0; i < 8; ++i) {
      h ^= (v >> (8 * i)) & 0xff;
      h *= 1099511628211ull;
    }
  };
  mix((uint64_t)bt->n_inst);
  mix((uint64_t)max_iters);
  for (const auto& in : bt->inst) {
    mix((uint64_t)in.n0);
    mix((uint64_t)in.n1);
    mix((uint64_t)in.n2);
    mix((uint64_t)in.R);
  }
  char buf[32];
  snprintf(buf, sizeof(buf), "%016llx", (unsigned long long)h);
  return buf;
}

bool cache_lookup(const char* path, const std::string& key, int* threads, int* spl, int* cps) {
  FILE* f = fopen(path, "r");
  if (!f) return false;
  char line[1024];
  bool found = false;
  const std::string needle = "\"" + key + "\":";
  while (fgets(line, sizeof(line), f)) {
    const char* p = strstr(line, needle.c_str());
    if (!p) continue;
    const char* t = strstr(p, "\"threads\":");
    const char* s = strstr(p, "\"sweeps_per_launch\":");
    const char* c = strstr(p, "\"ctas_per_sm\":");
    if (t && s && c && sscanf(t, "\"threads\": %d", threads) == 1 &&
        sscanf(s, "\"sweeps_per_launch\": %d", spl) == 1 &&
        sscanf(c, "\"ctas_per_sm\": %d", cps) == 1) {
      found = true;
      break;
    }
  }
  fclose(f);
  return found;
}

void cache_store(const char* path, const std::string& key, int threads, int spl, int cps,
                 double ms) {
  std::vector<std::string> entries;
  if (FILE* f = fopen(path, "r")) {
    char line[1024];
    const std::string needle = "\"" + key + "\":";
    while (fgets(line, sizeof(line), f)) {
      std::string l(line);
      if (l.find("\":") == std::string::npos || l.find(needle) != std::string::npos) continue;
      while (!l.empty() && (l.back() == '\n' || l.back() == ',' || l.back() == ' ')) l.pop_back();
      entries.push_back(l);
    }
    fclose(f);
  }
  char buf[512];
  snprintf(buf, sizeof(buf),
           " \"%s\": {\"threads\": %d, \"sweeps_per_launch\": %d, \"ctas_per_sm\": %d, "
           "\"ms\": %.4f}",
           key.c_str(), threads, spl, cps, ms);
  entries.push_back(buf);
  const std::string tmp = std::string(path) + ".tmp";
  FILE* f = fopen(tmp.c_str(), "w");
  if (!f) return;
  fprintf(f, "{\n");
  for (size_t i = 0; i < entries.size(); ++i)
    fprintf(f, "%s%s\n", entries[i].c_str(), i + 1 < entries.size() ? "," : "");
  fprintf(f, "}\n");
  fclose(f);
  rename(tmp.c_str(), path);
}

}  // namespace

extern "C" int tsr_batch_autotune(tsr_ctx* ctx, tsr_batch* bt, int max_iters,
                                  const float* d_init, const char* cache_path, int* from_cache) {
  if (!bt || !d_init || max_iters <= 0) return fail(TSR_E_INVALID_ARG, "invalid argument");
  TSR_TRY(check_ctx(ctx));
  if (from_cache) *from_cache = 0;
  cudaDeviceProp prop;
  TSR_CUDA(cudaGetDeviceProperties(&prop, ctx->device));
  std::string dev(prop.name);
  for (char& ch : dev)
    if (ch == '"' || ch == '|') ch = '_';
  const std::string key = dev + "|" + batch_signature(bt, max_iters);
  int t = 0, s = 0, c = 0;
  if (cache_path && cache_lookup(cache_path, key, &t, &s, &c) &&
      tsr_batch_set_config(bt, t, s, c) == TSR_OK) {
    if (from_cache) *from_cache = 1;
    return TSR_OK;
  }
  struct Cand {
    int threads, spl, cps;
  };
  const Cand cands[] = {{256, 0, 2}, {256, 0, 1}, {128, 0, 4}, {128, 0, 2}, {512, 0, 1},
                        {256, 1, 2}, {128, 1, 4}};
  void* scratch;
  TSR_TRY(slot_get(ctx, SLOT_MISC2, sizeof(float) * bt->f_floats, &scratch));
  cudaEvent_t e0, e1;
  TSR_CUDA(cudaEventCreate(&e0));
  TSR_CUDA(cudaEventCreate(&e1));
  double best = 1e300;
  Cand pick = cands[0];
  for (const Cand& cd : cands) {
    TSR_TRY(tsr_batch_set_config(bt, cd.threads, cd.spl, cd.cps));
    // warm-up run (captures the graph), then two timed runs
    TSR_TRY(tsr_cp_als_batched_dev_f32(ctx, bt, max_iters, 0.0, d_init, (float*)scratch,
                                       nullptr));
    TSR_CUDA(cudaEventRecord(e0, ctx->stream));
    for (int rep = 0; rep < 2; ++rep)
      TSR_TRY(tsr_cp_als_batched_dev_f32(ctx, bt, max_iters, 0.0, d_init, (float*)scratch,
                                         nullptr));
    TSR_CUDA(cudaEventRecord(e1, ctx->stream));
    TSR_CUDA(cudaEventSynchronize(e1));
    float ms = 0.f;
    TSR_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    if (ms / 2 < best) {
      best = ms / 2;
      pick = cd;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  TSR_TRY(tsr_batch_set_config(bt, pick.threads, pick.spl, pick.cps));
  if (cache_path) cache_store(cache_path, key, pick.threads, pick.spl, pick.cps, best);
  return TSR_OK;
}
