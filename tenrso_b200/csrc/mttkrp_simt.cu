// Dense MTTKRP, FP32 split-K form of the allocation-free entry point (every
// other FP32 MTTKRP runs the view kernels): M = X_(n) . KR with the unfolding
// X_(n) (I_n x K, row stride ld) resident in HBM and the KR rows generated into
// shared memory per K-step. Split-K over the grid: each CTA owns a K range
// and writes a partial I_n x R tile; the partials are summed in a fixed order
// (deterministic) by the consumer (the ALS solve, or mttkrp_reduce_kernel).
//
// Replaces the i/r/j triple loop of crates/tenrso-kernels/src/mttkrp.rs:135-143
// (same sum, different association: per-split partial sums, then a sum over
// splits).
#include <algorithm>

#include "kr.cuh"
#include "mttkrp.cuh"

namespace tsr {

namespace {
constexpr int BK = 32;

template <int BM, int BN>
constexpr int simt_threads() {
  return (BM / 8) * (BN / 4);
}
template <int BM, int BN>
constexpr int simt_min_blocks() {
  return 512 / simt_threads<BM, BN>() > 4 ? 4 : 512 / simt_threads<BM, BN>();
}

// BM x BN output tile per CTA, 8 x 4 per thread; NPF factor rows of each KR
// row are loaded one K-step ahead (the rest, for tensors of more than NPF + 1
// modes, after the FMA loop).
template <int BM, int BN, int NPF>
__global__ void __launch_bounds__(simt_threads<BM, BN>(), simt_min_blocks<BM, BN>())
mttkrp_f32_splitk_kernel(const float* __restrict__ A, int64_t rows, int64_t K, int64_t ld,
                         KRSpec kr, int64_t k_per_split, float* __restrict__ partials) {
  constexpr int NT = simt_threads<BM, BN>();
  constexpr int A_IT = BM * BK / 4 / NT;  // float4 of the A tile per thread
  constexpr int B_TPR = BN / 8;            // threads per KR row (8 columns each)
  constexpr int B_RPP = NT / B_TPR;        // KR rows per pass
  constexpr int B_IT = BK / B_RPP;         // passes per K-step
  static_assert(B_IT >= 1 && BK % B_RPP == 0, "tile");
  extern __shared__ __align__(16) float simt_smem[];
  float(*As)[BK][BM + 4] = reinterpret_cast<float(*)[BK][BM + 4]>(simt_smem);
  float(*Bs)[BK][BN] = reinterpret_cast<float(*)[BK][BN]>(simt_smem + 2 * BK * (BM + 4));
  const int tid = threadIdx.x;
  const int tx = tid % (BN / 4), ty = tid / (BN / 4);
  const int64_t m0 = (int64_t)blockIdx.y * BM;
  const int n0 = blockIdx.z * BN;
  const int R = kr.R;
  const int64_t kbeg = (int64_t)blockIdx.x * k_per_split;
  const int64_t kend = min(K, kbeg + k_per_split);
  const int nsteps = (int)((kend - kbeg + BK - 1) / BK);

  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  float4 areg[A_IT];
  float breg[B_IT][8];
  // A-tile mapping: 8 threads per row (32 floats = 128 B).
  auto load_a = [&](int64_t k0) {
#pragma unroll
    for (int it = 0; it < A_IT; ++it) {
      int idx = it * NT + tid;
      int m = idx / 8, kq = idx % 8;
      int64_t gm = m0 + m, gk = k0 + kq * 4;
      if (gm < rows && gk < kend)
        areg[it] = __ldg(reinterpret_cast<const float4*>(A + gm * ld + gk));
      else
        areg[it] = make_float4(0.f, 0.f, 0.f, 0.f);
      // columns past kend inside the same float4 belong to the next split
      if (gm < rows && gk < kend && gk + 4 > kend) {
        float* p = reinterpret_cast<float*>(&areg[it]);
        for (int e = (int)(kend - gk); e < 4; ++e) p[e] = 0.f;
      }
    }
  };
  auto store_a = [&](int buf) {
#pragma unroll
    for (int it = 0; it < A_IT; ++it) {
      int idx = it * NT + tid;
      int m = idx / 8, kq = idx % 8;
      As[buf][kq * 4 + 0][m] = areg[it].x;
      As[buf][kq * 4 + 1][m] = areg[it].y;
      As[buf][kq * 4 + 2][m] = areg[it].z;
      As[buf][kq * 4 + 3][m] = areg[it].w;
    }
  };
  // B-tile mapping: thread -> (KR row kk, 8 consecutive columns). The factor
  // values of the next K-step are loaded before the FMA loop of the current
  // one and multiplied after it, so the L2 latency overlaps the math.
  float braw[B_IT][NPF][8];
  uint32_t boff[B_IT][kMaxModes];
  bool bvalid[B_IT];
  auto gen_b_load = [&](int64_t k0) {
#pragma unroll
    for (int bi = 0; bi < B_IT; ++bi) {
      const int kk = bi * B_RPP + tid / B_TPR, c0 = (tid % B_TPR) * 8;
      const int64_t j = k0 + kk;
      bvalid[bi] = j < kend;
      kr_row_offsets(kr, (uint32_t)(bvalid[bi] ? j : kbeg), boff[bi]);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int c = n0 + c0 + e;
        const int cc = c < R ? c : 0;
#pragma unroll
        for (int q = 0; q < NPF; ++q)
          braw[bi][q][e] = q < kr.n_other ? __ldg(kr.f[q] + boff[bi][q] + cc) : 1.f;
      }
    }
  };
  auto gen_b_finish = [&]() {
#pragma unroll
    for (int bi = 0; bi < B_IT; ++bi) {
      const int c0 = (tid % B_TPR) * 8;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int c = n0 + c0 + e;
        float v = braw[bi][0][e];
#pragma unroll
        for (int q = 1; q < NPF; ++q) v *= braw[bi][q][e];
#pragma unroll
        for (int q = NPF; q < kMaxModes; ++q)
          if (q < kr.n_other) v *= __ldg(kr.f[q] + boff[bi][q] + (c < R ? c : 0));
        breg[bi][e] = (bvalid[bi] && c < R) ? v : 0.f;
      }
    }
  };
  auto store_b = [&](int buf) {
#pragma unroll
    for (int bi = 0; bi < B_IT; ++bi) {
      const int kk = bi * B_RPP + tid / B_TPR, c0 = (tid % B_TPR) * 8;
      *reinterpret_cast<float4*>(&Bs[buf][kk][c0]) =
          make_float4(breg[bi][0], breg[bi][1], breg[bi][2], breg[bi][3]);
      *reinterpret_cast<float4*>(&Bs[buf][kk][c0 + 4]) =
          make_float4(breg[bi][4], breg[bi][5], breg[bi][6], breg[bi][7]);
    }
  };

  if (nsteps > 0) {
    load_a(kbeg);
    gen_b_load(kbeg);
    gen_b_finish();
    store_a(0);
    store_b(0);
  }
  __syncthreads();
  for (int s = 0; s < nsteps; ++s) {
    const int buf = s & 1;
    const bool more = s + 1 < nsteps;
    if (more) {
      load_a(kbeg + (int64_t)(s + 1) * BK);
      gen_b_load(kbeg + (int64_t)(s + 1) * BK);
    }
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float4 a0 = *reinterpret_cast<const float4*>(&As[buf][kk][ty * 8]);
      float4 a1 = *reinterpret_cast<const float4*>(&As[buf][kk][ty * 8 + 4]);
      float4 b = *reinterpret_cast<const float4*>(&Bs[buf][kk][tx * 4]);
      float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      float bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    if (more) {
      gen_b_finish();
      store_a(buf ^ 1);
      store_b(buf ^ 1);
    }
    __syncthreads();
  }

  float* P = partials + (int64_t)blockIdx.x * rows * R;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    int64_t gm = m0 + ty * 8 + i;
    if (gm >= rows) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int c = n0 + tx * 4 + j;
      if (c < R) P[gm * R + c] = acc[i][j];
    }
  }
}

// out[e] = sum over splits of partials[s][e] (FP64), optionally times w[e % R].
// `groups` threads share an element, each summing every groups-th split with
// eight loads in flight; the groups combine through shared memory.
__global__ void __launch_bounds__(256)
mttkrp_reduce_kernel(const float* __restrict__ partials, int splits, int64_t n, int groups,
                     int R, const float* __restrict__ w, float* __restrict__ out) {
  __shared__ double red[256];
  const int per = 256 / groups;
  const int g = threadIdx.x / per, l = threadIdx.x % per;
  const int64_t k = (int64_t)blockIdx.x * per + l;
  double s = 0.0;
  if (k < n) {
    const float* p = partials + k;
    int q = g;
    for (; q + 7 * groups < splits; q += 8 * groups) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = __ldg(p + (int64_t)(q + u * groups) * n);
#pragma unroll
      for (int u = 0; u < 8; u += 2) s += (double)v[u] + (double)v[u + 1];
    }
    for (; q + groups < splits; q += 2 * groups) {
      const float v0 = __ldg(p + (int64_t)q * n), v1 = __ldg(p + (int64_t)(q + groups) * n);
      s += (double)v0 + (double)v1;
    }
    for (; q < splits; q += groups) s += (double)__ldg(p + (int64_t)q * n);
  }
  red[threadIdx.x] = s;
  __syncthreads();
  if (g != 0 || k >= n) return;
  for (int j = 1; j < groups; ++j) s += red[j * per + l];
  if (w) s *= (double)__ldg(w + (int)(k % R));
  out[k] = (float)s;
}

// khatri_rao.rs:56-89: C[a*J + b, k] = A[a, k] * B[b, k].
__global__ void khatri_rao_kernel(const float* __restrict__ A, int64_t I,
                                  const float* __restrict__ B, int64_t J, int64_t K,
                                  float* __restrict__ C) {
  int64_t n = I * J * K;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * blockDim.x) {
    int64_t k = e % K, row = e / K;
    int64_t a = row / J, b = row % J;
    C[e] = __ldg(A + a * K + k) * __ldg(B + b * K + k);
  }
}
}  // namespace

int launch_khatri_rao(tsr_ctx* ctx, const float* A, int64_t I, const float* B, int64_t J,
                      int64_t K, float* C) {
  int64_t n = I * J * K;
  unsigned grid = (unsigned)std::min<int64_t>(ceil_div(n, 256), (int64_t)ctx->sm_count * 8);
  khatri_rao_kernel<<<grid, 256, 0, ctx->stream>>>(A, I, B, J, K, C);
  ctx->launches++;
  TSR_CUDA(cudaGetLastError());
  return TSR_OK;
}

template <int BM, int BN>
constexpr size_t simt_smem_bytes() {
  return sizeof(float) * 2 * BK * (BM + 4 + BN);
}

void init_simt_attributes() {
  cudaFuncSetAttribute(mttkrp_f32_splitk_kernel<128, 64, 2>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)simt_smem_bytes<128, 64>());
  cudaFuncSetAttribute(mttkrp_f32_splitk_kernel<128, 64, 4>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)simt_smem_bytes<128, 64>());
  cudaFuncSetAttribute(mttkrp_f32_splitk_kernel<128, 32, 2>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)simt_smem_bytes<128, 32>());
  cudaFuncSetAttribute(mttkrp_f32_splitk_kernel<128, 32, 4>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)simt_smem_bytes<128, 32>());
}

SplitPlan plan_simt(const tsr_ctx* ctx, int64_t rows, int64_t K, int R) {
  SplitPlan p;
  p.bn = R <= 32 ? 32 : 64;
  const int64_t mt = ceil_div(rows, 128), nt = ceil_div(R, p.bn);
  // one full wave at the resident CTAs per SM (2 of 256 threads, 4 of 128)
  const int per_sm = p.bn == 32 ? 4 : 2;
  int64_t want =
      std::max<int64_t>(1, (int64_t)(ctx->sm_count - ctx->reserve_sms) * per_sm / (mt * nt));
  int64_t steps = ceil_div(K, BK);
  want = std::min<int64_t>(want, steps);
  p.k_per_split = round_up(ceil_div(K, want), BK);
  p.splits = (int)ceil_div(K, p.k_per_split);
  return p;
}

template <int BM, int BN, int NPF>
void launch_simt_tile(tsr_ctx* ctx, const float* A, const Unfolding& u, const KRSpec& kr,
                      const SplitPlan& plan, float* partials, dim3 grid) {
  mttkrp_f32_splitk_kernel<BM, BN, NPF>
      <<<grid, simt_threads<BM, BN>(), simt_smem_bytes<BM, BN>(), ctx->stream>>>(
          A, u.rows, u.cols, u.ld, kr, plan.k_per_split, partials);
}

int launch_mttkrp_simt(tsr_ctx* ctx, const float* A, const Unfolding& u, const KRSpec& kr,
                       const SplitPlan& plan, float* partials) {
  if (u.cols >= (int64_t)UINT32_MAX) return fail(TSR_E_UNSUPPORTED, "unfolding too wide");
  const int bn = plan.bn == 32 ? 32 : 64;
  dim3 grid(plan.splits, (unsigned)ceil_div(u.rows, 128), (unsigned)ceil_div(kr.R, bn));
  if (grid.y > 65535 || grid.z > 65535) return fail(TSR_E_UNSUPPORTED, "MTTKRP grid too large");
  const bool wide = kr.n_other > 2;
  if (bn == 32) {
    if (wide) launch_simt_tile<128, 32, 4>(ctx, A, u, kr, plan, partials, grid);
    else launch_simt_tile<128, 32, 2>(ctx, A, u, kr, plan, partials, grid);
  } else {
    if (wide) launch_simt_tile<128, 64, 4>(ctx, A, u, kr, plan, partials, grid);
    else launch_simt_tile<128, 64, 2>(ctx, A, u, kr, plan, partials, grid);
  }
  ctx->launches++;
  TSR_CUDA(cudaGetLastError());
  return TSR_OK;
}

int launch_mttkrp_reduce_scaled(tsr_ctx* ctx, const float* partials, int splits, int64_t rows,
                                int R, const float* w, float* out) {
  const int64_t n = rows * R;
  if (n == 0) return TSR_OK;
  // enough threads per element that a small result with many splits still
  // fills the SMs (32 groups leave 8 consecutive elements, one 32-byte sector,
  // per group), and no more: with 393216 elements of 6 splits, four groups
  // took 13.5 us, one 6
  int groups = 1;
  while (groups < 32 && 2 * groups <= splits &&
         ceil_div(n * groups, 256) < 4 * (int64_t)ctx->sm_count)
    groups *= 2;
  const int per = 256 / groups;
  mttkrp_reduce_kernel<<<(unsigned)ceil_div(n, per), 256, 0, ctx->stream>>>(
      partials, splits, n, groups, R > 0 ? R : 1, w, out);
  ctx->launches++;
  TSR_CUDA(cudaGetLastError());
  return TSR_OK;
}

int launch_mttkrp_reduce(tsr_ctx* ctx, const float* partials, int splits, int64_t n, float* out) {
  return launch_mttkrp_reduce_scaled(ctx, partials, splits, n, 1, nullptr, out);
}

}  // namespace tsr
