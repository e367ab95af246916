// The view kernel (see view.cuh), included by one translation unit per
// column-tile width.
//
// Tile: BM = 16 RPT rows x BN columns per CTA of 4 BN threads; a thread owns
// rows ty + 16 i and four neighbouring columns. Each step stages a chunk of up
// to 32 contracted columns: X's tile row by row (read back four columns at a
// time as 128-bit words) and the matching rows of K. The products are packed
// fp32 FMAs over column pairs, which have the scalar form's peak on sm_100a
// (about 70 TFLOP/s) at half the issue slots. Measured as T = X KR of a
// 12288 x 3072 matrix, 32 columns: 77 us (31 TFLOP/s) with 8 x 4 per thread
// and 16 warps per SM; 8 x 8 per thread at 12 warps 83 us, the copies spread
// between the FMAs 100 us, pairs over the contracted index 94 us. What holds
// it below peak is the duplication of X's values into pairs, the copies'
// address arithmetic and the barrier per step, at 50 % of the issue slots.
//
// X arrives by cp.async straight from its own layout, two buffers deep: 16
// bytes at a time where everything is aligned, else one float per lane (which
// also transposes on the way in when the row index is the contiguous
// direction). Odd sizes therefore cost no extra pass.
#pragma once
#include "view.cuh"

namespace tsr {
namespace {

constexpr int VK = 32;      // contracted columns per step, at most
constexpr int VPITCH = 36;  // floats per staged row of X (conflict-free reads)
// Products are summed in chains of 16 columns, the chains in a second set of
// accumulators: the rounding error stays that of short sums however long a
// split is (a tenth of the FMAs' adds, and less error than one long chain).
constexpr int VCHAIN = 16;

template <int BN, int RPT>
constexpr size_t view_smem() {
  const size_t stages = sizeof(float) * 2 * (16 * RPT * VPITCH + VK * BN);
  const size_t turned = sizeof(float) * (16 * RPT + 4) * BN;  // batched, transposed output
  return stages > turned ? stages : turned;
}
// Resident CTAs the register budget is held to: at most 128 registers.
template <int BN>
constexpr int view_min_blocks() {
  return BN == 64 ? 2 : BN == 48 ? 2 : BN == 32 ? 4 : 5;
}

__device__ __forceinline__ void view_cp16(float* dst, const float* src, bool ok) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = ok ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n)
               : "memory");
}
__device__ __forceinline__ void view_cp4(float* dst, const float* src, bool ok) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = ok ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n)
               : "memory");
}
__device__ __forceinline__ void view_fma2(uint64_t& d, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

__device__ __forceinline__ void view_add2(uint64_t& d, uint64_t a) {
  asm("add.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a));
}
__device__ __forceinline__ uint64_t view_dup(float a) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}

template <int V>
struct ViewInt {
  static constexpr int value = V;
};

// BATCHED: the matrix source, one product per batch entry, no split.
template <int BN, int RPT, int MAP, bool BATCHED>
__global__ void __launch_bounds__(4 * BN, view_min_blocks<BN>())
view_kernel(const __grid_constant__ ViewArgs g) {
  constexpr int TX = BN / 4, NT = 4 * BN, NW = NT / 32, BM = 16 * RPT;
  extern __shared__ __align__(16) float view_sm[];
  float* As = view_sm;                   // [2][BM][VPITCH]
  float* Bs = view_sm + 2 * BM * VPITCH;  // [2][VK][BN]
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int tx = tid % TX, ty = tid / TX;
  const int64_t i0 = (int64_t)blockIdx.x * BM;
  const int n0 = blockIdx.z * BN;
  const int R = g.R;
  const int rows_here = (int)min((int64_t)BM, g.rows - i0);
  const int64_t split = BATCHED ? 0 : blockIdx.y;
  const int64_t g0 = split * g.steps_per_split;
  const int nsteps = (int)min(g.steps_per_split, g.steps - g0);
  const int c0 = n0 + tx * 4;  // this thread's columns; it also stages them of K's tile

  // rows past the tensor are never loaded: zero them in both buffers once
  for (int e = rows_here * VPITCH + tid; e < BM * VPITCH; e += NT)
    As[e] = As[BM * VPITCH + e] = 0.f;

  for (int64_t z = BATCHED ? blockIdx.y : 0; z < (BATCHED ? g.batch : 1);
       z += BATCHED ? gridDim.y : 1) {
    const float* X = g.X + (BATCHED ? z * g.x_batch : 0) + i0 * g.row_stride;

    // the chunk being staged: run o, first column s0 of the run, its weights
    uint32_t o = (uint32_t)g0 / g.chunks, s0 = ((uint32_t)g0 - o * g.chunks) * g.kc;
    const float* run = X;
    float wt[4];
    bool new_run = true;
    int valid = 0;
    float4 braw[2];
    auto enter = [&]() {  // position and weights of the chunk (o, s0)
      if (new_run) {
        run = X;
        if (!BATCHED) {
#pragma unroll
          for (int e = 0; e < 4; ++e) wt[e] = 1.f;
          uint32_t q = o;
          for (int p = g.n_outer - 1; p >= 0; --p) {
            const uint32_t t = p > 0 ? q / g.size[p] : 0, i = q - t * g.size[p];
            run += i * g.stride[p];
            const float* f = g.f[p] + (int64_t)i * R + c0;
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (c0 + e < R) wt[e] *= __ldg(f + e);
            q = t;
          }
        }
        new_run = false;
      }
      valid = (int)min((uint32_t)g.kc, g.S - s0);
    };
    // rows m, m + step, .. of one staged column (or quad); columns past the
    // run (k >= valid) are zero-filled
    auto column = [&](float* dst, const float* src, int m, auto step, bool in) {
      constexpr int ST = decltype(step)::value;
      const int64_t inc = in ? ST * g.row_stride : 0;
      if (!in) src = g.X;
      dst += m * VPITCH;
#pragma unroll 4
      for (; m < rows_here; m += ST) {
        if (MAP == VIEW_VEC) view_cp16(dst, src, in);
        else view_cp4(dst, src, in);
        src += inc;
        dst += ST * VPITCH;
      }
    };
    auto load = [&](int buf) {
      float* dst = As + buf * BM * VPITCH;
      if (MAP == VIEW_VEC) {  // 8 quads of 4 rows
        const int k = (lane & 7) * 4, m = w * 4 + (lane >> 3);
        column(dst + k, run + s0 + k + m * g.row_stride, m, ViewInt<NW * 4>(), k < valid);
      } else if (MAP == VIEW_ALONG) {  // 32 columns of a row
        if (lane < g.kc)
          column(dst + lane, run + s0 + lane + w * g.row_stride, w, ViewInt<NW>(), lane < valid);
      } else {  // 4 columns of 8 rows; neighbouring rows (ACROSS) at constant offsets
        constexpr int ST = NW * 8, IT = (BM + ST - 1) / ST;
        const int64_t rs = MAP == VIEW_ACROSS ? 1 : g.row_stride;
        const int m = w * 8 + (lane & 7), kl = lane >> 3;
        const int n = m < rows_here ? (rows_here - m + ST - 1) / ST : 0;
        const float* src = run + m * rs + (s0 + kl) * g.k_stride;
        dst += m * VPITCH + kl;
        for (int k = kl; k < g.kc; k += 4) {
          const bool in = k < valid;
          const float* sp = in ? src : g.X;
#pragma unroll
          for (int q = 0; q < IT; ++q)
            if (q < n) view_cp4(dst + q * ST * VPITCH, sp + q * ST * rs, in);
          src += 4 * g.k_stride;
          dst += 4;
        }
      }
      // K's rows: columns past R and rows past the run are zero (the X values
      // the latter meet are zero-filled too: nothing non-finite leaks in)
      const float* ks = g.inner + (int64_t)(s0 + ty) * g.inner_s + (int64_t)c0 * g.inner_c;
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        braw[t] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ty + 16 * t < valid) {
          if (!BATCHED && g.inner_vec) {
            if (c0 < R) braw[t] = __ldg(reinterpret_cast<const float4*>(ks));
          } else {
            if (c0 < R) braw[t].x = __ldg(ks);
            if (c0 + 1 < R) braw[t].y = __ldg(ks + g.inner_c);
            if (c0 + 2 < R) braw[t].z = __ldg(ks + 2 * g.inner_c);
            if (c0 + 3 < R) braw[t].w = __ldg(ks + 3 * g.inner_c);
          }
        }
        ks += 16 * g.inner_s;
      }
    };
    auto store_b = [&](int buf) {
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int k = ty + 16 * t;
        float4 v = braw[t];
        if (!BATCHED) {
          v.x *= wt[0];
          v.y *= wt[1];
          v.z *= wt[2];
          v.w *= wt[3];
          if (k >= valid) v = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        *reinterpret_cast<float4*>(Bs + (buf * VK + k) * BN + tx * 4) = v;
      }
    };
    auto advance = [&]() {
      s0 += g.kc;
      if (s0 >= g.S) {
        s0 = 0;
        ++o;
        new_run = true;
      }
    };

    uint64_t tot[RPT][2];
#pragma unroll
    for (int i = 0; i < RPT; ++i) tot[i][0] = tot[i][1] = 0;

    enter();
    load(0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    store_b(0);
    for (int s = 0; s < nsteps; ++s) {
      const int buf = s & 1;
      const bool more = s + 1 < nsteps;
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      // after this barrier step s is staged and nobody reads the other buffer
      __syncthreads();
      if (more) {
        advance();
        enter();
        load(buf ^ 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
      }
      const float* a_row = As + buf * BM * VPITCH + ty * VPITCH;
      const float* b_col = Bs + buf * VK * BN + tx * 4;
#pragma unroll 1
      for (int k0 = 0; k0 < g.kc; k0 += VCHAIN) {
        uint64_t acc[RPT][2];
#pragma unroll
        for (int i = 0; i < RPT; ++i) acc[i][0] = acc[i][1] = 0;
        const int k1 = min(k0 + VCHAIN, g.kc);
#pragma unroll 1
        for (int kq = k0; kq < k1; kq += 4) {
          ulonglong2 b[4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            b[e] = *reinterpret_cast<const ulonglong2*>(b_col + (kq + e) * BN);
#pragma unroll
          for (int i = 0; i < RPT; ++i) {
            const float4 a = *reinterpret_cast<const float4*>(a_row + i * 16 * VPITCH + kq);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const uint64_t ad = view_dup(e == 0 ? a.x : e == 1 ? a.y : e == 2 ? a.z : a.w);
              view_fma2(acc[i][0], ad, b[e].x);
              view_fma2(acc[i][1], ad, b[e].y);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          view_add2(tot[i][0], acc[i][0]);
          view_add2(tot[i][1], acc[i][1]);
        }
      }
      if (more) store_b(buf ^ 1);
    }

    float* out = g.out + (BATCHED ? z * g.out_batch : split * g.out_split);
    auto value = [&](int i, int q) {
      const uint64_t v = tot[i][q >> 1];
      return __uint_as_float((uint32_t)((q & 1) ? v >> 32 : v));
    };
    if (!BATCHED || g.out_col == 1) {
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const int m = ty + 16 * i;
        if (m >= rows_here) continue;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (c0 + q < R) out[(i0 + m) * g.out_row + c0 + q] = value(i, q);
      }
      if (BATCHED) __syncthreads();  // the next batch entry refills the buffers
    } else {
      // rows are the output's contiguous direction: turn the tile through
      // shared memory and write whole runs of rows
      __syncthreads();
      constexpr int P = BM + 4;
#pragma unroll
      for (int i = 0; i < RPT; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) view_sm[(tx * 4 + q) * P + ty + 16 * i] = value(i, q);
      __syncthreads();
      for (int e = tid; e < BM * BN; e += NT) {
        const int m = e % BM, c = e / BM;
        if (m < rows_here && n0 + c < R)
          out[(i0 + m) * g.out_row + (n0 + c) * g.out_col] = view_sm[c * P + m];
      }
      __syncthreads();
      for (int e = rows_here * VPITCH + tid; e < BM * VPITCH; e += NT)
        As[e] = As[BM * VPITCH + e] = 0.f;
    }
  }
}

template <int BN, int RPT, int MAP>
int view_occ() {
  constexpr size_t sm = view_smem<BN, RPT>();
  cudaFuncSetAttribute(view_kernel<BN, RPT, MAP, false>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if constexpr (MAP != VIEW_STRIDED)  // batched products have a contiguous side
    cudaFuncSetAttribute(view_kernel<BN, RPT, MAP, true>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, view_kernel<BN, RPT, MAP, false>,
                                                4 * BN, sm);
  return n > 0 ? n : 1;
}
template <int BN, int RPT>
int view_occ_min() {
  const int n[4] = {view_occ<BN, RPT, VIEW_VEC>(), view_occ<BN, RPT, VIEW_ALONG>(),
                    view_occ<BN, RPT, VIEW_ACROSS>(), view_occ<BN, RPT, VIEW_STRIDED>()};
  int least = n[0];
  for (int v : n) least = v < least ? v : least;
  return least;
}

template <int BN, int RPT, bool BATCHED>
void view_map(cudaStream_t s, const ViewArgs& g, dim3 grid) {
  constexpr size_t sm = view_smem<BN, RPT>();
  constexpr int nt = 4 * BN;
  if (g.map == VIEW_VEC) view_kernel<BN, RPT, VIEW_VEC, BATCHED><<<grid, nt, sm, s>>>(g);
  else if (g.map == VIEW_ALONG)
    view_kernel<BN, RPT, VIEW_ALONG, BATCHED><<<grid, nt, sm, s>>>(g);
  else if (g.map == VIEW_ACROSS)
    view_kernel<BN, RPT, VIEW_ACROSS, BATCHED><<<grid, nt, sm, s>>>(g);
  else if constexpr (!BATCHED)
    view_kernel<BN, RPT, VIEW_STRIDED, false><<<grid, nt, sm, s>>>(g);
}
template <int BN, int RPT>
void view_go(cudaStream_t s, const ViewArgs& g, dim3 grid) {
  if (g.batch > 0) view_map<BN, RPT, true>(s, g, grid);
  else view_map<BN, RPT, false>(s, g, grid);
}

}  // namespace

template <int BN>
int view_ctas_per_sm(int bm) {
  switch (bm) {
    case 32: return view_occ_min<BN, 2>();
    case 48: return view_occ_min<BN, 3>();
    case 64: return view_occ_min<BN, 4>();
    case 96: return view_occ_min<BN, 6>();
    default: return view_occ_min<BN, 8>();
  }
}

template <int BN>
int launch_view_bn(tsr_ctx* ctx, cudaStream_t s, const ViewArgs& g, int bm, dim3 grid) {
  switch (bm) {
    case 32: view_go<BN, 2>(s, g, grid); break;
    case 48: view_go<BN, 3>(s, g, grid); break;
    case 64: view_go<BN, 4>(s, g, grid); break;
    case 96: view_go<BN, 6>(s, g, grid); break;
    default: view_go<BN, 8>(s, g, grid); break;
  }
  ctx->launches++;
  TSR_CUDA(cudaGetLastError());
  return TSR_OK;
}

}  // namespace tsr
