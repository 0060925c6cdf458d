// Dense small-dimension bucket: the Lindblad generator of a system of Hilbert dimension
// d <= 128 with dense operators, applied to rho (d x d):
//
//   L(t)[X] = A X + X A^dag + sum_i w_i C_i X C_i^dag,   A = sum_g a_g(t) A_g = -i H_nh,
//   w_i = |f_i(t)|^2,
//
// the reference's LindbladMatrixForm (qutip/core/cy/lindblad_matrix_form.pyx:105-204,
// full non-Hermitian branch) with dense operators, complex64 (the mixed form's generator).
//
// Bound: latency.  With two collapse operators the six d x d products are 50 million FP32
// multiply-adds at d = 128, 1.3 us of the whole GPU's FP32 units, so what counts is how many
// SMs share them and how long the chain of dependent pieces is.  An earlier form on the tensor
// cores (TF32 operands split hi + lo, three products each) spent 3 us per 32-wide K chunk
// on splitting and staging 128-row operands, for 0.55 us of MMAs, and its accumulation, which
// does not round to nearest, needed fresh accumulators for every chunk: 33 us per
// application on 24 SMs, 77 us on 8.  FP32 multiply-adds need no splitting, cut into any
// number of tiles and round to nearest.
//
// Work split: a cluster owns 8 output columns, its rank p the rows 16 p .. 16 p + 15 (128
// CTAs at d = 128).  Phase 1: every rank forms its 16 x 8 tile of w_i T_i, T_i = X C_i^dag;
// the ranks read one another's tiles through distributed shared memory.  Phase 2: A X,
// X A^dag and C_i (w_i T_i) go into one set of accumulators.  Within a CTA, half-warp s takes the
// k = s, s + 16, ... of every product, a thread a 4 x 2 tile (three 16-byte shared-memory
// loads for 8 complex multiply-adds); the 16 partial sums meet in a fixed order.
// Measured, d = 128, two collapse operators, a driven H: 33 -> 18 us per application (16 us with
// constant coefficients, 7 without collapse operators), the whole mixed solve 7.3 -> 4.7 ms,
// its error against the complex128 solution 2.1e-7..6.1e-7 over twelve systems where the
// tensor-core form had 4.6e-7..1.4e-6.
#include <cooperative_groups.h>
#include <mutex>

#include "capi_internal.h"
#include "common.cuh"
#include "stage.cuh"

namespace qg {

namespace cgrp = cooperative_groups;

constexpr int DN_THREADS = 256;
constexpr int DN_ROWS = 16;   // output rows of a CTA
constexpr int DN_COLS = 8;    // output columns of a cluster
constexpr int DN_SLICES = 16; // K slices (half-warps)
// Collapse operators staged at a time: two keep a CTA below half of an SM's shared memory.
// The GPU holds 15 clusters of 8 CTAs at one CTA per SM, and d = 128 has 16.
constexpr int DN_BATCH = 2;
static_assert(DN_BATCH * DN_ROWS * DN_COLS <= DN_THREADS, "a thread per T element");
// Strides between k of the operand tiles in shared memory: 16-byte aligned, and stores of
// consecutive k meet each bank twice at most.
constexpr int DN_RS = DN_ROWS + 2, DN_CS = DN_COLS + 2;

struct DenseSmem {  // offsets in float2
  int xr, xc, slot, slot_size, tm, part, total;
};
// Slot b: rows of an operator (DN_RS), then its conjugated column rows or T (DN_CS).
__host__ __device__ inline DenseSmem dense_layout(int kp) {
  DenseSmem s;
  s.xr = 0;
  s.xc = s.xr + kp * DN_RS;
  s.slot = s.xc + kp * DN_CS;
  s.slot_size = kp * (DN_RS + DN_CS);
  s.tm = s.slot + DN_BATCH * s.slot_size;
  s.part = s.tm + DN_BATCH * DN_ROWS * DN_COLS;
  s.total = s.part + DN_BATCH * (DN_THREADS / 32) * DN_ROWS * DN_COLS;
  return s;
}

__device__ __forceinline__ void cmac2(float2& a, float ar, float ai, float br, float bi) {
  a.x = fmaf(ar, br, a.x);
  a.x = fmaf(-ai, bi, a.x);
  a.y = fmaf(ar, bi, a.y);
  a.y = fmaf(ai, br, a.y);
}

// acc += rows^T cols over this half-warp's k: rows[k][r], cols[k][n] in shared memory.
__device__ __forceinline__ void mac_tile(float2 (&acc)[4][2], const float2* rows,
                                         const float2* cols, int kp, int slice, int rq, int cp) {
#pragma unroll 4
  for (int k = slice; k < kp; k += DN_SLICES) {
    const float4 a0 = *reinterpret_cast<const float4*>(rows + k * DN_RS + 4 * rq);
    const float4 a1 = *reinterpret_cast<const float4*>(rows + k * DN_RS + 4 * rq + 2);
    const float4 b = *reinterpret_cast<const float4*>(cols + k * DN_CS + 2 * cp);
    cmac2(acc[0][0], a0.x, a0.y, b.x, b.y);
    cmac2(acc[0][1], a0.x, a0.y, b.z, b.w);
    cmac2(acc[1][0], a0.z, a0.w, b.x, b.y);
    cmac2(acc[1][1], a0.z, a0.w, b.z, b.w);
    cmac2(acc[2][0], a1.x, a1.y, b.x, b.y);
    cmac2(acc[2][1], a1.x, a1.y, b.z, b.w);
    cmac2(acc[3][0], a1.z, a1.w, b.x, b.y);
    cmac2(acc[3][1], a1.z, a1.w, b.z, b.w);
  }
}

// This warp's two slices added, then its tile into part[r * DN_COLS + n].
__device__ __forceinline__ void put_tile(float2 (&acc)[4][2], float2* part, int lane, int rq,
                                         int cp) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      acc[i][j].x += __shfl_xor_sync(0xffffffffu, acc[i][j].x, 16);
      acc[i][j].y += __shfl_xor_sync(0xffffffffu, acc[i][j].y, 16);
      if (lane < 16) part[(4 * rq + i) * DN_COLS + 2 * cp + j] = acc[i][j];
    }
}

// Element e of a row-major operand tile of `width` rows: a warp covers 32 / 8 rows x 8 k.
__device__ __forceinline__ int tile_k(int e, int log2w) { return ((e >> (3 + log2w)) << 3) | (e & 7); }
__device__ __forceinline__ int tile_i(int e, int log2w) { return (e >> 3) & ((1 << log2w) - 1); }

template <int YDT, int EPI>
__global__ void __launch_bounds__(DN_THREADS, 2)
    dense_lindblad_kernel(qg_dense_lindblad L, double t, const float2* __restrict__ x,
                          AxpbyArgs ax, const __grid_constant__ RkArgs rk) {
  extern __shared__ __align__(16) float2 dn_smem[];
  __shared__ float2 ca[QG_MAX_GROUPS];
  __shared__ float wc[QG_MAX_COPS];
  __shared__ double red[DN_THREADS / 32];
  cgrp::cluster_group cl = cgrp::this_cluster();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ranks = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int d = L.d, kp = DN_ROWS * ranks;
  const int r0 = rank * DN_ROWS, n0 = (int)(blockIdx.x / (unsigned)ranks) * DN_COLS;
  const DenseSmem sm = dense_layout(kp);
  float2 *xr = dn_smem + sm.xr, *xc = dn_smem + sm.xc, *part = dn_smem + sm.part;
  auto slot_rows = [&](int b) { return dn_smem + sm.slot + b * sm.slot_size; };
  auto slot_cols = [&](int b) { return slot_rows(b) + kp * DN_RS; };
  const int slice = tid >> 4, rq = (tid >> 2) & 3, cp = tid & 3;
  const float2 zero = make_float2(0.f, 0.f);

  // Coefficient programs on warp 0 (a few microseconds of dependent FP64 work when there are
  // any) while the other warps stage what does not need them.
  const bool programs = L.a_coef_code || L.c_coef_code;
  const int skip = programs ? 32 : 0, step = DN_THREADS - skip, lt = tid - skip;
  if (!programs || warp == 0) {
    for (int i = tid; i < QG_MAX_GROUPS + L.n_cops; i += programs ? 32 : DN_THREADS) {
      if (i < L.n_groups) {
        const cplx a = L.a_coef_code
                           ? eval_coef(L.a_coef_code + L.a_coef_start[i], L.a_coef_consts, t)
                           : cplx{1.0, 0.0};
        ca[i] = make_float2((float)a.re, (float)a.im);
      } else if (i >= QG_MAX_GROUPS) {
        const int q = i - QG_MAX_GROUPS;
        const cplx f = L.c_coef_code
                           ? eval_coef(L.c_coef_code + L.c_coef_start[q], L.c_coef_consts, t)
                           : cplx{1.0, 0.0};
        wc[q] = (float)(f.re * f.re + f.im * f.im);
      }
    }
  }
  // collapse operators i0 .. i0 + m: rows of this rank, and conjugated rows of the columns
  auto stage_cops = [&](int i0, int m, int from, int stride) {
    for (int b = 0; b < m; ++b) {
      const float2* C = static_cast<const float2*>(L.c) + (size_t)(i0 + b) * d * d;
      float2 *cr = slot_rows(b), *cc = slot_cols(b);
#pragma unroll 8
      for (int e = from; e < DN_ROWS * kp; e += stride) {
        const int k = tile_k(e, 4), r = tile_i(e, 4);
        const bool in = r0 + r < d && k < d;
        cr[k * DN_RS + r] = in ? __ldg(C + (r0 + r) * d + k) : zero;
      }
#pragma unroll 4
      for (int e = from; e < DN_COLS * kp; e += stride) {
        const int k = tile_k(e, 3), n = tile_i(e, 3);
        const float2 v = n0 + n < d && k < d ? __ldg(C + (n0 + n) * d + k) : zero;
        cc[k * DN_CS + n] = make_float2(v.x, -v.y);
      }
    }
  };
  const int m0 = min(DN_BATCH, L.n_cops);
  if (lt >= 0) {
#pragma unroll 8
    for (int e = lt; e < DN_ROWS * kp; e += step) {  // X rows: X[r][k] at k d + r
      const int r = e & (DN_ROWS - 1), k = e >> 4;
      xr[k * DN_RS + r] = r0 + r < d && k < d ? __ldg(x + k * d + r0 + r) : zero;
    }
#pragma unroll 4
    for (int e = lt; e < DN_COLS * kp; e += step) {
      const int k = tile_k(e, 3), n = tile_i(e, 3);
      xc[k * DN_CS + n] = n0 + n < d && k < d ? __ldg(x + (n0 + n) * d + k) : zero;
    }
    stage_cops(0, m0, lt, step);
  }
  __syncthreads();
  // A(t) = sum_g a_g(t) A_g, rows of this rank and of the columns, in registers until the
  // collapse operators are done with the slots
  constexpr int AV = (DN_ROWS + DN_COLS) * QG_DENSE_MAX_D / DN_THREADS;
  float2 av[AV];
  auto a_place = [&](int q, bool& rows, int& k, int& i) {
    const int e = tid + q * DN_THREADS;
    rows = e < DN_ROWS * kp;
    const int f = rows ? e : e - DN_ROWS * kp, w = rows ? 4 : 3;
    k = tile_k(f, w);
    i = tile_i(f, w);
    return e < (DN_ROWS + DN_COLS) * kp;
  };
#pragma unroll
  for (int q = 0; q < AV; ++q) av[q] = zero;
#pragma unroll 1
  for (int g = 0; g < L.n_groups; ++g) {
    const float2* A = static_cast<const float2*>(L.a) + (size_t)g * d * d;
    const float2 c = ca[g];
    float2 v[AV];
#pragma unroll
    for (int q = 0; q < AV; ++q) {
      bool rows;
      int k, i;
      const bool in = a_place(q, rows, k, i);
      const int m = (rows ? r0 : n0) + i;
      v[q] = in && m < d && k < d ? __ldg(A + m * d + k) : zero;
    }
#pragma unroll
    for (int q = 0; q < AV; ++q) cmac2(av[q], c.x, c.y, v[q].x, v[q].y);
  }

  float2 acc[4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = zero;
  constexpr int TILE = DN_ROWS * DN_COLS, WARPS = DN_THREADS / 32;
  auto part_sum = [&](const float2* p) {
    float2 v = zero;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      v.x += p[w * TILE].x;
      v.y += p[w * TILE].y;
    }
    return v;
  };
  for (int i0 = 0; i0 < L.n_cops; i0 += DN_BATCH) {
    const int m = min(DN_BATCH, L.n_cops - i0);
    if (i0 > 0) {
      cl.sync();  // every rank has read the last batch's tiles
      stage_cops(i0, m, tid, DN_THREADS);
      __syncthreads();
    }
    // w_i X C_i^dag, this rank's rows
    for (int b = 0; b < m; ++b) {
      float2 p[4][2];
#pragma unroll
      for (int i = 0; i < 4; ++i) p[i][0] = p[i][1] = zero;
      mac_tile(p, xr, slot_cols(b), kp, slice, rq, cp);
      put_tile(p, part + (b * WARPS + warp) * TILE, lane, rq, cp);
    }
    __syncthreads();
    if (tid < m * TILE) {
      const int b = tid / TILE, o = tid - b * TILE;
      const float2 v = part_sum(part + b * WARPS * TILE + o);
      const float f = wc[i0 + b];
      dn_smem[sm.tm + tid] = make_float2(f * v.x, f * v.y);
    }
    cl.sync();  // every rank's tiles are in its shared memory
#pragma unroll 4
    for (int e = tid; e < m * kp * DN_COLS; e += DN_THREADS) {
      const int b = e / (kp * DN_COLS), f = e - b * kp * DN_COLS, k = f / DN_COLS, n = f % DN_COLS;
      const float2* remote = cl.map_shared_rank(dn_smem + sm.tm, k / DN_ROWS);
      slot_cols(b)[k * DN_CS + n] = remote[b * TILE + (k % DN_ROWS) * DN_COLS + n];
    }
    __syncthreads();
    for (int b = 0; b < m; ++b) mac_tile(acc, slot_rows(b), slot_cols(b), kp, slice, rq, cp);
  }
  __syncthreads();  // slot 0 is read
#pragma unroll
  for (int q = 0; q < AV; ++q) {
    bool rows;
    int k, i;
    if (!a_place(q, rows, k, i)) continue;
    if (rows) slot_rows(0)[k * DN_RS + i] = av[q];
    else slot_cols(0)[k * DN_CS + i] = make_float2(av[q].x, -av[q].y);
  }
  __syncthreads();
  mac_tile(acc, slot_rows(0), xc, kp, slice, rq, cp);  // A X
  mac_tile(acc, xr, slot_cols(0), kp, slice, rq, cp);  // X A^dag
  put_tile(acc, part + warp * TILE, lane, rq, cp);
  __syncthreads();
  double err_acc = 0.0;
  if (tid < TILE) {
    const int r = tid & (DN_ROWS - 1), n = tid >> 4;
    const float2 v = part_sum(part + r * DN_COLS + n);
    if (r0 + r < d && n0 + n < d)
      epilogue<QG_C64, YDT, EPI>((n0 + n) * d + r0 + r, cx<float>{v.x, v.y}, ax, rk, err_acc);
  }
  if constexpr (EPI == EPI_RK) {
    if (rk.stage == RK_STEP - 1) finish_error<DN_THREADS>(rk, err_acc, red);
  }
  if (L.n_cops > 0) cl.sync();  // no rank leaves while another may still read its tiles
}

template <int YDT, int EPI>
static int launch_dense(cudaStream_t st, const qg_dense_lindblad& L, double t, const void* x,
                        const AxpbyArgs& ax, const RkArgs& rk) {
  auto kern = dense_lindblad_kernel<YDT, EPI>;
  const int ranks = (L.d + DN_ROWS - 1) / DN_ROWS;
  const size_t smem = (size_t)dense_layout(DN_ROWS * ranks).total * sizeof(float2);
  static std::mutex mu;
  static size_t set_bytes[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
    return set_error(QG_ERR_CUDA, "no current CUDA device");
  {
    std::lock_guard<std::mutex> lock(mu);
    if (set_bytes[dev] < smem) {
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
          cudaSuccess)
        return set_error(QG_ERR_CUDA, "dense Lindblad kernel: shared memory opt-in failed");
      set_bytes[dev] = smem;
    }
  }
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ranks;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(ranks * ((L.d + DN_COLS - 1) / DN_COLS)));
  cfg.blockDim = dim3(DN_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, L, t, static_cast<const float2*>(x), ax, rk);
  return check_launch("dense_lindblad_kernel");
}

static int check_dense(const qg_dense_lindblad* L) {
  if (!L) return set_error(QG_ERR_ARG, "null generator");
  if (L->d < 1 || L->d > QG_DENSE_MAX_D)
    return set_error(QG_ERR_ARG, "dense bucket: need 1 <= d <= QG_DENSE_MAX_D (128)");
  if (L->n_groups < 1 || L->n_groups > QG_MAX_GROUPS)
    return set_error(QG_ERR_ARG, "n_groups out of range");
  if (L->n_cops < 0 || L->n_cops > QG_MAX_COPS)
    return set_error(QG_ERR_ARG, "collapse operator count out of range");
  if (!L->a || (L->n_cops > 0 && !L->c)) return set_error(QG_ERR_ARG, "null operator storage");
  if ((L->a_coef_code && (!L->a_coef_start || !L->a_coef_consts)) ||
      (L->c_coef_code && (!L->c_coef_start || !L->c_coef_consts)))
    return set_error(QG_ERR_ARG, "coefficient program tables incomplete");
  return QG_OK;
}

}  // namespace qg

using namespace qg;

extern "C" int qg_dense_lindblad_apply(const qg_dense_lindblad* L, double t, const void* x,
                                       void* y, double alpha_re, double alpha_im,
                                       double beta_re, double beta_im, void* stream) {
  int rc = check_dense(L);
  if (rc) return rc;
  if (!x || !y) return set_error(QG_ERR_ARG, "null vector");
  AxpbyArgs ax{y, alpha_re, alpha_im, beta_re, beta_im};
  RkArgs rk{};
  return launch_dense<QG_C64, EPI_AXPBY>((cudaStream_t)stream, *L, t, x, ax, rk);
}

extern "C" int qg_dense_lindblad_stage(const qg_dense_lindblad* L, const qg_rk_buffers* B,
                                       int stage, double t_prev, double dt, double atol,
                                       double rtol, void* stream) {
  int rc = check_dense(L);
  if (rc) return rc;
  RkArgs rk;
  const void* x = nullptr;
  rc = prepare_stage(B, QG_C64, (int64_t)L->d * L->d, stage, dt, atol, rtol, rk, x);
  if (rc) return rc;
  AxpbyArgs ax{};
  const double t = t_prev + VERN7_C_HOST[stage] * dt;
  cudaStream_t st = (cudaStream_t)stream;
  if (B->state_dtype == QG_C128) return launch_dense<QG_C128, EPI_RK>(st, *L, t, x, ax, rk);
  return launch_dense<QG_C64, EPI_RK>(st, *L, t, x, ax, rk);
}
