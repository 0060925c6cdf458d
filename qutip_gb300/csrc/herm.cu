// Vern7 stages of a Liouvillian on a Hermitian density matrix, evaluating half of it
// (qg_vern7_stage_herm), and the test that this applies (qg_hermitian_check).
//
// A Lindblad generator with real coefficients maps a Hermitian rho to a Hermitian matrix,
// so the element (c, r) of every stage vector is the conjugate of (r, c): the rows of the
// superoperator with r below c need not be evaluated.  Bound: the dictionary kernel of
// spmv.cu is bound by FP64 issue in complex128 (85 % of the pipe at a million rows) and by
// the gathers of x and the table lookups in complex64; both halve, as do the reads of the
// stage combination.
//
// Work split: vec(rho) is column-major and d a multiple of 32, so a 32-row slice of the
// dictionary layout is 32 consecutive r of one column c.  A block of 8 warps takes 32 rows
// x 8 columns on or below the diagonal: warp w evaluates column c0 + w, the values go out in
// place, and the block writes their conjugates to the mirrored 8 x 32 elements through
// shared memory, eight consecutive c (128 bytes in complex128) at a time.  Units of 8
// columns rather than 32 leave no SM with a fourth more work than the others (2112 units
// at d = 1024).  32 x 32 blocks on the diagonal are evaluated whole and not mirrored.
//
// Measured, whole solves of the L = 10 Ising chain (1,048,576 rows, 1646 right-hand sides):
// complex128 279 -> 168 ms, mixed 95 -> 66 ms (158 and 58 with the driver's loop and its
// coefficient table).  It is taken above 512 rows per SM, where the stages go out one by
// one; from 256 rows per SM up to there the fused step kernel (step.cu) evaluates the same
// units.
#include <mutex>

#include "capi_internal.h"
#include "common.cuh"
#include "herm.cuh"
#include "rows.cuh"
#include "stage.cuh"

namespace qg {

constexpr int HERM_BLOCK = 256;
constexpr int HERM_COLS = HERM_BLOCK / 32;

// ------------------------------------------------------------------ check ----
// Entry j of row `row` in group g: true and its code when j is below the slice's width.
template <int CB>
__device__ __forceinline__ int code_at(const qg_csr_groups& A, const unsigned char* codes, int g,
                                       int row, int j) {
  const int sl = row >> 5;
  const size_t i = (size_t)__ldg(A.row_ptr + g * (A.n_tiles + 1) + sl) + 128 * (size_t)(j >> 2) +
                   4 * (row & 31) + (j & 3);
  if (CB == 1) return codes[i];
  return reinterpret_cast<const unsigned short*>(codes)[i];
}

__device__ __forceinline__ double max_part(double2 v) { return fmax(fabs(v.x), fabs(v.y)); }
__device__ __forceinline__ double max_part(float2 v) {
  return fmax(fabs((double)v.x), fabs((double)v.y));
}

// Sets *flag when the operator does not commute with the Hermitian conjugate (an entry of
// row (r, c) without its conjugate at the mirrored place of row (c, r)), or rho is not
// Hermitian.  Entries are compared to the rounding of their row's largest value (the sums
// of a Liouvillian's terms round differently at mirrored places), rho element by element;
// a NaN or an infinity, in either, counts as not Hermitian.
template <int DT, int XDT, int CB, bool RI>
__global__ void __launch_bounds__(HERM_BLOCK)
    hermitian_check_kernel(qg_csr_groups A, int d, const typename elem<XDT>::T* x, int* flag) {
  using ST = typename elem<DT>::T;
  const int n = d * d;
  const ST* __restrict__ tval = static_cast<const ST*>(A.val);
  const unsigned char* codes = reinterpret_cast<const unsigned char*>(A.col);
  const double rel = DT == QG_C128 ? 0x1p-46 : 0x1p-22;
  const double relx = XDT == QG_C128 ? 0x1p-48 : 0x1p-21;
  for (int row = blockIdx.x * HERM_BLOCK + threadIdx.x; row < n;
       row += gridDim.x * HERM_BLOCK) {
    if (*(volatile int*)flag) return;
    const int c = row / d, r = row - c * d;
    const int mrow = c + r * d;
    bool ok = true;
    {
      const auto p = x[row], q = x[mrow];
      const double tol = relx * max_part(p);
      ok = isfinite(tol) && fabs((double)p.x - (double)q.x) <= tol &&
           fabs((double)p.y + (double)q.y) <= tol;
    }
    for (int g = 0; g < A.n_groups && ok; ++g) {
      const int t0 = __ldg(A.dict_start + g), tn = __ldg(A.dict_start + g + 1) - t0;
      const int w = __ldg(A.tile_row + (row >> 5) * A.n_groups + g);
      const int mw = __ldg(A.tile_row + (mrow >> 5) * A.n_groups + g);
      double top = 0.0;
      for (int j = 0; j < w; ++j) {
        const int k = code_at<CB>(A, codes, g, row, j);
        if (k <= 0 || k >= tn) continue;
        const ST v = tval[t0 + k];
        top = fmax(top, max_part(v));
        // a NaN beside a zero does not show in the maximum, an infinity leaves no tolerance
        if (!isfinite(v.x) || !isfinite(v.y)) ok = false;
      }
      const double tol = rel * top;
      for (int j = 0; j < w && ok; ++j) {
        const int k = code_at<CB>(A, codes, g, row, j);
        if (k <= 0 || k >= tn) continue;
        const ST v = tval[t0 + k];
        if (max_part(v) <= tol) continue;
        const int oc = __ldg(A.dict_off + t0 + k);
        const int col = row + (RI ? oc >> 1 : oc);
        if (col < 0 || col >= n) {
          ok = false;
          break;
        }
        const int cc = col / d, cr = col - cc * d;
        const int mo = cc + cr * d - mrow;  // offset of the mirrored entry
        const int want = RI ? (mo << 1) | (oc & 1) : mo;
        bool found = false;
        for (int i = 0; i < mw && !found; ++i) {
          const int mk = code_at<CB>(A, codes, g, mrow, i);
          if (mk <= 0 || mk >= tn || __ldg(A.dict_off + t0 + mk) != want) continue;
          const ST m = tval[t0 + mk];
          if (RI) {  // one real factor a in .y: the imaginary part changes sign
            const double a = v.y, b = m.y;
            found = fabs((oc & 1) ? a + b : a - b) <= tol;
          } else {
            found = fabs((double)v.x - (double)m.x) <= tol &&
                    fabs((double)v.y + (double)m.y) <= tol;
          }
        }
        ok = found;
      }
    }
    if (!ok) *flag = 1;
  }
}

// ------------------------------------------------------------------ stage ----
template <int DT>
struct HermBounds {
  static constexpr int MIN_BLOCKS = DT == QG_C64 ? 5 : 4;
};
template <int DT, int YDT, int CB, bool RI>
__global__ void __launch_bounds__(HERM_BLOCK, HermBounds<DT>::MIN_BLOCKS)
    vern7_herm_kernel(qg_csr_groups A, int d, double t, const typename elem<DT>::T* __restrict__ x,
                      const __grid_constant__ RkArgs rk) {
  using ST = typename elem<DT>::T;
  using YT = typename elem<YDT>::T;
  using CT = typename elem<DT>::R;
  using C4 = typename Codes4<CB>::T;
  extern __shared__ __align__(16) unsigned char dict_smem[];
  __shared__ cx<CT> coef[QG_MAX_GROUPS];
  __shared__ int ccls[QG_MAX_GROUPS];
  __shared__ int tstart[QG_MAX_GROUPS + 1];
  __shared__ double red[HERM_BLOCK / 32];
  // mirrored values of two units: k_s and the next stage input (or y_front, one unit)
  constexpr int PAD = HERM_PAD<ST>, YPAD = HERM_PAD<YT>;
  constexpr int TILE = HERM_COLS * PAD;
  __shared__ __align__(16) ST tiles[4 * TILE];
  static_assert(TILE * sizeof(ST) + HERM_COLS * YPAD * sizeof(YT) <= 4 * TILE * sizeof(ST),
                "the last stage's tiles fit");
  const int D = A.lanes, G = A.n_groups, S = A.n_tiles;
  ST* tval = reinterpret_cast<ST*>(dict_smem);
  int* toff = reinterpret_cast<int*>(dict_smem + (size_t)D * sizeof(ST));
  if (threadIdx.x < G) {
    const cplx k = rk.coefs ? rk.coefs[threadIdx.x] : group_coef(A, threadIdx.x, t);
    coef[threadIdx.x] = cx<CT>{(CT)k.re, (CT)k.im};
    ccls[threadIdx.x] = coef_class(coef[threadIdx.x]);
  }
  for (int i = threadIdx.x; i < D; i += HERM_BLOCK) {
    tval[i] = __ldg(static_cast<const ST*>(A.val) + i);
    toff[i] = __ldg(A.dict_off + i);
  }
  if (threadIdx.x <= (unsigned)G) tstart[threadIdx.x] = __ldg(A.dict_start + threadIdx.x);
  __syncthreads();
  const int lane = threadIdx.x & 31, w8 = threadIdx.x >> 5;
  const int nt = d >> 5;
  const int units = 2 * nt * (nt + 1);  // four per 32 x 32 block on or below the diagonal
  const int last_col = d * d - 1;
  const int s = rk.stage;
  const bool last = herm_last(rk), forms = herm_forms(rk);
  const size_t n64 = (size_t)rk.n;
  ST* kbuf = static_cast<ST*>(rk.k);
  const unsigned char* __restrict__ codes = reinterpret_cast<const unsigned char*>(A.col);
  double err_acc = 0.0;
  int tj = 0, tbase = 0;  // column block of the unit and the index of its first row block
  int buf = 0;
  for (int u = blockIdx.x; u < units; u += gridDim.x, buf ^= 1) {
    const int tau = u >> 2;
    while (tau >= tbase + (nt - tj)) {
      tbase += nt - tj;
      ++tj;
    }
    const int ti = tj + (tau - tbase);
    const int c0 = tj * 32 + (u & 3) * HERM_COLS;
    const int c = c0 + w8;
    const int sl = c * nt + ti;
    const int row = sl * 32 + lane;
    const bool mirrored = ti != tj;
    cx<CT> acc{0, 0};
    for (int g = 0; g < G; ++g) {  // as spmv_dict_kernel forms a row
      const int w = __ldg(A.tile_row + sl * G + g);
      const int wq = w >> 2, wr = w & 3;
      const int t0 = tstart[g], tn = tstart[g + 1] - t0;
      const C4* __restrict__ cp =
          reinterpret_cast<const C4*>(codes + (size_t)CB * __ldg(A.row_ptr + g * (S + 1) + sl)) +
          lane;
      const bool direct = sizeof(CT) == 8 && ccls[g] == 0;
      CT ar = direct ? acc.re : (CT)0, ai = direct ? acc.im : (CT)0;
#pragma unroll 2
      for (int q = 0; q < wq; ++q) {
        const C4 c4 = ld_stream(cp + 32 * q);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          int k = Codes4<CB>::at(c4, e);
          if constexpr (RI) {
            if (!__any_sync(0xffffffffu, k != 0)) continue;
          }
          k = t0 + (k < tn ? k : 0);
          dict_mac<RI, true>(tval, toff, x, k, row, last_col, ar, ai);
        }
      }
      if (wr) {
        const C4 c4 = ld_stream(cp + 32 * wq);
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          if (e < wr) {
            int k = Codes4<CB>::at(c4, e);
            if constexpr (RI) {
              if (!__any_sync(0xffffffffu, k != 0)) continue;
            }
            k = t0 + (k < tn ? k : 0);
            dict_mac<RI, true>(tval, toff, x, k, row, last_col, ar, ai);
          }
        }
      }
      if (direct) acc = cx<CT>{ar, ai};
      else coef_mac(acc, coef[g], ar, ai);
    }
    const HermValues<DT, YDT> o = herm_epilogue<DT, YDT>(row, acc, rk);
    const int at = w8 * PAD + lane;
    const int mc = threadIdx.x & (HERM_COLS - 1), mr = threadIdx.x / HERM_COLS;
    const size_t mrow = (size_t)(c0 + mc) + (size_t)(ti * 32 + mr) * d;
    if (!last) {
      ST* tk = tiles + buf * 2 * TILE;
      ST* tv = tk + TILE;
      tk[at] = ST{o.k.x, -o.k.y};
      if (forms) tv[at] = ST{o.v.x, -o.v.y};
      __syncthreads();
      if (mirrored) {
        kbuf[(size_t)s * n64 + mrow] = tk[mc * PAD + mr];
        if (forms) static_cast<ST*>(rk.ytmp_out)[mrow] = tv[mc * PAD + mr];
      }
    } else {
      ST* tk = tiles;
      YT* ty = reinterpret_cast<YT*>(tiles + TILE);
      err_acc += mirrored ? 2.0 * o.term : o.term;  // the mirrored element has the same term
      tk[at] = ST{o.k.x, -o.k.y};
      ty[w8 * YPAD + lane] = YT{o.y.x, -o.y.y};
      __syncthreads();
      if (mirrored) {
        kbuf[(size_t)s * n64 + mrow] = tk[mc * PAD + mr];
        herm_mirror_front<DT, YDT>(mrow, ty[mc * YPAD + mr], rk);
      }
      __syncthreads();  // one set of tiles: read before the next unit writes them
    }
  }
  if (last) finish_error<HERM_BLOCK>(rk, err_acc, red);
}

template <int DT, int YDT, int CB>
static int launch_herm(cudaStream_t st, const qg_csr_groups& A, int d, double t, const void* x,
                       const RkArgs& rk) {
  using ST = typename elem<DT>::T;
  auto kern = vern7_herm_kernel<DT, YDT, CB, DT == QG_C128>;
  const size_t smem = ((size_t)A.lanes * (sizeof(ST) + sizeof(int)) + 15) & ~(size_t)15;
  static OccCache cache;  // one per instantiation
  const int per_sm = launch_occupancy((const void*)kern, HERM_BLOCK, smem, cache);
  if (per_sm <= 0) return set_error(QG_ERR_ARG, "dictionary does not fit in shared memory");
  const int64_t nt = d / 32;
  int64_t grid = (int64_t)sm_count() * per_sm;
  if (grid > 2 * nt * (nt + 1)) grid = 2 * nt * (nt + 1);
  if (grid > qg_scratch_doubles()) grid = qg_scratch_doubles();
  kern<<<(int)grid, HERM_BLOCK, smem, st>>>(A, d, t, (const ST*)x, rk);
  return check_launch("vern7_herm_kernel");
}

template <int DT, int XDT, int CB>
static int launch_check(cudaStream_t st, const qg_csr_groups& A, int d, const void* x, int* flag) {
  const int64_t blocks = ((int64_t)d * d + HERM_BLOCK - 1) / HERM_BLOCK;
  const int64_t cap = (int64_t)sm_count() * 8;
  hermitian_check_kernel<DT, XDT, CB, DT == QG_C128>
      <<<(int)(blocks < cap ? blocks : cap), HERM_BLOCK, 0, st>>>(
          A, d, static_cast<const typename elem<XDT>::T*>(x), flag);
  return check_launch("hermitian_check_kernel");
}

// The layouts and shapes the half form takes: dictionary codes (split in complex128), a
// Hilbert dimension that is a multiple of 32.
int check_herm(const qg_csr_groups* A, int64_t d) {
  int rc = check_groups(A);
  if (rc) return rc;
  if (A->layout != (A->dtype == QG_C128 ? QG_LAYOUT_SLICED_DICT_RI : QG_LAYOUT_SLICED_DICT))
    return set_error(QG_ERR_UNSUPPORTED, "the Hermitian form needs the dictionary layout");
  if (d < 32 || d % 32 != 0 || d * d != A->n_rows || A->n_rows != A->n_cols ||
      A->n_rows >= INT32_MAX)
    return set_error(QG_ERR_ARG, "the Hermitian form needs d a multiple of 32 and d*d rows");
  return QG_OK;
}

}  // namespace qg

using namespace qg;

extern "C" int qg_hermitian_check(const qg_csr_groups* A, int64_t d, const void* rho, int rho_dtype,
                                  int* flag, void* stream) {
  int rc = check_herm(A, d);
  if (rc) return rc;
  if (!rho || !flag) return set_error(QG_ERR_ARG, "null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  const bool one = A->tile_nnz == 1;
  if (rho_dtype == QG_C128 && A->dtype == QG_C128)
    return one ? launch_check<QG_C128, QG_C128, 1>(st, *A, (int)d, rho, flag)
               : launch_check<QG_C128, QG_C128, 2>(st, *A, (int)d, rho, flag);
  if (rho_dtype == QG_C128 && A->dtype == QG_C64)
    return one ? launch_check<QG_C64, QG_C128, 1>(st, *A, (int)d, rho, flag)
               : launch_check<QG_C64, QG_C128, 2>(st, *A, (int)d, rho, flag);
  if (rho_dtype == QG_C64 && A->dtype == QG_C64)
    return one ? launch_check<QG_C64, QG_C64, 1>(st, *A, (int)d, rho, flag)
               : launch_check<QG_C64, QG_C64, 2>(st, *A, (int)d, rho, flag);
  return set_error(QG_ERR_UNSUPPORTED, "dtype");
}

int qg::stage_herm(const qg_csr_groups* A, int64_t d, const qg_rk_buffers* B, int stage,
                   double t_prev, double dt, double atol, double rtol, const void* coefs,
                   void* stream) {
  int rc = check_herm(A, d);
  if (rc) return rc;
  RkArgs rk;
  const void* x = nullptr;
  rc = prepare_stage(B, A->dtype, A->n_rows, stage, dt, atol, rtol, rk, x);
  if (rc) return rc;
  rk.coefs = static_cast<const cplx*>(coefs);
  cudaStream_t st = (cudaStream_t)stream;
  const double t = t_prev + VERN7_C_HOST[stage] * dt;
  const bool one = A->tile_nnz == 1;
  if (B->state_dtype == QG_C128 && B->stage_dtype == QG_C128)
    return one ? launch_herm<QG_C128, QG_C128, 1>(st, *A, (int)d, t, x, rk)
               : launch_herm<QG_C128, QG_C128, 2>(st, *A, (int)d, t, x, rk);
  if (B->state_dtype == QG_C128)
    return one ? launch_herm<QG_C64, QG_C128, 1>(st, *A, (int)d, t, x, rk)
               : launch_herm<QG_C64, QG_C128, 2>(st, *A, (int)d, t, x, rk);
  return one ? launch_herm<QG_C64, QG_C64, 1>(st, *A, (int)d, t, x, rk)
             : launch_herm<QG_C64, QG_C64, 2>(st, *A, (int)d, t, x, rk);
}

extern "C" int qg_vern7_stage_herm(const qg_csr_groups* A, int64_t d, const qg_rk_buffers* B,
                                   int stage, double t_prev, double dt, double atol, double rtol,
                                   void* stream) {
  return stage_herm(A, d, B, stage, t_prev, dt, atol, rtol, nullptr, stream);
}
