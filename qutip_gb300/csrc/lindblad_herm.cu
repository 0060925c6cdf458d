// The matrix-free Lindblad generator on a Hermitian rho: the elements (r, c) with r >= c of
//   A rho + rho A^dag + sum_i w_i C_i rho C_i^dag
// (lindblad_kernel in spmv.cu has the element's formula), each also written to its mirror
// (c, r) as its conjugate, with a real diagonal: the reference's assume_hermitian_state
// branch (qutip/core/cy/lindblad_matrix_form.pyx:171-188).
//
// Bound: load latency and instruction issue.  The d x d operators stay in L1 and rho in L2, so
// HBM carries the stage vectors only, and an element is some 30 dependent pairs of loads
// (operator entry, then the rho element it names).  So a warp evaluates four columns at once:
// 32 consecutive r of columns c .. c + 3, whose row-r entries are loaded once for the four and
// whose gathers are in flight together, and the block's row-c entries are staged in shared
// memory once per unit as (c' d, value) pairs, read as broadcasts.  A unit is 32 rows x 16
// columns for a block of 4 warps; its conjugates go out through shared memory, 16 consecutive
// elements at a time, and the mirrored elements' k_j are not read again.
// Measured: the L = 10 Ising chain's solve, mixed form, 92 -> 74 ms (31 us a stage, the full
// form 51; with one element per thread, 32 x 32 tiles and the mirrors through an epilogue of
// their own, 43); complex128 stages 313 us against 409 in the full form.
#include <mutex>

#include "capi_internal.h"
#include "common.cuh"
#include "herm.cuh"
#include "lindblad_herm.cuh"
#include "rows.cuh"
#include "stage.cuh"

namespace qg {

constexpr int LH_BLOCK = 128;
constexpr int LH_Q = 4;                        // columns of a warp
constexpr int LH_COLS = LH_Q * LH_BLOCK / 32;  // columns of a unit
// row-c entries kept in shared memory: operators up to this many entries a row in all
constexpr int LH_KEEP = 48;

template <int DT>
struct LhBounds {
  static constexpr int MIN_BLOCKS = DT == QG_C64 ? 8 : 4;
};

template <int DT, int YDT, int EPI>
__global__ void __launch_bounds__(LH_BLOCK, LhBounds<DT>::MIN_BLOCKS)
    lindblad_herm_kernel(const __grid_constant__ qg_lindblad L, double t,
                         const typename elem<DT>::T* __restrict__ x, AxpbyArgs ax,
                         const __grid_constant__ RkArgs rk, int wa, int wtot) {
  using ST = typename elem<DT>::T;
  using YT = typename elem<YDT>::T;
  using R = typename elem<DT>::R;
  constexpr int Q = LH_Q;
  extern __shared__ __align__(16) unsigned char lh_smem[];  // row-c entries: values, offsets
  __shared__ cx<R> ca[QG_MAX_GROUPS];
  __shared__ R wc[QG_MAX_COPS];
  __shared__ double red[LH_BLOCK / 32];
  constexpr int PAD = HERM_PAD<ST>, YPAD = HERM_PAD<YT>;
  __shared__ __align__(16) ST tk[LH_COLS * PAD];
  __shared__ __align__(16) YT ty[LH_COLS * YPAD];  // the stage input as ST, or y_front
  ST* tv = reinterpret_cast<ST*>(ty);
  const bool keep = wtot <= LH_KEEP;
  ST* sv = reinterpret_cast<ST*>(lh_smem);
  int* so = reinterpret_cast<int*>(lh_smem + (keep ? (size_t)wtot * LH_COLS * sizeof(ST) : 0));
  const int G = L.n_groups, ND = L.n_diag_cops, NE = L.n_cops - L.n_diag_cops;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const cplx* table = stage_coefs<EPI>(rk);
  if (tid < G) {
    const cplx k = table ? table[tid]
                         : prog_coef(L.a_coef_code, L.a_coef_start, L.a_coef_consts, tid, t);
    ca[tid] = cx<R>{(R)k.re, (R)k.im};
  }
  for (int i = tid; i < L.n_cops; i += LH_BLOCK) {
    const cplx f = table ? table[G + i]
                         : prog_coef(L.c_coef_code, L.c_coef_start, L.c_coef_consts, i, t);
    wc[i] = (R)(f.re * f.re + f.im * f.im);
  }
  const int d = (int)L.d;
  const ST* __restrict__ dconst = static_cast<const ST*>(L.d_const);
  const ST* __restrict__ adiag = static_cast<const ST*>(L.a_diag);
  const int* __restrict__ acol = L.a_col;
  const ST* __restrict__ aval = static_cast<const ST*>(L.a_val);
  const ST* __restrict__ cdiag = static_cast<const ST*>(L.c_diag);
  const int* __restrict__ ccol = L.c_col;
  const ST* __restrict__ cval = static_cast<const ST*>(L.c_val);
  const int dmask = L.a_diag_const, nd0 = L.n_const_diag;
  int nw1 = 0;  // leading general collapse operators of width 1
  while (nw1 < NE && L.c_width[nw1] == 1) ++nw1;
  double err_acc = 0.0;
  const int nt = (d + 31) / 32;
  const int units = nt * (nt + 1);  // two per 32 x 32 block on or below the diagonal
  int tj = 0, tbase = 0;
  for (int u = blockIdx.x; u < units; u += gridDim.x) {
    const int tau = u >> 1;
    while (tau >= tbase + (nt - tj)) {
      tbase += nt - tj;
      ++tj;
    }
    const int r0 = (tj + (tau - tbase)) * 32, c0 = tj * 32 + (u & 1) * LH_COLS;
    if (c0 >= d) continue;  // uniform: the last block's second half of a ragged d
    __syncthreads();        // the previous unit's entries and tiles are read (and ca, wc written)
    if (keep) {
      for (int e = tid; e < wtot * LH_COLS; e += LH_BLOCK) {
        const int j = e / LH_COLS, c = min(c0 + (e % LH_COLS), d - 1);
        const bool a = j < wa;
        const int i = (a ? j : j - wa) * d + c;
        sv[e] = __ldg((a ? aval : cval) + i);
        so[e] = __ldg((a ? acol : ccol) + i) * d;
      }
      __syncthreads();
    }
    // row-c entry j (those of A first, then the collapse operators') of column c0 + cl
    auto centry = [&](int j, int cl, ST& v, int& o) {
      if (keep) {
        v = sv[j * LH_COLS + cl];
        o = so[j * LH_COLS + cl];
      } else {
        const bool a = j < wa;
        const int i = (a ? j : j - wa) * d + min(c0 + cl, d - 1);
        v = __ldg((a ? aval : cval) + i);
        o = __ldg((a ? acol : ccol) + i) * d;
      }
    };
    const int r = min(r0 + lane, d - 1);  // lanes past d repeat the last row and write nothing
    const int q0 = w * Q;
    cx<R> acc[Q];
    int cd[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) cd[q] = min(c0 + q0 + q, d - 1) * d;
    // diagonal factor: the precomputed constant part plus the time-dependent rest
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int c = min(c0 + q0 + q, d - 1);
      R dr = 0, di = 0;
      if (dconst) {
        const ST p = __ldg(dconst + (r + cd[q]));
        dr = p.x;
        di = p.y;
      }
      for (int g = 0; g < G; ++g) {
        if ((dmask >> g) & 1) continue;
        const cx<R> k = ca[g];
        const ST p = __ldg(adiag + g * d + r), s = __ldg(adiag + g * d + c);
        dr += k.re * (p.x + s.x) - k.im * (p.y - s.y);  // k p + conj(k s)
        di += k.re * (p.y - s.y) + k.im * (p.x + s.x);
      }
      for (int i = nd0; i < ND; ++i) {
        const R f = wc[i];
        const ST p = __ldg(cdiag + i * d + r), s = __ldg(cdiag + i * d + c);
        dr += f * (p.x * s.x + p.y * s.y);  // w p conj(s)
        di += f * (p.y * s.x - p.x * s.y);
      }
      const ST xe = ld_gather(x + (r + cd[q]));
      acc[q] = cx<R>{dr * xe.x - di * xe.y, dr * xe.y + di * xe.x};
    }
    // off-diagonal A: A rho (row r against column c) and rho A^dag (row c against row r)
    int j = 0;
    for (int g = 0; g < G; ++g) {
      const int W = L.a_width[g];
      if (W == 0) continue;
      R lr[Q], li[Q], qr[Q], qi[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) lr[q] = li[q] = qr[q] = qi[q] = 0;
      for (int e = j + W; j < e; ++j) {
        const int cr = __ldg(acol + j * d + r);
        const ST vr = __ldg(aval + j * d + r);
        ST x1[Q], x2[Q], vc[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          int o;
          centry(j, q0 + q, vc[q], o);
          x1[q] = ld_gather(x + (cr + cd[q]));
          x2[q] = ld_gather(x + (r + o));
        }
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          cmac_any(lr[q], li[q], vr, x1[q]);
          cmac_conj(qr[q], qi[q], vc[q], x2[q]);
        }
      }
      const cx<R> k = ca[g];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        acc[q].re += k.re * lr[q] - k.im * li[q] + k.re * qr[q] + k.im * qi[q];
        acc[q].im += k.re * li[q] + k.im * lr[q] + k.re * qi[q] - k.im * qr[q];
      }
    }
    // general collapse operators: C rho C^dag.  The leading width-1 operators (s-, a, ...)
    // run branch-free in complex64 (a padding entry has value 0 and a valid column); the
    // FP64-bound complex128 form skips padding instead.
    int base = 0, i = 0;
#pragma unroll 2
    for (; i < nw1; ++i, base += d) {
      const R f = wc[ND + i];
      const ST v = __ldg(cval + base + r);
      const int cr = __ldg(ccol + base + r);
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        ST b;
        int o;
        centry(wa + i, q0 + q, b, o);
        if constexpr (DT == QG_C128) {
          if ((b.x == (R)0 && b.y == (R)0) || (v.x == (R)0 && v.y == (R)0)) continue;
        }
        const ST xv = ld_gather(x + (cr + o));
        const R pr = f * (v.x * b.x + v.y * b.y), pi = f * (v.y * b.x - v.x * b.y);  // f v conj(b)
        acc[q].re += pr * xv.x - pi * xv.y;
        acc[q].im += pr * xv.y + pi * xv.x;
      }
    }
    int cj = wa + nw1;
    for (; i < NE; ++i) {
      const int W = L.c_width[i];
      const R f = wc[ND + i];
      for (int q = 0; q < Q; ++q) {
        R sr2 = 0, si2 = 0;
        for (int m = 0; m < W; ++m) {
          ST b;
          int o;
          centry(cj + m, q0 + q, b, o);
          if (b.x == (R)0 && b.y == (R)0) continue;  // warp-uniform: padding of row c
          R ir = 0, ii = 0;
          for (int p = 0; p < W; ++p) {
            const int ep = base + p * d + r;
            const ST v = __ldg(cval + ep);
            if (v.x != (R)0 || v.y != (R)0)
              cmac_any(ir, ii, v, ld_gather(x + (__ldg(ccol + ep) + o)));
          }
          sr2 += b.x * ir + b.y * ii;  // conj(b) * inner
          si2 += b.x * ii - b.y * ir;
        }
#pragma unroll
        for (int qq = 0; qq < Q; ++qq)
          if (qq == q) {
            acc[qq].re += f * sr2;
            acc[qq].im += f * si2;
          }
      }
      base += W * d;
      cj += W;
    }
    // in place, and the conjugates into the tiles (through which a thread's four values also
    // reach the one copy of the epilogue's code)
#pragma unroll
    for (int q = 0; q < Q; ++q) tk[(q0 + q) * PAD + lane] = ST{acc[q].re, acc[q].im};
#pragma unroll 1
    for (int q = 0; q < Q; ++q) {
      const int cl = q0 + q, c = c0 + cl;
      const bool valid = r0 + lane < d && c < d && r >= c;
      if (valid) {
        const ST a = tk[cl * PAD + lane];
        const cx<R> v{a.x, r == c ? (R)0 : a.y};  // A + A^dag: real diagonal
        const int row = r + c * d;
        if constexpr (EPI == EPI_AXPBY) {
          epilogue<DT, YDT, EPI>(row, v, ax, rk, err_acc);
          tk[cl * PAD + lane] = ST{v.re, -v.im};
        } else {
          const HermValues<DT, YDT> o = herm_epilogue<DT, YDT>(row, v, rk);
          tk[cl * PAD + lane] = ST{o.k.x, -o.k.y};
          if (herm_last(rk)) {
            ty[cl * YPAD + lane] = YT{o.y.x, -o.y.y};
            err_acc += r == c ? o.term : 2.0 * o.term;  // the mirrored element has the same term
          } else if (herm_forms(rk)) {
            tv[cl * PAD + lane] = ST{o.v.x, -o.v.y};
          }
        }
      }
    }
    __syncthreads();
    const int mc = tid % LH_COLS;
#pragma unroll
    for (int p = 0; p < 32 * LH_COLS / LH_BLOCK; ++p) {
      const int mr = tid / LH_COLS + p * (LH_BLOCK / LH_COLS);
      const int cc = c0 + mc, rr = r0 + mr;
      if (rr < d && cc < d && rr > cc) {
        const size_t mrow = (size_t)cc + (size_t)rr * d;
        const ST kv = tk[mc * PAD + mr];
        if constexpr (EPI == EPI_AXPBY) {
          epilogue<DT, YDT, EPI>((int)mrow, cx<R>{kv.x, kv.y}, ax, rk, err_acc);
        } else {
          static_cast<ST*>(rk.k)[(size_t)rk.stage * (size_t)rk.n + mrow] = kv;
          if (herm_last(rk))
            herm_mirror_front<DT, YDT>(mrow, ty[mc * YPAD + mr], rk);
          else if (herm_forms(rk))
            static_cast<ST*>(rk.ytmp_out)[mrow] = tv[mc * PAD + mr];
        }
      }
    }
  }
  if constexpr (EPI == EPI_RK) {
    if (rk.stage == RK_STEP - 1) finish_error<LH_BLOCK>(rk, err_acc, red);
  }
}

template <int DT, int YDT, int EPI>
int launch_lindblad_herm(cudaStream_t st, const qg_lindblad& L, double t, const void* x,
                         const AxpbyArgs& ax, const RkArgs& rk) {
  using ST = typename elem<DT>::T;
  auto kern = lindblad_herm_kernel<DT, YDT, EPI>;
  int wa = 0, wtot = 0;
  for (int g = 0; g < L.n_groups; ++g) wa += L.a_width[g];
  wtot = wa;
  for (int i = 0; i < L.n_cops - L.n_diag_cops; ++i) wtot += L.c_width[i];
  const size_t smem = wtot <= LH_KEEP ? (size_t)wtot * LH_COLS * (sizeof(ST) + 4) : 0;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, LH_BLOCK, smem) !=
          cudaSuccess ||
      per_sm <= 0)
    return set_error(QG_ERR_CUDA, "occupancy query failed");
  const int64_t nt = (L.d + 31) / 32;
  int64_t grid = (int64_t)sm_count() * per_sm;
  if (grid > nt * (nt + 1)) grid = nt * (nt + 1);
  if (grid > qg_scratch_doubles()) grid = qg_scratch_doubles();
  kern<<<(int)grid, LH_BLOCK, smem, st>>>(L, t, (const ST*)x, ax, rk, wa, wtot);
  return check_launch("lindblad_herm_kernel");
}

#define QG_LH(DT, YDT, EPI)                                                                   \
  template int launch_lindblad_herm<DT, YDT, EPI>(cudaStream_t, const qg_lindblad&, double,   \
                                                  const void*, const AxpbyArgs&, const RkArgs&);
QG_LH(QG_C128, QG_C128, EPI_AXPBY)
QG_LH(QG_C64, QG_C64, EPI_AXPBY)
QG_LH(QG_C128, QG_C128, EPI_RK)
QG_LH(QG_C64, QG_C128, EPI_RK)
QG_LH(QG_C64, QG_C64, EPI_RK)
#undef QG_LH

}  // namespace qg
