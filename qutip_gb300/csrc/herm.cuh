// The fused Vern7 epilogue of the forms that evaluate half of a Hermitian matrix: the values of
// an element are written in place and returned, so that the caller can write their conjugates
// to the mirrored element without reading its k_j again.
#pragma once
#include "stage.cuh"

namespace qg {

template <int DT, int YDT>
struct HermValues {
  typename elem<DT>::T k;  // k_s
  typename elem<DT>::T v;  // the next stage's input (stages that form one)
  typename elem<YDT>::T y; // y_front (stage 9)
  double term;             // WRMS term of the element (stage 9)
};

__device__ __forceinline__ bool herm_last(const RkArgs& rk) { return rk.stage == RK_STEP - 1; }
__device__ __forceinline__ bool herm_forms(const RkArgs& rk) {
  return rk.stage != RK_STEP - 1 && rk.stage != RK_EXTRA_STEP - 1;
}

// epilogue() of stage.cuh for EPI_RK, operation by operation, returning what it wrote.
template <int DT, int YDT>
__device__ __forceinline__ HermValues<DT, YDT> herm_epilogue(int row, cx<typename elem<DT>::R> acc,
                                                             const RkArgs& rk) {
  using ST = typename elem<DT>::T;
  using YT = typename elem<YDT>::T;
  using CT = typename elem<DT>::R;
  constexpr bool MIXED = DT != YDT;
  HermValues<DT, YDT> o;
  const int s = rk.stage;
  const size_t n64 = (size_t)rk.n;
  ST* kbuf = static_cast<ST*>(rk.k);
  st_cx(&o.k, acc);
  kbuf[(size_t)s * n64 + row] = o.k;
  if (!herm_last(rk)) {
    if (!herm_forms(rk)) return o;
    cx<CT> v;
    if constexpr (MIXED) v = ld_cx<CT>(static_cast<const ST*>(rk.y_prev_s) + row);
    else v = ld_cx<CT>(static_cast<const YT*>(rk.y_prev) + row);
#pragma unroll
    for (int j = 0; j < RK_EXTRA_STEP - 1; ++j) {
      if (j > s) break;
      if ((rk.nz_a >> j) & 1u)
        cx_axpy(v, fa<CT>(rk, j), j == s ? acc : ld_cx<CT>(kbuf + (size_t)j * n64 + row));
    }
    st_cx(&o.v, v);
    static_cast<ST*>(rk.ytmp_out)[row] = o.v;
    return o;
  }
  if constexpr (MIXED) {
    cx<CT> inc{0, 0};
    float erh = 0.f, erl = 0.f, eih = 0.f, eil = 0.f;
#pragma unroll
    for (int j = 0; j < RK_STEP; ++j) {
      const bool ub = (rk.nz_a >> j) & 1u, uq = (rk.nz_e >> j) & 1u;
      if (!ub && !uq) continue;
      const cx<CT> kj = (j == s) ? acc : ld_cx<CT>(kbuf + (size_t)j * n64 + row);
      if (ub) cx_axpy(inc, fa<CT>(rk, j), kj);
      if (uq) {  // the error estimate in float-float
        ff_acc(erh, erl, fe<CT>(rk, j), rk.fe_l[j], (float)kj.re);
        ff_acc(eih, eil, fe<CT>(rk, j), rk.fe_l[j], (float)kj.im);
      }
    }
    const double2 yp = static_cast<const double2*>(rk.y_prev)[row];
    o.y = make_double2(yp.x + (double)inc.re, yp.y + (double)inc.im);
    static_cast<float2*>(rk.y_front_s)[row] = make_float2((float)o.y.x, (float)o.y.y);
    const double er = (double)erh + (double)erl, ei = (double)eih + (double)eil;
    o.term = wrms_term(er * er + ei * ei, o.y.x * o.y.x + o.y.y * o.y.y, rk.atol, rk.rtol);
  } else {
    cx<CT> y = ld_cx<CT>(static_cast<const YT*>(rk.y_prev) + row), e{0, 0};
#pragma unroll
    for (int j = 0; j < RK_STEP; ++j) {
      const bool ub = (rk.nz_a >> j) & 1u, uq = (rk.nz_e >> j) & 1u;
      if (!ub && !uq) continue;
      const cx<CT> kj = (j == s) ? acc : ld_cx<CT>(kbuf + (size_t)j * n64 + row);
      if (ub) cx_axpy(y, fa<CT>(rk, j), kj);
      if (uq) cx_axpy(e, fe<CT>(rk, j), kj);
    }
    st_cx(&o.y, y);
    const cx<CT> ys = ld_cx<CT>(&o.y);
    const double mag2 = (double)ys.re * ys.re + (double)ys.im * ys.im;
    const double sc = rk.atol + rk.rtol * sqrt(mag2);
    o.term = ((double)e.re * e.re + (double)e.im * e.im) / (sc * sc);
  }
  static_cast<YT*>(rk.y_front)[row] = o.y;
  return o;
}

// y_front at the mirrored element (and its complex64 copy in the mixed form).
template <int DT, int YDT>
__device__ __forceinline__ void herm_mirror_front(size_t mrow, typename elem<YDT>::T y,
                                                  const RkArgs& rk) {
  static_cast<typename elem<YDT>::T*>(rk.y_front)[mrow] = y;
  if constexpr (DT != YDT)
    static_cast<float2*>(rk.y_front_s)[mrow] = make_float2((float)y.x, (float)y.y);
}

// Row stride of a shared-memory tile of elements T: odd multiples of 16 bytes apart for
// 16-byte elements, 34 for 8-byte ones, so that the transposed reads meet no bank twice.
template <typename T>
constexpr int HERM_PAD = sizeof(T) == 16 ? 33 : 34;

}  // namespace qg
