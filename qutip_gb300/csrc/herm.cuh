// The fused Vern7 epilogue of the forms that evaluate half of a Hermitian matrix: the values of
// an element are written in place and returned, so that the caller can write their conjugates
// to the mirrored element without reading its k_j again.
#pragma once
#include "stage.cuh"

namespace qg {

// A weighted sum of stages on top of a start value, f + fl the weight.
template <typename CT>
struct PlainSum {
  cx<CT> v;
  __device__ __forceinline__ void add(CT f, float, cx<CT> k) { cx_axpy(v, f, k); }
  __device__ __forceinline__ cx<CT> value() const { return v; }
  __device__ __forceinline__ double2 wide() const { return make_double2(v.re, v.im); }
};
// The half form's: in complex64 the low parts of the weights have a sum of their own.  Vern7's
// weights are large and of both signs; rounded to floats they leave an error that the full
// form averages with the other roundings of an element and its mirror, which are the same ones
// here.  Measured against complex128, mixed form, largest error of the outputs, means of 16
// random Ising chains each of L = 6, 7, 8 and of 8 of L = 9: full form 1.8, 1.5, 1.6 and 1.7e-7,
// half form with plain sums 1.9, 1.7, 1.6 and 2.0e-7, with this 1.3, 1.0, 0.9 and 0.7e-7 (0.7e-7
// of each is the rounding of the operator's entries); the L = 10 solve 57.7 -> 58.8 ms.  Sums
// in pairs throughout (two-sum) gain another fifth and cost 61.2 ms.
template <typename CT>
struct HermSum : PlainSum<CT> {};
template <>
struct HermSum<float> {
  cx<float> v, low{0.f, 0.f};
  __device__ __forceinline__ HermSum(cx<float> start) : v(start) {}
  __device__ __forceinline__ void add(float f, float fl, cx<float> k) {
    cx_axpy(v, f, k);
    cx_axpy(low, fl, k);
  }
  __device__ __forceinline__ cx<float> value() const { return cx_add(v, low); }
  __device__ __forceinline__ double2 wide() const {
    return make_double2((double)v.re + (double)low.re, (double)v.im + (double)low.im);
  }
};

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

// epilogue() of stage.cuh for EPI_RK, operation by operation but for the complex64 sums,
// returning what it wrote.
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
    cx<CT> base;
    if constexpr (MIXED) base = ld_cx<CT>(static_cast<const ST*>(rk.y_prev_s) + row);
    else base = ld_cx<CT>(static_cast<const YT*>(rk.y_prev) + row);
    HermSum<CT> v{base};
#pragma unroll
    for (int j = 0; j < RK_EXTRA_STEP - 1; ++j) {
      if (j > s) break;
      if ((rk.nz_a >> j) & 1u)
        v.add(fa<CT>(rk, j), rk.fa_l[j], j == s ? acc : ld_cx<CT>(kbuf + (size_t)j * n64 + row));
    }
    st_cx(&o.v, v.value());
    static_cast<ST*>(rk.ytmp_out)[row] = o.v;
    return o;
  }
  if constexpr (MIXED) {
    HermSum<CT> inc{cx<CT>{0, 0}};
    float erh = 0.f, erl = 0.f, eih = 0.f, eil = 0.f;
#pragma unroll
    for (int j = 0; j < RK_STEP; ++j) {
      const bool ub = (rk.nz_a >> j) & 1u, uq = (rk.nz_e >> j) & 1u;
      if (!ub && !uq) continue;
      const cx<CT> kj = (j == s) ? acc : ld_cx<CT>(kbuf + (size_t)j * n64 + row);
      if (ub) inc.add(fa<CT>(rk, j), rk.fa_l[j], kj);
      if (uq) {  // the error estimate in float-float
        ff_acc(erh, erl, fe<CT>(rk, j), rk.fe_l[j], (float)kj.re);
        ff_acc(eih, eil, fe<CT>(rk, j), rk.fe_l[j], (float)kj.im);
      }
    }
    const double2 yp = static_cast<const double2*>(rk.y_prev)[row];
    const double2 dy = inc.wide();
    o.y = make_double2(yp.x + dy.x, yp.y + dy.y);
    static_cast<float2*>(rk.y_front_s)[row] = make_float2((float)o.y.x, (float)o.y.y);
    const double er = (double)erh + (double)erl, ei = (double)eih + (double)eil;
    o.term = wrms_term(er * er + ei * ei, o.y.x * o.y.x + o.y.y * o.y.y, rk.atol, rk.rtol);
  } else {
    HermSum<CT> y{ld_cx<CT>(static_cast<const YT*>(rk.y_prev) + row)};
    cx<CT> e{0, 0};
#pragma unroll
    for (int j = 0; j < RK_STEP; ++j) {
      const bool ub = (rk.nz_a >> j) & 1u, uq = (rk.nz_e >> j) & 1u;
      if (!ub && !uq) continue;
      const cx<CT> kj = (j == s) ? acc : ld_cx<CT>(kbuf + (size_t)j * n64 + row);
      if (ub) y.add(fa<CT>(rk, j), rk.fa_l[j], kj);
      if (uq) cx_axpy(e, fe<CT>(rk, j), kj);
    }
    st_cx(&o.y, y.value());
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
