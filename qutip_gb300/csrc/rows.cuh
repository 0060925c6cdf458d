// Row arithmetic shared by the matvec kernels (spmv.cu) and the fused step kernel
// (step.cu): complex multiply-accumulates, sub-warp sums, dictionary codes and the
// coefficient product, in one place so that both take the same operations in the same
// order and a row's sum has the same bits whichever kernel forms it.
#pragma once
#include "common.cuh"
#include "stage.cuh"

namespace qg {

// Complex multiply-accumulate in the accumulation precision.
__device__ __forceinline__ void cmac_any(double& ar, double& ai, double2 v, double2 x) {
  ar = fma(v.x, x.x, ar);
  ar = fma(-v.y, x.y, ar);
  ai = fma(v.x, x.y, ai);
  ai = fma(v.y, x.x, ai);
}
__device__ __forceinline__ void cmac_any(float& ar, float& ai, float2 v, float2 x) {
  ar = fmaf(v.x, x.x, ar);
  ar = fmaf(-v.y, x.y, ar);
  ai = fmaf(v.x, x.y, ai);
  ai = fmaf(v.y, x.x, ai);
}

// acc += conj(v) * x
__device__ __forceinline__ void cmac_conj(double& ar, double& ai, double2 v, double2 x) {
  ar = fma(v.x, x.x, ar);
  ar = fma(v.y, x.y, ar);
  ai = fma(v.x, x.y, ai);
  ai = fma(-v.y, x.x, ai);
}
__device__ __forceinline__ void cmac_conj(float& ar, float& ai, float2 v, float2 x) {
  ar = fmaf(v.x, x.x, ar);
  ar = fmaf(v.y, x.y, ar);
  ai = fmaf(v.x, x.y, ai);
  ai = fmaf(-v.y, x.x, ai);
}

__device__ __forceinline__ cplx prog_coef(const int* code, const int* start, const double* consts,
                                          int g, double t) {
  if (code == nullptr) return cplx{1.0, 0.0};
  return eval_coef(code + start[g], consts, t);
}

template <int LANES, typename R>
__device__ __forceinline__ cx<R> sub_reduce(R ar, R ai) {
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) {
    ar += __shfl_xor_sync(0xffffffffu, ar, o);
    ai += __shfl_xor_sync(0xffffffffu, ai, o);
  }
  return cx<R>{ar, ai};
}

// Class of each group's coefficient, decided once per block: 0 = exactly one (the
// group's sum goes straight into the row's), 1 = real, 2 = complex.
template <typename CT>
__device__ __forceinline__ int coef_class(cx<CT> c) {
  return (c.re == (CT)1 && c.im == (CT)0) ? 0 : (c.im == (CT)0 ? 1 : 2);
}

template <int CB>
struct Codes4;
template <>
struct Codes4<1> {
  using T = unsigned int;
  __device__ static int at(T c, int u) { return (int)((c >> (8 * u)) & 0xffu); }
};
template <>
struct Codes4<2> {
  using T = uint2;
  __device__ static int at(T c, int u) {
    const unsigned w = u < 2 ? c.x : c.y;
    return (int)((w >> (16 * (u & 1))) & 0xffffu);
  }
};

// One stored code: the table pair k applied to x[row + offset].  Whole complex values
// (QG_LAYOUT_SLICED_DICT) cost four multiply-adds.  With the real/imaginary split
// (QG_LAYOUT_SLICED_DICT_RI, complex128) a table entry is one real factor: toff holds
// (offset << 1) | imag and tval the pair (c1, c2) = (a, a) for a real part or (-a, a) for
// an imaginary part, applied as (c1 p, c2 q) with (p, q) = x, or x's parts exchanged for
// an imaginary part -- two FP64 multiply-adds, GB300's scarce FP64 rate being the bound.
// NC: x is constant for the launch (read-only path); otherwise it was written by the same
// launch and is read with ordinary loads.
template <bool RI, bool NC, typename ST, typename R>
__device__ __forceinline__ void dict_mac(const ST* tval, const int* toff, const ST* x, int k,
                                         int row, int last_col, R& ar, R& ai) {
  if constexpr (RI) {
    const int oc = toff[k];
    const int col = min(max(row + (oc >> 1), 0), last_col);
    const ST v = tval[k];
    ST xv;
    if constexpr (NC) xv = ld_gather(x + col);
    else xv = x[col];
    const bool sw = (oc & 1) != 0;
    ar = fma(v.x, sw ? xv.y : xv.x, ar);
    ai = fma(v.y, sw ? xv.x : xv.y, ai);
  } else {
    const int col = min(max(row + toff[k], 0), last_col);
    ST xv;
    if constexpr (NC) xv = ld_gather(x + col);
    else xv = x[col];
    cmac_any(ar, ai, tval[k], xv);
  }
}

// acc += c * (ar, ai).  In FP64 a real coefficient (every group of a Liouvillian with a
// real time dependence, and the constant group) takes two multiply-adds, not four; the
// branch is uniform (one coefficient per group).  FP32 keeps the plain product.
template <typename R>
__device__ __forceinline__ void coef_mac(cx<R>& acc, cx<R> c, R ar, R ai) {
  if constexpr (sizeof(R) == 8) {
    if (c.im == (R)0) {
      acc.re = fma(c.re, ar, acc.re);
      acc.im = fma(c.re, ai, acc.im);
      return;
    }
  }
  acc = cx_add(acc, cx_mul(c, cx<R>{ar, ai}));
}

}  // namespace qg
