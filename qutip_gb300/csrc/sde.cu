// Stochastic Schrodinger and master equations with the reference's explicit Platen scheme
// (qutip/solver/sode/_sode.pyx:58-120, Breuer & Petruccione eq. 7.47), drift and diffusion
// of qutip/solver/sode/ssystem.pyx:119-250.  A group of threads integrates one trajectory
// through n_steps fixed steps with the Wiener increments the host drew (the reference's own
// generator stream), so a launch covers a whole output interval of one or many
// trajectories.  States of up to 640 entries with one stochastic operator (512 with two) take
// a thread per entry (sde_row_kernel, below).  With more operators a state of up to 64 entries
// is integrated by one warp (4 trajectories per CTA; syncs are __syncwarp), and a larger one by a
// CTA of 256 threads; there every vector operation follows the reference's order of operations
// (`_data.add(a, b, s)` is a + s b element by element, the complex scalars formed the way
// the reference forms them), where the row kernel contracts to fused multiply-adds.  CSR rows
// are summed in column order in both.
#include "capi_internal.h"
#include "common.cuh"

namespace qg {

constexpr int SDE_BLOCK = 256;   // CTA shape: one trajectory per CTA
constexpr int SDE_WARPS = 4;     // warp shape: one trajectory per warp, 4 per CTA
constexpr int SDE_WARP_MAX_N = 64;  // states up to this length take the warp shape

// A group of GS threads integrating one trajectory: a warp (GS = 32, syncs are
// __syncwarp, sums are XOR butterflies) or a CTA (GS = SDE_BLOCK).  Sums come back to
// every thread with the same bits.
template <int GS>
struct SdeGroup;
template <>
struct SdeGroup<32> {
  int rank;
  __device__ __forceinline__ void sync() const { __syncwarp(); }
  __device__ __forceinline__ double2 sum(double2 v, double*) const {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
      v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    return v;
  }
};
template <>
struct SdeGroup<SDE_BLOCK> {
  int rank;
  __device__ __forceinline__ void sync() const { __syncthreads(); }
  __device__ double2 sum(double2 v, double* red) const {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      v.x += __shfl_down_sync(0xffffffffu, v.x, o);
      v.y += __shfl_down_sync(0xffffffffu, v.y, o);
    }
    constexpr int W = SDE_BLOCK / 32;
    __syncthreads();  // earlier readers of red are done
    if ((threadIdx.x & 31) == 0) {
      red[threadIdx.x >> 5] = v.x;
      red[W + (threadIdx.x >> 5)] = v.y;
    }
    __syncthreads();
    double re = 0.0, im = 0.0;
    for (int w = 0; w < W; ++w) {
      re += red[w];
      im += red[W + w];
    }
    return make_double2(re, im);
  }
};

struct Sde {
  const qg_sde* S;
  int n, m;
  double2* F;   // drift output
  double2* D1;  // state + dt drift
  double2* VT;  // Platen support vector
  double2* TMP;
  double2* D2;  // m diffusion vectors
  double2* VP;  // m support vectors (+)
  double2* VM;  // m support vectors (-)
  double2* D2P; // m diffusions at VP_i
  double2* D2M; // m diffusions at VM_i
  double* red;  // reduction scratch (CTA shape)
};

__device__ __forceinline__ double2 cmul2(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a + s b
__device__ __forceinline__ double2 axpy(double2 a, double2 s, double2 b) {
  const double2 t = cmul2(s, b);
  return make_double2(a.x + t.x, a.y + t.y);
}
__device__ __forceinline__ double2 axpy(double2 a, double s, double2 b) {
  return make_double2(a.x + s * b.x, a.y + s * b.y);
}

// y = rows [row0, row0 + n) of a CSR operator times x (x complete on entry)
template <int GS>
__device__ void csr_mv(const SdeGroup<GS>& g, const int* __restrict__ rp,
                       const int* __restrict__ col, const double2* __restrict__ val,
                       int64_t row0, const double2* x, double2* y, int n) {
  for (int r = g.rank; r < n; r += GS) {
    const int s = __ldg(rp + row0 + r), e = __ldg(rp + row0 + r + 1);
    double ar = 0.0, ai = 0.0;
    for (int p = s; p < e; ++p) {
      const double2 v = __ldg(val + p);
      const double2 z = x[__ldg(col + p)];
      ar += v.x * z.x - v.y * z.y;
      ai += v.x * z.y + v.y * z.x;
    }
    y[r] = make_double2(ar, ai);
  }
}

// SSE: <x| M_i |x> (M_i x goes through TMP)
template <int GS>
__device__ double2 expect_m(const SdeGroup<GS>& g, const Sde& q, int i, const double2* x) {
  const qg_sde& S = *q.S;
  g.sync();
  csr_mv(g, S.m_rp, S.m_col, static_cast<const double2*>(S.m_val), (int64_t)i * q.n, x, q.TMP,
         q.n);
  double2 acc = make_double2(0.0, 0.0);
  for (int r = g.rank; r < q.n; r += GS) {
    const double2 a = x[r], b = q.TMP[r];
    acc.x += a.x * b.x + a.y * b.y;  // conj(a) b
    acc.y += a.x * b.y - a.y * b.x;
  }
  return g.sum(acc, q.red);
}

// SME: tr of the d x d matrix whose column-stacked form is v
template <int GS>
__device__ double2 trace_vec(const SdeGroup<GS>& g, const Sde& q, const double2* v) {
  const int d = q.S->d;
  double2 acc = make_double2(0.0, 0.0);
  for (int k = g.rank; k < d; k += GS) {
    const double2 a = v[(int64_t)k * (d + 1)];
    acc.x += a.x;
    acc.y += a.y;
  }
  return g.sum(acc, q.red);
}

// out = drift(x)   (ssystem.pyx:141-154 closed, 227-228 open)
template <int GS>
__device__ void drift(const SdeGroup<GS>& g, const Sde& q, const double2* x, double2* out) {
  const qg_sde& S = *q.S;
  g.sync();
  csr_mv(g, S.l_rp, S.l_col, static_cast<const double2*>(S.l_val), 0, x, out, q.n);
  if (S.open) return;
  for (int i = 0; i < q.m; ++i) {
    const double2 e = expect_m(g, q, i, x);
    g.sync();
    csr_mv(g, S.c_rp, S.c_col, static_cast<const double2*>(S.c_val), (int64_t)i * q.n, x,
           q.TMP, q.n);
    const double2 s1 = cmul2(make_double2(-0.125 * e.x, -0.125 * e.y), e);  // -0.125 * e * e
    const double2 s2 = make_double2(0.5 * e.x, 0.5 * e.y);
    for (int r = g.rank; r < q.n; r += GS) {
      const double2 o = axpy(out[r], s1, x[r]);
      out[r] = axpy(o, s2, q.TMP[r]);
    }
  }
}

// d2[i] = diffusion_i(x) for every i   (ssystem.pyx:156-166 closed, 230-240 open)
template <int GS>
__device__ void diffusion(const SdeGroup<GS>& g, const Sde& q, const double2* x, double2* d2) {
  const qg_sde& S = *q.S;
  for (int i = 0; i < q.m; ++i) {
    double2* out = d2 + (int64_t)i * q.n;
    g.sync();
    csr_mv(g, S.c_rp, S.c_col, static_cast<const double2*>(S.c_val), (int64_t)i * q.n, x, out,
           q.n);
    double2 e;
    if (S.open) {
      g.sync();
      e = trace_vec(g, q, out);
      e = make_double2(-e.x, -e.y);
    } else {
      e = expect_m(g, q, i, x);
      e = make_double2(-0.5 * e.x, -0.5 * e.y);
    }
    for (int r = g.rank; r < q.n; r += GS) out[r] = axpy(out[r], e, x[r]);
  }
}

// One Platen step from X into OUT (_sode.pyx:62-120).
template <int GS>
__device__ void platen_step(const SdeGroup<GS>& g, const Sde& q, const double2* X, double2* OUT,
                            const double* dW, double dt) {
  const int n = q.n, m = q.m;
  const double sqrt_dt = sqrt(dt);
  const double sqrt_dt_inv = 0.25 / sqrt_dt;
  drift(g, q, X, q.F);
  for (int r = g.rank; r < n; r += GS) q.D1[r] = axpy(X[r], dt, q.F[r]);
  diffusion(g, q, X, q.D2);
  for (int r = g.rank; r < n; r += GS) {
    const double2 d1 = q.D1[r];
    OUT[r] = make_double2(d1.x * 0.5, d1.y * 0.5);
    double2 vt = d1;
    for (int i = 0; i < m; ++i) {
      const double2 d2 = q.D2[(int64_t)i * n + r];
      q.VP[(int64_t)i * n + r] = axpy(d1, sqrt_dt, d2);
      q.VM[(int64_t)i * n + r] = axpy(d1, -sqrt_dt, d2);
      vt = axpy(vt, dW[i], d2);
    }
    q.VT[r] = vt;
  }
  drift(g, q, q.VT, q.F);
  for (int r = g.rank; r < n; r += GS) {
    const double2 o = axpy(OUT[r], 0.5 * dt, q.F[r]);
    OUT[r] = axpy(o, 0.5, X[r]);
  }
  for (int i = 0; i < m; ++i) {
    diffusion(g, q, q.VP + (int64_t)i * n, q.D2P);
    diffusion(g, q, q.VM + (int64_t)i * n, q.D2M);
    const double dw = dW[i] * 0.25;
    for (int r = g.rank; r < n; r += GS) {
      double2 o = axpy(OUT[r], 2 * dw, q.D2[(int64_t)i * n + r]);
      for (int j = 0; j < m; ++j) {
        double dw2p, dw2m;
        if (i == j) {
          const double dw2 = sqrt_dt_inv * (dW[i] * dW[j] - dt);
          dw2p = dw2 + dw;
          dw2m = -dw2 + dw;
        } else {
          dw2p = sqrt_dt_inv * dW[i] * dW[j];
          dw2m = -dw2p;
        }
        o = axpy(o, dw2p, q.D2P[(int64_t)j * n + r]);
        o = axpy(o, dw2m, q.D2M[(int64_t)j * n + r]);
      }
      OUT[r] = o;
    }
  }
}

// One Euler-Maruyama step from X into OUT (_sode.pyx:32-55): X + dt drift + sum_i dW_i d2_i.
template <int GS>
__device__ void euler_step(const SdeGroup<GS>& g, const Sde& q, const double2* X, double2* OUT,
                           const double* dW, double dt) {
  drift(g, q, X, q.F);
  diffusion(g, q, X, q.D2);
  for (int r = g.rank; r < q.n; r += GS) {
    double2 o = axpy(X[r], dt, q.F[r]);
    for (int i = 0; i < q.m; ++i) o = axpy(o, dW[i], q.D2[(int64_t)i * q.n + r]);
    OUT[r] = o;
  }
}

constexpr int SDE_PLATEN = 0, SDE_EULER = 1;

template <int GS, int SCHEME>
__device__ void run_trajectory(const SdeGroup<GS>& g, const qg_sde& S, int traj,
                               double2* states, const double* dW, int n_steps, double dt,
                               int64_t work_values, double* red) {
  Sde q;
  q.S = &S;
  q.n = (int)S.n;
  q.m = S.n_sc;
  q.red = red;
  const int64_t n = S.n, m = S.n_sc;
  double2* w = static_cast<double2*>(S.work) + (int64_t)traj * work_values;
  q.F = w;
  q.D1 = w + n;
  q.VT = w + 2 * n;
  q.TMP = w + 3 * n;
  double2* spare = w + 4 * n;  // the other half of the state double buffer
  q.D2 = w + 5 * n;
  q.VP = q.D2 + m * n;
  q.VM = q.VP + m * n;
  q.D2P = q.VM + m * n;
  q.D2M = q.D2P + m * n;
  double2* home = states + (int64_t)traj * n;
  double2* X = home;
  double2* OUT = spare;
  const double* dwt = dW + (int64_t)traj * n_steps * m;
  for (int k = 0; k < n_steps; ++k) {
    if constexpr (SCHEME == SDE_EULER)
      euler_step(g, q, X, OUT, dwt + (int64_t)k * m, dt);
    else
      platen_step(g, q, X, OUT, dwt + (int64_t)k * m, dt);
    g.sync();
    double2* t = X;
    X = OUT;
    OUT = t;
  }
  if (X != home) {  // odd step count: the state ended in the spare
    for (int r = g.rank; r < q.n; r += GS) home[r] = X[r];
  }
}

template <int SCHEME>
__global__ void __launch_bounds__(SDE_BLOCK) sde_cta_kernel(qg_sde S, double2* states,
                                                            const double* __restrict__ dW,
                                                            int n_steps, double dt,
                                                            int64_t work_values) {
  __shared__ double red[2 * SDE_BLOCK / 32];
  const SdeGroup<SDE_BLOCK> g{(int)threadIdx.x};
  run_trajectory<SDE_BLOCK, SCHEME>(g, S, blockIdx.x, states, dW, n_steps, dt, work_values, red);
}

template <int SCHEME>
__global__ void __launch_bounds__(32 * SDE_WARPS) sde_warp_kernel(
    qg_sde S, int n_traj, double2* states, const double* __restrict__ dW, int n_steps, double dt,
    int64_t work_values) {
  const int traj = blockIdx.x * SDE_WARPS + (threadIdx.x >> 5);
  if (traj >= n_traj) return;  // whole warps leave together
  const SdeGroup<32> g{(int)(threadIdx.x & 31)};
  run_trajectory<32, SCHEME>(g, S, traj, states, dW, n_steps, dt, work_values, nullptr);
}

// --------------------------------------------- short states, few operators ----
// States of up to SDE_ROW_THREADS entries with one or two stochastic operators: one thread per
// entry, the CTA's trajectories side by side (n threads each, so 40-entry kets fill 35 of 40
// warps instead of half of every second), all steps of the launch in shared memory and
// registers.  Bound: FP64 issue (an SM does two multiply-adds a clock, a warp's instruction
// takes 16).  So the steps share what they can -- one product each of L, C_i and M_i with the
// state serves both drift and diffusion; L, C and M meet the supports in one pass -- a
// value's zero real or imaginary part is not multiplied (Liouvillians of real operators have
// few other values), and a sum over the state is taken by a few lanes, its other warps not
// issuing FP64 adds.  A Platen step has 6 barriers; the kernels above, 15.
// Measured, 100 steps: 256 master-equation trajectories of 400 entries 5.63 -> 2.90
// ms (29 us a step); 1000 kets of 40 entries 4.67 -> 1.58 ms.  Longer states and more
// operators keep the kernels above: their vectors outgrow shared memory and registers.
// A launch reserves what its operators need; a block still waits for an SM with that room (and
// registers for up to 640 threads) to spare, so beside a batch that holds every SM in part a
// launch of kets with a CTA each ran at once (0.35 ms for 0.23 alone), one of 400-entry states
// or of seven kets a CTA at the batch's end, where the kernels above found room.
// Most threads of a CTA: 96 registers for one operator, 128 for two.  CTAs of up to
// SDE_ROW_PAIR threads with one operator are compiled for two on an SM (72 registers): one
// alone leaves the FP64 pipe idle behind its barriers.
template <int M>
constexpr int SDE_ROW_THREADS = M == 1 ? 640 : 512;
constexpr int SDE_ROW_PAIR = 448;
constexpr int SDE_ROW_MAX_M = 2;
constexpr int SDE_ROW_OP_SMEM = 72 * 1024;  // operators kept in shared memory up to this size

// A row's entries: kept transposed in shared memory (entry j of row r at j * n + r) or read
// from the CSR arrays.
struct RowOp {
  const double2* v;
  const int* c;
  int stride, len;
};
__device__ __forceinline__ bool nonzero(double a) {
  return ((__double2hiint(a) << 1) | __double2loint(a)) != 0;
}
__device__ __forceinline__ double2 row_mv(const RowOp& o, const double2* x) {
  double ar = 0.0, ai = 0.0;
  for (int j = 0; j < o.len; ++j) {
    const double2 v = o.v[j * o.stride];
    const double2 z = x[o.c[j * o.stride]];
    if (nonzero(v.x)) {
      ar = fma(v.x, z.x, ar);
      ai = fma(v.x, z.y, ai);
    }
    if (nonzero(v.y)) {
      ar = fma(-v.y, z.y, ar);
      ai = fma(v.y, z.x, ai);
    }
  }
  return make_double2(ar, ai);
}

// a + s b in four multiply-adds
__device__ __forceinline__ double2 fma_axpy(double2 a, double2 s, double2 b) {
  return make_double2(fma(s.x, b.x, fma(-s.y, b.y, a.x)), fma(s.x, b.y, fma(s.y, b.x, a.y)));
}

template <int M, bool OPEN>
constexpr int SDE_ROW_SUMS = (OPEN ? 0 : M) + 2 * M * M;

template <int M, bool OPEN, int SCHEME, int NT>
__global__ void __launch_bounds__(NT, NT <= SDE_ROW_PAIR ? 2 : 1)
    sde_row_kernel(qg_sde S, int n_traj, double2* states, const double* __restrict__ dW,
                   int n_steps, double dt, int T, int op_smem) {
  constexpr int K = SDE_ROW_SUMS<M, OPEN>;
  extern __shared__ __align__(16) unsigned char sde_smem[];
  __shared__ int need_s, off_s;
  const int n = (int)S.n, d = S.d;
  const int tid = threadIdx.x, threads = blockDim.x;
  const int t = tid / n, r = tid - t * n;
  const int traj = blockIdx.x * T + t;
  const bool on = t < T && traj < n_traj;
  const int cnt = OPEN ? d : n;  // terms of a sum over the state
  double2* X = reinterpret_cast<double2*>(sde_smem);
  double2* VT = X + (size_t)T * n;
  double2* VP = VT + (size_t)T * n;        // VP[i], then VM[i]
  double2* col = VP + (size_t)2 * M * T * n;
  double2* res = col + (size_t)K * T * cnt;
  double2* sq = res + (size_t)K * T;
  unsigned char* ops = reinterpret_cast<unsigned char*>(sq + (OPEN ? 0 : (size_t)K * T));

  // ---- the rows' operator entries: every operator's longest row, then the copies ----
  RowOp L, C[M], Mx[M];
  const int n_ops = 1 + M + (OPEN ? 0 : M);
  if (tid == 0) off_s = 0;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 1 + 2 * M; ++q) {
    if (q >= n_ops) break;
    const bool isl = q == 0, isc = q >= 1 && q <= M;
    const int* rp = isl ? S.l_rp : (isc ? S.c_rp : S.m_rp);
    const int* gc = isl ? S.l_col : (isc ? S.c_col : S.m_col);
    const double2* gv = static_cast<const double2*>(isl ? S.l_val : (isc ? S.c_val : S.m_val));
    const int block = isl ? 0 : (isc ? q - 1 : q - 1 - M);
    int s = 0, len = 0;
    if (t < T) {
      s = __ldg(rp + (size_t)block * n + r);
      len = __ldg(rp + (size_t)block * n + r + 1) - s;
    }
    if (tid == 0) need_s = 0;
    __syncthreads();
    atomicMax(&need_s, len);
    __syncthreads();
    const int w = need_s, at = off_s;
    const size_t bytes = ((size_t)w * n * 20 + 15) & ~(size_t)15;
    RowOp o{gv + s, gc + s, 1, len};
    if (at + bytes <= (size_t)op_smem) {
      double2* v = reinterpret_cast<double2*>(ops + at);
      int* c = reinterpret_cast<int*>(v + (size_t)w * n);
      if (t == 0) {
        for (int j = 0; j < len; ++j) {
          v[j * n + r] = __ldg(gv + s + j);
          c[j * n + r] = __ldg(gc + s + j);
        }
      }
      o = RowOp{v + r, c + r, n, len};
    }
    __syncthreads();
    if (tid == 0 && at + bytes <= (size_t)op_smem) off_s = at + (int)bytes;
    __syncthreads();
    if (isl) L = o;
#pragma unroll
    for (int i = 0; i < M; ++i) {
      if (q == 1 + i) C[i] = o;
      if (q == 1 + M + i) Mx[i] = o;
    }
  }

  const size_t base = (size_t)t * n;
  const size_t own = base + r;
  const bool diag = OPEN && r % (d + 1) == 0;
  const int slot = OPEN ? r / (d + 1) : r;
  // sums over the state: term s of this thread, then of each of `k` totals e the scalars
  // that meet vectors: -e (open) or -e/2 in res, and -e^2/8 (closed) in sq
  auto put = [&](int s, double2 v) {
    if (on && (!OPEN || diag)) col[((size_t)s * T + t) * cnt + slot] = v;
  };
  auto bra = [](double2 a, double2 b) {  // conj(a) b
    return make_double2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
  };
  // lanes per sum: the adds of a warp instruction cost 16 clocks whatever its lanes
  const int lanes = cnt > 64 ? 32 : 4;
  auto reduce = [&](int k) {
    __syncthreads();
    const int jobs = k * T * lanes;
    for (int j0 = (tid & ~31); j0 < jobs; j0 += threads) {
      const int j = j0 + (tid & 31);
      const int s = j / lanes, l = j - s * lanes;
      double2 a = make_double2(0.0, 0.0);
      if (s < k * T) {
        const double2* c = col + (size_t)s * cnt;
        for (int i = l; i < cnt; i += lanes) {
          a.x += c[i].x;
          a.y += c[i].y;
        }
      }
      for (int o = lanes >> 1; o > 0; o >>= 1) {
        a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
        a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
      }
      if (s < k * T && l == 0) {
        const double h = OPEN ? -1.0 : -0.5;
        res[s] = make_double2(h * a.x, h * a.y);
        if constexpr (!OPEN) sq[s] = cmul2(make_double2(-0.125 * a.x, -0.125 * a.y), a);
      }
    }
    __syncthreads();
  };
  double2 xr = make_double2(0.0, 0.0);
  if (t < T) {
    if (on) xr = states[(size_t)traj * n + r];
    X[own] = xr;
  }
  const double sqrt_dt = sqrt(dt);
  const double sqrt_dt_inv = 0.25 / sqrt_dt;
  const double* dwt = dW + (size_t)(on ? traj : 0) * n_steps * M;
  for (int k = 0; k < n_steps; ++k) {
    double dw[M];
#pragma unroll
    for (int i = 0; i < M; ++i) dw[i] = __ldg(dwt + (size_t)k * M + i);
    __syncthreads();  // X complete
    // drift and diffusion at X
    double2 F = make_double2(0.0, 0.0), D2[M];
    if (on) {
      F = row_mv(L, X + base);
#pragma unroll
      for (int i = 0; i < M; ++i) {
        D2[i] = row_mv(C[i], X + base);
        put(i, OPEN ? D2[i] : bra(xr, row_mv(Mx[i], X + base)));
      }
    }
    reduce(M);
    double2 out = make_double2(0.0, 0.0), d1 = out, vp[M], vm[M];
    if (on) {
#pragma unroll
      for (int i = 0; i < M; ++i) {
        const double2 h = res[i * T + t];
        if constexpr (!OPEN)
          F = fma_axpy(fma_axpy(F, sq[i * T + t], xr), make_double2(-h.x, -h.y), D2[i]);
        D2[i] = fma_axpy(D2[i], h, xr);
      }
      d1 = axpy(xr, dt, F);
    }
    if constexpr (SCHEME == SDE_EULER) {
      if (on) {
        out = d1;
#pragma unroll
        for (int i = 0; i < M; ++i) out = axpy(out, dw[i], D2[i]);
        xr = out;
        X[own] = out;
      }
      continue;
    } else {
      double2 vt = d1;
      if (on) {
        out = make_double2(d1.x * 0.5, d1.y * 0.5);
#pragma unroll
        for (int i = 0; i < M; ++i) {
          vp[i] = axpy(d1, sqrt_dt, D2[i]);
          vm[i] = axpy(d1, -sqrt_dt, D2[i]);
          vt = axpy(vt, dw[i], D2[i]);
          VP[(size_t)i * T * n + own] = vp[i];
          VP[(size_t)(M + i) * T * n + own] = vm[i];
        }
        VT[own] = vt;
      }
      __syncthreads();
      // drift at VT, diffusions at VP_i and VM_i
      double2 CT[M], P[M][M], Q[M][M];
      if (on) {
        F = row_mv(L, VT + base);
        if constexpr (!OPEN) {
#pragma unroll
          for (int i = 0; i < M; ++i) {
            CT[i] = row_mv(C[i], VT + base);
            put(2 * M * M + i, bra(vt, row_mv(Mx[i], VT + base)));
          }
        }
#pragma unroll
        for (int i = 0; i < M; ++i) {
          const double2* vpi = VP + (size_t)i * T * n + base;
          const double2* vmi = VP + (size_t)(M + i) * T * n + base;
#pragma unroll
          for (int j = 0; j < M; ++j) {
            P[i][j] = row_mv(C[j], vpi);
            Q[i][j] = row_mv(C[j], vmi);
            put(2 * (i * M + j), OPEN ? P[i][j] : bra(vp[i], row_mv(Mx[j], vpi)));
            put(2 * (i * M + j) + 1, OPEN ? Q[i][j] : bra(vm[i], row_mv(Mx[j], vmi)));
          }
        }
      }
      reduce(K);
      if (on) {
        if constexpr (!OPEN) {
#pragma unroll
          for (int i = 0; i < M; ++i) {
            const double2 h = res[(2 * M * M + i) * T + t];
            F = fma_axpy(fma_axpy(F, sq[(2 * M * M + i) * T + t], vt), make_double2(-h.x, -h.y),
                         CT[i]);
          }
        }
        out = axpy(out, 0.5 * dt, F);
        out = axpy(out, 0.5, xr);
#pragma unroll
        for (int i = 0; i < M; ++i) {
          const double w = dw[i] * 0.25;
          out = axpy(out, 2 * w, D2[i]);
#pragma unroll
          for (int j = 0; j < M; ++j) {
            const double2 dp = fma_axpy(P[i][j], res[(2 * (i * M + j)) * T + t], vp[i]);
            const double2 dm = fma_axpy(Q[i][j], res[(2 * (i * M + j) + 1) * T + t], vm[i]);
            double wp, wm;
            if (i == j) {
              const double w2 = sqrt_dt_inv * (dw[i] * dw[j] - dt);
              wp = w2 + w;
              wm = -w2 + w;
            } else {
              wp = sqrt_dt_inv * dw[i] * dw[j];
              wm = -wp;
            }
            out = axpy(out, wp, dp);
            out = axpy(out, wm, dm);
          }
        }
        xr = out;
        X[own] = out;
      }
    }
  }
  if (on) states[(size_t)traj * n + r] = xr;
}

constexpr int SDE_ROW_SMEM = 220 * 1024;  // most dynamic shared memory of a CTA

// Launch shape of the row kernel: trajectories and threads of a CTA, the bytes of its vectors
// and of its operators in shared memory, and whether the form for two CTAs on an SM takes it.
struct SdeRowShape {
  int T, threads, vecs, ops;
  bool pair;
};
static SdeRowShape sde_row_shape(int n, int d, int m, bool open, int n_traj, int sms,
                                 int op_bytes) {
  const int most = m == 1 ? SDE_ROW_THREADS<1> : SDE_ROW_THREADS<2>;
  const int sums = (open ? 0 : m) + 2 * m * m;  // SDE_ROW_SUMS
  const int per = 16 * (n * (2 + 2 * m) + sums * ((open ? d : n) + (open ? 1 : 2)));
  // trajectories per CTA: enough CTAs for every SM first, then full CTAs
  int T = (n_traj - 1) / sms + 1;
  if (T > most / n) T = most / n;
  // one CTA per SM at most: no second one to make room for
  const bool pair = m == 1 && n <= SDE_ROW_PAIR && (n_traj - 1) / T + 1 > sms;
  if (pair && T > SDE_ROW_PAIR / n) T = SDE_ROW_PAIR / n;
  // the sums of kets of one entry and two operators outgrow the vectors: 576 bytes a trajectory
  if (T > SDE_ROW_SMEM / per) T = SDE_ROW_SMEM / per;
  const int vecs = T * per, room = SDE_ROW_SMEM - vecs;
  // what the operators need where that is known: blocks find room beside other work and one
  // another
  int ops = room < SDE_ROW_OP_SMEM ? room : SDE_ROW_OP_SMEM;
  if (op_bytes > 0 && op_bytes < ops) ops = op_bytes;
  return SdeRowShape{T, (T * n + 31) / 32 * 32, vecs, ops, pair};
}

template <int M, bool OPEN, int SCHEME, int NT>
static int launch_sde_rows(const qg_sde& S, int n_traj, double2* states, const double* dW,
                           int n_steps, double dt, const SdeRowShape& sh, cudaStream_t st) {
  const int smem = sh.vecs + sh.ops;
  auto kern = sde_row_kernel<M, OPEN, SCHEME, NT>;
  if (!allow_smem((const void*)kern, (size_t)smem))
    return set_error(QG_ERR_CUDA, "stochastic kernel: shared memory opt-in failed");
  kern<<<(n_traj - 1) / sh.T + 1, sh.threads, smem, st>>>(S, n_traj, states, dW, n_steps, dt, sh.T,
                                                         sh.ops);
  return check_launch("sde_row_kernel");
}

template <bool OPEN, int SCHEME>
static int launch_sde_rows_shape(const qg_sde& S, int n_traj, double2* states, const double* dW,
                                 int n_steps, double dt, cudaStream_t st) {
  const SdeRowShape sh = sde_row_shape((int)S.n, S.d, S.n_sc, OPEN, n_traj, sm_count(),
                                       S.op_bytes);
  if (S.n_sc == 2)
    return launch_sde_rows<2, OPEN, SCHEME, SDE_ROW_THREADS<2>>(S, n_traj, states, dW, n_steps, dt,
                                                                sh, st);
  if (!sh.pair)
    return launch_sde_rows<1, OPEN, SCHEME, SDE_ROW_THREADS<1>>(S, n_traj, states, dW, n_steps, dt,
                                                                sh, st);
  return launch_sde_rows<1, OPEN, SCHEME, SDE_ROW_PAIR>(S, n_traj, states, dW, n_steps, dt, sh, st);
}

static int check_sde(const qg_sde* S) {
  if (!S) return set_error(QG_ERR_ARG, "null system");
  if (S->n < 1 || S->n >= (int64_t)INT32_MAX / (QG_MAX_COPS + 1))
    return set_error(QG_ERR_ARG, "state length out of range");
  if (S->n_sc < 1 || S->n_sc > QG_MAX_COPS) return set_error(QG_ERR_ARG, "n_sc out of range");
  if (S->open != 0 && S->open != 1) return set_error(QG_ERR_ARG, "open must be 0 or 1");
  if (S->open && (int64_t)S->d * S->d != S->n)
    return set_error(QG_ERR_ARG, "SME: the state length must be d*d");
  if (!S->open && S->d != S->n) return set_error(QG_ERR_ARG, "SSE: the state length must be d");
  if (!S->l_rp || !S->l_col || !S->l_val || !S->c_rp || !S->c_col || !S->c_val || !S->work)
    return set_error(QG_ERR_ARG, "null operator or workspace");
  if (!S->open && (!S->m_rp || !S->m_col || !S->m_val))
    return set_error(QG_ERR_ARG, "SSE needs the expectation operators");
  return QG_OK;
}

template <int SCHEME>
static int launch_sde(const qg_sde* S, int32_t n_traj, void* states, const double* dW,
                      int32_t n_steps, double dt, void* stream) {
  int rc = check_sde(S);
  if (rc) return rc;
  if (n_traj < 0 || n_steps < 0 || !(dt > 0.0)) return set_error(QG_ERR_ARG, "bad launch");
  if (n_traj == 0 || n_steps == 0) return QG_OK;
  if (!states || !dW) return set_error(QG_ERR_ARG, "null states or noise");
  if (S->n_sc <= SDE_ROW_MAX_M &&
      S->n <= (S->n_sc == 1 ? SDE_ROW_THREADS<1> : SDE_ROW_THREADS<2>)) {
    double2* x = static_cast<double2*>(states);
    cudaStream_t st = (cudaStream_t)stream;
    return S->open ? launch_sde_rows_shape<true, SCHEME>(*S, n_traj, x, dW, n_steps, dt, st)
                   : launch_sde_rows_shape<false, SCHEME>(*S, n_traj, x, dW, n_steps, dt, st);
  }
  const int64_t wv = (5 + 5 * (int64_t)S->n_sc) * S->n;
  if (S->n <= SDE_WARP_MAX_N) {
    sde_warp_kernel<SCHEME><<<(n_traj + SDE_WARPS - 1) / SDE_WARPS, 32 * SDE_WARPS, 0,
                              (cudaStream_t)stream>>>(*S, n_traj, static_cast<double2*>(states),
                                                      dW, n_steps, dt, wv);
    return check_launch("sde_warp_kernel");
  }
  sde_cta_kernel<SCHEME><<<n_traj, SDE_BLOCK, 0, (cudaStream_t)stream>>>(
      *S, static_cast<double2*>(states), dW, n_steps, dt, wv);
  return check_launch("sde_cta_kernel");
}

}  // namespace qg

using namespace qg;

extern "C" int64_t qg_sde_work_values(int64_t n, int32_t n_sc) {
  return (5 + 5 * (int64_t)n_sc) * n;
}

extern "C" int qg_sde_row_shape(int64_t n, int32_t n_sc, int32_t open, int32_t n_traj,
                                int32_t n_sms, int32_t op_bytes, int32_t* shape) {
  if (!shape) return set_error(QG_ERR_ARG, "null shape");
  if (n < 1 || n_sc < 1 || n_traj < 1 || n_sms < 1) return set_error(QG_ERR_ARG, "bad launch");
  if (n_sc > SDE_ROW_MAX_M || n > (n_sc == 1 ? SDE_ROW_THREADS<1> : SDE_ROW_THREADS<2>)) return 1;
  int d = (int)n;
  if (open)
    for (d = 1; (int64_t)d * d < n;) ++d;
  const SdeRowShape s = sde_row_shape((int)n, d, n_sc, open != 0, n_traj, n_sms, op_bytes);
  const int32_t v[4] = {s.T, s.threads, s.vecs, s.ops};
  for (int i = 0; i < 4; ++i) shape[i] = v[i];
  return QG_OK;
}

extern "C" int qg_sde_platen(const qg_sde* S, int32_t n_traj, void* states, const double* dW,
                             int32_t n_steps, double dt, void* stream) {
  return launch_sde<SDE_PLATEN>(S, n_traj, states, dW, n_steps, dt, stream);
}

extern "C" int qg_sde_euler(const qg_sde* S, int32_t n_traj, void* states, const double* dW,
                            int32_t n_steps, double dt, void* stream) {
  return launch_sde<SDE_EULER>(S, n_traj, states, dW, n_steps, dt, stream);
}
