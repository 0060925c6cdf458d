// Several Vern7 stages of one system in one launch (qg_vern7_range): a trial step (stages
// 0..9 with the error norm) or the dense-output stages (10..15) of a system whose rows all
// fit the GPU at once, one row per sub-warp of LANES threads.
//
// What bounds it: latency.  A stage of a system of up to some 70,000 rows is a few
// microseconds of dependent loads and FP64 work, so ten launches a step, each with its own
// host call, launch gap and re-read of the row's data, cost more than the arithmetic:
// 21.6 us per right-hand side at 65,536 rows, whose FP64 work takes 6.4 us.  Here the
// stages follow one another behind a grid barrier; a row keeps its operator entries (or
// codes), its k_j and its state in shared memory and registers for the whole launch, and
// only the stage input crosses between SMs.
//
// Complex128 rows are bound by FP64 issue once the launches are gone: an FP64 instruction holds
// its SM for 16 clocks however few lanes it has, so a row goes to fewer threads than the
// matvec kernel's sub-warp and a coefficient that is one is not multiplied.  A Hermitian
// density matrix (herm_d) is evaluated by half as in herm.cu, 8 warps to a unit of 32 rows x
// 8 columns on or below the diagonal: the L = 8 Ising chain puts 8 warps on an SM that way
// instead of 14.
//
// Measured, whole complex128 solves: the L = 8 Ising chain (65,536 rows) 39.1 -> 27.9 ms in
// one launch a step, and 24.9 -> 21.5 ms by half; the d = 125 Bose-Hubbard trimer (15,625
// rows, odd) 9.8 -> 6.2 ms.  An operator with more rows than the GPU has resident threads at
// 512 a block keeps one launch a stage: there a stage is 40 us and more, and the launches no
// longer count.
//
// The blocks take the shared memory that their rows need, but all of them at once: beside a
// batch on another stream that holds every SM in part, a solve waits until its blocks fit.  One
// block per SM with 100 KB of batch on each: the N = 10 Jaynes-Cummings solve runs beside it
// (4.3 ms, 2.5 alone), at 30 or 170 KB (the SM keeps its split between L1 and shared memory
// while a block runs) it waits for the batch's end, as does the L = 6 Ising solve, whose
// stages one by one ran beside it.  A CSR operator that should not wait takes a launch shape
// without this kernel (sub-warps of 16).
//
// The launch is cooperative (all blocks resident), and every wait at the barrier is bounded:
// a wait that gives up sets *result to -1, every block leaves, and the launch's stages hold NaN
// in its rows: what is read from them before the host sees the word is no value.  A row's sum
// and its stage combination are formed by the operations of the per-stage kernels in their
// order.
#include <mutex>
#include <type_traits>

#include "capi_internal.h"
#include "common.cuh"
#include "herm.cuh"
#include "rows.cuh"
#include "stage.cuh"

namespace qg {

// Layouts: row-major CSR with LANES threads per row, 32-row slices, dictionary codes.
enum Kind { KIND_CSR = 0, KIND_SLICED = 1, KIND_DICT1 = 2, KIND_DICT2 = 3 };

constexpr int STEP_THREADS = 512;   // most threads of a block (one block per SM)
constexpr int STEP_MIN_WARPS = 4;   // fewer warps per block only spread the barrier wider
// most entries (CSR, sliced) or code words a thread keeps in shared memory; rows longer than
// that read the rest from global memory at every stage
constexpr int STEP_KEEP = 32;
// A thread's share of the longest row, where that is known: the launch waits until all its
// blocks fit beside whatever else the GPU runs, so it takes no more than it uses (the
// four-entry rows of a Jaynes-Cummings system: 27 KB a block where 32 entries take 98).
static int step_keep(const qg_csr_groups& A, int kind, int lanes) {
  if (A.row_words <= 0) return STEP_KEEP;
  const int most = kind == KIND_CSR ? (A.row_words + A.n_groups * (lanes - 1)) / lanes : A.row_words;
  return most < STEP_KEEP ? most : STEP_KEEP;
}
constexpr int HERM_WARPS = 8;       // a unit of the half form: 32 rows x 8 columns
constexpr long long STEP_WAIT_CYCLES = 16 * WAIT_CYCLES;  // the GPU may be shared meanwhile

struct StepArgs {
  qg_csr_groups A;
  RkArgs rk;           // buffers and tolerances (factors are formed on the device)
  const void* x0;      // input of stage 0
  void* ytmp;          // both stage-input buffers
  double t_prev, dt;
  int s0, s1;          // stages [s0, s1)
  int keep;            // entries or code words kept per thread
  int herm_d;          // > 0: half form of a Hermitian d x d state (HERM instantiations)
  unsigned int* bar;   // arrivals of every earlier launch and of this one
  unsigned int bar_base;
  long long wait;      // most SM clocks at a barrier
};

__device__ unsigned int g_step_fault = 0u;

// Shared memory of a block, in bytes from its start (every part 16-byte aligned).
struct StepSmem {
  int tval, toff, k, val, idx, rp, tile, total;
};
template <typename ST>
__host__ __device__ inline StepSmem step_smem(const qg_csr_groups& A, int kind, int threads,
                                              int rows, int keep, bool herm) {
  const int D = kind >= KIND_DICT1 ? A.lanes : 0;
  auto up = [](size_t b) { return (int)((b + 15) & ~(size_t)15); };
  StepSmem L;
  L.tval = 0;
  L.toff = up((size_t)D * sizeof(ST));
  L.k = L.toff + up((size_t)D * 4);
  L.val = L.k + up((size_t)rows * RK_EXTRA_STEP * sizeof(ST));
  const int vb = kind >= KIND_DICT1 ? 0 : (int)sizeof(ST);
  const int ib = kind == KIND_DICT2 ? 8 : 4;
  L.idx = L.val + up((size_t)threads * keep * vb);
  L.rp = L.idx + up((size_t)threads * keep * ib);
  L.tile = L.rp + up((size_t)rows * (kind == KIND_CSR ? A.n_groups + 1 : 2 * A.n_groups) * 4);
  // half form: the conjugates of a unit's k and of its stage input or y_front
  L.total = L.tile + (herm ? (threads / 32) * 2 * HERM_PAD<double2> * 16 : 0);
  return L;
}

// Grid barrier: block arrivals counted in one word that only grows; this launch's n-th
// barrier completes at base + n * blocks.  False when the bounded wait gave up.
__device__ __forceinline__ bool grid_barrier(unsigned int* bar, unsigned int target,
                                             long long wait, bool* ok_s) {
  if (gridDim.x == 1) {
    __syncthreads();
    return true;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    const long long t0 = clock64();
    unsigned int v;
    bool ok;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      ok = (int)(v - target) >= 0;
    } while (!ok && clock64() - t0 < wait);
    __threadfence();
    *ok_s = ok;
  }
  __syncthreads();
  return *ok_s;
}

// LANES: threads of a row.  PARTS: sums of each thread (CSR); entry p goes to lane
// p % (LANES * PARTS) and the lanes are added pairwise, as in the matvec kernel.
template <int DT, int YDT, int KIND, int LANES, int PARTS, bool HERM>
__global__ void __launch_bounds__(STEP_THREADS, 1)
    vern7_range_kernel(const __grid_constant__ StepArgs a) {
  using ST = typename elem<DT>::T;
  using YT = typename elem<YDT>::T;
  using R = typename elem<DT>::R;
  constexpr bool MIXED = DT != YDT;
  constexpr bool RI = DT == QG_C128;
  constexpr bool DICT = KIND >= KIND_DICT1;
  constexpr int CB = KIND == KIND_DICT2 ? 2 : 1;
  using Sum = typename std::conditional<HERM, HermSum<R>, PlainSum<R>>::type;
  using C4 = typename Codes4<CB>::T;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ cx<R> coef[RK_EXTRA_STEP][QG_MAX_GROUPS];
  __shared__ int ccls[RK_EXTRA_STEP][QG_MAX_GROUPS];
  __shared__ R fac[RK_EXTRA_STEP][RK_EXTRA_STEP];  // dt a of the combination after stage s
  constexpr bool FF = HERM && sizeof(R) == 4;      // their low parts, for HermSum
  __shared__ float fac_l[FF ? RK_EXTRA_STEP : 1][RK_EXTRA_STEP];
  __shared__ R fe_s[RK_STEP];
  __shared__ float fel_s[RK_STEP];
  __shared__ unsigned int nz_s[RK_EXTRA_STEP + 1];
  __shared__ int tstart[QG_MAX_GROUPS + 1];
  __shared__ double red[STEP_THREADS / 32];
  __shared__ bool ok_s, last_s;
  const qg_csr_groups& A = a.A;
  const RkArgs& rk = a.rk;
  const int G = A.n_groups, n = (int)A.n_rows;
  const int tid = threadIdx.x, threads = blockDim.x;
  const int rows = threads / LANES;
  const int lrow = tid / LANES, lane = tid % LANES;
  int row = blockIdx.x * rows + lrow;
  bool valid = row < n;
  bool mirrored = false;
  int mirror = 0;  // element this thread writes the conjugate of (half form)
  if constexpr (HERM) {
    const int d = a.herm_d, nt = d >> 5;
    const int u = blockIdx.x * (threads / (32 * HERM_WARPS)) + (tid >> 5) / HERM_WARPS;
    valid = u < 2 * nt * (nt + 1);
    int tj = 0, tau = valid ? u >> 2 : 0;
    while (tau >= nt - tj) {
      tau -= nt - tj;
      ++tj;
    }
    const int ti = tj + tau, c0 = tj * 32 + (u & 3) * HERM_WARPS;
    row = ((c0 + ((tid >> 5) % HERM_WARPS)) * nt + ti) * 32 + (tid & 31);
    if (!valid) row = tid & 31;
    mirrored = valid && ti != tj;
    const int e = tid % (32 * HERM_WARPS);
    mirror = (c0 + e % HERM_WARPS) + (ti * 32 + e / HERM_WARPS) * d;
  }
  const StepSmem L = step_smem<ST>(A, KIND, threads, rows, a.keep, HERM);
  ST* tval = reinterpret_cast<ST*>(smem + L.tval);
  int* toff = reinterpret_cast<int*>(smem + L.toff);
  ST* ksm = reinterpret_cast<ST*>(smem + L.k) + lrow;  // k_j of this row at ksm[j * rows]
  ST* vsm = reinterpret_cast<ST*>(smem + L.val) + tid;  // kept entry i at [i * threads]
  int* csm = reinterpret_cast<int*>(smem + L.idx) + tid;
  C4* wsm = reinterpret_cast<C4*>(smem + L.idx) + tid;
  int* rpsm = reinterpret_cast<int*>(smem + L.rp) + lrow;  // row bounds, [g * rows]
  // half form: tiles of this thread's unit; its own place and the one it mirrors from
  ST* tk = reinterpret_cast<ST*>(smem + L.tile);
  YT* ty = reinterpret_cast<YT*>(smem + L.tile + (threads / 32) * HERM_PAD<double2> * 16);
  ST* tv = reinterpret_cast<ST*>(ty);
  constexpr int PAD = HERM_PAD<ST>, YPAD = HERM_PAD<YT>;
  const int unit0 = (tid >> 5) / HERM_WARPS * HERM_WARPS;  // first warp (tile column) of the unit
  const int t_own = (tid >> 5), t_from = unit0 + tid % HERM_WARPS,
            l_from = tid % (32 * HERM_WARPS) / HERM_WARPS;

  // ---- once per launch: factors, coefficients, the row's operator data ----
  for (int e = tid; e < (a.s1 - a.s0) * G; e += threads) {
    const int s = a.s0 + e / G, g = e % G;
    const cplx c = group_coef(A, g, a.t_prev + VERN7_C[s] * a.dt);
    coef[s][g] = cx<R>{(R)c.re, (R)c.im};
    ccls[s][g] = coef_class(coef[s][g]);
  }
  for (int e = tid; e < RK_EXTRA_STEP * RK_EXTRA_STEP; e += threads) {
    const int s = e / RK_EXTRA_STEP, j = e % RK_EXTRA_STEP;
    double v = 0.0;
    if (s == RK_STEP - 1 && a.s0 == 0) v = j < RK_STEP ? a.dt * VERN7_B[j] : 0.0;
    else if (s + 1 < RK_EXTRA_STEP && j <= s) v = a.dt * VERN7_A[s + 1][j];
    fac[s][j] = (R)v;
    if constexpr (FF) fac_l[s][j] = (float)(v - (double)(float)v);
    const double w = s == 0 && j < RK_STEP ? a.dt * VERN7_E[j] : 0.0;
    if (s == 0 && j < RK_STEP) {
      fe_s[j] = (R)w;
      fel_s[j] = (float)(w - (double)(float)w);
    }
    // the masks are of the double factors, as the per-stage kernels take them
    const unsigned int nz = __ballot_sync(0xffffffffu, v != 0.0);
    const unsigned int ne = __ballot_sync(0xffffffffu, w != 0.0);
    if ((tid & 31) == 0) {  // a warp covers two rows of the table
      nz_s[s] = nz & 0xffffu;
      nz_s[s + 1 < RK_EXTRA_STEP ? s + 1 : s] = nz >> 16;
      if (s == 0) nz_s[RK_EXTRA_STEP] = ne & 0xffffu;
    }
  }
  if constexpr (DICT) {
    for (int i = tid; i < A.lanes; i += threads) {
      tval[i] = __ldg(static_cast<const ST*>(A.val) + i);
      toff[i] = __ldg(A.dict_off + i);
    }
    if (tid <= G) tstart[tid] = __ldg(A.dict_start + tid);
  }
  const int sl = row >> 5;  // slice (sliced layouts: LANES == 1, a warp is a slice)
  const int S = A.n_tiles;
  const ST* __restrict__ gval = static_cast<const ST*>(A.val);
  const int* __restrict__ gcol = A.col;
  const unsigned char* __restrict__ codes = reinterpret_cast<const unsigned char*>(A.col);
  if constexpr (KIND == KIND_CSR) {
    int i = 0;
    int s = valid ? __ldg(A.row_ptr + row * G) : 0;
    if (lane == 0) rpsm[0] = s;
    for (int g = 0; g < G; ++g) {
      const int e = valid ? __ldg(A.row_ptr + row * G + g + 1) : 0;
      if (lane == 0) rpsm[(g + 1) * rows] = e;
      for (int p = s + lane; p < e; p += LANES, ++i)
        if (i < a.keep) {
          vsm[i * threads] = __ldg(gval + p);
          csm[i * threads] = __ldg(gcol + p);
        }
      s = e;
    }
  } else if (sl < S) {
    int i = 0;
    int off = 0;
    if constexpr (KIND == KIND_SLICED) off = __ldg(A.row_ptr + sl) + (tid & 31);
    for (int g = 0; g < G; ++g) {
      const int w = __ldg(A.tile_row + sl * G + g);
      if constexpr (DICT) off = __ldg(A.row_ptr + g * (S + 1) + sl);
      rpsm[(2 * g) * rows] = w;
      rpsm[(2 * g + 1) * rows] = off;
      if constexpr (DICT) {
        const C4* cp = reinterpret_cast<const C4*>(codes + (size_t)CB * off) + (tid & 31);
        for (int q = 0; q < (w + 3) / 4; ++q, ++i)
          if (i < a.keep) wsm[i * threads] = __ldg(cp + 32 * q);
      } else {
        for (int j = 0; j < w; ++j, ++i)
          if (i < a.keep) {
            vsm[i * threads] = __ldg(gval + off + 32 * j);
            csm[i * threads] = __ldg(gcol + off + 32 * j);
          }
        off += 32 * w;
      }
    }
  }
  const bool owner = valid && lane == 0;
  const size_t n64 = (size_t)n;
  ST* kg = static_cast<ST*>(rk.k) + row;
  cx<R> base{0, 0};
  if (owner) {
    if constexpr (MIXED) base = ld_cx<R>(static_cast<const ST*>(rk.y_prev_s) + row);
    else base = ld_cx<R>(static_cast<const YT*>(rk.y_prev) + row);
    for (int j = 0; j < a.s0; ++j) ksm[j * rows] = kg[(size_t)j * n64];
  }
  __syncthreads();
  ST* ytmp = static_cast<ST*>(a.ytmp);
  unsigned int target = a.bar_base;
  bool ok = true;
  // out = base + sum_{j <= s} (dt a_{s+1,j}) k_j, in the reference's order
  auto low = [&](int s, int j) { return FF ? fac_l[FF ? s : 0][j] : 0.f; };
  auto form_input = [&](int s) {
    Sum v{base};
    const unsigned int nz = nz_s[s];
    for (int j = 0; j <= s; ++j)
      if ((nz >> j) & 1u) v.add(fac[s][j], low(s, j), ld_cx<R>(ksm + j * rows));
    ST q;
    st_cx(&q, v.value());
    ytmp[(size_t)((s + 1) & 1) * n64 + row] = q;
    if constexpr (HERM) tv[t_own * PAD + (tid & 31)] = ST{q.x, -q.y};
  };
  auto mirror_input = [&](int s) {  // after a barrier that follows form_input
    if (mirrored) ytmp[(size_t)((s + 1) & 1) * n64 + mirror] = tv[t_from * PAD + l_from];
  };
  if (a.s0 > 0) {  // the first stage's input (stages 10..15 follow an accepted step)
    if (owner) form_input(a.s0 - 1);
    if constexpr (HERM) {
      __syncthreads();
      mirror_input(a.s0 - 1);
    }
    target += gridDim.x;
    ok = grid_barrier(a.bar, target, a.wait, &ok_s);
  }

  // ---- stages ----
  double err_acc = 0.0;
  const int last_col = (int)A.n_cols - 1;
  for (int s = a.s0; s < a.s1 && ok; ++s) {
    const ST* x = s == 0 ? static_cast<const ST*>(a.x0) : ytmp + (size_t)(s & 1) * n64;
    cx<R> acc{0, 0};
    if constexpr (KIND == KIND_CSR) {
      int i = 0;
      int ps = rpsm[0];
      for (int g = 0; g < G; ++g) {
        const int pe = rpsm[(g + 1) * rows];
        const int i0 = i;
        R ar[PARTS] = {}, ai[PARTS] = {};
        for (int p = ps + lane; p < pe; p += LANES * PARTS, i += PARTS) {
          ST v[PARTS], xv[PARTS];
#pragma unroll
          for (int l = 0; l < PARTS; ++l) {
            if (p + l * LANES >= pe) break;
            int c;
            if (i + l < a.keep) {
              v[l] = vsm[(i + l) * threads];
              c = csm[(i + l) * threads];
            } else {
              v[l] = __ldg(gval + p + l * LANES);
              c = __ldg(gcol + p + l * LANES);
            }
            xv[l] = x[c];
          }
#pragma unroll
          for (int l = 0; l < PARTS; ++l)
            if (p + l * LANES < pe) cmac_any(ar[l], ai[l], v[l], xv[l]);
        }
        i = i0 + (pe - ps - lane + LANES - 1) / LANES;  // this thread's entries so far
#pragma unroll
        for (int o = PARTS / 2; o > 0; o >>= 1)
          for (int l = 0; l < o; ++l) {
            ar[l] += ar[l + o];
            ai[l] += ai[l + o];
          }
        const cx<R> sum = sub_reduce<LANES>(ar[0], ai[0]);
        if (sizeof(R) == 8 && ccls[s][g] == 0) acc = cx_add(acc, sum);
        else acc = cx_add(acc, cx_mul(coef[s][g], sum));
        ps = pe;
      }
    } else if constexpr (KIND == KIND_SLICED) {
      if (sl < S) {
        int i = 0;
        for (int g = 0; g < G; ++g) {
          const int w = rpsm[(2 * g) * rows], off = rpsm[(2 * g + 1) * rows];
          R ar = 0, ai = 0;
          for (int j = 0; j < w; ++j, ++i) {
            ST v;
            int c;
            if (i < a.keep) {
              v = vsm[i * threads];
              c = csm[i * threads];
            } else {
              v = __ldg(gval + off + 32 * j);
              c = __ldg(gcol + off + 32 * j);
            }
            cmac_any(ar, ai, v, x[c]);
          }
          acc = cx_add(acc, cx_mul(coef[s][g], cx<R>{ar, ai}));
        }
      }
    } else {
      if (sl < S) {
        int i = 0;
        for (int g = 0; g < G; ++g) {
          const int w = rpsm[(2 * g) * rows], off = rpsm[(2 * g + 1) * rows];
          const int t0 = tstart[g], tn = tstart[g + 1] - t0;
          const C4* cp = reinterpret_cast<const C4*>(codes + (size_t)CB * off) + (tid & 31);
          const bool direct = sizeof(R) == 8 && ccls[s][g] == 0;
          R ar = direct ? acc.re : (R)0, ai = direct ? acc.im : (R)0;
          for (int q = 0; 4 * q < w; ++q, ++i) {
            const C4 c4 = i < a.keep ? wsm[i * threads] : __ldg(cp + 32 * q);
            const int m = min(4, w - 4 * q);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              if (u < m) {
                int k = Codes4<CB>::at(c4, u);
                if constexpr (RI) {  // FP64-bound: skip a position that is padding everywhere
                  if (!__any_sync(0xffffffffu, k != 0)) continue;
                }
                k = t0 + (k < tn ? k : 0);  // a table index of this group whatever the code
                dict_mac<RI, false>(tval, toff, x, k, row, last_col, ar, ai);
              }
            }
          }
          if (direct) acc = cx<R>{ar, ai};
          else coef_mac(acc, coef[s][g], ar, ai);
        }
      }
    }
    if (owner) {
      st_cx(ksm + s * rows, acc);
      const ST kq = ksm[s * rows];
      kg[(size_t)s * n64] = kq;
      if constexpr (HERM) tk[t_own * PAD + (tid & 31)] = ST{kq.x, -kq.y};
      if (s == RK_STEP - 1) {
        const unsigned int nz = nz_s[s], ne = nz_s[RK_EXTRA_STEP];
        if constexpr (MIXED) {
          Sum inc{cx<R>{0, 0}};
          float erh = 0.f, erl = 0.f, eih = 0.f, eil = 0.f;
          for (int j = 0; j < RK_STEP; ++j) {
            const cx<R> kj = ld_cx<R>(ksm + j * rows);
            if ((nz >> j) & 1u) inc.add(fac[s][j], low(s, j), kj);
            if ((ne >> j) & 1u) {  // the error estimate in float-float
              ff_acc(erh, erl, fe_s[j], fel_s[j], (float)kj.re);
              ff_acc(eih, eil, fe_s[j], fel_s[j], (float)kj.im);
            }
          }
          const double2 yp = static_cast<const double2*>(rk.y_prev)[row];
          const double2 dy = inc.wide();
          const double2 yf = make_double2(yp.x + dy.x, yp.y + dy.y);
          static_cast<double2*>(rk.y_front)[row] = yf;
          static_cast<float2*>(rk.y_front_s)[row] = make_float2((float)yf.x, (float)yf.y);
          if constexpr (HERM) ty[t_own * YPAD + (tid & 31)] = make_double2(yf.x, -yf.y);
          const double er = (double)erh + (double)erl, ei = (double)eih + (double)eil;
          err_acc = wrms_term(er * er + ei * ei, yf.x * yf.x + yf.y * yf.y, rk.atol, rk.rtol);
        } else {
          Sum y{base};
          cx<R> e{0, 0};
          for (int j = 0; j < RK_STEP; ++j) {
            const cx<R> kj = ld_cx<R>(ksm + j * rows);
            if ((nz >> j) & 1u) y.add(fac[s][j], low(s, j), kj);
            if ((ne >> j) & 1u) cx_axpy(e, fe_s[j], kj);
          }
          YT yq;
          st_cx(&yq, y.value());
          static_cast<YT*>(rk.y_front)[row] = yq;
          if constexpr (HERM) ty[t_own * YPAD + (tid & 31)] = YT{yq.x, -yq.y};
          const cx<R> ys = ld_cx<R>(&yq);
          const double mag2 = (double)ys.re * ys.re + (double)ys.im * ys.im;
          const double sc = rk.atol + rk.rtol * sqrt(mag2);
          err_acc = ((double)e.re * e.re + (double)e.im * e.im) / (sc * sc);
        }
      } else if (s + 1 < a.s1) {
        form_input(s);
      }
      if constexpr (HERM) {
        if (mirrored) err_acc *= 2.0;  // the mirrored element has the same term
      }
    }
    if constexpr (HERM) {
      __syncthreads();
      if (mirrored) {
        static_cast<ST*>(rk.k)[(size_t)s * n64 + mirror] = tk[t_from * PAD + l_from];
        if (s == RK_STEP - 1) herm_mirror_front<DT, YDT>(mirror, ty[t_from * YPAD + l_from], rk);
        else if (s + 1 < a.s1) mirror_input(s);
      }
    }
    if (s + 1 < a.s1) {
      target += gridDim.x;
      ok = grid_barrier(a.bar, target, a.wait, &ok_s);
    }
  }
  if (!ok) {
    const R none = (R)__longlong_as_double(0x7ff8000000000000LL);
    for (int s = a.s0; s < a.s1; ++s) {
      if (owner) kg[(size_t)s * n64] = ST{none, none};
      if constexpr (HERM) {
        if (mirrored) static_cast<ST*>(rk.k)[(size_t)s * n64 + mirror] = ST{none, none};
      }
    }
    if (tid == 0) {
      atomicOr(&g_step_fault, 1u);
      if (rk.result) *rk.result = -1.0;
    }
    return;
  }
  if (a.s1 != RK_STEP) return;
  // WRMS error: block partials, summed in block order by the block that finishes last
  __syncthreads();
  double v = err_acc;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((tid & 31) == 0) red[tid >> 5] = v;
  __syncthreads();
  if (tid == 0) {
    double t = 0.0;
    for (int w = 0; w < threads / 32; ++w) t += red[w];
    rk.scratch[blockIdx.x] = t;
    __threadfence();
    last_s = atomicAdd(rk.counter, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last_s || tid >= 32) return;
  __threadfence();
  double t = 0.0;
  for (int i = tid; i < (int)gridDim.x; i += 32) t += __ldcg(rk.scratch + i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
  if (tid == 0) {
    *rk.result = sqrt(t / (double)n);
    *rk.counter = 0u;
  }
}

constexpr int STEP_MAX_SMEM = 220 * 1024;

// 1 when the launch does not fit (the caller then takes one launch per stage).
template <int DT, int YDT, int KIND, int LANES, int PARTS = 1, bool HERM = false>
static int launch_range(StepArgs& a, uint32_t* bar_base, cudaStream_t st) {
  using ST = typename elem<DT>::T;
  const int64_t sms = sm_count();
  int64_t warps = (a.A.n_rows * LANES + 31) / 32;
  if (HERM) {
    const int64_t nt = a.herm_d / 32;
    warps = 2 * nt * (nt + 1) * HERM_WARPS;
  }
  int64_t per = (warps + sms - 1) / sms;  // warps of a block, one block per SM
  if (per < STEP_MIN_WARPS) per = STEP_MIN_WARPS;
  if (HERM) per = (per + HERM_WARPS - 1) / HERM_WARPS * HERM_WARPS;
  if (per * 32 > STEP_THREADS) return 1;
  const int threads = (int)per * 32, rows = threads / LANES;
  const int grid = (int)((warps + per - 1) / per);
  a.keep = step_keep(a.A, KIND, LANES);
  auto bytes = [&] { return step_smem<ST>(a.A, KIND, threads, rows, a.keep, HERM).total; };
  int smem = bytes();
  for (; smem > STEP_MAX_SMEM && a.keep > 2; smem = bytes()) a.keep = a.keep > 4 ? a.keep / 2 : 2;
  if (smem > STEP_MAX_SMEM) return 1;
  auto kern = vern7_range_kernel<DT, YDT, KIND, LANES, PARTS, HERM>;
  static std::mutex mu;
  static bool opted[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
    return set_error(QG_ERR_CUDA, "no current CUDA device");
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!opted[dev]) {
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               STEP_MAX_SMEM) != cudaSuccess)
        return set_error(QG_ERR_CUDA, "fused step kernel: shared memory opt-in failed");
      opted[dev] = true;
    }
  }
  a.bar_base = *bar_base;
  void* args[] = {&a};
  if (cudaLaunchCooperativeKernel((const void*)kern, dim3((unsigned)grid), dim3((unsigned)threads),
                                  args, (size_t)smem, st) != cudaSuccess)
    return check_launch("vern7_range_kernel");
  const int barriers = (a.s1 - a.s0 - 1) + (a.s0 > 0 ? 1 : 0);
  if (grid > 1) *bar_base += (uint32_t)(barriers * grid);
  return check_launch("vern7_range_kernel");
}

template <int DT, int YDT, int KIND>
static int launch_range_dict(StepArgs& a, uint32_t* bar_base, cudaStream_t st) {
  return a.herm_d > 0 ? launch_range<DT, YDT, KIND, 1, 1, true>(a, bar_base, st)
                      : launch_range<DT, YDT, KIND, 1>(a, bar_base, st);
}

template <int DT, int YDT>
static int launch_range_layout(StepArgs& a, uint32_t* bar_base, cudaStream_t st) {
  const qg_csr_groups& A = a.A;
  switch (A.layout) {
    case QG_LAYOUT_ROW_MAJOR:
      // Four lanes as two threads of two sums each: half the FP64 instructions of the
      // coefficients and the stage combination, where one thread of four sums leaves too few
      // warps to hide the gathers (Bose-Hubbard, d = 125: 4 x 1 5.05 ms a solve, 2 x 2
      // 4.48, 1 x 4 5.57).
      switch (A.lanes) {
        case 2: return launch_range<DT, YDT, KIND_CSR, 2>(a, bar_base, st);
        case 4: return launch_range<DT, YDT, KIND_CSR, 2, 2>(a, bar_base, st);
        case 8: return launch_range<DT, YDT, KIND_CSR, 8>(a, bar_base, st);
        default: return 1;
      }
    case QG_LAYOUT_SLICED: return launch_range<DT, YDT, KIND_SLICED, 1>(a, bar_base, st);
    case QG_LAYOUT_SLICED_DICT:
      if constexpr (DT == QG_C128) return 1;  // complex128 dictionaries are split
      return A.tile_nnz == 1 ? launch_range_dict<DT, YDT, KIND_DICT1>(a, bar_base, st)
                             : launch_range_dict<DT, YDT, KIND_DICT2>(a, bar_base, st);
    case QG_LAYOUT_SLICED_DICT_RI:
      if constexpr (DT != QG_C128) return 1;
      return A.tile_nnz == 1 ? launch_range_dict<DT, YDT, KIND_DICT1>(a, bar_base, st)
                             : launch_range_dict<DT, YDT, KIND_DICT2>(a, bar_base, st);
    default: return 1;
  }
}

}  // namespace qg

using namespace qg;

int step_fault_take() {
  unsigned int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_step_fault, sizeof(v)) != cudaSuccess) return 0;
  if (v) cudaMemcpyToSymbol(g_step_fault, &zero, sizeof(zero));
  return (int)v;
}

// d > 0: the half form of a d x d state; A has been checked.
static int vern7_range(const qg_csr_groups* A, const qg_rk_buffers* B, int stage0, int stage1,
                       double t_prev, double dt, double atol, double rtol, int64_t d,
                       int32_t wait_mcycles, unsigned int* barrier, uint32_t* barrier_base,
                       void* stream) {
  if (!barrier || !barrier_base) return set_error(QG_ERR_ARG, "null barrier word");
  if (A->n_rows != A->n_cols) return set_error(QG_ERR_ARG, "operator must be square with n rows");
  if (!((stage0 == 0 && stage1 == RK_STEP) || (stage0 == RK_STEP && stage1 == RK_EXTRA_STEP)))
    return set_error(QG_ERR_ARG, "stages must be a whole trial step or the dense-output stages");
  StepArgs a{};
  const void* x = nullptr;
  const int rc = prepare_stage(B, A->dtype, A->n_rows, stage0 == 0 ? RK_STEP - 1 : stage0, dt, atol,
                               rtol, a.rk, x);
  if (rc) return rc;
  if (B->n == 0) return 1;
  a.A = *A;
  a.x0 = B->state_dtype != B->stage_dtype ? B->y_prev_s : B->y_prev;
  a.ytmp = B->ytmp;
  a.t_prev = t_prev;
  a.dt = dt;
  a.s0 = stage0;
  a.s1 = stage1;
  a.bar = barrier;
  a.herm_d = (int)d;
  a.wait = wait_mcycles > 0 ? 1000000LL * wait_mcycles : STEP_WAIT_CYCLES;
  cudaStream_t st = (cudaStream_t)stream;
  if (B->state_dtype == QG_C128 && B->stage_dtype == QG_C128)
    return launch_range_layout<QG_C128, QG_C128>(a, barrier_base, st);
  if (B->state_dtype == QG_C128) return launch_range_layout<QG_C64, QG_C128>(a, barrier_base, st);
  return launch_range_layout<QG_C64, QG_C64>(a, barrier_base, st);
}

int qg::range_csr(const qg_csr_groups* A, const qg_rk_buffers* B, int stage0, int stage1,
                  double t_prev, double dt, double atol, double rtol, int64_t d,
                  int32_t wait_mcycles, unsigned int* barrier, uint32_t* barrier_base,
                  void* stream) {
  const int rc = d > 0 ? check_herm(A, d) : check_groups(A);
  return rc ? rc : vern7_range(A, B, stage0, stage1, t_prev, dt, atol, rtol, d, wait_mcycles,
                               barrier, barrier_base, stream);
}

extern "C" int qg_vern7_range(const qg_csr_groups* A, const qg_rk_buffers* B, int stage0,
                              int stage1, double t_prev, double dt, double atol, double rtol,
                              unsigned int* barrier, uint32_t* barrier_base, void* stream) {
  return range_csr(A, B, stage0, stage1, t_prev, dt, atol, rtol, 0, 0, barrier, barrier_base,
                   stream);
}

extern "C" int qg_vern7_range_herm(const qg_csr_groups* A, const qg_rk_buffers* B, int stage0,
                                   int stage1, double t_prev, double dt, double atol, double rtol,
                                   int64_t d, unsigned int* barrier, uint32_t* barrier_base,
                                   void* stream) {
  const int rc = check_herm(A, d);  // d <= 0 among what it refuses
  return rc ? rc : range_csr(A, B, stage0, stage1, t_prev, dt, atol, rtol, d, 0, barrier,
                             barrier_base, stream);
}
