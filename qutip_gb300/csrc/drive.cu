// Host driver of one system's integration (qg_vern7_integrate, qg_vern7_run_dm): the control
// flow of Explicit_RungeKutta (qutip/solver/integrator/explicit_rk.pyx:278-467) around the
// stage launches of this library.  A step of a small system is tens of microseconds on the
// GPU; the same loop in the host language above spent 65 us a step between the launches, on
// building arguments, reading the error norm back and asking for the outputs.  The error
// norm goes straight to a word of pinned host memory that the loop watches; a second word
// tells of a dense-output launch that gave up, which the loop does not wait for.  Measured, whole
// solves: Jaynes-Cummings N = 10 5.4 -> 2.8 ms, Bose-Hubbard d = 125 6.2 -> 4.8, Ising L = 8
// 27.4 -> 24.9, L = 10 mixed 66 -> 61 (matrix form 98 -> 92), dense d = 128 7.9 -> 7.3.
#include <math.h>

#include <atomic>
#include <chrono>

#include "capi_internal.h"
#include "common.cuh"
#include "qutip_gb300.h"
#include "rows.cuh"
#include "vern7_tableau.cuh"

namespace qg {

// The watched word holds this until the step's error norm (>= 0, or -1) arrives.
constexpr double NOT_YET = -2.0;
constexpr int WATCH = 200000;  // looks at the word before the stream is waited for instead

// Coefficients of the stages that go out one launch each, evaluated in one launch before them.
// A program is 2 to 4 us of dependent loads and FP64 work (one multiplication and a cosine:
// 2 us beyond a constant's 1) that every block of every stage repeated at its start, several
// at once on an SM's FP64 pipe; here the stages of a step are evaluated side by side, by the
// same operations at the same t.  (The dense generator evaluates them beside its loads: no
// gain there, and no table.)  Measured, whole solves of the L = 10 Ising chain: complex128
// 165 -> 158 ms, mixed 61 -> 58, mixed in matrix form 74 -> 70.
struct CoefProgram {
  const int *code, *start;
  const double* consts;
  int n;
};
struct CoefPrograms {
  CoefProgram groups, cops;
  double t[RK_EXTRA_STEP];
};
constexpr int COEF_THREADS = (QG_MAX_GROUPS + QG_MAX_COPS + 31) / 32 * 32;

__global__ void __launch_bounds__(COEF_THREADS)
    coef_table_kernel(const __grid_constant__ CoefPrograms p, int s0, cplx* out) {
  const int s = s0 + blockIdx.x, i = threadIdx.x, n = p.groups.n + p.cops.n;
  if (i >= n) return;
  const CoefProgram& q = i < p.groups.n ? p.groups : p.cops;
  const int g = i < p.groups.n ? i : i - p.groups.n;
  out[s * n + i] = prog_coef(q.code, q.start, q.consts, g, p.t[s]);
}

struct Drive {
  const qg_generator* gen;
  qg_rk_buffers* B;
  qg_vern7_ctl* c;
  void* stream;

  using Clock = std::chrono::steady_clock;
  const Clock::time_point start = Clock::now();
  // Whether the call has run for its slice of time: a caller that waits for signals (an
  // interrupt) gets them between calls.
  bool late() const {
    return c->slice > 0.0 &&
           std::chrono::duration<double>(Clock::now() - start).count() >= c->slice;
  }

  int n_coefs = 0;  // coefficients of a stage in the table; 0: no table

  // The coefficients of stages [s0, s1), one block a stage.
  int coefs(int s0, int s1, double dt) {
    CoefPrograms p{};
    if (gen->kind == QG_GEN_CSR) {
      const auto* A = static_cast<const qg_csr_groups*>(gen->op);
      p.groups = {A->coef_code, A->coef_start, A->coef_consts, A->n_groups};
    } else if (gen->kind == QG_GEN_LINDBLAD) {
      const auto* L = static_cast<const qg_lindblad*>(gen->op);
      p.groups = {L->a_coef_code, L->a_coef_start, L->a_coef_consts, L->n_groups};
      p.cops = {L->c_coef_code, L->c_coef_start, L->c_coef_consts, L->n_cops};
    }
    const int n = p.groups.n + p.cops.n;
    n_coefs = 0;
    if (!c->coef_table || (!p.groups.code && !p.cops.code) || n < 1 ||
        n > QG_MAX_GROUPS + QG_MAX_COPS)
      return QG_OK;
    for (int s = s0; s < s1; ++s) p.t[s] = c->t_prev + VERN7_C_HOST[s] * dt;
    coef_table_kernel<<<s1 - s0, COEF_THREADS, 0, (cudaStream_t)stream>>>(
        p, s0, reinterpret_cast<cplx*>(c->coef_table));
    ++c->launches;
    n_coefs = n;
    return check_launch("coef_table_kernel");
  }

  int stage(int s, double dt) {
    ++c->launches;
    const double* k = n_coefs ? c->coef_table + 2 * (size_t)s * n_coefs : nullptr;
    switch (gen->kind) {
      case QG_GEN_CSR: {
        const qg_csr_groups* A = static_cast<const qg_csr_groups*>(gen->op);
        if (gen->hermitian_d > 0)
          return stage_herm(A, gen->hermitian_d, B, s, c->t_prev, dt, c->atol, c->rtol, k, stream);
        return stage_csr(A, B, s, c->t_prev, dt, c->atol, c->rtol, k, stream);
      }
      case QG_GEN_LINDBLAD:
        return stage_lindblad(static_cast<const qg_lindblad*>(gen->op), B, s, c->t_prev, dt,
                              c->atol, c->rtol, k, stream);
      default:
        return qg_dense_lindblad_stage(static_cast<const qg_dense_lindblad*>(gen->op), B, s,
                                       c->t_prev, dt, c->atol, c->rtol, stream);
    }
  }

  // stages [s0, s1): 0 when they went out in one launch, 1 when they do not fit one
  int range(int s0, int s1, double dt) {
    if (gen->kind != QG_GEN_CSR) return 1;
    const auto* A = static_cast<const qg_csr_groups*>(gen->op);
    const int rc = range_csr(A, B, s0, s1, c->t_prev, dt, c->atol, c->rtol,
                             gen->hermitian_d > 0 ? gen->hermitian_d : 0, c->wait_mcycles,
                             c->barrier, &c->barrier_base, stream);
    if (rc == 0) ++c->launches;
    return rc;
  }

  int trial(double dt, double& err) {
    volatile double* word = c->host_result;
    double* const device_result = B->result;
    *word = NOT_YET;
    B->result = c->host_result;
    int rc = range(0, RK_STEP, dt);
    if (rc == 1) {
      rc = coefs(0, RK_STEP, dt);
      for (int s = 0; s < RK_STEP && rc == QG_OK; ++s) rc = stage(s, dt);
    }
    B->result = device_result;
    if (rc != QG_OK) return rc;
    c->rhs += RK_STEP;
    c->t_front = c->t_prev + dt;
    for (int i = 0; i < WATCH && *word == NOT_YET; ++i) {
    }
    if (*word == NOT_YET && cudaStreamSynchronize((cudaStream_t)stream) != cudaSuccess)
      return check_launch("vern7 trial step");
    err = *word;
    if (err == NOT_YET) return set_error(QG_ERR_CUDA, "the step's error norm did not arrive");
    std::atomic_thread_fence(std::memory_order_acquire);
    if (err < 0.0 || dense_gave_up()) return gave_up();
    return QG_OK;
  }

  // The waits of a dense-output launch: known once the launch is over, so looked at after the
  // next trial step's wait, and by the caller after its own.
  bool dense_gave_up() const {
    return const_cast<volatile double*>(c->host_result)[1] < 0.0;
  }

  int gave_up() {
    // every block leaves within the same limit, and may still write the words until then
    cudaStreamSynchronize((cudaStream_t)stream);
    c->host_result[1] = 0.0;
    c->status = QG_DEVICE_WAIT;
    return set_error(QG_ERR_CUDA,
                     "a device wait of the fused step kernel gave up; the GPU may be unhealthy");
  }

  // _prep_dense_out (explicit_rk.pyx:399-410)
  int dense_out() {
    const double dt = c->dt_int;
    double* const device_result = B->result;
    B->result = c->host_result + 1;  // written when a wait gives up
    int rc = range(RK_STEP, RK_EXTRA_STEP, dt);
    B->result = device_result;
    if (rc == 1) {
      qg_state_view v = {};
      const bool mixed = B->state_dtype != B->stage_dtype;
      v.n = B->n;
      v.base_dtype = v.k_dtype = B->stage_dtype;
      v.base = mixed ? B->y_prev_s : B->y_prev;
      v.k = B->k;
      v.n_k = RK_STEP;
      for (int j = 0; j < RK_STEP; ++j) v.f[j] = dt * VERN7_A_HOST[RK_STEP][j];
      const size_t es = B->stage_dtype == QG_C128 ? 16 : 8;
      ++c->launches;
      rc = qg_rk_combine(&v, (char*)B->ytmp + (RK_STEP & 1) * (size_t)B->n * es, B->stage_dtype,
                         stream);
      if (rc == QG_OK) rc = coefs(RK_STEP, RK_EXTRA_STEP, dt);
      for (int s = RK_STEP; s < RK_EXTRA_STEP && rc == QG_OK; ++s) rc = stage(s, dt);
    }
    c->rhs += RK_EXTRA_STEP - RK_STEP;
    return rc;
  }

  // _get_timestep (explicit_rk.pyx:440-449)
  double timestep(double t) const {
    const double need = t - c->t_prev;
    if (c->interpolate || need <= c->dt_safe) return c->interpolate ? c->dt_safe : need;
    return need / (trunc(need / c->dt_safe) + 1.0);
  }

  // _recompute_safe_step (explicit_rk.pyx:451-467)
  void safe_step(double err, double dt) {
    double factor = 10.0;
    if (err != 0.0) {
      factor = 0.9 * pow(err, -1.0 / (RK_ORDER + 1));
      factor = factor < 10.0 ? factor : 10.0;
      factor = factor > 0.2 ? factor : 0.2;
    }
    c->dt_safe = dt * factor;
    if (c->max_step != 0.0 && !(c->dt_safe < c->max_step)) c->dt_safe = c->max_step;
    if (c->min_step != 0.0 && !(c->dt_safe > c->min_step)) c->dt_safe = c->min_step;
  }

  // _step_in_err (explicit_rk.pyx:333-356)
  int step_in_err(double t, int64_t limit, int64_t& nsteps) {
    double err = 1.0;
    nsteps = 0;
    while (err >= 1.0) {
      const double dt = timestep(t);
      const int rc = trial(dt, err);
      if (rc != QG_OK) return rc;
      c->dt_int = dt;
      safe_step(err, dt);
      if (dt == c->min_step && err > 1.0) {
        c->status = QG_DT_UNDERFLOW;
        break;
      }
      ++nsteps;
      ++c->steps;
      if (err >= 1.0) ++c->rejected;
      if (nsteps > limit) {
        c->status = QG_TOO_MUCH_WORK;
        break;
      }
    }
    return QG_OK;
  }

  void swap() {
    void* y = const_cast<void*>(B->y_prev);
    B->y_prev = B->y_front;
    B->y_front = y;
    void* s = const_cast<void*>(B->y_prev_s);
    B->y_prev_s = B->y_front_s;
    B->y_front_s = s;
    c->swaps ^= 1;
  }

  // integrate (explicit_rk.pyx:278-331)
  int integrate(double t, int step) {
    int64_t left = c->left;
    if (c->paused == 1) {
      c->paused = 0;  // goes on in the loop below
    } else {
      if (t == c->t) return QG_OK;
      if (t < c->t_prev) {
        c->status = QG_OUTSIDE_RANGE;
        return QG_OK;
      }
      if (c->interpolate && t < c->t_front) {
        if (c->status != QG_INTERPOLATED) {
          const int rc = dense_out();
          if (rc != QG_OK) return rc;
          c->status = QG_INTERPOLATED;
        }
        c->interp = 1;
        c->t = t;
        return QG_OK;
      }
      left = c->max_numsteps;
      c->status = QG_NORMAL;
      if (step && c->t < c->t_front && t > c->t_front) t = c->t_front;
    }
    while (c->t_front < t && c->status >= 0) {
      swap();
      c->t_prev = c->t_front;
      int64_t n = 0;
      const int rc = step_in_err(t, left, n);
      if (rc != QG_OK) return rc;
      left -= n;
      if (step) break;
      if (c->t_front < t && c->status >= 0 && late()) {
        c->left = left;
        c->paused = 1;
        return QG_OK;
      }
    }
    if (c->status < 0) return QG_OK;
    if (c->t_front > t) {
      const int rc = dense_out();
      if (rc != QG_OK) return rc;
      c->status = QG_INTERPOLATED;
      c->t = t;
      c->interp = 1;
    } else {
      c->status = QG_AT_FRONT;
      c->t = c->t_front;
      c->interp = 0;
    }
    return QG_OK;
  }
};

static int check_drive(const qg_generator* gen, const qg_rk_buffers* B, const qg_vern7_ctl* c) {
  if (!gen || !gen->op || !B || !c || !c->host_result || !c->barrier)
    return set_error(QG_ERR_ARG, "null pointer");
  if (gen->kind != QG_GEN_CSR && gen->kind != QG_GEN_LINDBLAD && gen->kind != QG_GEN_DENSE)
    return set_error(QG_ERR_ARG, "unknown generator kind");
  return QG_OK;
}

}  // namespace qg

using namespace qg;

extern "C" int qg_vern7_integrate(const qg_generator* gen, qg_rk_buffers* B, qg_vern7_ctl* c,
                                  double t, int step, void* stream) {
  const int rc = check_drive(gen, B, c);
  if (rc) return rc;
  Drive d{gen, B, c, stream};
  return d.integrate(t, step);
}

extern "C" int qg_vern7_run_dm(const qg_generator* gen, qg_rk_buffers* B, qg_vern7_ctl* c,
                               const double* tlist, int n_times, const qg_csr_groups* ops,
                               int64_t d, double* out, void* stream) {
  int rc = check_drive(gen, B, c);
  if (rc) return rc;
  if (n_times < 0 || (n_times > 0 && (!tlist || !ops || !out)))
    return set_error(QG_ERR_ARG, "null pointer");
  Drive dr{gen, B, c, stream};
  const int64_t row = n_times > 0 ? 2 * ((int64_t)ops->n_groups + 1) : 0;
  qg_state_view v = {};
  v.n = B->n;
  v.base_dtype = B->state_dtype;
  v.k_dtype = B->stage_dtype;
  v.k = B->k;
  int i = c->paused ? c->n_done : 0;
  if (c->paused == 2) c->paused = 0;
  while (i < n_times) {
    rc = dr.integrate(tlist[i], 0);
    c->n_done = i;
    if (rc != QG_OK || c->status < 0 || c->paused) return rc;
    ++c->launches;
    if (c->status != QG_INTERPOLATED) {
      // the state at the end of a step, or the time asked for again
      v.base = B->y_front;
      rc = qg_expect_dm(ops, d, &v, out + i * row, stream);
      if (rc != QG_OK) return rc;
      c->n_done = ++i;
      if (i < n_times && dr.late()) {
        c->paused = 2;
        return QG_OK;
      }
      continue;
    }
    // every following output time inside this step is read from its dense output
    double tau[QG_EXPECT_TIMES];
    int m = 0;
    while (m < QG_EXPECT_TIMES && i + m < n_times &&
           (m == 0 || (c->t_prev <= tlist[i + m] && tlist[i + m] < c->t_front))) {
      tau[m] = (tlist[i + m] - c->t_prev) / c->dt_int;
      ++m;
    }
    v.base = B->y_prev;
    rc = qg_expect_dm_times(ops, d, &v, m, tau, c->dt_int, out + i * row, B->scratch, B->counter,
                            stream);
    if (rc != QG_OK) return rc;
    c->t = tlist[i + m - 1];
    c->n_done = i += m;
    if (i < n_times && dr.late()) {
      c->paused = 2;
      return QG_OK;
    }
  }
  return QG_OK;
}
