"""Adaptive Verner-7 integrator on the GPU for one (large) system.

The control flow mirrors ``Explicit_RungeKutta`` (qutip/solver/integrator/explicit_rk.pyx:47-530)
step for step -- first-step estimate, ``integrate`` with ``step=True`` for
Monte-Carlo stepping, ``_step_in_err`` retries, interpolation past the target
with the 7th-order dense output -- so that the step sequence, and therefore the
result, is the reference's.  The vector work runs in these kinds of launches:

* ``qg_vern7_range`` -- all ten stages of a trial step, or the six dense-output stages, in
  one launch, for operators whose rows all fit the GPU at once;
* ``qg_vern7_stage`` -- otherwise one per stage: the matvec ``k_s = A(t_s) x_s`` fused
  with the next stage's input combination; the tenth fuses ``y_front`` and the
  FP64 WRMS error reduction (``wrmn_error_dense``, qutip/core/data/ode.pyx:27-52);
* ``qg_rk_combine`` -- dense-output stage input and materialised outputs;
* ``qg_norm2`` -- norms of the first-step estimate.

Precision forms: ``"double"`` (complex128 operator, stages and state),
``"mixed"`` (complex64 operator and stages with FP32 matvec accumulation, the
state ``y``, the stage combinations and the error control in FP64) and
``"single"`` (complex64 state as well; error control still FP64).  The scalar
step-size recurrences run on the host in IEEE double; the only per-step
device-to-host transfer is the 8-byte error norm.  For the library's own operators that
host loop is the library's (``qg_vern7_integrate``); the methods below are the same loop for
subclasses of them, for objects with a ``vern7_stage`` of their own and for any other operator
with ``matvec`` and ``vern7_stage``.  The package itself has none of these: there the loop below
is what the tests hold the library's against.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from . import _lib
from . import vern7_tableau as T
from .operator import DeviceOperator, qg_dtype, stream_ptr, torch_dtype

AT_FRONT, INTERPOLATED, NORMAL = 2, 1, 0
TOO_MUCH_WORK, DT_UNDERFLOW, OUTSIDE_RANGE, NOT_INITIATED = -1, -2, -3, -4
DEVICE_WAIT = _lib.QG_DEVICE_WAIT
STATUS_MESSAGES = {
    AT_FRONT: "Internal state at the desired time.",
    INTERPOLATED: "Internal state past the desired time and interpolation to step done.",
    NORMAL: "No work done.",
    TOO_MUCH_WORK: ("Too much work done in one call. Try to increase the nsteps parameter or "
                    "increasing the tolerance."),
    DT_UNDERFLOW: "Step size becomes too small. Try increasing tolerance.",
    OUTSIDE_RANGE: "Step outside available range.",
    NOT_INITIATED: "Not initialized.",
    DEVICE_WAIT: ("a device wait of the fused step kernel gave up; the GPU may be unhealthy"),
}
PRECISIONS = {"double": ("c128", "c128"), "mixed": ("c128", "c64"), "single": ("c64", "c64")}


class IntegratorError(RuntimeError):
    """Integration failure; the plugin layer re-raises it as ``IntegratorException``."""


class GpuVern7:
    """Single-system adaptive Vern7 on device buffers.

    ``op`` is a :class:`DeviceOperator` or a
    :class:`~qutip_gb300.lindblad.LindbladOperator` whose dtype is the stage dtype
    of ``precision``.
    """

    def __init__(self, op: DeviceOperator, atol=1e-8, rtol=1e-6, nsteps=1000, first_step=0.0,
                 min_step=0.0, max_step=0.0, interpolate=True, precision="double"):
        if precision not in PRECISIONS:
            raise ValueError(f"precision must be one of {sorted(PRECISIONS)}")
        self.state_dt, self.stage_dt = PRECISIONS[precision]
        if op.dtype != self.stage_dt:
            raise TypeError(f"precision {precision!r} needs a {self.stage_dt} operator")
        if op.n_rows != op.n_cols:
            raise ValueError("the generator must be square")
        self.op = op
        self.precision = precision
        self.atol, self.rtol = float(atol), float(rtol)
        # 64 bits in the library: what no integration counts to is as good as any larger limit
        self.max_numsteps = max(min(int(nsteps), 2**63 - 1), -2**63)
        self.first_step = float(first_step)
        self.min_step = float(min_step) or 1e-15       # explicit_rk.pyx:133
        self.max_step = float(max_step)
        self.interpolate = bool(interpolate)
        self.order = T.ORDER
        self.a = np.zeros((16, 16))
        for i, row in enumerate(T.A):
            self.a[i, :len(row)] = row
        self.b, self.c, self.e, self.bi = np.array(T.B), np.array(T.C), np.array(T.E), np.array(T.BI)
        n = op.n_rows
        self.n = n
        dev = op.device
        sdt, kdt = torch_dtype(self.state_dt), torch_dtype(self.stage_dt)
        self._ya = torch.zeros(n, dtype=sdt, device=dev)
        self._yb = torch.zeros(n, dtype=sdt, device=dev)
        self.y_out = torch.zeros(n, dtype=sdt, device=dev)
        self.k = torch.zeros(16 * n, dtype=kdt, device=dev)
        self.ytmp = torch.zeros(2 * n, dtype=kdt, device=dev)
        self.scratch = torch.zeros(int(_lib.load().qg_scratch_doubles()), dtype=torch.float64,
                                   device=dev)
        # word 0: reductions (left zero); word 1: arrivals at the fused step kernel's barrier
        self.counter = torch.zeros(4, dtype=torch.int32, device=dev)
        self._barrier_base = C.c_uint32(0)
        self.result = torch.zeros(4, dtype=torch.float64, device=dev)
        # word 0: the error norm; word 1: negative when a dense-output launch gave up
        self._host = torch.zeros(4, dtype=torch.float64).pin_memory()
        self._words = self._host.numpy()
        self._wait_mcycles = 0           # limit of a wait; 0: the library's
        self._slice = 0.05               # seconds between looks at the interpreter's signals
        self._coefs = torch.empty(_lib.QG_COEF_TABLE, dtype=torch.float64, device=dev)
        self.y_prev, self.y_front = self._ya, self._yb
        # mixed form: complex64 copies of y_prev / y_front (stage inputs), swapped with them
        self.mixed = self.state_dt != self.stage_dt
        if self.mixed:
            self.y_prev_s = torch.zeros(n, dtype=kdt, device=dev)
            self.y_front_s = torch.zeros(n, dtype=kdt, device=dev)
        else:
            self.y_prev_s = self.y_front_s = None
        self._set = False
        self._hermitian = False   # decided for each initial value
        self.status = NOT_INITIATED
        self.stats = {"steps": 0, "rejected": 0, "rhs": 0}
        self._out = ("front", None)  # how the state at self.t is obtained

    # -- buffers ---------------------------------------------------------
    def _rk(self) -> _lib.RkBuffers:
        ps = self.y_prev_s.data_ptr() if self.mixed else None
        fs = self.y_front_s.data_ptr() if self.mixed else None
        return _lib.RkBuffers(self.n, qg_dtype(self.state_dt), qg_dtype(self.stage_dt),
                              self.y_prev.data_ptr(), self.y_front.data_ptr(), ps, fs,
                              self.k.data_ptr(), self.ytmp.data_ptr(), self.scratch.data_ptr(),
                              self.counter.data_ptr(), self.result.data_ptr())

    def _swap(self):
        self.y_prev, self.y_front = self.y_front, self.y_prev
        if self.mixed:
            self.y_prev_s, self.y_front_s = self.y_front_s, self.y_prev_s

    def _view(self, base: torch.Tensor, factors=()) -> _lib.StateView:
        f = (C.c_double * 16)(*([float(x) for x in factors] + [0.0] * (16 - len(factors))))
        return _lib.StateView(self.n, qg_dtype(self.state_dt if base.dtype == torch_dtype(
            self.state_dt) else self.stage_dt), qg_dtype(self.stage_dt), base.data_ptr(),
            self.k.data_ptr(), len(factors), 0, f)

    def _combine(self, base, factors, out):
        v = self._view(base, factors)
        _lib.call("qg_rk_combine", C.byref(v), out.data_ptr(),
                  qg_dtype("c128" if out.dtype == torch.complex128 else "c64"), stream_ptr())

    def _read_result(self) -> float:
        self._host[:1].copy_(self.result[:1], non_blocking=True)
        torch.cuda.current_stream().synchronize()
        return float(self._host[0])

    def _norm(self, x: torch.Tensor) -> float:
        _lib.call("qg_norm2", x.data_ptr(), qg_dtype("c128" if x.dtype == torch.complex128 else "c64"),
                  x.numel(), self.scratch.data_ptr(), self.counter.data_ptr(),
                  self.result.data_ptr(), stream_ptr())
        return math.sqrt(self._read_result())

    def _k(self, j) -> torch.Tensor:
        return self.k[j * self.n:(j + 1) * self.n]

    def _ytmp(self, j) -> torch.Tensor:
        return self.ytmp[j * self.n:(j + 1) * self.n]

    def _deriv_into(self, t, x_stage: torch.Tensor, j: int):
        self.op.matvec(t, x_stage, self._k(j))
        self.stats["rhs"] += 1

    # -- reference algorithm ----------------------------------------------
    def set_initial_value(self, y0, t: float):
        """``set_initial_value`` (explicit_rk.pyx:204-230); copies ``y0``."""
        y0 = torch.as_tensor(y0)
        if y0.numel() != self.n:
            raise ValueError(f"state of size {y0.numel()} for a generator of size {self.n}")
        if self._words[1] < 0:                      # of the state before: nothing to it any more
            self._reset_waits()
        self.y_prev.copy_(y0.reshape(-1).to(self.y_prev.device, self.y_prev.dtype))
        self.y_front.copy_(self.y_prev)
        if self.mixed:
            self._combine(self.y_prev, (), self.y_prev_s)
            self.y_front_s.copy_(self.y_prev_s)
        self.t = self.t_prev = self.t_front = float(t)
        self.dt_int = 0.0
        self._out = ("front", None)
        self.status = NORMAL
        self._set = True
        dim = getattr(self.op, "hermitian_dim", None)
        self._hermitian = (dim is not None and dim() > 0 and self.op.real_coefficients()
                           and self.op.check_hermitian(self.y_prev))
        self.dt_safe = self._estimate_first_step(self.t, self.y_prev) if not self.first_step \
            else self.first_step

    def _stage_input(self, y: torch.Tensor) -> torch.Tensor:
        if y.dtype == torch_dtype(self.stage_dt):
            return y
        self._combine(y, (), self._ytmp(0))
        return self._ytmp(0)

    def _stage_base(self) -> torch.Tensor:
        """Base of the stage combinations: y_prev, or its complex64 copy when mixed."""
        return self.y_prev_s if self.mixed else self.y_prev

    def _estimate_first_step(self, t, y0):
        # explicit_rk.pyx:232-276
        norm = self._norm(y0)
        tol = self.atol + norm * self.rtol
        self._deriv_into(t, self._stage_input(y0), 0)
        if norm <= self.atol:
            norm = 1
        tmp = self._norm(self._k(0))
        fact = math.factorial(self.order)
        if tmp >= self.atol * 1e-6:
            dt1 = (tol * fact * norm ** self.order) ** (1 / (self.order + 1)) / tmp
        else:
            dt1 = (tol * fact) ** (1 / (self.order + 1)) * norm * 0.5
        t1 = t + dt1 / 100
        self._combine(y0, [dt1 / 100], self._ytmp(1))
        self._deriv_into(t1, self._ytmp(1), 1)
        tmp = self._norm(self._k(1))
        if tmp >= self.atol * 1e-6:
            dt2 = (tol * fact * norm ** self.order) ** (1 / (self.order + 1)) / tmp
        else:
            dt2 = dt1
        dt = min(dt1, dt2)
        if self.max_step:
            dt = min(self.max_step, dt)
        if self.min_step:
            dt = max(self.min_step, dt)
        return dt

    def integrate(self, t: float, step: bool = False):
        """``integrate`` (explicit_rk.pyx:278-331)."""
        t = float(t)
        nsteps_left = self.max_numsteps
        if not self._set:
            self.status = NOT_INITIATED
            return
        self._check_waits()
        gen = self._generator()
        if gen is not None:
            self._drive("qg_vern7_integrate", gen, t, int(step))
            return
        if t == self.t:
            return
        if t < self.t_prev:
            self.status = OUTSIDE_RANGE
            return
        if self.interpolate and t < self.t_front:
            if self.status != INTERPOLATED:
                self._prep_dense_out()
                self.status = INTERPOLATED
            self._set_interp(t)
            self.t = t
            return
        self.status = NORMAL
        if step and self.t < self.t_front and t > self.t_front:
            t = self.t_front
        while self.t_front < t and self.status >= 0:
            # y_prev <- y_front: swap the buffers (the old y_prev is dead)
            self._swap()
            self.t_prev = self.t_front
            nsteps_left -= self._step_in_err(t, nsteps_left)
            if step:
                break
        if self.status < 0:
            return
        if self.t_front > t:
            self._prep_dense_out()
            self.status = INTERPOLATED
            self.t = t
            self._set_interp(t)
        else:
            self.status = AT_FRONT
            self.t = self.t_front
            self._out = ("front", None)

    # -- the same loop in the library ---------------------------------------
    def _generator(self):
        """The operator as the library's driver takes it (``qg_vern7_integrate``); None for
        an operator that is not one of the library's own or whose ``vern7_stage`` was replaced,
        which the loops here then drive."""
        from .dense import DenseLindbladOperator
        from .lindblad import LindbladOperator
        cls = type(self.op)
        kind = {DeviceOperator: _lib.QG_GEN_CSR, LindbladOperator: _lib.QG_GEN_LINDBLAD,
                DenseLindbladOperator: _lib.QG_GEN_DENSE}.get(cls)
        if kind is None or not self._stages_of(cls):
            return None
        return _lib.Generator(kind, 0, C.addressof(self.op.struct),
                              math.isqrt(self.n) if self._half() else 0)

    def _drive(self, name, gen, *args):
        """Call a driver of the library on this integrator's buffers and scalar state."""
        rk = self._rk()
        c = _lib.Vern7Ctl(self.t, self.t_prev, self.t_front, self.dt_safe, self.dt_int, self.atol,
                          self.rtol, self.min_step, self.max_step, self.max_numsteps,
                          self.stats["steps"], self.stats["rejected"], self.stats["rhs"], 0,
                          self.status, int(self.interpolate), int(self._out[0] == "interp"), 0,
                          self._barrier_base.value, self._wait_mcycles,
                          self.counter.data_ptr() + 4,
                          self._host.data_ptr(), self._coefs.data_ptr())
        c.slice = self._slice
        run = getattr(_lib.load(), name)
        while True:                   # an interrupt is raised between the calls
            try:
                rc = run(C.byref(gen), C.byref(rk), C.byref(c), *args, stream_ptr())
            finally:
                self._take(c)
            if not c.paused:
                break
        if rc != _lib.QG_OK and c.status == DEVICE_WAIT:
            self._wait_gave_up()
        _lib.check(rc, name)
        if c.status >= 0:
            if c.interp:
                self._set_interp(self.t)
            else:
                self._out = ("front", None)

    def _take(self, c):
        """The scalar state after a call of the library's driver."""
        _lib.LAUNCHES[0] += c.launches
        if c.swaps:
            self._swap()
        c.launches = c.swaps = 0
        self.t, self.t_prev, self.t_front = c.t, c.t_prev, c.t_front
        self.dt_safe, self.dt_int, self.status = c.dt_safe, c.dt_int, c.status
        self.stats.update(steps=c.steps, rejected=c.rejected, rhs=c.rhs)
        self._barrier_base.value = c.barrier_base

    def run_dm(self, tlist, ops, d: int, out: torch.Tensor) -> bool:
        """Integrate to each of ``tlist`` and record ``ops``' expectation values, one row of
        ``out`` per time, up to the first failure; False when the loops here must do it.
        :meth:`check` after ``out`` was read tells whether all of it is valid."""
        gen = self._generator()
        if gen is None or not self._set:
            return False
        self._check_waits()
        tl = np.ascontiguousarray(tlist, dtype=np.float64)
        self._drive("qg_vern7_run_dm", gen, tl.ctypes.data, len(tl), C.byref(ops.struct), d,
                    out.data_ptr())
        return True

    def _step_in_err(self, t, max_step):
        # explicit_rk.pyx:333-356
        error = 1.0
        nsteps = 0
        while error >= 1:
            dt = self._get_timestep(t)
            error = self._compute_step(dt)
            self.dt_int = dt
            self._recompute_safe_step(error, dt)
            if dt == self.min_step and error > 1:
                self.status = DT_UNDERFLOW
                break
            nsteps += 1
            self.stats["steps"] += 1
            if error >= 1:
                self.stats["rejected"] += 1
            if nsteps > max_step:
                self.status = TOO_MUCH_WORK
                break
        return nsteps

    def _compute_step(self, dt):
        # explicit_rk.pyx:358-397: ten fused stages; the last returns the error
        rk = self._rk()
        s = stream_ptr()
        fused = self._range(rk, 0, T.RK_STEP, dt, s)
        if not fused:
            stage = self._stage()
            for i in range(T.RK_STEP):
                stage(rk, i, self.t_prev, dt, self.atol, self.rtol, s)
        self.stats["rhs"] += T.RK_STEP
        self.t_front = self.t_prev + dt
        error = self._read_result()
        if fused and error < 0:
            self._wait_gave_up()
        return error

    def _check_waits(self):
        """Raise when a wait of an earlier dense-output launch gave up (its stages hold NaN)."""
        if self._words[1] < 0:
            self._wait_gave_up()

    def _reset_waits(self):
        torch.cuda.current_stream().synchronize()   # every block has left and written its word
        self.counter.zero_()
        self._barrier_base.value = 0
        self._words[1] = 0.0

    def _wait_gave_up(self):
        self._reset_waits()
        self.status = DEVICE_WAIT
        self._set = False                           # no step to go on from
        raise IntegratorError(STATUS_MESSAGES[DEVICE_WAIT])

    def _stage(self):
        """The operator's stage launch, by half where that applies."""
        return self.op.vern7_stage_herm if self._half() else self.op.vern7_stage

    def _stages_of(self, cls) -> bool:
        """Whether the operator's stages are those of ``cls``: a subclass or an object with a
        ``vern7_stage`` of its own gets every stage through it."""
        return getattr(self.op.vern7_stage, "__func__", None) is cls.vern7_stage

    def _half(self) -> bool:
        """Whether the state is a Hermitian density matrix that the generator keeps Hermitian
        (the coefficients may have been replaced since the state was set, so their part is
        looked at again)."""
        return (self._hermitian and self.op.real_coefficients()
                and self._stages_of(DeviceOperator))

    def _range(self, rk, stage0, stage1, dt, s) -> bool:
        """The stages in one launch where the operator's rows all fit the GPU at once."""
        if not self._stages_of(DeviceOperator):
            return False
        run = self.op.vern7_range_herm if self._half() else self.op.vern7_range
        return run(rk, stage0, stage1, self.t_prev, dt, self.atol, self.rtol,
                   self.counter.data_ptr() + 4, self._barrier_base, s)

    def _prep_dense_out(self):
        # explicit_rk.pyx:399-410
        dt = self.dt_int
        rk = self._rk()
        rk.result = self._host.data_ptr() + 8       # written when a wait gives up
        s = stream_ptr()
        if not self._range(rk, T.RK_STEP, T.RK_EXTRA_STEP, dt, s):
            self._combine(self._stage_base(),
                          [dt * self.a[T.RK_STEP, j] for j in range(T.RK_STEP)],
                          self._ytmp(T.RK_STEP & 1))
            stage = self._stage()
            for i in range(T.RK_STEP, T.RK_EXTRA_STEP):
                stage(rk, i, self.t_prev, dt, self.atol, self.rtol, s)
        self.stats["rhs"] += T.RK_EXTRA_STEP - T.RK_STEP

    def dense_factors(self, t):
        # explicit_rk.pyx:412-430 (Horner in tau, highest degree first)
        tau = (t - self.t_prev) / self.dt_int
        out = []
        for i in range(T.RK_EXTRA_STEP):
            acc = 0.0
            for j in range(T.DENSEOUT_ORDER - 1, -1, -1):
                acc += self.bi[i, j]
                acc *= tau
            out.append(self.dt_int * acc)
        return out

    def _set_interp(self, t):
        self._out = ("interp", self.dense_factors(t))

    def _get_timestep(self, t):
        # explicit_rk.pyx:440-449
        dt_needed = t - self.t_prev
        if self.interpolate:
            return self.dt_safe
        if dt_needed <= self.dt_safe:
            return dt_needed
        return dt_needed / (int(dt_needed / self.dt_safe) + 1)

    def _recompute_safe_step(self, err, dt):
        # explicit_rk.pyx:451-467
        if err == 0:
            factor = 10.0
        else:
            factor = 0.9 * err ** (-1 / (self.order + 1))
            factor = min(10.0, factor)
            factor = max(0.2, factor)
        self.dt_safe = dt * factor
        if self.max_step:
            self.dt_safe = min(self.max_step, self.dt_safe)
        if self.min_step:
            self.dt_safe = max(self.min_step, self.dt_safe)

    # -- outputs ------------------------------------------------------------
    def successful(self) -> bool:
        return self.status >= 0 and self._words[1] >= 0

    def check(self):
        self._check_waits()
        if not self.successful():
            raise IntegratorError(STATUS_MESSAGES[self.status])

    def state_view(self) -> _lib.StateView:
        """The state at ``self.t`` as a lazy view (valid until the next step)."""
        if self._out[0] == "front":
            return self._view(self.y_front)
        return self._view(self.y_prev, self._out[1])

    def step_view(self) -> _lib.StateView:
        """The current step's dense output: ``y_prev`` and the 16 stages, no factors."""
        return self._view(self.y_prev)

    def get_state(self) -> torch.Tensor:
        """Materialise the state at ``self.t`` into ``self.y_out`` (state dtype)."""
        if self._out[0] == "front":
            self.y_out.copy_(self.y_front)
        else:
            self._combine(self.y_prev, self._out[1], self.y_out)
        return self.y_out
