// Error reporting and device queries shared by the C-ABI translation units.
#pragma once
#include <cuda_runtime.h>

#include <mutex>

#include "qutip_gb300.h"

namespace qg {
// Record a message for qg_last_error() on this thread and return code.
int set_error(int code, const char* msg);
// Check cudaGetLastError() after a launch; QG_OK or QG_ERR_CUDA.
int check_launch(const char* what);
// Multiprocessor count of the current device (cached per device).
int sm_count();
// Opt a kernel into `bytes` of dynamic shared memory on the current device.  Any size is opted
// in: the 48 KB default counts a kernel's static shared memory too (17 KB of tiles or 5.6 KB of
// factor slices had launches of 32 to 47 KB refused).  The limit only grows: host threads
// with launches of different sizes would otherwise lower it between one another's call and
// launch.
bool allow_smem(const void* kernel, size_t bytes);
// The same, and the resident blocks per SM (<= 0 on failure).  The caller keeps one cache
// per kernel instantiation, an entry per device, shared by host threads under its mutex.
constexpr int OCC_MAX_DEVICES = 64;
struct OccCache {
  std::mutex mu;
  int occ[OCC_MAX_DEVICES] = {};
  size_t smem[OCC_MAX_DEVICES] = {};
};
int launch_occupancy(const void* kernel, int block, size_t smem, OccCache& c);
// Validate a grouped operator (shape, layout and tables); QG_OK or an error code.
int check_groups(const qg_csr_groups* A);
// The same for an operator of the Hermitian half form on d x d states.
int check_herm(const qg_csr_groups* A, int64_t d);
// One stage with the coefficients of that stage already on the device (coefs: the operator's
// groups, then the collapse operators, complex double each; null: the launch evaluates them).
int stage_csr(const qg_csr_groups* A, const qg_rk_buffers* B, int stage, double t_prev, double dt,
              double atol, double rtol, const void* coefs, void* stream);
int stage_herm(const qg_csr_groups* A, int64_t d, const qg_rk_buffers* B, int stage, double t_prev,
               double dt, double atol, double rtol, const void* coefs, void* stream);
int stage_lindblad(const qg_lindblad* L, const qg_rk_buffers* B, int stage, double t_prev,
                   double dt, double atol, double rtol, const void* coefs, void* stream);
// qg_vern7_range (d = 0) or qg_vern7_range_herm, with the limit of a wait in millions of SM
// clocks (0: the default).
int range_csr(const qg_csr_groups* A, const qg_rk_buffers* B, int stage0, int stage1,
              double t_prev, double dt, double atol, double rtol, int64_t d, int32_t wait_mcycles,
              unsigned int* barrier, uint32_t* barrier_base, void* stream);
}  // namespace qg

// The fault flag of the fused step kernel's barrier waits, read and cleared (for
// qg_device_fault).
int step_fault_take();
