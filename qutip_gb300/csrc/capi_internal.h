// Error reporting and device queries shared by the C-ABI translation units.
#pragma once
#include <cuda_runtime.h>

#include "qutip_gb300.h"

namespace qg {
// Record a message for qg_last_error() on this thread and return code.
int set_error(int code, const char* msg);
// Check cudaGetLastError() after a launch; QG_OK or QG_ERR_CUDA.
int check_launch(const char* what);
// Multiprocessor count of the current device (cached per device).
int sm_count();
// Validate a grouped operator (shape, layout and tables); QG_OK or an error code.
int check_groups(const qg_csr_groups* A);
// The same for an operator of the Hermitian half form on d x d states.
int check_herm(const qg_csr_groups* A, int64_t d);
}  // namespace qg

// The fault flag of the fused step kernel's barrier waits, read and cleared (for
// qg_device_fault).
int step_fault_take();
