// Declarations shared between the translation units of the library.
#pragma once
#include <cuda_runtime.h>

#include "../../include/cswap_b200.h"

namespace csw {

// records the runtime error for csw_last_cuda_error() and returns CSW_ERR_CUDA
csw_status cuda_fail(cudaError_t e);

// the status word of the CURRENT device (created on first use; it is zero unless a
// kernel gave up on a bounded wait)
csw_status device_state(int** d_status);

// SMs of the CURRENT device: 148, or what a partition of it has.  Touches no memory of the
// device and synchronises nothing.
int sm_count();

}  // namespace csw
