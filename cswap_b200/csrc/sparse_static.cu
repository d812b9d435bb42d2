// An allocation-free way into the sparse compressor.
//
// Some callers may not allocate device memory at the moment they need to
// compress: a swap hook that runs while the framework's caching allocator is
// locked or already out of memory (which is exactly when swapping is wanted),
// a callback on a path where cudaMalloc's implicit device synchronisation
// would stall other streams, or an embedding with a fixed memory budget handed
// over at start-up.  The compressor keeps all of its working state in the
// output buffer, so for them this is csw_sparse_compress within the size limit
// they were promised.  (The driver places the kernels on a device when they are
// first used there; the warm-up call at start-up, n = 0, gets that over with while
// memory is still available.)
#include <cuda_runtime.h>

#include "../../include/cswap_b200.h"
#include "internal.h"
#include "sparse_kernels.h"

extern "C" csw_status csw_sparse_compress_static(const float* d_in, size_t n, void* d_out, size_t cap,
                                                 uint32_t* nnz_out, csw_stream_t stream) {
  if (n > CSW_SPARSE_STATIC_MAX_ELEMS) return CSW_ERR_LIMIT;
  if (n == 0) {
    const cudaError_t e = csw::sparse_compress_preload();
    if (e != cudaSuccess) return csw::cuda_fail(e);
  }
  return csw_sparse_compress(d_in, n, d_out, cap, nnz_out, stream);
}
