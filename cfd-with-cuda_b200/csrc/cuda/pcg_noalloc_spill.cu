// Vectors of the allocation-free PCG (pcg_noalloc.cu) that the shared memory of a
// device or partition with few SMs cannot hold.  A module of its own: with
// CUDA's lazy loading (the default) its 12 MiB are placed on a device only when
// the address is asked for.
#include <cuda_runtime.h>

#include "../../../include/cfdfs.h"

namespace cfd {

static __device__ __align__(256) double g_noalloc_spill[3 * (size_t)CFD_NOALLOC_MAX_N];

cudaError_t noalloc_spill(double** p) { return cudaGetSymbolAddress(reinterpret_cast<void**>(p), g_noalloc_spill); }

}  // namespace cfd
