// Radix sort: the kernels for keys of 8 byte(s) (see radix.cuh).
#include "radix.cuh"

namespace clo {
namespace radix {

template cudaError_t sort<uint64_t>(const void *, void *, void *, size_t, int, int, CCLContext *,
	cudaStream_t, GError **);
template cudaError_t msd_partition<uint64_t>(const void *, void *, size_t, int, uint32_t *,
	CCLContext *, cudaStream_t, GError **);

}  // namespace radix
}  // namespace clo
