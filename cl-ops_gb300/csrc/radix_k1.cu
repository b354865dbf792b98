// Radix sort: the kernels for keys of 1 byte(s) (see radix.cuh).
#include "radix.cuh"

namespace clo {
namespace radix {

template cudaError_t sort<uint8_t>(const void *, void *, void *, size_t, int, int, CCLContext *,
	cudaStream_t, GError **);

}  // namespace radix
}  // namespace clo
