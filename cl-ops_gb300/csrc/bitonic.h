// Declarations shared by the bitonic sorters' dispatch (bitonic.cu) and
// their per-element-width kernel units (bitonic_k{1,2,4,8}.cu, built from
// bitonic.cuh).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "clo_internal.h"

namespace clo {
namespace bitonic {

struct Half16 {
	uint16_t bits;
};

// The network over src's n (>= 2) elements into dst, for the element types
// of one width.
#define CLO_BITONIC_WIDTH(W) \
	cudaError_t sort_width##W(const void *src, void *dst, size_t n, CloType type, int max_ps, \
		int max_sfs, BitonicUser user, CCLContext *ctx, cudaStream_t s, GError **err);
CLO_BITONIC_WIDTH(1)
CLO_BITONIC_WIDTH(2)
CLO_BITONIC_WIDTH(4)
CLO_BITONIC_WIDTH(8)
#undef CLO_BITONIC_WIDTH

}  // namespace bitonic
}  // namespace clo
