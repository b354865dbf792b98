// Dispatch of the bitonic sorters ("sbitonic", "abitonic") by element width;
// the kernels are in bitonic.cuh.
#include "bitonic.h"

#include "clo_internal.h"

namespace clo {

cudaError_t bitonic_sort(const void *src, void *dst, size_t n, CloType type, int max_ps,
	int max_sfs, BitonicUser user, CCLContext *ctx, cudaStream_t s, GError **err) {
	const size_t eb = clo_type_sizeof(type);
	if (eb != 1 && eb != 2 && eb != 4 && eb != 8) {
		set_error(err, CLO_ERROR_ARGS, "Unsupported element type %d", (int)type);
		return cudaErrorInvalidValue;
	}
	// Too short to sort, or buffers that overlap in part: copied first.
	const char *a = (const char *)src, *b = (const char *)dst;
	const bool overlap = a != b && a < b + n * eb && b < a + n * eb;
	if (a != b && (n < 2 || overlap)) {
		cudaError_t e = n ? cudaMemcpyAsync(dst, src, n * eb, cudaMemcpyDeviceToDevice, s)
						  : cudaSuccess;
		if (e != cudaSuccess) {
			cuda_ok(e, err, "sort copy");
			return e;
		}
		src = dst;
	}
	if (n < 2) return cudaSuccess;
	switch (eb) {
	case 1: return bitonic::sort_width1(src, dst, n, type, max_ps, max_sfs, user, ctx, s, err);
	case 2: return bitonic::sort_width2(src, dst, n, type, max_ps, max_sfs, user, ctx, s, err);
	case 4: return bitonic::sort_width4(src, dst, n, type, max_ps, max_sfs, user, ctx, s, err);
	default: return bitonic::sort_width8(src, dst, n, type, max_ps, max_sfs, user, ctx, s, err);
	}
}

}  // namespace clo
