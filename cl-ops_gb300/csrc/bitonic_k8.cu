// Bitonic sorters: the kernels for elements of 8 byte(s) (see bitonic.cuh).
#include "bitonic.cuh"

namespace clo {
namespace bitonic {

cudaError_t sort_width8(const void *src, void *dst, size_t n, CloType type, int max_ps,
	int max_sfs, BitonicUser user, CCLContext *ctx, cudaStream_t s, GError **err) {
	auto go = [&](auto t) {
		using T = decltype(t);
		return sort_typed<T>((const T *)src, (T *)dst, n, max_ps, max_sfs, user, ctx, s, err);
	};
	switch (type) {
	case CLO_LONG: return go(int64_t());
	case CLO_ULONG: return go(uint64_t());
	case CLO_DOUBLE: return go(double());
	default: return cudaErrorInvalidValue;
	}
}

}  // namespace bitonic
}  // namespace clo
