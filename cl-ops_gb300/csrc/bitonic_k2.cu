// Bitonic sorters: the kernels for elements of 2 byte(s) (see bitonic.cuh).
#include "bitonic.cuh"

namespace clo {
namespace bitonic {

cudaError_t sort_width2(const void *src, void *dst, size_t n, CloType type, int max_ps,
	int max_sfs, BitonicUser user, CCLContext *ctx, cudaStream_t s, GError **err) {
	auto go = [&](auto t) {
		using T = decltype(t);
		return sort_typed<T>((const T *)src, (T *)dst, n, max_ps, max_sfs, user, ctx, s, err);
	};
	switch (type) {
	case CLO_SHORT: return go(int16_t());
	case CLO_USHORT: return go(uint16_t());
	case CLO_HALF: return go(Half16());
	default: return cudaErrorInvalidValue;
	}
}

}  // namespace bitonic
}  // namespace clo
