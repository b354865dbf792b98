// Dispatch of the radix sort by key width; the kernels are in radix.cuh.
#include "radix.h"

#include "clo_internal.h"

namespace clo {

cudaError_t radix_msd_partition(const void *keys_in, void *keys_out, size_t n, int key_bytes,
	int sort_bits, uint32_t *counts, CCLContext *ctx, cudaStream_t s, GError **err) {
	if (sort_bits < radix::kRadixBits || n >= (size_t)radix::kStValue) {
		set_error(err, CLO_ERROR_ARGS, "satradix partition: %d sort bits, %zu keys", sort_bits, n);
		return cudaErrorInvalidValue;
	}
	switch (key_bytes) {
	case 2: return radix::msd_partition<uint16_t>(keys_in, keys_out, n, sort_bits, counts, ctx, s, err);
	case 4: return radix::msd_partition<uint32_t>(keys_in, keys_out, n, sort_bits, counts, ctx, s, err);
	case 8: return radix::msd_partition<uint64_t>(keys_in, keys_out, n, sort_bits, counts, ctx, s, err);
	}
	set_error(err, CLO_ERROR_ARGS, "satradix partition: key width %d", key_bytes);
	return cudaErrorInvalidValue;
}

cudaError_t radix_sort(const void *src, void *dst, void *vals, size_t n, int key_bytes,
	int val_bytes, int sort_bits, CCLContext *ctx, cudaStream_t s, GError **err) {
	if (val_bytes && src != dst) {
		set_error(err, CLO_ERROR_ARGS, "satradix: values are sorted in place, with their keys");
		return cudaErrorInvalidValue;
	}
	// Nothing to sort, or buffers that overlap in part: copied first.
	const char *a = (const char *)src, *b = (const char *)dst;
	const size_t bytes = n * (size_t)key_bytes;
	const bool none = n < 2 || sort_bits < radix::kRadixBits;
	if (a != b && (none || (a < b + bytes && b < a + bytes))) {
		cudaError_t e = n ? cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, s)
						  : cudaSuccess;
		if (e != cudaSuccess) {
			cuda_ok(e, err, "sort copy");
			return e;
		}
		src = dst;
	}
	if (none) return cudaSuccess;
	const int passes = sort_bits / radix::kRadixBits;
	if (src == dst && passes > 1 && passes % 2) {
		set_error(err, CLO_ERROR_ARGS, "satradix: %d passes in place", passes);
		return cudaErrorInvalidValue;
	}
	// Small whole-key sorts without values: equal keys are the same bits, so
	// any sort gives the stable one's result, and the bitonic tiles are faster
	// while launches and latencies, not bytes, are what a sort costs (us,
	// bitonic / the radix sort's best: u32 2^10 4.4 / 8.2, 2^15 14 / 25, 2^17 24
	// / 27.5, 2^18 30 / 28; u64 2^10 6.2 / 15, 2^15 22 / 44, 2^18 41 / 58, 2^20
	// 101 / 80; keys of one and two bytes are faster by radix).
	if (val_bytes == 0 && key_bytes >= 4 && sort_bits == 8 * key_bytes &&
		n <= ((size_t)1 << (key_bytes == 8 ? 18 : 17)))
		return bitonic_sort(src, dst, n, key_bytes == 8 ? CLO_ULONG : CLO_UINT, 4, 0,
			BITONIC_SATRADIX, ctx, s, err);
	switch (key_bytes) {
	case 1: return radix::sort<uint8_t>(src, dst, vals, n, val_bytes, sort_bits, ctx, s, err);
	case 2: return radix::sort<uint16_t>(src, dst, vals, n, val_bytes, sort_bits, ctx, s, err);
	case 4: return radix::sort<uint32_t>(src, dst, vals, n, val_bytes, sort_bits, ctx, s, err);
	case 8: return radix::sort<uint64_t>(src, dst, vals, n, val_bytes, sort_bits, ctx, s, err);
	}
	set_error(err, CLO_ERROR_ARGS, "Unsupported key width %d", key_bytes);
	return cudaErrorInvalidValue;
}

}  // namespace clo
