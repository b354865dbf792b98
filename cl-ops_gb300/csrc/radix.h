// Declarations shared by the radix sort's dispatch (radix.cu) and its
// per-key-width kernel units (radix_k{1,2,4,8}.cu, built from radix.cuh).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "clo_internal.h"

namespace clo {
namespace radix {

constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;

// Tile status word: 2-bit flag | 30-bit count.
constexpr uint32_t kStAgg = 1u << 30;
constexpr uint32_t kStPrefix = 2u << 30;
constexpr uint32_t kStValue = (1u << 30) - 1u;

// radix_sort and radix_msd_partition (clo_internal.h) for keys of type K.
template <typename K>
cudaError_t sort(const void *src, void *dst, void *vals, size_t n, int val_bytes, int sort_bits,
	CCLContext *ctx, cudaStream_t s, GError **err);
template <typename K>
cudaError_t msd_partition(const void *keys_in, void *keys_out, size_t n, int sort_bits,
	uint32_t *counts, CCLContext *ctx, cudaStream_t s, GError **err);

}  // namespace radix
}  // namespace clo
