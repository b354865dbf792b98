// Register layout of the plain scan's tiles: a warp owns a stretch of
// consecutive elements in rows of 32 x kE: in row r lane l
// holds elements kE l .. kE l + kE - 1, kE being as many as fill a 32-byte
// store of outputs. Loads and stores are whole vectors between global memory
// and registers, and a row's scan is a warp scan of the lanes' sums: nothing
// is transposed through shared memory (some shapes park a tile's registers
// there, scan.cu).
#pragma once

#include <stddef.h>
#include <stdint.h>

#include "dev_common.cuh"

namespace clo {
namespace scanrows {

template <typename InT, typename OutT, int THREADS, int TILE>
struct Rows {
	static constexpr int kThreads = THREADS, kTile = TILE;
	static constexpr int kWarps = kThreads / 32, kWarpElems = kTile / kWarps;
	static constexpr int kE = 32 / sizeof(OutT);          // a lane's run in one row
	static constexpr int kRows = kWarpElems / (32 * kE);
	static constexpr int kInBytes = kE * sizeof(InT);     // 4 .. 256
	static constexpr int kWords = (kInBytes + 3) / 4;     // registers of a run
	uint32_t w[kRows][kWords];

	__device__ __forceinline__ InT at(int r, int e) const {
		if constexpr (sizeof(InT) == 8)
			return (InT)((uint64_t)w[r][2 * e] | (uint64_t)w[r][2 * e + 1] << 32);
		else if constexpr (sizeof(InT) == 4) return (InT)w[r][e];
		else if constexpr (sizeof(InT) == 2) return (InT)(uint16_t)(w[r][e / 2] >> (16 * (e % 2)));
		else return (InT)(uint8_t)(w[r][e / 4] >> (8 * (e % 4)));
	}

	// The warp's kWarpElems elements at p, all valid, as vectors: 32 bytes where
	// `wide` (p 32-byte aligned), else 16 (p 16-byte aligned).
	__device__ __forceinline__ void load(const InT *p, int lane, bool wide) {
#pragma unroll
		for (int r = 0; r < kRows; ++r) {
			const char *q = reinterpret_cast<const char *>(p) + (size_t)(32 * r + lane) * kInBytes;
			if constexpr (kInBytes >= 32) {
				if (wide) {
#pragma unroll
					for (int i = 0; i < kWords / 8; ++i)
						dev::ld_stream_v8(q + 32 * i, *reinterpret_cast<uint32_t(*)[8]>(&w[r][8 * i]));
				} else {
#pragma unroll
					for (int i = 0; i < kWords / 4; ++i) put4(r, 4 * i, q + 16 * i);
				}
			} else if constexpr (kInBytes == 16) {
				put4(r, 0, q);
			} else if constexpr (kInBytes == 8) {
				const uint2 v = __ldcs(reinterpret_cast<const uint2 *>(q));
				w[r][0] = v.x;
				w[r][1] = v.y;
			} else {
				w[r][0] = __ldcs(reinterpret_cast<const uint32_t *>(q));
			}
		}
	}
	__device__ __forceinline__ void put4(int r, int at, const char *q) {
		const uint4 v = dev::ld_stream_v4(reinterpret_cast<const uint4 *>(q));
		w[r][at] = v.x;
		w[r][at + 1] = v.y;
		w[r][at + 2] = v.z;
		w[r][at + 3] = v.w;
	}
	// Element by element; those from `valid` on are zero.
	__device__ __forceinline__ void load_some(const InT *p, int lane, size_t valid) {
#pragma unroll
		for (int r = 0; r < kRows; ++r) {
#pragma unroll
			for (int i = 0; i < kWords; ++i) w[r][i] = 0;
#pragma unroll
			for (int e = 0; e < kE; ++e) {
				const size_t i = (size_t)(32 * r + lane) * kE + e;
				const InT v = i < valid ? p[i] : (InT)0;
				if constexpr (sizeof(InT) == 8) {
					w[r][2 * e] = (uint32_t)(uint64_t)v;
					w[r][2 * e + 1] = (uint32_t)((uint64_t)v >> 32);
				} else if constexpr (sizeof(InT) == 4) {
					w[r][e] = (uint32_t)v;
				} else if constexpr (sizeof(InT) == 2) {
					w[r][e / 2] |= (uint32_t)(uint16_t)v << (16 * (e % 2));
				} else {
					w[r][e / 4] |= (uint32_t)(uint8_t)v << (8 * (e % 4));
				}
			}
		}
	}
};

// A lane's run of outputs, 32 bytes.
template <typename OutT>
__device__ __forceinline__ void store_run(OutT *q, const uint32_t (&o)[8], bool wide) {
	if (wide) {
		dev::st_stream_v8(q, o);
	} else {
		uint4 *p = reinterpret_cast<uint4 *>(q);
		dev::st_stream_v4(p, make_uint4(o[0], o[1], o[2], o[3]));
		dev::st_stream_v4(p + 1, make_uint4(o[4], o[5], o[6], o[7]));
	}
}

// Packs output e of a run into its words.
template <typename OutT>
__device__ __forceinline__ void pack(uint32_t (&o)[8], int e, OutT v) {
	if constexpr (sizeof(OutT) == 8) {
		o[2 * e] = (uint32_t)(uint64_t)v;
		o[2 * e + 1] = (uint32_t)((uint64_t)v >> 32);
	} else if constexpr (sizeof(OutT) == 4) {
		o[e] = (uint32_t)v;
	} else if constexpr (sizeof(OutT) == 2) {
		if (e % 2 == 0) o[e / 2] = (uint16_t)v;
		else o[e / 2] |= (uint32_t)(uint16_t)v << 16;
	} else {
		if (e % 4 == 0) o[e / 4] = (uint8_t)v;
		else o[e / 4] |= (uint32_t)(uint8_t)v << (8 * (e % 4));
	}
}

}  // namespace scanrows
}  // namespace clo
