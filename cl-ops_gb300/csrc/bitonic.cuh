// "sbitonic" and "abitonic": the reference's bitonic sorting network,
// replayed exactly on sm_103a. Included by one unit per element width
// (bitonic_k{1,2,4,8}.cu), which compile in parallel.
//
// Network (src/cl_ops/sort/clo_sort_sbitonic.cl:38-69 and the grouped
// kernels of clo_sort_abitonic.cl:31-1067): over N = nlpo2(n) elements,
// for stage s = 1..log2 N and step t = s..1, elements i and i + 2^(t-1)
// with bit t-1 of i clear are compared; the block direction is bit s of i
// (1 = descending); they swap iff COMPARE(key_i, key_j) XOR desc, with
// COMPARE(a, b) = a > b. Every step touches disjoint pairs, so any
// implementation that applies the same steps in the same order produces
// the same array, bit for bit, including where the compare is not a total
// order (equal keys, NaN, -0.0/+0.0).
//
// Launches (both sorters):
//   - bitonic_tile<.., SORT>: stages 1..T of every tile of 2^T elements;
//   - bitonic_global_steps<g>: g consecutive steps with strides >= the
//     tile, 2^g elements per thread held in registers;
//   - bitonic_tile<.., finish>: the remaining steps T..1 of a stage.
// A tile is the work of one CTA (2^K elements). Sorts that one tile holds may
// take a cluster of 2^LOGC CTAs, which exchange elements through distributed
// shared memory.
// The option settings that limit the grouping (maxps, maxsfs) take the
// shared-memory rounds at the end of this file.
// Sizes that are not a power of two are padded with the element type's
// maximum, which the final ascending stage moves past the real elements;
// the reference requires power-of-two sizes.
//
// HBM roofline: 2 x sizeof(T) x N bytes per launch (one read, one write).
#pragma once

#include <cuda_fp16.h>

#include <algorithm>
#include <climits>
#include <type_traits>

#include "bitonic.h"
#include "clo_internal.h"
#include "dev_common.cuh"
#include "launch.h"
#include "timing.h"

namespace clo {
namespace bitonic {
namespace {

template <typename T>
struct BT {
	__device__ __forceinline__ static bool gt(T a, T b) { return a > b; }
};
template <>
struct BT<Half16> {
	__device__ __forceinline__ static bool gt(Half16 a, Half16 b) {
		return __hgt(__ushort_as_half(a.bits), __ushort_as_half(b.bits));
	}
};

template <typename T> __host__ __device__ constexpr T max_value();
template <> constexpr int8_t max_value<int8_t>() { return INT8_MAX; }
template <> constexpr uint8_t max_value<uint8_t>() { return UINT8_MAX; }
template <> constexpr int16_t max_value<int16_t>() { return INT16_MAX; }
template <> constexpr uint16_t max_value<uint16_t>() { return UINT16_MAX; }
template <> constexpr int32_t max_value<int32_t>() { return INT32_MAX; }
template <> constexpr uint32_t max_value<uint32_t>() { return UINT32_MAX; }
template <> constexpr int64_t max_value<int64_t>() { return INT64_MAX; }
template <> constexpr uint64_t max_value<uint64_t>() { return UINT64_MAX; }
template <> constexpr Half16 max_value<Half16>() { return Half16{0x7c00}; }  // +inf
template <> constexpr float max_value<float>() { return __builtin_huge_valf(); }
template <> constexpr double max_value<double>() { return __builtin_huge_val(); }

// Doubles are compared as integers where that gives the network's result: the
// SM compares two doubles a clock. ord() maps the bits to integers of the same
// order (its own inverse); the two orders agree but for NaN (unordered) and
// for -0 (equal to +0), so data holding one of those keeps the compare.
__device__ __forceinline__ int64_t ord(int64_t bits) {
	return bits ^ (int64_t)((uint64_t)(bits >> 63) >> 1);
}
__device__ __forceinline__ bool ord_special(int64_t bits) {
	const uint32_t hi = (uint32_t)((uint64_t)bits >> 32), lo = (uint32_t)bits;
	const uint32_t mag = hi & 0x7fffffffu;
	return mag > 0x7ff00000u || (mag == 0x7ff00000u && lo != 0) || (hi == 0x80000000u && lo == 0);
}

template <typename T>
__device__ __forceinline__ void cmpxchg(T &a, T &b, bool desc) {
	if (BT<T>::gt(a, b) != desc) {
		T t = a;
		a = b;
		b = t;
	}
}

// --------------------------------------------------------- global steps
// Steps step .. step-G+1 of `stage`, 2^G elements per thread.
// Threads per CTA: 128 where a thread holds 128 32-bit words (168 registers
// a thread, three CTAs per SM), else 256.
template <typename T, int G>
constexpr int gs_words() { return (1 << G) * (sizeof(T) == 8 ? 2 : 1); }
template <typename T, int G>
constexpr int gs_threads() { return gs_words<T, G>() >= 128 ? 128 : 256; }
template <typename T, int G>
constexpr int gs_min_blocks() {
	return gs_words<T, G>() >= 128 ? 3 : gs_words<T, G>() >= 64 ? 2 : 1;
}

// G steps over 2^G groups of V elements each, in registers.
template <typename T, int G, int V>
__device__ __forceinline__ void steps_in_regs(T (&r)[V << G], bool desc) {
	if constexpr (std::is_same<T, double>::value) {
		int64_t o[V << G];
		bool special = false;
#pragma unroll
		for (int m = 0; m < (V << G); ++m) {
			o[m] = __double_as_longlong(r[m]);
			special = special || ord_special(o[m]);
		}
		if (!special) {
#pragma unroll
			for (int m = 0; m < (V << G); ++m) o[m] = ord(o[m]);
			steps_in_regs<int64_t, G, V>(o, desc);
#pragma unroll
			for (int m = 0; m < (V << G); ++m) r[m] = __longlong_as_double(ord(o[m]));
			return;
		}
	}
#pragma unroll
	for (int s = G - 1; s >= 0; --s)
#pragma unroll
		for (int m = 0; m < (1 << G); ++m)
			if (!(m & (1 << s)))
#pragma unroll
				for (int v = 0; v < V; ++v)
					cmpxchg(r[m * V + v], r[(m | (1 << s)) * V + v], desc);
}

template <typename T, int G>
__global__ void __launch_bounds__((gs_threads<T, G>()), (gs_min_blocks<T, G>()))
bitonic_global_steps(T *data, size_t groups, int stage, int step) {
	dev::pdl_wait();
	size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
	if (q >= groups) return;
	const int lo_bits = step - G;
	size_t low = q & (((size_t)1 << lo_bits) - 1);
	size_t high = q >> lo_bits;
	size_t base = (high << step) | low;
	const size_t inc = (size_t)1 << lo_bits;
	const bool desc = (base >> stage) & 1;
	T r[1 << G];
	T *p = data + base;
#pragma unroll
	for (int m = 0; m < (1 << G); ++m) r[m] = p[m * inc];
	steps_in_regs<T, G, 1>(r, desc);
	// With 64 or more words a thread, the store addresses are computed
	// afresh rather than kept from the loads (as many more live registers).
	if constexpr (gs_words<T, G>() >= 64) asm volatile("" : "+l"(p));
#pragma unroll
	for (int m = 0; m < (1 << G); ++m) p[m * inc] = r[m];
}

// The same for few steps, a thread taking 16 consecutive bytes of each of
// its 2^G strides: one element a stride leaves too few bytes in flight (the
// sort of 2^24 ints: 627 -> 617 us). Takes a 16-byte aligned array and
// strides of at least 16 bytes.
template <typename T, int G>
__global__ void __launch_bounds__(256)
bitonic_global_steps_v(T *data, size_t groups, int stage, int step) {
	constexpr int V = 16 / sizeof(T);
	dev::pdl_wait();
	const size_t q = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) * V;
	if (q >= groups) return;
	const int lo_bits = step - G;
	const size_t low = q & (((size_t)1 << lo_bits) - 1);
	const size_t base = ((q >> lo_bits) << step) | low;
	const size_t inc = (size_t)1 << lo_bits;
	const bool desc = (base >> stage) & 1;
	struct alignas(16) Vec {
		T e[V];
	};
	T r[V << G];
	T *p = data + base;
#pragma unroll
	for (int m = 0; m < (1 << G); ++m) {
		const Vec v = *reinterpret_cast<const Vec *>(p + m * inc);
#pragma unroll
		for (int i = 0; i < V; ++i) r[m * V + i] = v.e[i];
	}
	steps_in_regs<T, G, V>(r, desc);
#pragma unroll
	for (int m = 0; m < (1 << G); ++m) {
		Vec v;
#pragma unroll
		for (int i = 0; i < V; ++i) v.e[i] = r[m * V + i];
		*reinterpret_cast<Vec *>(p + m * inc) = v;
	}
}

// ------------------------------------------------------- register tiles
// A thread holds 2^RE elements in registers. In layout L(B) register m of thread g (its id within the tile:
// cluster rank above the thread index) holds tile element
//   ((g >> B) << (B + RE)) | (m << B) | (g & (2^B - 1)),
// so the steps on index bits B .. B + RE - 1 are compare-exchanges between
// a thread's own registers. A stage's steps run in phases of up to RE bits,
// from the stage's top bit down to L(0), joined by transposes through the
// padded shared tile (element i of a CTA's part at i + (i >> RE): a warp's
// 32 accesses of any layout fall in 32 banks). The steps and their order
// are those of the network, so the result is the reference's.
//
// With LOGC > 0 the tile spans a cluster, each CTA's shared memory holding
// its 2^K consecutive elements. The phase on the cluster's bits takes the
// layout L(T - RE), whose registers span the CTAs: it is entered by reading
// the other CTAs' shared memory and left by writing into it. 2^15 4-byte
// elements sort in one launch on 8 SMs in 14.6 us, against 17 in five launches
// of one-CTA tiles.
//
// No barrier is needed before a transpose's writes: a thread writes exactly
// the slots it read itself in the transpose before (each slot has one owner
// per layout). After them the barrier covers the threads that read them:
// the warp for layouts up to L(5) (a warp holds the same 2^(RE+5)
// consecutive elements in each of them), the CTA, or the cluster.
template <typename T, int K_, int LOGC_, int RE_>
struct TileCfg {
	static constexpr int kK = K_, LOGC = LOGC_, RE = RE_, R = 1 << RE, TL = kK + LOGC;
	static constexpr int kThreads = 1 << (kK - RE), kCluster = 1 << LOGC;
	static constexpr int LR = TL - RE;  // the cluster phase's layout
	static constexpr size_t kSmem = ((size_t)(1 << kK) + (1 << (kK - RE))) * sizeof(T);
	// (64 registers a thread, 80 with 16 8-byte elements.)
	static constexpr int kMinBlocks = (sizeof(T) == 8 && RE == 4 ? 768 : 1024) / kThreads;
};

template <typename T, typename CFG>
struct RegTile {
	using C = CFG;
	static constexpr int RE = C::RE, R = C::R, TL = C::TL, K = C::kK, LOGC = C::LOGC;
	T r[R];
	T *s;
	uint32_t tid, rank, g;

	__device__ __forceinline__ static constexpr uint32_t pad(uint32_t i) { return i + (i >> RE); }
	template <int B>
	__device__ __forceinline__ static uint32_t idx(uint32_t t, uint32_t m) {
		return ((t >> B) << (B + RE)) | (m << B) | (t & ((1u << B) - 1u));
	}
	// Offset of register m's slot from register 0's: the register bits never
	// carry into the padding term.
	template <int B>
	__device__ __forceinline__ static constexpr uint32_t off(uint32_t m) {
		return (m << B) + ((m << B) >> RE);
	}
	template <int B>
	static constexpr bool remote = LOGC > 0 && B + RE > K;

	template <int B>
	__device__ __forceinline__ void put() {
		if constexpr (remote<B>) {
			static_assert(!remote<B> || B == C::LR, "one cluster layout");
			const uint32_t a = dev::smem_u32(s) + pad(g) * (uint32_t)sizeof(T);
			constexpr int PER = R >> LOGC;  // registers per CTA's part
#pragma unroll
			for (int c = 0; c < (1 << LOGC); ++c) {
				const uint32_t ra = dev::map_shared(a, c);
#pragma unroll
				for (int m = 0; m < PER; ++m)
					dev::st_dsmem<T>(ra + off<B>(m) * (uint32_t)sizeof(T), r[c * PER + m]);
			}
		} else {
			T *p = s + pad(idx<B>(tid, 0));
#pragma unroll
			for (int m = 0; m < R; ++m) p[off<B>(m)] = r[m];
		}
	}
	template <int B>
	__device__ __forceinline__ void get() {
		if constexpr (remote<B>) {
			const uint32_t a = dev::smem_u32(s) + pad(g) * (uint32_t)sizeof(T);
			constexpr int PER = R >> LOGC;
#pragma unroll
			for (int c = 0; c < (1 << LOGC); ++c) {
				const uint32_t ra = dev::map_shared(a, c);
#pragma unroll
				for (int m = 0; m < PER; ++m)
					r[c * PER + m] = dev::ld_dsmem<T>(ra + off<B>(m) * (uint32_t)sizeof(T));
			}
		} else {
			const T *p = s + pad(idx<B>(tid, 0));
#pragma unroll
			for (int m = 0; m < R; ++m) r[m] = p[off<B>(m)];
		}
	}
	template <int FROM, int TO>
	__device__ __forceinline__ void transpose() {
		put<FROM>();
		if constexpr (remote<FROM> || remote<TO>) {
			dev::cluster_arrive();
			dev::cluster_wait();
		} else if constexpr (FROM <= 5 && TO <= 5) {
			__syncwarp();
		} else {
			__syncthreads();
		}
		get<TO>();
	}

	// Integers run every step ascending as a min/max pair, with the elements
	// of descending blocks complemented for the stage (equal elements are the
	// same bits, so which of them swaps does not show). Floating types keep
	// the network's compare, whose NaN and signed-zero outcomes depend on it.
	static constexpr bool kInt = std::is_integral<T>::value;
	// Complements the elements whose index bit S is set (in L(0)); S == TL:
	// the whole tile by its own direction.
	template <int S>
	__device__ __forceinline__ void flip(bool tile_desc) {
		if constexpr (kInt) {
			if constexpr (S < RE) {
#pragma unroll
				for (int m = 0; m < R; ++m)
					if ((m >> S) & 1) r[m] = (T)~r[m];
			} else {
				const bool d = S == TL ? tile_desc : (bool)((g >> (S - RE)) & 1u);
				const T x = d ? (T)~(T)0 : (T)0;
#pragma unroll
				for (int m = 0; m < R; ++m) r[m] = (T)(r[m] ^ x);
			}
		}
	}
	// Steps on bits HI .. LO of stage S in L(B).
	template <int S, int B, int HI, int LO>
	__device__ __forceinline__ void phase(bool tile_desc) {
		bool d = tile_desc;
		if constexpr (!kInt && S < TL && !(S >= B && S < B + RE))
			d = (g >> (S < B ? S : S - RE)) & 1u;
#pragma unroll
		for (int b = HI; b >= LO; --b) {
			const int sb = 1 << (b - B);
#pragma unroll
			for (int m = 0; m < R; ++m) {
				if (m & sb) continue;
				if constexpr (kInt) {
					const T x = r[m], y = r[m | sb];
					r[m] = x < y ? x : y;
					r[m | sb] = x < y ? y : x;
				} else if constexpr (S < TL && S >= B && S < B + RE) {
					cmpxchg(r[m], r[m | sb], (bool)((m >> (S - B)) & 1));
				} else {
					cmpxchg(r[m], r[m | sb], d);
				}
			}
		}
	}
	static constexpr int lay(int hi) { return hi - RE + 1 > 0 ? hi - RE + 1 : 0; }
	// Steps HI .. 0 of stage S, coming from layout FROM and ending in L(0).
	template <int S, int FROM, int HI>
	__device__ __forceinline__ void down(bool tile_desc) {
		if constexpr (HI >= 0) {
			constexpr int B = lay(HI);
			transpose<FROM, B>();
			phase<S, B, HI, B>(tile_desc);
			down<S, B, B - 1>(tile_desc);
		}
	}
	// Stage S (L(0) before and after).
	template <int S>
	__device__ __forceinline__ void stage(bool tile_desc) {
		flip<S>(tile_desc);
		if constexpr (S - 1 < RE) {
			phase<S, 0, S - 1, 0>(tile_desc);
		} else if constexpr (S > K) {
			transpose<0, C::LR>();
			phase<S, C::LR, S - 1, C::LR>(tile_desc);
			down<S, C::LR, C::LR - 1>(tile_desc);
		} else {
			down<S, 0, S - 1>(tile_desc);
		}
		flip<S>(tile_desc);
	}
	template <int S>
	__device__ __forceinline__ void stages(int last, bool tile_desc) {
		if (S > last) return;
		stage<S>(tile_desc);
		if constexpr (S < TL) stages<S + 1>(last, tile_desc);
	}
};

// A CTA's 2^K elements between global memory and L(0). A thread's
// consecutive elements move as 32-byte vectors when the part is 32-byte aligned
// (half the requests of 16-byte vectors, whose lanes 64 or 128 bytes apart each
// touch a line of their own) and wholly valid, else coalesced element by
// element through a transpose, elements from `valid` on reading as the pad.
template <typename Tile, typename T>
__device__ __forceinline__ void tile_load(Tile &t, const T *p, size_t valid, T pad) {
	constexpr int K = Tile::K, B = K - Tile::RE, R = Tile::R;
	if (sizeof(T) >= 4 && valid >= ((size_t)1 << K) && ((uintptr_t)p % 32) == 0) {
		const char *src = reinterpret_cast<const char *>(p) + (size_t)t.tid * (R * sizeof(T));
		uint32_t w[R * sizeof(T) / 4 + 1];
#pragma unroll
		for (int q = 0; q < (int)(R * sizeof(T) / 32); ++q)
			dev::ld_v8(src + 32 * q, *reinterpret_cast<uint32_t(*)[8]>(w + 8 * q));
#pragma unroll
		for (int m = 0; m < R; ++m) {
			if constexpr (sizeof(T) == 8)
				t.r[m] = __builtin_bit_cast(T, (uint64_t)w[2 * m] | (uint64_t)w[2 * m + 1] << 32);
			else if constexpr (sizeof(T) == 4)
				t.r[m] = __builtin_bit_cast(T, w[m]);
		}
	} else {
#pragma unroll
		for (int m = 0; m < R; ++m) {
			const uint32_t i = ((uint32_t)m << B) | t.tid;
			t.r[m] = i < valid ? p[i] : pad;
		}
		t.template transpose<B, 0>();
	}
}

template <typename Tile, typename T>
__device__ __forceinline__ void tile_store(Tile &t, T *p, size_t valid) {
	constexpr int K = Tile::K, B = K - Tile::RE, R = Tile::R;
	if (sizeof(T) >= 4 && valid >= ((size_t)1 << K) && ((uintptr_t)p % 32) == 0) {
		char *dst = reinterpret_cast<char *>(p) + (size_t)t.tid * (R * sizeof(T));
		uint32_t w[R * sizeof(T) / 4 + 1];
#pragma unroll
		for (int m = 0; m < R; ++m) {
			if constexpr (sizeof(T) == 8) {
				uint64_t v = __builtin_bit_cast(uint64_t, t.r[m]);
				w[2 * m] = (uint32_t)v;
				w[2 * m + 1] = (uint32_t)(v >> 32);
			} else if constexpr (sizeof(T) == 4) {
				w[m] = __builtin_bit_cast(uint32_t, t.r[m]);
			}
		}
#pragma unroll
		for (int q = 0; q < (int)(R * sizeof(T) / 32); ++q)
			dev::st_v8(dst + 32 * q, *reinterpret_cast<const uint32_t(*)[8]>(w + 8 * q));
	} else {
		t.template transpose<0, B>();
#pragma unroll
		for (int m = 0; m < R; ++m) {
			const uint32_t i = ((uint32_t)m << B) | t.tid;
			if (i < valid) p[i] = t.r[m];
		}
	}
}

// SORT: stages 1 .. min(T, stage) of every tile of `src` (elements from
// n_src on are the pad) into `dst`. Otherwise: steps T .. 1 of `stage` (> T)
// of every tile of `src` into `dst` (the same array, or in the last stage
// the caller's). Elements of `dst` from n_dst on are not written.
template <typename T, typename C, bool SORT>
__global__ void __launch_bounds__(C::kThreads, C::kMinBlocks)
bitonic_tile(const T *src, T *dst, size_t n_src, size_t n_dst, int stage) {
	constexpr int K = C::kK, LOGC = C::LOGC;
	// Doubles travel as their bits (see ord).
	constexpr bool kOrd = std::is_same<T, double>::value;
	static_assert(LOGC == 0 || (SORT && !kOrd), "clusters sort up to 4-byte elements");
	using U = typename std::conditional<kOrd, int64_t, T>::type;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	RegTile<U, C> t;
	t.s = reinterpret_cast<U *>(smem_raw);
	t.tid = threadIdx.x;
	t.rank = LOGC ? dev::cluster_rank() : 0u;
	t.g = (t.rank << (K - C::RE)) | t.tid;
	const size_t part = (size_t)blockIdx.x << K;              // this CTA's elements
	const size_t tile = part >> C::TL << C::TL;               // its tile's
	dev::pdl_wait();
	const U *usrc = reinterpret_cast<const U *>(src);
	U *udst = reinterpret_cast<U *>(dst);
	U pad = __builtin_bit_cast(U, max_value<T>());
	if constexpr (SORT) {
		if (tile >= n_src) {
			// A tile of padding alone (the whole cluster's) needs no sorting.
#pragma unroll
			for (int m = 0; m < C::R; ++m) {
				const size_t i = part + (size_t)m * C::kThreads + t.tid;
				if (i < n_dst) udst[i] = pad;
			}
			return;
		}
		tile_load(t, usrc + part, part < n_src ? n_src - part : 0, pad);
	} else {
#pragma unroll
		for (int m = 0; m < C::R; ++m) t.r[m] = usrc[tile + (((size_t)m << C::LR) | t.g)];
	}
	auto work = [&](auto &w) {
		if constexpr (SORT) {
			w.template stages<1>(stage, (tile >> C::TL) & 1);
		} else {
			const bool desc = (tile >> stage) & 1;
			w.template flip<C::TL>(desc);
			w.template phase<C::TL, C::LR, C::TL - 1, C::LR>(desc);
			w.template down<C::TL, C::LR, C::LR - 1>(desc);
			w.template flip<C::TL>(desc);
		}
	};
	if constexpr (kOrd) {
		bool special = false;
#pragma unroll
		for (int m = 0; m < C::R; ++m) special = special || ord_special(t.r[m]);
		special = __syncthreads_or(special);
		if (!special) {
#pragma unroll
			for (int m = 0; m < C::R; ++m) t.r[m] = ord(t.r[m]);
			work(t);
#pragma unroll
			for (int m = 0; m < C::R; ++m) t.r[m] = ord(t.r[m]);
		} else {
			RegTile<T, C> f;
			f.s = reinterpret_cast<T *>(smem_raw);
			f.tid = t.tid;
			f.rank = t.rank;
			f.g = t.g;
#pragma unroll
			for (int m = 0; m < C::R; ++m) f.r[m] = __longlong_as_double(t.r[m]);
			work(f);
#pragma unroll
			for (int m = 0; m < C::R; ++m) t.r[m] = __double_as_longlong(f.r[m]);
		}
	} else {
		work(t);
	}
	tile_store(t, udst + part, part < n_dst ? n_dst - part : 0);
}

// ------------------------------------- shared-memory rounds (options)
// Tiles of up to 2^14 elements (2^13 of 8 bytes) for the settings that
// bound the grouping: at most maxg (<= 4) steps per register round.
constexpr int kRoundThreads = 512;

__device__ __forceinline__ uint32_t spad(uint32_t i) { return i + (i >> 5); }

// Applies steps j .. j-g+1 of a stage to the tile in shared memory, in
// groups of 2^g elements held in registers. `desc_fn(i)` gives the
// direction of element i (tile-local index).
template <typename T, int G, typename DescFn>
__device__ __forceinline__ void smem_steps(T *s, uint32_t tile_n, int j,
	DescFn desc_fn) {
	const int lo_bits = j - G;
	const uint32_t groups = tile_n >> G;
	const uint32_t inc = 1u << lo_bits;
	for (uint32_t q = threadIdx.x; q < groups; q += blockDim.x) {
		uint32_t low = q & (inc - 1);
		uint32_t base = ((q >> lo_bits) << j) | low;
		bool desc = desc_fn(base);
		T r[1 << G];
#pragma unroll
		for (int m = 0; m < (1 << G); ++m) r[m] = s[spad(base + m * inc)];
#pragma unroll
		for (int b = G - 1; b >= 0; --b) {
#pragma unroll
			for (int m = 0; m < (1 << G); ++m)
				if (!(m & (1 << b))) cmpxchg(r[m], r[m | (1 << b)], desc);
		}
#pragma unroll
		for (int m = 0; m < (1 << G); ++m) s[spad(base + m * inc)] = r[m];
	}
}

// Steps j..1 of one stage, at most maxg (<= 4) per barrier interval.
template <typename T, typename DescFn>
__device__ __forceinline__ void smem_stage_tail(T *s, uint32_t tile_n, int j,
	int maxg, DescFn desc_fn) {
	while (j >= 1) {
		int g = j < maxg ? j : maxg;
		switch (g) {
		case 4: smem_steps<T, 4>(s, tile_n, j, desc_fn); break;
		case 3: smem_steps<T, 3>(s, tile_n, j, desc_fn); break;
		case 2: smem_steps<T, 2>(s, tile_n, j, desc_fn); break;
		default: smem_steps<T, 1>(s, tile_n, j, desc_fn); break;
		}
		__syncthreads();
		j -= g;
	}
}

// FIRST: stages 1..t of every tile of 2^t elements; otherwise steps t..1 of
// `stage` (> t).
template <typename T, bool FIRST>
__global__ void __launch_bounds__(kRoundThreads, sizeof(T) <= 4 ? 3 : 2)
bitonic_rounds(T *data, int t, int stage, int maxg) {
	extern __shared__ __align__(16) unsigned char smem_raw[];
	T *s = reinterpret_cast<T *>(smem_raw);
	const uint32_t tile_n = 1u << t;
	const size_t tile_base = (size_t)blockIdx.x << t;
	T *g = data + tile_base;
	for (uint32_t i = threadIdx.x; i < tile_n; i += blockDim.x) s[spad(i)] = g[i];
	__syncthreads();
	if constexpr (FIRST) {
		for (int st = 1; st <= t; ++st) {
			if (st < t) {
				smem_stage_tail(s, tile_n, st, maxg, [st](uint32_t i) { return (bool)((i >> st) & 1); });
			} else {
				const bool d = (tile_base >> st) & 1;
				smem_stage_tail(s, tile_n, st, maxg, [d](uint32_t) { return d; });
			}
		}
	} else {
		const bool d = (tile_base >> stage) & 1;
		smem_stage_tail(s, tile_n, t, maxg, [d](uint32_t) { return d; });
	}
	for (uint32_t i = threadIdx.x; i < tile_n; i += blockDim.x) g[i] = s[spad(i)];
}

template <typename T>
__global__ void fill_value(T *p, size_t n, T v) {
	size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
	if (i < n) p[i] = v;
}

// ------------------------------------------------------------- launches
// What the per-kernel timing calls them, by BitonicUser.
struct TimerNames {
	const char *tile_sort, *global_steps, *tile_finish;
};
constexpr TimerNames kTimerNames[] = {
	{"abitonic_tile_sort", "abitonic_global_steps", "abitonic_tile_finish"},
	{"sbitonic_tile_sort", "sbitonic_global_steps", "sbitonic_tile_finish"},
	{"satradix_tile_sort", "satradix_global_steps", "satradix_tile_finish"}};

inline int ilog2(size_t v) {
	int r = 0;
	while (((size_t)1 << r) < v) ++r;
	return r;
}

// The global passes of `stage` down to stride 2^t, over the first `elems`
// elements, at most maxg steps each, in balanced groups (6 steps as 3 + 3,
// not 5 + 1): a pass of few steps per thread is the slowest per byte.
template <typename T>
cudaError_t global_passes(T *d, size_t elems, int stage, int t, int maxg, double bytes,
	const TimerNames &names, cudaStream_t s, unsigned &launches) {
	cudaError_t e = cudaSuccess;
	for (int j = stage; j > t && e == cudaSuccess;) {
		const int rem = j - t;
		const int npass = (rem + maxg - 1) / maxg;
		const int g = (rem + npass - 1) / npass;
		const size_t groups = elems >> g;
		KernelTimer tm(names.global_steps, s, bytes);
		auto go = [&](auto G) {
			constexpr int g_ = decltype(G)::value;
			constexpr int V = 16 / sizeof(T);
			if constexpr (g_ <= 3) {
				if ((uintptr_t)d % 16 == 0 && ((size_t)1 << (j - g_)) >= V)
					return launch_chained(bitonic_global_steps_v<T, g_>,
						(unsigned)((groups / V + 255) / 256), 256, 0, s, 1, d, groups, stage, j);
			}
			constexpr int th = gs_threads<T, g_>();
			return launch_chained(bitonic_global_steps<T, g_>, (unsigned)((groups + th - 1) / th),
				th, 0, s, 1, d, groups, stage, j);
		};
		switch (g) {
		case 7:
			if constexpr (sizeof(T) == 4) e = go(std::integral_constant<int, 7>());
			break;
		case 6:
			if constexpr (sizeof(T) >= 2) e = go(std::integral_constant<int, 6>());
			break;
		case 5: e = go(std::integral_constant<int, 5>()); break;
		case 4: e = go(std::integral_constant<int, 4>()); break;
		case 3: e = go(std::integral_constant<int, 3>()); break;
		case 2: e = go(std::integral_constant<int, 2>()); break;
		default: e = go(std::integral_constant<int, 1>()); break;
		}
		tm.stop();
		launches++;
		j -= g;
	}
	return e;
}

// Most steps of a global pass: a pass moves the whole array whatever its
// step count, so fewer, longer passes cut the bytes (1-byte types spill at
// 64 elements a thread).
template <typename T>
constexpr int kGlobalSteps = sizeof(T) == 4 ? 7 : sizeof(T) == 1 ? 5 : 6;

// Stages 1 .. min(T, stages) of every tile of src's n elements into out, of
// which n_out are written.
template <typename T, typename C>
cudaError_t launch_tile_sort(const T *src, T *out, size_t n, size_t n_out, size_t parts, int stages,
	double bytes, const TimerNames &names, cudaStream_t s, unsigned &launches) {
	auto kern = bitonic_tile<T, C, true>;
	cudaError_t e = cudaSuccess;
	if (C::kSmem > 48 * 1024)
		e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::kSmem);
	if (e != cudaSuccess) return e;
	KernelTimer tm(names.tile_sort, s, bytes);
	e = launch_chained(kern, (unsigned)parts, C::kThreads, C::kSmem, s, C::kCluster, src, out, n, n_out,
		std::min(stages, C::TL));
	tm.stop();
	launches++;
	return e;
}

// The sort with one-CTA tiles. `work` holds N elements (it is `dst` when
// n == N or one tile holds everything).
template <typename T, typename C>
cudaError_t run_tiles(const T *src, T *dst, T *work, size_t n, int logN,
	const TimerNames &names, cudaStream_t s, unsigned &launches) {
	constexpr int K = C::kK;
	const size_t N = (size_t)1 << logN;
	const double pass_bytes = 2.0 * (double)N * sizeof(T);
	if (logN <= K)
		return launch_tile_sort<T, C>(src, dst, n, n, 1, logN, pass_bytes, names, s, launches);
	auto fin_k = bitonic_tile<T, C, false>;
	cudaError_t e = cudaSuccess;
	if (C::kSmem > 48 * 1024)
		e = cudaFuncSetAttribute(fin_k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::kSmem);
	if (e == cudaSuccess)
		e = launch_tile_sort<T, C>(src, work, n, N, N >> K, logN, pass_bytes, names, s, launches);
	for (int stage = K + 1; stage <= logN && e == cudaSuccess; ++stage) {
		// A stage leaves blocks of padding alone as they are.
		const size_t elems = ((n + ((size_t)1 << stage) - 1) >> stage) << stage;
		e = global_passes<T>(work, elems, stage, K, kGlobalSteps<T>, pass_bytes, names, s, launches);
		if (e != cudaSuccess) break;
		const bool last = stage == logN;
		KernelTimer tf(names.tile_finish, s, pass_bytes);
		e = launch_chained(fin_k, (unsigned)(elems >> K), C::kThreads, C::kSmem, s, 1,
			(const T *)work, last ? dst : work, N, last ? n : N, stage);
		tf.stop();
		launches++;
	}
	return e;
}

// Settings that bound the grouping: at most max_ps steps per round and tiles
// of 2^max_sfs elements, on N elements in place.
template <typename T>
cudaError_t run_rounds(T *d, int logN, int max_ps, int max_sfs,
	const TimerNames &names, cudaStream_t s, unsigned &launches) {
	const size_t N = (size_t)1 << logN;
	int t = std::min(sizeof(T) >= 8 ? 13 : 14, logN);
	if (max_sfs >= 1 && max_sfs < t) t = max_sfs;
	const int maxg = std::max(1, std::min(4, max_ps));
	const int gmaxg = max_ps >= 4 ? kGlobalSteps<T> : maxg;
	const uint32_t tile_n = 1u << t;
	const size_t smem = (size_t)(tile_n + tile_n / 32 + 1) * sizeof(T);
	const unsigned threads = std::min<uint32_t>(kRoundThreads, std::max<uint32_t>(tile_n / 2, 32));
	cudaError_t e = cudaFuncSetAttribute(bitonic_rounds<T, true>,
		cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
	if (e == cudaSuccess)
		e = cudaFuncSetAttribute(bitonic_rounds<T, false>,
			cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
	const size_t tiles = N >> t;
	const double pass_bytes = 2.0 * (double)N * sizeof(T);
	for (int stage = t; stage <= logN && e == cudaSuccess; ++stage) {
		const bool first = stage == t;
		if (!first) e = global_passes<T>(d, N, stage, t, gmaxg, pass_bytes, names, s, launches);
		if (e != cudaSuccess) break;
		KernelTimer tm(first ? names.tile_sort : names.tile_finish, s, pass_bytes);
		auto kern = first ? bitonic_rounds<T, true> : bitonic_rounds<T, false>;
		kern<<<(unsigned)tiles, threads, smem, s>>>(d, t, stage, maxg);
		tm.stop();
		launches++;
		e = cudaGetLastError();
	}
	return e;
}

// Tiles by size and type. Up to kOneTile elements one tile does the whole
// sort: one CTA of 2^kSmallK elements, or (types up to 4 bytes) a cluster of
// eight of those. Beyond, tiles of one such CTA; small ones keep all SMs busy
// and their launches, chained, are cheap. us a sort:
//   float, tiles of 2^12 / 2^13 / 2^14 (16 elements a thread): 2^16 20.3 / 26.4
//   / -, 2^20 55.3 / 54.9 / -, 1.5 x 10^6 78.2 / 89.3 / -, 2^24 596 / 635 / -;
//   32 elements a thread: 2^16 22.7 / 27.3 / 41, 2^24 657 / 632 / 659; clusters
//   of eight over 2^12: 2^16 26, 2^20 63, 2^24 755; 2^15 14.6 in one cluster
//   against 17 in five launches.
//   double, 2^11 by 8 / 2^13 by 16: 2^16 37 / 63, 2^19 86 / 110, 2^20 138 / 132,
//   1.5 x 10^6 206 / 236, 2^22 496 / 499, 5 x 10^6 746 / 721, 2^24 2357 / 2145
//   (the compares bound the large sorts); clusters of eight over 2^12 by 16:
//   2^16 44. long: 2^20 102 / 105, 2^22 346 / 392, 5 x 10^6 488 / 560, 2^23 680
//   / 729, 2^24 1789 / 1797, 2^25 3833 / 3771.
//   char, 32 / 16 elements a thread: 2^16 27 / 26, 2^24 673 / 729.
template <typename T>
using SmallTile = typename std::conditional<sizeof(T) == 8, TileCfg<T, 11, 0, 3>,
	TileCfg<T, 12, 0, sizeof(T) == 1 ? 5 : 4>>::type;
template <typename T>
using ClusterTile = TileCfg<T, 12, 3, sizeof(T) == 1 ? 5 : 4>;
template <typename T>
constexpr int kOneTile = sizeof(T) == 8 ? 11 : 15;
// log2 of the padded size from which 8-byte elements take tiles of 2^13.
template <typename T>
constexpr int kBigTileMin = std::is_same<T, double>::value ? 23 : 25;

template <typename T>
cudaError_t sort_typed(const T *src, T *dst, size_t n, int max_ps, int max_sfs,
	BitonicUser user, CCLContext *ctx, cudaStream_t s, GError **err) {
	cudaError_t e = cudaSuccess;
	const int logN = ilog2(n);
	const size_t N = (size_t)1 << logN;
	const TimerNames &names = kTimerNames[user];
	unsigned launches = 0;
	T *tmp = nullptr;
	const int t0 = std::min(sizeof(T) >= 8 ? 13 : 14, logN);
	const bool rounds = max_ps < 4 || (max_sfs >= 1 && max_sfs < t0);
	if (N != n && (rounds || logN > kOneTile<T>)) {
		tmp = (T *)tmp_alloc(ctx, N * sizeof(T), s, err);
		if (!tmp) return cudaErrorMemoryAllocation;
	}
	T *work = tmp ? tmp : dst;
	if (rounds) {
		if (work != src)
			e = cudaMemcpyAsync(work, src, n * sizeof(T), cudaMemcpyDeviceToDevice, s);
		if (e == cudaSuccess && N != n) {
			const size_t pad = N - n;
			fill_value<T><<<(unsigned)((pad + 255) / 256), 256, 0, s>>>(tmp + n, pad,
				max_value<T>());
			launches++;
			e = cudaGetLastError();
		}
		if (e == cudaSuccess) e = run_rounds<T>(work, logN, max_ps, max_sfs, names, s, launches);
		if (e == cudaSuccess && tmp)
			e = cudaMemcpyAsync(dst, tmp, n * sizeof(T), cudaMemcpyDeviceToDevice, s);
	} else if (logN > SmallTile<T>::kK && logN <= kOneTile<T>) {
		if constexpr (sizeof(T) <= 4)
			e = launch_tile_sort<T, ClusterTile<T>>(src, dst, n, n, ClusterTile<T>::kCluster, logN,
				2.0 * (double)N * sizeof(T), names, s, launches);
	} else {
		bool big = false;
		if constexpr (sizeof(T) == 8) {
			big = logN >= kBigTileMin<T>;
			if (big) e = run_tiles<T, TileCfg<T, 13, 0, 4>>(src, dst, work, n, logN, names, s, launches);
		}
		if (!big) e = run_tiles<T, SmallTile<T>>(src, dst, work, n, logN, names, s, launches);
	}
	if (tmp) tmp_free(tmp, s);
	count_launches(launches);
	if (e != cudaSuccess) cuda_ok(e, err, "bitonic sort");
	return e;
}

}  // namespace
}  // namespace bitonic
}  // namespace clo
