// "satradix": stable LSD radix sort, onesweep style, 8-bit digits. Included by
// one unit per key width (radix_k{1,2,4,8}.cu), which compile in parallel.
//
// Result contract (src/cl_ops/sort/clo_sort_satradix.c:117-335 with the
// kernels of clo_sort_satradix.cl:34-258): a stable sort, ascending by the
// unsigned bit pattern of the key. The reference sorts with
// log2(radix)-bit digits; any digit width gives the same stable order, so
// the width here is a tuning choice (8 bits: 4 passes for 32-bit keys).
//
// Per sort, launches chained by programmatic serialisation (launch.h):
//   1. radix_prep clears the histograms and counters;
//   2. radix_upsweep_w reads the keys once, builds the 256-bin histogram of every digit position, and
//      its last CTA scans them into digit bases and writes the plan: which
//      passes run and between which buffers;
//   3. per digit position, radix_pass_tiles (one launch per pass), a CTA for
//      each tile or, in large sorts, resident CTAs that take tile after tile
//      (15360 32-bit keys; 7168 pairs of a 64-bit key and a 32-bit value),
//      tiles claimed in order from a counter:
//      a. keys are loaded in half-warp units (a unit's keys are in index
//         order; full tiles of 32-bit keys arrive by bulk copy into shared
//         memory), the tile's digit counts are published for the decoupled
//         lookback before the tile is ranked;
//      b. keys are ranked among equal digits of their unit, stably (lanes
//         in order, rounds in order): peers found through a shared-memory
//         OR mask in the low half of the unit's word for the digit, whose
//         high half holds the unit's next position; keys (and values) are
//         staged in shared memory in tile-sorted order;
//      c. one thread per digit looks back over the preceding tiles
//         (bounded waits) for the digit's global offset;
//      d. the staged tile is written out so that consecutive threads write
//         consecutive addresses of a digit's run.
// Passes whose digit has a single populated bin are skipped (the order of
// a stable sort by a constant digit is the identity): their CTAs end at
// once. The first pass reads the caller's input and the last one writes its
// output, whatever the number of passes between, so a sort into another
// buffer takes no copy (2^28 32-bit keys: 3.61 ms with one).
//
// HBM roofline per 32-bit key: 4 B (upsweep) + P x 8 B (passes), i.e.
// 36 B/key for P = 4.
#pragma once

#include <algorithm>
#include <type_traits>

#include "clo_internal.h"
#include "dev_common.cuh"
#include "launch.h"
#include "radix.h"
#include "timing.h"

namespace clo {
namespace radix {
namespace {

template <typename K>
__device__ __forceinline__ uint32_t digit_of(K k, int shift) {
	return (uint32_t)(k >> shift) & (kRadix - 1);
}

// --------------------------------------------------------------- plan
// One word per pass: how it runs and its buffers (0 the input, 1 the output,
// 2 the alternate), and which status buffer it uses.
constexpr uint32_t kPlanRun = 0, kPlanSkip = 1, kPlanCopy = 2;
__host__ __device__ constexpr uint32_t plan_word(uint32_t mode, uint32_t src, uint32_t dst,
	uint32_t st) {
	return mode | src << 2 | dst << 4 | st << 6;
}

// Control words of one sort: [hist][base][counters 8][plan 8][ticket], the
// first two of passes * 256 words. radix_prep clears all but the bases.
struct Control {
	uint32_t *hist;     // counts by pass and digit
	uint32_t *base;     // their exclusive sums over the digits of a pass
	uint32_t *counter;  // next tile of each pass
	uint32_t *plan;     // plan words
	uint32_t *ticket;   // upsweep CTAs that have added their counts
};
inline size_t control_words(int passes) { return 2 * (size_t)passes * kRadix + 32; }
inline Control control_at(uint32_t *w, int passes) {
	Control c;
	c.base = w;
	c.hist = w + (size_t)passes * kRadix;
	c.counter = c.hist + (size_t)passes * kRadix;
	c.plan = c.counter + 8;
	c.ticket = c.plan + 8;
	return c;
}

__global__ void __launch_bounds__(256) radix_prep(uint32_t *words, uint32_t count) {
	dev::pdl_wait();
	for (uint32_t i = threadIdx.x; i < count; i += 256) words[i] = 0;
}

// What the upsweep does besides counting: its CTAs clear the first pass's
// tile statuses between them, and the last one to finish writes the digit
// bases and the plan.
struct UpTail {
	Control c;
	uint4 *clear;      // status words to clear, in 16-byte units
	size_t clear_n;
	size_t n;
	bool in_place;     // input and output are one buffer
};

// The passes in the order they run alternate between the output and the
// alternate buffer so that the last one writes the output. In place, the
// first pass must not write its own input, so an odd number of passes is
// made even by letting one skipped pass copy; with nothing to do out of
// place, the first pass copies.
__device__ __forceinline__ void write_plan(uint32_t *plan, uint32_t trivial, int passes,
	bool in_place) {
	const uint32_t all = (1u << passes) - 1u;
	const int act = __popc(all & ~trivial);
	int copy = -1;
	if (in_place ? (act & 1) : act == 0) copy = __ffs(all & trivial) - 1;
	const int total = act + (copy >= 0);
	uint32_t prev = 0, run = 0;
	int i = 0;
	for (int p = 0; p < passes; ++p) {
		const bool active = !((trivial >> p) & 1u);
		if (!active && p != copy) {
			plan[p] = plan_word(kPlanSkip, 0, 0, 0);
			continue;
		}
		const uint32_t dst = ((total - 1 - i) & 1) ? 2u : 1u;
		plan[p] = plan_word(active ? kPlanRun : kPlanCopy, prev, dst, run & 1u);
		run += active;
		prev = dst;
		++i;
	}
}

__device__ __forceinline__ void upsweep_clear(const UpTail &t, uint32_t threads) {
	for (size_t i = blockIdx.x * (size_t)threads + threadIdx.x; i < t.clear_n;
		 i += (size_t)gridDim.x * threads)
		t.clear[i] = make_uint4(0, 0, 0, 0);
}

// Called by every CTA after its adds to the histograms (THREADS a multiple
// of 256).
template <int PASSES, int THREADS>
__device__ __forceinline__ void upsweep_tail(const UpTail &t) {
	__shared__ uint32_t s_last, s_trivial, s_tot[THREADS / 32];
	__threadfence();
	__syncthreads();
	if (threadIdx.x == 0) {
		s_last = atomicAdd(t.c.ticket, 1u) == gridDim.x - 1;
		s_trivial = 0;
	}
	__syncthreads();
	if (!s_last) return;
	__threadfence();
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	for (int b0 = 0; b0 < PASSES * kRadix; b0 += THREADS) {  // whole passes at a time
		const int b = b0 + (int)threadIdx.x;
		const bool valid = b < PASSES * kRadix;
		const uint32_t v = valid ? dev::ld_relaxed_u32(t.c.hist + b) : 0u;
		uint32_t inc = v;
#pragma unroll
		for (int d = 1; d < 32; d <<= 1) {
			const uint32_t u = __shfl_up_sync(0xffffffffu, inc, d);
			if (lane >= d) inc += u;
		}
		if (lane == 31) s_tot[warp] = inc;
		if (valid && v == (uint32_t)t.n) atomicOr(&s_trivial, 1u << (b / kRadix));
		__syncthreads();
		uint32_t base = inc - v;
		for (int w = warp & ~7; w < warp; ++w) base += s_tot[w];
		if (valid) t.c.base[b] = base;
		__syncthreads();
	}
	if (threadIdx.x == 0) write_plan(t.c.plan, s_trivial, PASSES, t.in_place);
}

// ----------------------------------------------------------- upsweep
// Histograms of all `passes` digit positions in one read, counted into
// lane columns shared by the CTA's warps through shared-memory adds: the
// counter of digit d of lane l lives in bank l, so a warp's 32 adds hit 32
// different banks whatever the digits. Each thread keeps kUpsweepInFlight
// 16-byte loads in flight.
constexpr int kUpsweepInFlight = 8;

// 1024-thread CTAs. The first four digit positions count into full 32-bit
// words (digit d of lane l at word d * 32 + l per position: one byte
// extract, one address computation and one shared add per key and
// position, and no overflow bound, 32 KB a position); positions five to
// eight (64-bit keys) into 16-bit halves of word (d >> 1) * 32 + l, 16 KB
// per position, with the grid keeping a thread at kUpwHalfKeysPerThread
// keys so that a half, which all 32 warps of a CTA add to, stays below
// 2^16 (eight positions: 192 KB, one CTA per SM).
constexpr int kUpwThreads = 1024;
constexpr size_t kUpwHalfKeysPerThread = 2000;

template <int PASSES>
constexpr size_t upw_smem() {
	return (size_t)(PASSES < 4 ? PASSES : 4) * kRadix * 32 * 4 +
		(size_t)(PASSES > 4 ? PASSES - 4 : 0) * (kRadix / 2) * 32 * 4;
}
// Word offset of position p's columns.
__host__ __device__ constexpr int upw_pos_base(int p) {
	return p <= 4 ? p * kRadix * 32 : 4 * kRadix * 32 + (p - 4) * (kRadix / 2) * 32;
}

template <typename K, int PASSES>
__global__ void __launch_bounds__(kUpwThreads, 1)
radix_upsweep_w(const K *keys, size_t n, int base_shift, UpTail tail) {
	extern __shared__ __align__(16) uint32_t up_smem[];
	for (int i = threadIdx.x; i < upw_pos_base(PASSES); i += kUpwThreads) up_smem[i] = 0;
	dev::pdl_wait();
	upsweep_clear(tail, kUpwThreads);
	__syncthreads();
	const int lane = threadIdx.x & 31;
	uint32_t *col = up_smem + lane;
	auto count = [&](int p, K key) {
		const uint32_t d = digit_of(key, base_shift + p * kRadixBits);
		if (p >= 4) atomicAdd(col + upw_pos_base(p) + (d >> 1) * 32, 1u << ((d & 1) << 4));
		else atomicAdd(col + upw_pos_base(p) + d * 32, 1u);
	};
	constexpr int PER = 16 / sizeof(K);  // keys per 16-byte load
	const bool aligned = ((uintptr_t)keys % 16) == 0;
	const size_t nvec = aligned ? n / PER : 0;
	const uint4 *kv4 = reinterpret_cast<const uint4 *>(keys);
	const size_t stride = (size_t)gridDim.x * kUpwThreads;
	size_t i = blockIdx.x * (size_t)kUpwThreads + threadIdx.x;
	for (; i + (kUpsweepInFlight - 1) * stride < nvec; i += kUpsweepInFlight * stride) {
		uint4 v[kUpsweepInFlight];
#pragma unroll
		for (int u = 0; u < kUpsweepInFlight; ++u) v[u] = dev::ld_stream_v4(kv4 + i + u * stride);
#pragma unroll
		for (int u = 0; u < kUpsweepInFlight; ++u) {
			const K *e = reinterpret_cast<const K *>(&v[u]);
#pragma unroll
			for (int q = 0; q < PER; ++q)
#pragma unroll
				for (int p = 0; p < PASSES; ++p) count(p, e[q]);
		}
	}
	for (; i < nvec; i += stride) {
		uint4 v = dev::ld_stream_v4(kv4 + i);
		const K *e = reinterpret_cast<const K *>(&v);
#pragma unroll
		for (int q = 0; q < PER; ++q)
#pragma unroll
			for (int p = 0; p < PASSES; ++p) count(p, e[q]);
	}
	for (size_t j = nvec * PER + blockIdx.x * (size_t)kUpwThreads + threadIdx.x; j < n;
		 j += stride) {
		const K key = keys[j];
#pragma unroll
		for (int p = 0; p < PASSES; ++p) count(p, key);
	}
	__syncthreads();
	for (int b = threadIdx.x; b < PASSES * kRadix; b += kUpwThreads) {
		const int p = b / kRadix, d = b % kRadix;
		const bool half = p >= 4;
		// Digit d's 32 columns, from a rotated start (no bank conflicts).
		const uint32_t *row = up_smem + upw_pos_base(p) + (half ? d >> 1 : d) * 32;
		const int hs = half ? (d & 1) << 4 : 0;
		uint32_t v = 0;
#pragma unroll 8
		for (int c = 0; c < 32; ++c) {
			const uint32_t w = row[(c + lane) & 31];
			v += half ? (w >> hs) & 0xFFFFu : w;
		}
		if (v) atomicAdd(tail.c.hist + b, v);
	}
	upsweep_tail<PASSES, kUpwThreads>(tail);
}

// ------------------------------------------------------- one-byte keys
// Writes the sorted bytes from the digit bases: byte i is the digit whose run
// holds i. A thread writes 16 bytes at a time, found by a search in the 256
// bases. Bound by the writes: a sort reads and writes each key once (2^26
// keys: 37 us against 217 with a ranked pass and, in place, a copy back).
constexpr int kFillBytesThreads = 256;
__global__ void __launch_bounds__(kFillBytesThreads)
radix_fill_bytes(uint8_t *out, size_t n, const uint32_t *base, bool in_place) {
	__shared__ uint32_t s_base[kRadix + 1];
	dev::pdl_wait();
	s_base[threadIdx.x] = base[threadIdx.x];
	if (threadIdx.x == 0) s_base[kRadix] = (uint32_t)n;
	__syncthreads();
	// In place, one key alone stays as it is (2^28 equal keys 100 -> 53 us).
	if (in_place && __syncthreads_or(s_base[threadIdx.x] == 0 && s_base[threadIdx.x + 1] == n)) return;
	const bool vec = ((uintptr_t)out % 16) == 0;
	const size_t stride = (size_t)gridDim.x * kFillBytesThreads * 16;
	for (size_t i0 = (blockIdx.x * (size_t)kFillBytesThreads + threadIdx.x) * 16; i0 < n; i0 += stride) {
		// The last digit whose base is at most i0.
		uint32_t d = 0;
#pragma unroll
		for (uint32_t step = kRadix / 2; step; step >>= 1)
			if (s_base[d + step] <= i0) d += step;
		const size_t end = i0 + 16 < n ? i0 + 16 : n;
		uint32_t w[4];
		if (s_base[d + 1] >= end) {
			w[0] = w[1] = w[2] = w[3] = d * 0x01010101u;
		} else {
#pragma unroll
			for (int q = 0; q < 16; ++q) {
				while (i0 + q < end && s_base[d + 1] <= i0 + q) ++d;
				if (q % 4 == 0) w[q / 4] = 0;
				w[q / 4] |= d << (8 * (q % 4));
			}
		}
		if (vec && end - i0 == 16) {
			*reinterpret_cast<uint4 *>(out + i0) = make_uint4(w[0], w[1], w[2], w[3]);
		} else {
#pragma unroll
			for (int q = 0; q < 16; ++q)
				if (i0 + q < end) out[i0 + q] = (uint8_t)(w[q / 4] >> (8 * (q % 4)));
		}
	}
}

// ------------------------------------------------------- two-byte keys
// Sorts of two-byte keys without values, from their histogram of 65536 bins:
// radix_count16 counts a stretch of the keys per CTA (one CTA an SM) into
// 16-bit counters in shared memory (128 KB) and stores its histogram;
// radix_sum16 adds the CTAs' histograms per bin and scans the bins of its
// block; radix_fill16 writes the sorted keys. The keys are read once and
// written once. 2^26 keys: 111 us against 442 with two ranked passes.
//
// Every kC16Step keys the counters of 32768 and more, of which there can be
// few, move to the 32-bit counters `over`, so that none overflows.
constexpr int kC16Threads = 1024, kC16Bins = 65536, kC16Step = 32760;
constexpr size_t kC16Smem = kC16Bins * 2;

__global__ void __launch_bounds__(kC16Threads, 1)
radix_count16(const uint16_t *keys, size_t n, size_t per_cta,
	uint32_t *parts, uint32_t *over) {
	extern __shared__ __align__(16) uint32_t c16[];  // bin b: half b & 1 of word b >> 1
	for (int i = threadIdx.x; i < kC16Bins / 8; i += kC16Threads)
		reinterpret_cast<uint4 *>(c16)[i] = make_uint4(0, 0, 0, 0);
	dev::pdl_wait();
	__syncthreads();
	auto count = [&](uint32_t k) { atomicAdd(c16 + (k >> 1), 1u << ((k & 1u) << 4)); };
	const size_t begin = blockIdx.x * per_cta;
	const size_t finish = begin + per_cta < n ? begin + per_cta : n;
	for (size_t a = begin; a < finish; a += kC16Step) {
		const size_t e = a + kC16Step < finish ? a + kC16Step : finish;
		// Keys up to a 16-byte boundary, whole vectors, the rest.
		const size_t head = (16 - ((uintptr_t)(keys + a) % 16)) % 16 / 2;
		const size_t v0 = a + head < e ? a + head : e;
		const uint32_t nv = (uint32_t)(e - v0) / 8;
		for (size_t i = a + threadIdx.x; i < v0; i += kC16Threads) count(keys[i]);
		const uint4 *v4 = reinterpret_cast<const uint4 *>(keys + v0);
		constexpr int U = (kC16Step / 8 + kC16Threads - 1) / kC16Threads;  // 4
		uint4 v[U];
		auto held = [&](int u) { return threadIdx.x + u * kC16Threads < nv; };
#pragma unroll
		for (int u = 0; u < U; ++u)
			if (held(u)) v[u] = dev::ld_stream_v4(v4 + threadIdx.x + u * kC16Threads);
		auto one_key = [](const uint4 &x) {
			return x.x == x.y && x.x == x.z && x.x == x.w && x.x >> 16 == (x.x & 0xFFFFu);
		};
		auto count_all = [&](const uint4 &x) {
			const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
			for (int q = 0; q < 4; ++q) {
				count(w[q] & 0xFFFFu);
				count(w[q] >> 16);
			}
		};
		// Where a thread's first eight keys are one key (sorted keys, few
		// values) its warp looks for such vectors and adds them up before
		// the shared counter, on which the lanes' adds would queue: us, 2^26
		// equal keys 293 without, sorted ones 296.
		if (__any_sync(0xffffffffu, held(0) && one_key(v[0]))) {
#pragma unroll
			for (int u = 0; u < U; ++u) {
				const bool same = held(u) && one_key(v[u]);
				const uint32_t m = __ballot_sync(0xffffffffu, same);
				if (same) {
					const uint32_t k = v[u].x & 0xFFFFu, peers = __match_any_sync(m, k);
					if ((peers & dev::lanemask_lt()) == 0)
						atomicAdd(c16 + (k >> 1), 8u * __popc(peers) << ((k & 1u) << 4));
				} else if (held(u)) {
					count_all(v[u]);
				}
			}
		} else {
#pragma unroll
			for (int u = 0; u < U; ++u)
				if (held(u)) count_all(v[u]);
		}
		for (size_t i = v0 + (size_t)nv * 8 + threadIdx.x; i < e; i += kC16Threads) count(keys[i]);
		__syncthreads();
		if (e < finish) {
			for (int i = threadIdx.x; i < kC16Bins / 8; i += kC16Threads) {
				const uint4 c = reinterpret_cast<const uint4 *>(c16)[i];
				if ((c.x | c.y | c.z | c.w) & 0x80008000u) {
					const uint32_t w[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
					for (int q = 0; q < 4; ++q) {
						const uint32_t high = (w[q] >> 15) & 0x00010001u;
						if (high & 1u) atomicAdd(over + 8 * i + 2 * q, 32768u);
						if (high >> 16) atomicAdd(over + 8 * i + 2 * q + 1, 32768u);
						c16[4 * i + q] = w[q] & 0x7FFF7FFFu;
					}
				}
			}
			__syncthreads();
		}
	}
	uint4 *dst = reinterpret_cast<uint4 *>(parts + (size_t)blockIdx.x * (kC16Bins / 2));
	for (int i = threadIdx.x; i < kC16Bins / 8; i += kC16Threads)
		dst[i] = reinterpret_cast<const uint4 *>(c16)[i];
}

// 128 CTAs of 512 bins: 256 words across, four histograms at a time. Writes
// each bin's start within its block and the block's total.
constexpr int kS16Bins = 512, kS16Blocks = kC16Bins / kS16Bins;
__global__ void __launch_bounds__(1024)
radix_sum16(const uint32_t *parts, uint32_t histograms,
	const uint32_t *over, uint32_t *start, uint32_t *block_total) {
	constexpr int W = kS16Bins / 2;
	__shared__ uint32_t s_lo[4][W], s_hi[4][W], s_warp[8];
	const int x = threadIdx.x % W, y = threadIdx.x / W, lane = threadIdx.x & 31;
	dev::pdl_wait();
	const uint32_t *p = parts + blockIdx.x * W + x;
	uint32_t lo = 0, hi = 0;
#pragma unroll 8
	for (uint32_t t = y; t < histograms; t += 4) {
		const uint32_t w = p[(size_t)t * (kC16Bins / 2)];
		lo += w & 0xFFFFu;
		hi += w >> 16;
	}
	s_lo[y][x] = lo;
	s_hi[y][x] = hi;
	__syncthreads();
	if (y == 0) {
		const uint2 o = *reinterpret_cast<const uint2 *>(over + blockIdx.x * kS16Bins + 2 * x);
		lo = o.x;
		hi = o.y;
#pragma unroll
		for (int q = 0; q < 4; ++q) {
			lo += s_lo[q][x];
			hi += s_hi[q][x];
		}
	}
	uint32_t inc = lo + hi;
#pragma unroll
	for (int d = 1; d < 32; d <<= 1) {
		const uint32_t t = __shfl_up_sync(0xffffffffu, inc, d);
		if (lane >= d) inc += t;
	}
	if (y == 0 && lane == 31) s_warp[x / 32] = inc;
	__syncthreads();
	if (y == 0) {
		uint32_t at = inc - lo - hi;
		for (int w = 0; w < x / 32; ++w) at += s_warp[w];
		*reinterpret_cast<uint2 *>(start + blockIdx.x * kS16Bins + 2 * x) = make_uint2(at, at + lo);
		if (x == W - 1) block_total[blockIdx.x] = at + lo + hi;
	}
}

// Each CTA writes an equal stretch of the output, a window of kF16Window
// bins' starts (a scan of the block totals, made by every CTA, plus the
// in-block starts) in shared memory at a time; a warp searches there for the
// bins of 1024 keys, its lanes between those for theirs.
constexpr int kF16Threads = 512, kF16Window = 2048, kF16Chunk = 1024;
__global__ void __launch_bounds__(kF16Threads)
radix_fill16(uint16_t *out, size_t n, size_t per_cta, const uint32_t *start,
	const uint32_t *block_total, bool in_place) {
	__shared__ uint32_t s_block[kS16Blocks + 1], s_warp[4], s_win[kF16Window + 1];
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	dev::pdl_wait();
	uint32_t v = tid < kS16Blocks ? block_total[tid] : 0u, inc = v;
#pragma unroll
	for (int d = 1; d < 32; d <<= 1) {
		const uint32_t t = __shfl_up_sync(0xffffffffu, inc, d);
		if (lane >= d) inc += t;
	}
	if (tid < kS16Blocks && lane == 31) s_warp[tid / 32] = inc;
	__syncthreads();
	if (tid < kS16Blocks) {
		uint32_t at = inc - v;
		for (int w = 0; w < tid / 32; ++w) at += s_warp[w];
		s_block[tid] = at;
	}
	if (tid == 0) s_block[kS16Blocks] = (uint32_t)n;
	__syncthreads();
	const bool vec = ((uintptr_t)out % 16) == 0;
	auto bin_start = [&](uint32_t b) {
		return b >= (uint32_t)kC16Bins ? (uint32_t)n : s_block[b / kS16Bins] + start[b];
	};
	const size_t o0 = blockIdx.x * per_cta, o1 = o0 + per_cta < n ? o0 + per_cta : n;
	if (o0 >= o1) return;
	// The last bin that starts at or before i (every thread alike).
	auto bin_of = [&](size_t i) {
		uint32_t b = 0;
#pragma unroll
		for (uint32_t step = kS16Blocks / 2; step; step >>= 1)
			if (s_block[b + step] <= i) b += step;
		b *= kS16Bins;
#pragma unroll
		for (uint32_t step = kS16Bins / 2; step; step >>= 1)
			if (bin_start(b + step) <= i) b += step;
		return b;
	};
	uint32_t wb = bin_of(o0);
	// In place, one key alone stays as it is (2^28 equal keys 314 -> 178 us).
	if (in_place && bin_start(wb) == 0 && bin_start(wb + 1) == n) return;
	for (size_t at = o0; at < o1; wb += kF16Window) {
		// A window of empty bins is jumped over.
		if (bin_start(wb + kF16Window) <= at) wb = bin_of(at);
		__syncthreads();
		for (int i = tid; i <= kF16Window; i += kF16Threads) s_win[i] = bin_start(wb + i);
		__syncthreads();
		// Whole vectors whose first key lies in the window's bins.
		const size_t wend = std::min<size_t>(o1, s_win[kF16Window]);
		// Last bin of the window that starts at or before i, among lo .. hi.
		auto find = [&](size_t i, uint32_t lo, uint32_t hi) {
			while (lo < hi) {
				const uint32_t mid = (lo + hi + 1) / 2;
				if (s_win[mid] <= i) lo = mid;
				else hi = mid - 1;
			}
			return lo;
		};
		for (size_t c = at + (size_t)warp * kF16Chunk; c < wend; c += (kF16Threads / 32) * kF16Chunk) {
			const uint32_t b0 = find(c, 0, kF16Window - 1);
			const uint32_t b1 = find(c + kF16Chunk - 1, b0, kF16Window - 1);
#pragma unroll
			for (int r = 0; r < kF16Chunk / 256; ++r) {
				const size_t i0 = c + r * 256 + lane * 8;
				if (i0 >= wend) break;
				const size_t end = i0 + 8 < o1 ? i0 + 8 : o1;
				uint32_t b = find(i0, b0, b1), next = s_win[b + 1];
				uint32_t w[4];
				if (next >= end) {
					w[0] = w[1] = w[2] = w[3] = (wb + b) * 0x00010001u;
				} else {
					b += wb;
#pragma unroll
					for (int q = 0; q < 8; ++q) {
						while (i0 + q < end && next <= i0 + q) {
							++b;
							next = b + 1 - wb <= (uint32_t)kF16Window ? s_win[b + 1 - wb] : bin_start(b + 1);
						}
						if (q % 2 == 0) w[q / 2] = b;
						else w[q / 2] |= b << 16;
					}
				}
				if (vec && end - i0 == 8) {
					*reinterpret_cast<uint4 *>(out + i0) = make_uint4(w[0], w[1], w[2], w[3]);
				} else {
#pragma unroll
					for (int q = 0; q < 8; ++q)
						if (i0 + q < end) out[i0 + q] = (uint16_t)(w[q / 2] >> (16 * (q % 2)));
				}
			}
		}
		if (wend > at) at += (wend - at + 7) / 8 * 8;
	}
}

// ------------------------------------------------- pass state and lookback
template <typename K, typename V>
struct PassArgs {
	K *keys[3];             // input, output, alternate
	V *vals[3];
	const uint32_t *plan;   // this pass's plan word
	const uint32_t *base;   // digit bases of this digit position
	uint32_t *status[2];    // tiles * 256 words each
	uint32_t *tile_counter;
	int *dev_status;
	size_t n;
	int shift;
};

// Lookback window: predecessor statuses read per round trip per digit. A
// tile's nearest inclusive predecessor is a few tiles back; wider windows
// measured slower.
#ifndef CLO_RADIX_LOOK_WINDOW
#define CLO_RADIX_LOOK_WINDOW 8
#endif
constexpr int kLookWindow = CLO_RADIX_LOOK_WINDOW;

// Threads per CTA of the pass: at least one per digit (threads below 256
// own a digit in the per-tile scans, the lookback and the output bases).
#ifndef CLO_RADIX_PASS_THREADS
#define CLO_RADIX_PASS_THREADS 256
#endif
constexpr int kPassThreads = CLO_RADIX_PASS_THREADS;
static_assert(kPassThreads >= 256 && kPassThreads <= 1024 && kPassThreads % 32 == 0,
	"pass CTA size");
// Keys per thread for one-word keys (0: the 256-thread shape scaled to the
// CTA size).
#ifndef CLO_RADIX_PASS_KPT1
#define CLO_RADIX_PASS_KPT1 0
#endif
// Resident CTAs per SM the pass is compiled for (registers a thread:
// 65536 / (CTAs x threads)).
#ifndef CLO_RADIX_PASS_MINB
#define CLO_RADIX_PASS_MINB 2
#endif

// Reads the statuses of tiles base, base-1, ..., base-W+1 for one digit
// (independent loads, one round trip), adds them in order to `excl` up to
// and including the first inclusive prefix. Returns true when a prefix was
// reached; otherwise moves `base` to the first unpublished predecessor
// (or past the window).
template <int W>
__device__ __forceinline__ bool lookback_window(const uint32_t *status, int digit,
	long long &base, uint32_t &excl) {
	uint32_t sv[W];
#pragma unroll
	for (int i = 0; i < W; ++i) {
		long long j = base - i;
		sv[i] = j >= 0 ? dev::ld_relaxed_u32(status + (size_t)j * kRadix + digit)
					   : kStPrefix;
	}
	int consumed = W;
	bool done = false;
#pragma unroll
	for (int i = 0; i < W; ++i) {
		if (!done && consumed == W) {
			if ((sv[i] & ~kStValue) == 0) {
				consumed = i;
			} else {
				excl += sv[i] & kStValue;
				if (sv[i] & kStPrefix) done = true;
			}
		}
	}
	if (!done) base -= consumed;
	return done;
}

// Lookback of sorts with few tiles (grouped_tiles), which all run at about the
// same time: with windows a tile's prefix waits for its predecessors'
// prefixes, a chain of tiles / 16 round trips. Here every tile also adds its
// counts to its group's row (kGroup tiles; arrivals in the top bits), and a
// tile sums the rows of the groups before its own and the counts of its own
// group's earlier tiles: no tile waits for another's prefix, and a tile reads
// tiles / 16 + 8 rows on average instead of tiles / 2. 2^20 32-bit keys (274
// tiles of 3840): 42.9 us a sort against 48.2.
constexpr uint32_t kGroup = 16;
constexpr uint32_t kGroupOne = 1u << 20;  // an arrival; kGroup tiles' keys stay below
__device__ __forceinline__ uint32_t group_lookback(const uint32_t *status, uint32_t num_tiles,
	uint32_t t, int digit, int *dev_status) {
	const uint32_t g = t / kGroup, first = g * kGroup;
	const uint32_t *groups = status + (size_t)num_tiles * kRadix + digit;
	const uint32_t *tiles = status + (size_t)first * kRadix + digit;
	const uint32_t rows = g + (t - first);
	uint32_t excl = 0, iter = 0;
	constexpr int B = 8;  // rows per round trip
	for (uint32_t r0 = 0; r0 < rows; r0 += B) {
		uint32_t v[B];
		bool ready;
		do {
			ready = true;
#pragma unroll
			for (int i = 0; i < B; ++i) {
				const uint32_t r = r0 + i;
				v[i] = r >= rows ? kStAgg
					: dev::ld_relaxed_u32((r < g ? groups + (size_t)r * kRadix
												 : tiles + (size_t)(r - g) * kRadix));
			}
#pragma unroll
			for (int i = 0; i < B; ++i) {
				const bool group_row = r0 + i < g;
				ready = ready && (group_row ? v[i] / kGroupOne == kGroup : (v[i] & ~kStValue) != 0);
			}
			if (!ready) {
				if (++iter >= dev::kSpinLimit) {
					dev::report_timeout(dev_status, DEV_ERR_LOOKBACK_TIMEOUT, (int)t);
					return excl;
				}
				dev::backoff(iter);
			}
		} while (!ready);
#pragma unroll
		for (int i = 0; i < B; ++i) excl += v[i] & (r0 + i < g ? kGroupOne - 1u : kStValue);
	}
	return excl;
}

// Ranking and count rows: 256 digits each, 264 words apart, odd rows 8
// words later, so rows 2w and 2w + 1 (the two units of warp w) hold a digit
// 16 banks apart and a digit both halves of a warp hold does not conflict.
constexpr int kRowWords = kRadix + 8;
__device__ __forceinline__ int row_of(int r) { return r * kRowWords + (r & 1) * 8; }

// ------------------------------------------------------- onesweep pass
// Tiles are claimed in order from an atomic counter, one per CTA or, in large
// sorts, one after the other by resident CTAs (the next one claimed once the
// tile's status is out), so every tile a CTA waits on belongs to a CTA that is
// running and waits on lower tiles only. Per tile:
//  1. keys (and values) are loaded in half-warp units: unit u holds the
//     tile's keys u * 16 KPT .. (u + 1) * 16 KPT - 1, round j of lane l the
//     key 16 j + l, so a unit's (round, lane) order is index order;
//  2. the digits are counted into per-unit rows (16-bit halves, units u and
//     u + 8 sharing a row); the thread of digit d turns them into unit
//     prefixes and the tile's count of d, and publishes the count as the
//     tile's lookback status (tile 0: its inclusive prefix) before the
//     tile is ranked;
//  3. ranking: the unit's word for digit d holds the unit's next tile
//     position for d in its upper half and the round's peer mask in its
//     lower half, so a round is one OR, one read and one store by the
//     lowest peer (stable: lanes in order, rounds in order); keys and
//     values are staged in shared memory at their tile-sorted positions;
//  4. the thread of digit d looks back over the preceding tiles' statuses
//     (windows of kLookWindow, bounded waits), publishes the inclusive
//     prefix and sets the digit's output base;
//  5. the staged tile is written out so that consecutive threads write
//     consecutive addresses of a digit's run.
// Consecutive tiles fill consecutive stretches of every digit's output, so
// output lines complete in L2 while they are hot, and the pass moves one
// read and one write of each key (and value). Tiles are large (TilesCfg)
// because each costs one lookback.
//
// Shared memory: a ranking row per half-warp unit and a count row per two
// units (row_of), the tile offsets and a scan array (256 words each), 64
// misc words, the staged tile (keys, then values).
// Full tiles of 32- or 64-bit keys (with 32- or 64-bit values, if any) are
// taken in with bulk copies (per half-warp unit one of its keys and one of
// its values, into the staging area; the copy engine, not the load/store
// pipe) and read from shared memory: a warp round of 32-bit elements is
// one conflict-free wavefront instead of two global ones (the two units
// of a warp are KPT x 64 bytes apart). 32-bit keys: 0.808 -> 0.790 ms a
// pass at 2^28.
#ifndef CLO_RADIX_BULK_LOAD
#define CLO_RADIX_BULK_LOAD 1
#endif
// 64-bit values as well: (u32, u64) pairs at 2^27 4.31 -> 3.26 ms a sort,
// (u64, u64) 10.28 -> 8.30 ms with the larger tiles the freed registers
// allow.
#ifndef CLO_RADIX_BULK_V8
#define CLO_RADIX_BULK_V8 1
#endif
template <typename K, typename V, bool HAS_V>
constexpr bool bulk_tile_load() {
	return CLO_RADIX_BULK_LOAD && (sizeof(K) == 4 || sizeof(K) == 8) &&
		(!HAS_V || sizeof(V) == 4 || (CLO_RADIX_BULK_V8 && sizeof(V) == 8));
}
// Landing-area elements per unit: the unit's elements, plus 16 where 4-byte
// elements of both units of a warp would otherwise fall in the same banks.
template <int KPT, int BYTES>
constexpr int land_unit_elems() {
	return 16 * KPT + (BYTES == 4 && (16 * KPT) % 32 == 0 ? 16 : 0);
}
// Landing-area bytes of the keys (the values follow them).
template <typename K, int THREADS, int KPT>
constexpr size_t land_key_bytes() {
	return (size_t)(THREADS / 16) * land_unit_elems<KPT, (int)sizeof(K)>() * sizeof(K);
}

template <typename K, typename V, bool HAS_V, int THREADS, int KPT>
constexpr size_t tiles_smem() {
	const size_t stage = (size_t)THREADS * KPT * (sizeof(K) + (HAS_V ? sizeof(V) : 0));
	const size_t land = bulk_tile_load<K, V, HAS_V>()
		? land_key_bytes<K, THREADS, KPT>() + (HAS_V
			? (size_t)(THREADS / 16) * land_unit_elems<KPT, (int)sizeof(V)>() * sizeof(V) : 0)
		: 0;
	return ((size_t)(THREADS / 16 + THREADS / 32) * kRowWords + 2 * kRadix + 64) *
		sizeof(uint32_t) + (stage > land ? stage : land);
}

// How a pass takes its tiles: one a CTA, looking back by windows or by groups,
// or tile after tile by resident CTAs.
constexpr int kTilesOne = 0, kTilesGrouped = 1, kTilesLoop = 2;

// n elements copied by the whole grid, eight 16-byte vectors a thread in
// flight where both sides are aligned.
template <typename T>
__device__ __forceinline__ void copy_elements(const T *in, T *out, size_t n) {
	const size_t threads = (size_t)gridDim.x * blockDim.x;
	const size_t self = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	size_t done = 0;
	if ((((uintptr_t)in | (uintptr_t)out) & 15) == 0) {
		const size_t vecs = n * sizeof(T) / 16;
		const uint4 *a = reinterpret_cast<const uint4 *>(in);
		uint4 *b = reinterpret_cast<uint4 *>(out);
		constexpr int B = 8;
		for (size_t i = self; i < vecs; i += B * threads) {
			uint4 r[B];
#pragma unroll
			for (int j = 0; j < B; ++j)
				if (i + j * threads < vecs) r[j] = a[i + j * threads];
#pragma unroll
			for (int j = 0; j < B; ++j)
				if (i + j * threads < vecs) b[i + j * threads] = r[j];
		}
		done = vecs * (16 / sizeof(T));
	}
	for (size_t i = done + self; i < n; i += threads) out[i] = in[i];
}

template <typename K, typename V, bool HAS_V, int THREADS, int KPT, int MINB, int MODE>
__global__ void __launch_bounds__(THREADS, MINB)
radix_pass_tiles(const __grid_constant__ PassArgs<K, V> a, uint32_t num_tiles) {
	constexpr int TILE = THREADS * KPT;
	constexpr int UNITS = THREADS / 16;
	constexpr int HALF = UNITS / 2;
	constexpr int UKEYS = 16 * KPT;  // a unit's keys
	static_assert(UKEYS <= 0xFFFF && TILE <= 0xFFFF, "16-bit unit and tile counts");
	extern __shared__ __align__(16) unsigned char smem[];
	uint32_t *s_rank = reinterpret_cast<uint32_t *>(smem);   // [UNITS] rows
	uint32_t *s_cnt = s_rank + UNITS * kRowWords;            // [HALF] rows
	uint32_t *s_tile_off = s_cnt + HALF * kRowWords;         // [256]
	uint32_t *s_part = s_tile_off + kRadix;                  // [256]
	uint32_t *s_misc = s_part + kRadix;                      // [64]
	unsigned char *s_stage = reinterpret_cast<unsigned char *>(s_misc + 64);

	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int unit = 2 * warp + (lane >> 4);
	const uint32_t l16 = lane & 15;
	const uint32_t lt16 = (1u << l16) - 1u;
	uint32_t *my_rank = s_rank + row_of(unit);
	uint32_t *my_cnt = s_cnt + row_of(unit % HALF);
	const uint32_t cnt_inc = 1u << ((unit / HALF) * 16);
	const int shift = a.shift;
	// Threads below 256 (whole warps) own digit pd in the per-digit steps.
	const bool owner = THREADS == kRadix || tid < kRadix;
	const int pd = tid & (kRadix - 1);
	const int dw = pd >> 5;

	constexpr bool BULK = bulk_tile_load<K, V, HAS_V>();
	constexpr int LK = land_unit_elems<KPT, (int)sizeof(K)>();
	constexpr int LV = land_unit_elems<KPT, (int)sizeof(V)>();
	uint64_t *bar = reinterpret_cast<uint64_t *>(s_misc + 32);
	K *land_k = reinterpret_cast<K *>(s_stage);
	V *land_v = reinterpret_cast<V *>(s_stage + land_key_bytes<K, THREADS, KPT>());
	// (Selected, not indexed: the parameters stay in the constant bank.)
	auto pick = [](auto *const (&b)[3], uint32_t i) { return i == 0 ? b[0] : i == 1 ? b[1] : b[2]; };
	auto bulk_ok_for = [&](const K *k, const V *v) {
		return BULK && ((uintptr_t)k % 16) == 0 && (!HAS_V || ((uintptr_t)v % 16) == 0);
	};
	// Tile tt's bulk copies (one thread).
	auto issue = [&](const K *kin, const V *vin, uint32_t tt) {
		dev::mbar_expect_tx(bar, (uint32_t)(TILE * (sizeof(K) + (HAS_V ? sizeof(V) : 0))));
		const size_t t0 = (size_t)tt * TILE;
#pragma unroll 1
		for (int u = 0; u < UNITS; ++u) {
			dev::bulk_g2s(land_k + u * LK, kin + t0 + u * UKEYS, (uint32_t)(UKEYS * sizeof(K)), bar);
			if constexpr (HAS_V)
				dev::bulk_g2s(land_v + u * LV, vin + t0 + u * UKEYS, (uint32_t)(UKEYS * sizeof(V)), bar);
		}
	};
	if (owner) {
#pragma unroll
		for (int i = 0; i < HALF; ++i) s_cnt[row_of(i) + pd] = 0;
	}
	dev::pdl_wait();
	if (tid == 0) {
		const uint32_t tt = atomicAdd(a.tile_counter, 1u);
		const uint32_t plan = *a.plan;
		s_misc[0] = tt;
		s_misc[1] = plan;
		const K *kin = pick(a.keys, (plan >> 2) & 3u);
		const V *vin = pick(a.vals, (plan >> 2) & 3u);
		if ((plan & 3u) == kPlanRun && bulk_ok_for(kin, vin) && tt < num_tiles &&
			(size_t)(tt + 1) * TILE <= a.n) {
			dev::mbar_init(bar, 1);
			issue(kin, vin, tt);
		}
	}
	const uint32_t gbase = owner ? a.base[pd] : 0;
	__syncthreads();
	uint32_t t = s_misc[0];
	// The plan's buffers: held where the registers allow it, else worked out
	// where they are used (us a sort, held / not: u32 2^28 3163 / 3236, u64 2^27
	// 4602 / 4566, (u32, u32) 2^27 2562 / 2466).
	const uint32_t plan = s_misc[1];
	const K *const kin0 = pick(a.keys, (plan >> 2) & 3u);
	K *const kout0 = pick(a.keys, (plan >> 4) & 3u);
	const V *const vin0 = pick(a.vals, (plan >> 2) & 3u);
	V *const vout0 = pick(a.vals, (plan >> 4) & 3u);
	uint32_t *const status0 = (plan >> 6) & 1u ? a.status[1] : a.status[0];
	uint32_t *const status1 = (plan >> 6) & 1u ? a.status[0] : a.status[1];
	if ((plan & 3u) == kPlanSkip) return;
	if ((plan & 3u) == kPlanCopy) {
		copy_elements(kin0, kout0, a.n);
		if constexpr (HAS_V) copy_elements(vin0, vout0, a.n);
		return;
	}
	constexpr bool HOLD = MODE != kTilesLoop || (sizeof(K) <= 4 && !HAS_V);
	auto keys_in = [&] { return HOLD ? kin0 : pick(a.keys, (s_misc[1] >> 2) & 3u); };
	auto keys_out = [&] { return HOLD ? kout0 : pick(a.keys, (s_misc[1] >> 4) & 3u); };
	auto vals_in = [&] { return HOLD ? vin0 : pick(a.vals, (s_misc[1] >> 2) & 3u); };
	auto vals_out = [&] { return HOLD ? vout0 : pick(a.vals, (s_misc[1] >> 4) & 3u); };
	auto status_now = [&] { return HOLD ? status0 : (s_misc[1] >> 6) & 1u ? a.status[1] : a.status[0]; };
	auto status_nxt = [&] { return HOLD ? status1 : (s_misc[1] >> 6) & 1u ? a.status[0] : a.status[1]; };
	if (t >= num_tiles) return;
	uint32_t parity = 0;

	do {
	// Keys (and values) of this thread's unit, round-major (index order).
	K k[KPT];
	V v[HAS_V ? KPT : 1];
	const K *__restrict__ kin = keys_in();
	const V *__restrict__ vin = vals_in();
	const size_t ubase = (size_t)t * TILE + (size_t)unit * UKEYS;
	if (bulk_ok_for(kin, vin) && (size_t)(t + 1) * TILE <= a.n) {
		if (!dev::mbar_wait_bounded(bar, parity)) {
			if (tid == 0) dev::report_timeout(a.dev_status, DEV_ERR_COPY_TIMEOUT, (int)t);
			dev::mbar_wait_bounded(bar, parity);  // the copies still in flight
		}
#pragma unroll
		for (int j = 0; j < KPT; ++j) {
			k[j] = land_k[unit * LK + j * 16 + l16];
			if constexpr (HAS_V) v[j] = land_v[unit * LV + j * 16 + l16];
		}
	} else {
#pragma unroll
		for (int j = 0; j < KPT; ++j) {
			const size_t idx = ubase + (size_t)j * 16 + l16;
			k[j] = idx < a.n ? kin[idx] : (K)~(K)0;
			if constexpr (HAS_V) v[j] = idx < a.n ? vin[idx] : (V)0;
		}
	}
#pragma unroll
	for (int j = 0; j < KPT; ++j) atomicAdd(my_cnt + digit_of(k[j], shift), cnt_inc);
	__syncthreads();
	// Unit prefixes of digit pd in unit order (written to the units' rank
	// words, the tile offset added below) and the tile's count.
	uint32_t sum = 0;
	uint32_t *st = HOLD ? status0 + (size_t)t * kRadix + pd : nullptr;
	if (owner) {
		uint32_t *status = status_now(), *status_next = status_nxt();
		uint32_t run = 0;
#pragma unroll
		for (int i = 0; i < HALF; ++i) {
			s_rank[row_of(i) + pd] = run << 16;
			run += s_cnt[row_of(i) + pd] & 0xFFFFu;
		}
#pragma unroll
		for (int i = 0; i < HALF; ++i) {
			s_rank[row_of(i + HALF) + pd] = run << 16;
			run += s_cnt[row_of(i) + pd] >> 16;
		}
		sum = run;
		// Publish the tile's count of digit pd (tile 0: its inclusive prefix).
		dev::st_relaxed_u32(HOLD ? st : status + (size_t)t * kRadix + pd, (t == 0 ? kStPrefix : kStAgg) | sum);
		status_next[(size_t)t * kRadix + pd] = 0;
		if constexpr (MODE == kTilesGrouped) {
			const size_t g = ((size_t)num_tiles + t / kGroup) * kRadix + pd;
			atomicAdd(status + g, kGroupOne + sum);
			if (t % kGroup == 0) status_next[g] = 0;
		}
		// Tile offsets of the digits: exclusive scan of the counts.
		uint32_t inc = sum;
#pragma unroll
		for (int d = 1; d < 32; d <<= 1) {
			uint32_t tt = __shfl_up_sync(0xffffffffu, inc, d);
			if (lane >= d) inc += tt;
		}
		if (lane == 31) s_misc[8 + dw] = inc;
		s_part[pd] = inc - sum;
	}
	__syncthreads();
	if (owner) {
		uint32_t to = s_part[pd];
#pragma unroll
		for (int w = 0; w < 8; ++w)
			if (w < dw) to += s_misc[8 + w];
#pragma unroll
		for (int i = 0; i < UNITS; ++i) s_rank[row_of(i) + pd] += to << 16;
		// Output index of staged position q of digit d is q + G[d] (mod
		// 2^32), G[d] = global base + lookback prefix - tile offset; the
		// prefix is added after the lookback.
		s_tile_off[pd] = gbase - to;
	}
	__syncthreads();
	K *sk = reinterpret_cast<K *>(s_stage);
	V *sv = reinterpret_cast<V *>(s_stage + (size_t)TILE * sizeof(K));
#pragma unroll
	for (int j = 0; j < KPT; ++j) {
		const uint32_t pos = dev::unit_rank_digit(my_rank + digit_of(k[j], shift), l16, lt16);
		if (pos < (uint32_t)TILE) {
			sk[pos] = k[j];
			if (HAS_V) sv[pos] = v[j];
		}
	}
	// Lookback over the preceding tiles for digit pd (bounded waits).
	uint32_t excl = 0;
	if (owner && t > 0) {
		uint32_t *status = status_now();
		if constexpr (MODE == kTilesGrouped) {
			excl = group_lookback(status, num_tiles, t, pd, a.dev_status);
		} else {
			long long base = (long long)t - 1;
			uint32_t iter = 0;
			bool done = lookback_window<kLookWindow>(status, pd, base, excl);
			while (!done && base >= 0) {
				uint32_t sw = dev::ld_relaxed_u32(status + (size_t)base * kRadix + pd);
				while ((sw & ~kStValue) == 0) {
					if (++iter >= dev::kSpinLimit) break;
					dev::backoff(iter);
					sw = dev::ld_relaxed_u32(status + (size_t)base * kRadix + pd);
				}
				if ((sw & ~kStValue) == 0) {
					dev::report_timeout(a.dev_status, DEV_ERR_LOOKBACK_TIMEOUT, (int)t);
					break;
				}
				done = lookback_window<kLookWindow>(status, pd, base, excl);
			}
			dev::st_relaxed_u32(HOLD ? st : status + (size_t)t * kRadix + pd, kStPrefix | (excl + sum));
		}
	}
	if (owner) s_tile_off[pd] += excl;
	__syncthreads();
	// The next tile is claimed (its status comes after this tile's, which is
	// out) and the counts cleared while the staged tile is written out.
	uint32_t next = 0;
	if constexpr (MODE == kTilesLoop) {
		if (tid == 0) next = atomicAdd(a.tile_counter, 1u);
		if (owner) {
#pragma unroll
			for (int i = 0; i < HALF; ++i) s_cnt[row_of(i) + pd] = 0;
		}
	}
	K *__restrict__ kout = keys_out();
	V *__restrict__ vout = vals_out();
#pragma unroll
	for (int i = 0; i < KPT; ++i) {
		const int q = i * THREADS + tid;
		const K key = sk[q];
		const size_t o = (uint32_t)(s_tile_off[digit_of(key, shift)] + (uint32_t)q);
		if (o < a.n) {
			kout[o] = key;
			if (HAS_V) vout[o] = sv[q];
		}
	}
	if constexpr (MODE != kTilesLoop) return;
	if (tid == 0) s_misc[0] = next;
	// The staging area was written by plain stores; bulk copies write it next.
	if constexpr (BULK) dev::fence_proxy_async();
	__syncthreads();
	t = s_misc[0];
	if (t >= num_tiles) return;
	parity ^= 1;
	if (tid == 0 && (size_t)(t + 1) * TILE <= a.n) {
		const K *ki = keys_in();
		const V *vi = vals_in();
		if (bulk_ok_for(ki, vi)) issue(ki, vi, t);
	}
	} while (MODE == kTilesLoop);
}

// ------------------------------------------------- small sorts in a cluster
// Small sorts in one launch: a cluster of CL CTAs (one for the smallest) holds the keys, CTA c the slice
// [c * slice, (c + 1) * slice) in its shared memory. Per digit: keys into
// registers by half-warp units as in radix_pass_tiles, unit counts, the
// CTA's digit totals read by every CTA through distributed shared memory,
// each unit's first position of every digit, ranks, and each key (and value)
// stored straight to its place in the slice that holds it. Two cluster
// barriers a digit take the place of a launch, a tile claim, a load, a
// lookback and a store to memory. A digit that holds every key is skipped.
constexpr int kClThreads = 512, kClUnits = kClThreads / 16, kClRounds = 16;
// Largest sort of one CTA and of a cluster of eight (0: the multi-launch sort
// or, for whole 4- and 8-byte keys, the bitonic tiles are faster). us a sort,
// this / multi-launch, pairs with two client copies: (u32, u32) 2^10 15.8 /
// 23.6, 2^12 20.5 / 31.8, 2^14 30.7 / 33.8, 2^15 41 / 36; (u64, u64) 2^12 34.8
// / 53.3, 2^14 51.7 / 59.4, 2^15 75.8 / 59.4; u16 keys 2^13 8.7 / 12.2; u8 keys
// 2^13 5.0 / 7.9. At 2^12 one CTA and eight are equal.
template <typename K>
constexpr size_t kOneCtaKeys = sizeof(K) <= 2 ? 8192 : 4096;
template <typename K, bool HAS_V>
constexpr size_t kClusterKeys = HAS_V || sizeof(K) == 8 ? 16384 : 0;

template <typename K, typename V, bool HAS_V>
constexpr size_t cluster_smem(size_t slice) {
	return ((size_t)(kClUnits + kClUnits / 2) * kRowWords + 2 * kRadix) * 4 +
		(slice * (sizeof(K) + (HAS_V ? sizeof(V) : 0)) + 15) / 16 * 16;
}

template <typename K, typename V, bool HAS_V, int CL>
__global__ void __launch_bounds__(kClThreads, 1)
radix_cluster(const K *kin, K *kout, const V *vin, V *vout, uint32_t n, uint32_t rounds,
	int passes) {
	constexpr int HALF = kClUnits / 2, R = kClRounds;
	extern __shared__ __align__(16) unsigned char cl_shared[];
	uint32_t *s_rank = reinterpret_cast<uint32_t *>(cl_shared);  // [units] rows
	uint32_t *s_cnt = s_rank + kClUnits * kRowWords;             // [HALF] rows
	uint32_t *s_own = s_cnt + HALF * kRowWords;                  // [2][256] digit totals
	const uint32_t slice = rounds * kClThreads;
	// 8-byte parts first, so that both are aligned (a slice is a multiple of
	// 512 elements).
	unsigned char *s_data = reinterpret_cast<unsigned char *>(s_own + 2 * kRadix);
	K *s_key = reinterpret_cast<K *>(s_data);
	V *s_val = reinterpret_cast<V *>(s_data + (size_t)slice * sizeof(K));
	__shared__ uint32_t s_scan[8];

	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int unit = 2 * warp + (lane >> 4);
	const uint32_t l16 = lane & 15, lt16 = (1u << l16) - 1u;
	const uint32_t rank = CL > 1 ? dev::cluster_rank() : 0u;
	uint32_t *my_rank = s_rank + row_of(unit);
	uint32_t *my_cnt = s_cnt + row_of(unit % HALF);
	const uint32_t cnt_inc = 1u << ((unit / HALF) * 16);
	const bool owner = tid < kRadix;
	const uint32_t first = rank * slice;                     // of this CTA's slice
	const uint32_t local = (uint32_t)unit * 16 * rounds + l16;  // of this thread, round 0
	const uint32_t held = first < n ? std::min<uint32_t>(slice, n - first) : 0;
	const uint32_t per_slice = (uint32_t)((1ull << 32) / slice) + 1u;  // pos / slice as a product
	auto barrier = [] {
		if constexpr (CL > 1) {
			dev::cluster_arrive();
			dev::cluster_wait();
		} else {
			__syncthreads();
		}
	};
	K k[R];
	V v[HAS_V ? R : 1];
	dev::pdl_wait();
#pragma unroll
	for (int j = 0; j < R; ++j) {
		const uint32_t i = local + j * 16;
		const bool ok = (uint32_t)j < rounds && i < held;
		k[j] = ok ? kin[first + i] : (K)0;
		if constexpr (HAS_V) v[j] = ok ? vin[first + i] : (V)0;
	}
	bool moved = false;  // the slice is in shared memory
	for (int p = 0; p < passes; ++p) {
		const int shift = p * kRadixBits;
		uint32_t *own = s_own + (p & 1) * kRadix;
		if (owner)
#pragma unroll
			for (int i = 0; i < HALF; ++i) s_cnt[row_of(i) + tid] = 0;
		__syncthreads();
#pragma unroll
		for (int j = 0; j < R; ++j)
			if ((uint32_t)j < rounds && local + j * 16 < held)
				atomicAdd(my_cnt + digit_of(k[j], shift), cnt_inc);
		__syncthreads();
		uint32_t c[HALF];
		uint32_t mine = 0;
		if (owner) {
#pragma unroll
			for (int i = 0; i < HALF; ++i) {
				c[i] = s_cnt[row_of(i) + tid];
				mine += (c[i] & 0xFFFFu) + (c[i] >> 16);
			}
			own[tid] = mine;
		}
		// Every CTA's totals are out, and every CTA has its keys in registers.
		barrier();
		uint32_t total = mine, before = 0, inc = 0;
		if (owner) {
			if constexpr (CL > 1) {
				const uint32_t a = dev::smem_u32(own + tid);
				total = 0;
#pragma unroll
				for (int r = 0; r < CL; ++r) {
					const uint32_t x = dev::ld_dsmem<uint32_t>(dev::map_shared(a, r));
					total += x;
					if ((uint32_t)r < rank) before += x;
				}
			}
			inc = total;
#pragma unroll
			for (int d = 1; d < 32; d <<= 1) {
				const uint32_t t = __shfl_up_sync(0xffffffffu, inc, d);
				if (lane >= d) inc += t;
			}
			if (lane == 31) s_scan[warp] = inc;
		}
		// (The same in every CTA.) One digit holds every key: nothing moves.
		if (__syncthreads_or(owner && total == n)) continue;
		if (owner) {
			uint32_t at = inc - total + before;
			for (int w = 0; w < warp; ++w) at += s_scan[w];
#pragma unroll
			for (int i = 0; i < HALF; ++i) {
				s_rank[row_of(i) + tid] = at << 16;
				at += c[i] & 0xFFFFu;
			}
#pragma unroll
			for (int i = 0; i < HALF; ++i) {
				s_rank[row_of(i + HALF) + tid] = at << 16;
				at += c[i] >> 16;
			}
		}
		__syncthreads();
#pragma unroll
		for (int j = 0; j < R; ++j) {
			if ((uint32_t)j < rounds) {
				const bool ok = local + j * 16 < held;
				const uint32_t pos = dev::unit_rank_digit_if(ok, my_rank + digit_of(k[j], shift), l16,
					lt16);
				if (ok) {
					if constexpr (CL > 1) {
						const uint32_t to = __umulhi(pos, per_slice), o = pos - to * slice;
						dev::st_dsmem<K>(dev::map_shared(dev::smem_u32(s_key + o), to), k[j]);
						if constexpr (HAS_V)
							dev::st_dsmem<V>(dev::map_shared(dev::smem_u32(s_val + o), to), v[j]);
					} else {
						s_key[pos] = k[j];
						if constexpr (HAS_V) s_val[pos] = v[j];
					}
				}
			}
		}
		barrier();
		moved = true;
		if (p + 1 < passes) {
#pragma unroll
			for (int j = 0; j < R; ++j) {
				const uint32_t i = local + j * 16;
				if ((uint32_t)j < rounds && i < held) {
					k[j] = s_key[i];
					if constexpr (HAS_V) v[j] = s_val[i];
				}
			}
		}
	}
	if (moved) {
		for (uint32_t i = tid; i < held; i += kClThreads) {
			kout[first + i] = s_key[i];
			if constexpr (HAS_V) vout[first + i] = s_val[i];
		}
	} else {
#pragma unroll
		for (int j = 0; j < R; ++j) {
			const uint32_t i = local + j * 16;
			if ((uint32_t)j < rounds && i < held) {
				kout[first + i] = k[j];
				if constexpr (HAS_V) vout[first + i] = v[j];
			}
		}
	}
	// No CTA leaves while another may still read its totals.
	if constexpr (CL > 1) barrier();
}

// Tile shape of the pass by the 32-bit register words a key (and value)
// takes: keys per thread and resident CTAs per SM, each the measured best
// at 2^27 - 2^28 elements (larger tiles spread the per-tile work -- row
// clears and scans, the lookback -- over more keys; the limits are 128
// registers a thread, without spills but for the 12 to 16 bytes of (u32, u64)
// pairs, and two CTAs' shared memory per SM).
// 32-bit keys: 15360-key tiles; 64-bit keys or 32-bit pairs: 10240;
// 12-byte pairs (bulk-loaded): 7168, 5120 for those loaded lane by lane
// (8- and 16-bit keys with 64-bit values); 16-byte pairs 5120.
template <typename K, typename V, bool HAS_V>
struct TilesCfg {
	static constexpr int kWords = (int)((sizeof(K) + 3) / 4) + (HAS_V ? (int)((sizeof(V) + 3) / 4) : 0);
	static constexpr int kThreads = kPassThreads;
#ifndef CLO_RADIX_PASS_KPT2
#define CLO_RADIX_PASS_KPT2 40
#endif
#ifndef CLO_RADIX_PASS_KPT3
#define CLO_RADIX_PASS_KPT3 28
#endif
#ifndef CLO_RADIX_PASS_KPT4
#define CLO_RADIX_PASS_KPT4 20
#endif
	static constexpr int kKpt256 = kWords == 1 ? 60 : kWords == 2 ? CLO_RADIX_PASS_KPT2
		: kWords == 3 ? (bulk_tile_load<K, V, HAS_V>() ? CLO_RADIX_PASS_KPT3 : 20)
		: (bulk_tile_load<K, V, HAS_V>() ? CLO_RADIX_PASS_KPT4 : 16);
	static constexpr int kKpt = (kWords == 1 && CLO_RADIX_PASS_KPT1 > 0) ? CLO_RADIX_PASS_KPT1
		: kKpt256 * 256 / kThreads;
	static constexpr int kMinBlocks = CLO_RADIX_PASS_MINB;
	static constexpr int kTile = kThreads * kKpt;
};

// Smaller tiles for smaller sorts: Q eighths of the keys per thread. A sort
// takes the smallest tile that leaves at most one tile per SM: fewer rounds a
// tile, and two tiles on an SM share its one shared-memory pipe. 32-bit keys,
// us a sort with 1 / 2 / 4 eighths: 2^18 27.9 / 30.4 / 35.8, 2^19 36.5 / 31.5
// / 36.9, 2^20 64.7 / 42.9 / 37.3.
template <typename K, typename V, bool HAS_V, int Q>
struct TilesCfgPart {
	using Big = TilesCfg<K, V, HAS_V>;
	static constexpr int kThreads = Big::kThreads;
	static constexpr int kKpt = Big::kKpt * Q / 8 < 4 ? 4 : Big::kKpt * Q / 8;
	static constexpr int kMinBlocks = Big::kMinBlocks;
	static constexpr int kTile = kThreads * kKpt;
};
// Most large tiles that look back by groups: one-word keys only up to a tile
// per SM (2^21 keys 54.0 us against 56.4 with windows, but 2^22, two tiles an
// SM, 90.4 against 83.3: that shape has no registers left), others through
// about two waves (2^22 (u64, u32) pairs 305 against 323, (u32, u32) 143
// against 159; 2^23 and 1100 tiles 610 against 576).
template <int WORDS>
size_t grouped_tiles(CCLContext *ctx) {
	return WORDS == 1 ? ctx->sm_count : ctx->sm_count * 21 / 5;
}

template <typename K, int PASSES>
cudaError_t launch_upsweep_p(cudaStream_t s, const K *keys, size_t n, int base_shift,
	int sm_count, const UpTail &tail) {
	constexpr size_t smem = upw_smem<PASSES>();
	auto kern = radix_upsweep_w<K, PASSES>;
	if (smem > 48 * 1024) {
		cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
			(int)smem);
		if (e != cudaSuccess) return e;
	}
	// 2048 threads per SM: two CTAs where shared memory allows (228 KB per
	// SM, 1 KB reserved per CTA); at least enough CTAs for the key cap of
	// the 16-bit halves.
	const int per_sm = (int)std::min<size_t>(2, (228 * 1024) / (smem + 1024));
	size_t grid = (size_t)sm_count * std::max(per_sm, 1);
	const size_t need = ((n * sizeof(K) + 15) / 16 + kUpwThreads - 1) / kUpwThreads;
	if (grid > need) grid = std::max<size_t>(need, 1);
	if (PASSES > 4) {
		const size_t cap = kUpwThreads * kUpwHalfKeysPerThread;
		grid = std::max(grid, (n + cap - 1) / cap);
	}
	return launch_chained(kern, (unsigned)grid, kUpwThreads, smem, s, 1, keys, n, base_shift, tail);
}

// The control words' clearing and the upsweep (2 launches).
template <typename K>
cudaError_t launch_upsweep(int passes, cudaStream_t s, const K *keys, size_t n,
	int sm_count, const UpTail &tail, int base_shift = 0) {
	cudaError_t e = launch_chained(radix_prep, 1, 256, 0, s, 1, tail.c.hist,
		(uint32_t)(passes * kRadix + 32));
	if (e != cudaSuccess) return e;
	switch (passes) {
	case 1: return launch_upsweep_p<K, 1>(s, keys, n, base_shift, sm_count, tail);
	case 2: return launch_upsweep_p<K, 2>(s, keys, n, base_shift, sm_count, tail);
	case 3: return launch_upsweep_p<K, 3>(s, keys, n, base_shift, sm_count, tail);
	case 4: return launch_upsweep_p<K, 4>(s, keys, n, base_shift, sm_count, tail);
	case 5: return launch_upsweep_p<K, 5>(s, keys, n, base_shift, sm_count, tail);
	case 6: return launch_upsweep_p<K, 6>(s, keys, n, base_shift, sm_count, tail);
	case 7: return launch_upsweep_p<K, 7>(s, keys, n, base_shift, sm_count, tail);
	default: return launch_upsweep_p<K, 8>(s, keys, n, base_shift, sm_count, tail);
	}
}

// Passes of at least three waves of tiles run as resident CTAs that take tile
// after tile: no gaps between CTAs, and a pass that the plan skips costs one
// wave of empty CTAs instead of one per tile (2^28 equal keys 353 -> 178 us a
// sort). Below, one CTA a tile is faster. us, one / loop: u32 keys 5 x 10^6
// 113 / 127, 10^7 193 / 192, 1.4 x 10^7 231 / 225, 2^27 1682 / 1622; u64 keys 4 x
// 10^6 228 / 239, 10^7 458 / 453, 2^27 4721 / 4597; (u32, u32) 10^7 286 / 295, 2 x
// 10^7 505 / 498, 2^27 2781 / 2796; (u64, u32) 7 x 10^6 488 / 498, 1.4 x 10^7
// 872 / 857, 2^27 6835 / 6856; (u64, u64) 10^7 796 / 781, 2^27 8692 / 8675. Pairs
// of 3 to 5 waves lose up to 3% and (u32, u64) 1 to 3% throughout (2 x 10^7 636 /
// 651, 2^27 3658 / 3723); they loop all the same, for the passes that are skipped.
constexpr size_t kLoopWaves = 3;
template <typename TC>
bool loop_tiles(size_t n, CCLContext *ctx) {
	return (n + TC::kTile - 1) / TC::kTile >= kLoopWaves * TC::kMinBlocks * ctx->sm_count;
}
template <typename TC, int MODE>
unsigned pass_grid(size_t ctiles, CCLContext *ctx) {
	return (unsigned)(MODE == kTilesLoop ? std::min<size_t>(ctiles,
		(size_t)TC::kMinBlocks * ctx->sm_count) : ctiles);
}

template <typename K, typename V, bool HAS_V, typename TC, int MODE>
cudaError_t sort_tiles(const K *src, K *dst, V *vals, size_t n, int passes,
	CCLContext *ctx, cudaStream_t s, GError **err) {
	// Tiles of TC's size.
	const size_t ctiles = (n + TC::kTile - 1) / TC::kTile;
	const unsigned grid = pass_grid<TC, MODE>(ctiles, ctx);
	const size_t smem = tiles_smem<K, V, HAS_V, TC::kThreads, TC::kKpt>();
	auto kern = radix_pass_tiles<K, V, HAS_V, TC::kThreads, TC::kKpt, TC::kMinBlocks, MODE>;
	cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
		(int)smem);
	if (e != cudaSuccess) {
		cuda_ok(e, err, "satradix");
		return e;
	}
	// In place with a single pass the result is made in the alternate buffer
	// and copied back.
	const bool in_place = src == dst;
	const bool copy_back = in_place && passes == 1;
	// Scratch: [control][status0][status1][alt keys][alt vals], a status row
	// per tile (and per group of tiles).
	const size_t status_words = (ctiles + (MODE == kTilesGrouped ? (ctiles + kGroup - 1) / kGroup : 0)) * kRadix;
	const size_t off_st0 = (control_words(passes) * 4 + 255) / 256 * 256;
	const size_t off_st1 = off_st0 + status_words * 4;
	const size_t off_keys = (off_st1 + status_words * 4 + 255) / 256 * 256;
	const size_t off_vals = (off_keys + n * sizeof(K) + 255) / 256 * 256;
	const size_t total = off_vals + (HAS_V ? n * sizeof(V) : 0);
	char *tmp = (char *)tmp_alloc(ctx, total, s, err);
	if (!tmp) return cudaErrorMemoryAllocation;
	UpTail tail;
	tail.c = control_at((uint32_t *)tmp, passes);
	tail.clear = (uint4 *)(tmp + off_st0);
	tail.clear_n = status_words / 4;
	tail.n = n;
	tail.in_place = in_place && !copy_back;
	K *alt_k = (K *)(tmp + off_keys);
	V *alt_v = HAS_V ? (V *)(tmp + off_vals) : nullptr;
	{
		KernelTimer t("satradix_upsweep", s, (double)n * sizeof(K));
		e = launch_upsweep<K>(passes, s, src, n, ctx->sm_count, tail);
		t.stop();
	}
	PassArgs<K, V> pa;
	pa.keys[0] = const_cast<K *>(src);
	pa.keys[1] = copy_back ? alt_k : dst;
	pa.keys[2] = alt_k;
	pa.vals[0] = vals;
	pa.vals[1] = copy_back ? alt_v : vals;
	pa.vals[2] = alt_v;
	pa.status[0] = (uint32_t *)(tmp + off_st0);
	pa.status[1] = (uint32_t *)(tmp + off_st1);
	pa.dev_status = ctx->d_status;
	pa.n = n;
	for (int p = 0; p < passes && e == cudaSuccess; ++p) {
		pa.plan = tail.c.plan + p;
		pa.base = tail.c.base + (size_t)p * kRadix;
		pa.tile_counter = tail.c.counter + p;
		pa.shift = p * kRadixBits;
		KernelTimer t("satradix_onesweep", s,
			2.0 * (double)n * (sizeof(K) + (HAS_V ? sizeof(V) : 0)));
		e = launch_chained(kern, grid, TC::kThreads, smem, s, 1, pa, (uint32_t)ctiles);
		t.stop();
	}
	if (copy_back && e == cudaSuccess) {
		e = cudaMemcpyAsync(dst, alt_k, n * sizeof(K), cudaMemcpyDeviceToDevice, s);
		if (e == cudaSuccess && HAS_V)
			e = cudaMemcpyAsync(vals, alt_v, n * sizeof(V), cudaMemcpyDeviceToDevice, s);
	}
	count_launches(2 + passes);
	tmp_free(tmp, s);
	if (e != cudaSuccess) cuda_ok(e, err, "satradix");
	return e;
}

// One-byte keys without values: their sorted order is their histogram.
inline cudaError_t sort_bytes(const uint8_t *src, uint8_t *dst, size_t n, CCLContext *ctx,
	cudaStream_t s, GError **err) {
	char *tmp = (char *)tmp_alloc(ctx, control_words(1) * 4, s, err);
	if (!tmp) return cudaErrorMemoryAllocation;
	UpTail tail = {};
	tail.c = control_at((uint32_t *)tmp, 1);
	tail.n = n;
	cudaError_t e;
	{
		KernelTimer t("satradix_upsweep", s, (double)n);
		e = launch_upsweep<uint8_t>(1, s, src, n, ctx->sm_count, tail);
		t.stop();
	}
	if (e == cudaSuccess) {
		const size_t vecs = (n + 15) / 16;
		const unsigned grid = (unsigned)std::min<size_t>((vecs + kFillBytesThreads - 1) /
			kFillBytesThreads, 8 * (size_t)ctx->sm_count);
		KernelTimer t("satradix_fill", s, (double)n);
		e = launch_chained(radix_fill_bytes, grid, kFillBytesThreads, 0, s, 1, dst, n,
			(const uint32_t *)tail.c.base, src == dst);
		t.stop();
	}
	count_launches(3);
	tmp_free(tmp, s);
	if (e != cudaSuccess) cuda_ok(e, err, "satradix");
	return e;
}

// Two-byte keys without values, from kC16Min keys (us, this / two ranked
// passes: 2^19 20.2 / 16.8, 2^20 21.0 / 20.7, 2^21 21.4 / 31.6, 2^24 48 / 136).
constexpr size_t kC16Min = (size_t)5 << 18;
inline cudaError_t sort_16(const uint16_t *src, uint16_t *dst, size_t n, CCLContext *ctx,
	cudaStream_t s, GError **err) {
	// One CTA an SM, each with at least a step of keys.
	const size_t ctas = std::max<size_t>(1, std::min<size_t>(ctx->sm_count, n / kC16Step));
	const size_t per_cta = ((n + ctas - 1) / ctas + 7) / 8 * 8;
	const size_t off_over = ctas * kC16Smem, off_start = off_over + kC16Bins * 4;
	const size_t off_total = off_start + kC16Bins * 4;
	char *tmp = (char *)tmp_alloc(ctx, off_total + kS16Blocks * 4, s, err);
	if (!tmp) return cudaErrorMemoryAllocation;
	uint32_t *over = (uint32_t *)(tmp + off_over), *start = (uint32_t *)(tmp + off_start);
	uint32_t *total = (uint32_t *)(tmp + off_total);
	cudaError_t e = cudaFuncSetAttribute(radix_count16, cudaFuncAttributeMaxDynamicSharedMemorySize,
		(int)kC16Smem);
	if (e == cudaSuccess) e = clear_chained(over, kC16Bins * 4, s);
	if (e == cudaSuccess) {
		KernelTimer t("satradix_upsweep", s, 2.0 * (double)n);
		e = launch_chained(radix_count16, (unsigned)ctas, kC16Threads, kC16Smem, s, 1, src, n, per_cta,
			(uint32_t *)tmp, over);
		t.stop();
	}
	if (e == cudaSuccess)
		e = launch_chained(radix_sum16, kS16Blocks, 1024, 0, s, 1, (const uint32_t *)tmp,
			(uint32_t)ctas, (const uint32_t *)over, start, total);
	if (e == cudaSuccess) {
		const size_t cap = 2 * (size_t)ctx->sm_count;
		const size_t out_per = std::max<size_t>((n + cap - 1) / cap, kF16Chunk * 4) / 8 * 8 + 8;
		const unsigned grid = (unsigned)((n + out_per - 1) / out_per);
		KernelTimer t("satradix_fill", s, 2.0 * (double)n);
		e = launch_chained(radix_fill16, grid, kF16Threads, 0, s, 1, dst, n, out_per, (const uint32_t *)start,
			(const uint32_t *)total, src == dst);
		t.stop();
	}
	count_launches(3);
	tmp_free(tmp, s);
	if (e != cudaSuccess) cuda_ok(e, err, "satradix");
	return e;
}

template <typename K, typename V, bool HAS_V, int CL>
cudaError_t sort_cluster(const K *src, K *dst, V *vals, size_t n, int passes, cudaStream_t s,
	GError **err) {
	const size_t rounds = (n + (size_t)CL * kClThreads - 1) / ((size_t)CL * kClThreads);
	const size_t smem = cluster_smem<K, V, HAS_V>(rounds * kClThreads);
	auto kern = radix_cluster<K, V, HAS_V, CL>;
	cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
		(int)cluster_smem<K, V, HAS_V>(kClThreads * kClRounds));
	if (e == cudaSuccess) {
		KernelTimer t("satradix_cluster", s, 2.0 * (double)n * (sizeof(K) + (HAS_V ? sizeof(V) : 0)));
		e = launch_chained(kern, CL, kClThreads, smem, s, CL, src, dst, (const V *)vals, vals,
			(uint32_t)n, (uint32_t)rounds, passes);
		t.stop();
		count_launches(1);
	}
	if (e != cudaSuccess) cuda_ok(e, err, "satradix");
	return e;
}

template <typename K, typename V, bool HAS_V>
cudaError_t sort_typed(const void *src, void *dst, void *vals, size_t n, int sort_bits,
	CCLContext *ctx, cudaStream_t s, GError **err) {
	const int passes = sort_bits / kRadixBits;
	if (n >= (size_t)kStValue) {
		set_error(err, CLO_ERROR_ARGS,
			"satradix: %zu elements exceed the single-sort limit of 2^30 - 1", n);
		return cudaErrorInvalidValue;
	}
	const K *ks = (const K *)src;
	K *kd = (K *)dst;
	V *v = (V *)vals;
	if (n <= kOneCtaKeys<K>) return sort_cluster<K, V, HAS_V, 1>(ks, kd, v, n, passes, s, err);
	if constexpr (kClusterKeys<K, HAS_V> > 0) {
		if (n <= kClusterKeys<K, HAS_V>)
			return sort_cluster<K, V, HAS_V, 8>(ks, kd, v, n, passes, s, err);
	}
	if constexpr (sizeof(K) == 1 && !HAS_V) return sort_bytes(ks, kd, n, ctx, s, err);
	if constexpr (sizeof(K) == 2 && !HAS_V) {
		if (passes == 2 && n >= kC16Min) return sort_16(ks, kd, n, ctx, s, err);
	}
	// The smallest tile that leaves at most one tile per SM; beyond, large
	// tiles.
	const size_t sms = (size_t)ctx->sm_count;
	auto fits = [&](size_t tile) { return (n + tile - 1) / tile <= sms; };
	auto go = [&](auto tc, auto mode) {
		return sort_tiles<K, V, HAS_V, decltype(tc), decltype(mode)::value>(ks, kd, v, n, passes,
			ctx, s, err);
	};
	using Yes = std::integral_constant<int, kTilesGrouped>;
	using One = std::integral_constant<int, kTilesOne>;
	using Loop = std::integral_constant<int, kTilesLoop>;
	using P1 = TilesCfgPart<K, V, HAS_V, 1>;
	using P2 = TilesCfgPart<K, V, HAS_V, 2>;
	using P4 = TilesCfgPart<K, V, HAS_V, 4>;
	using P6 = TilesCfgPart<K, V, HAS_V, 6>;
	using Big = TilesCfg<K, V, HAS_V>;
	if (fits(P1::kTile)) return go(P1(), Yes());
	if (fits(P2::kTile)) return go(P2(), Yes());
	if (fits(P4::kTile)) return go(P4(), Yes());
	if (fits(P6::kTile)) return go(P6(), Yes());
	if (n <= Big::kTile * grouped_tiles<Big::kWords>(ctx)) return go(Big(), Yes());
	return loop_tiles<Big>(n, ctx) ? go(Big(), Loop()) : go(Big(), One());
}

// Stable partition of n keys by the top 8 of their sort_bits low bits:
// keys_out receives the keys grouped by that digit, in input order within a
// digit; counts (host) receives the 256 group sizes. One histogram kernel
// for the digit, one pass, a host readback of its 256 counts.
template <typename K>
cudaError_t msd_partition_typed(const K *keys_in, K *keys_out, size_t n, int sort_bits,
	uint32_t *counts, CCLContext *ctx, cudaStream_t s, GError **err) {
	using TC = TilesCfg<K, uint32_t, false>;
	const int shift = sort_bits - kRadixBits;
	const size_t ctiles = (n + TC::kTile - 1) / TC::kTile;
	const unsigned grid = pass_grid<TC, kTilesLoop>(ctiles, ctx);
	const size_t smem = tiles_smem<K, uint32_t, false, TC::kThreads, TC::kKpt>();
	auto kern = radix_pass_tiles<K, uint32_t, false, TC::kThreads, TC::kKpt, TC::kMinBlocks,
		kTilesLoop>;
	cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
		(int)smem);
	if (e != cudaSuccess) {
		cuda_ok(e, err, "satradix partition");
		return e;
	}
	const size_t status_words = ctiles * kRadix;
	const size_t off_st0 = (control_words(1) * 4 + 255) / 256 * 256;
	const size_t off_st1 = off_st0 + status_words * 4;
	char *tmp = (char *)tmp_alloc(ctx, off_st1 + status_words * 4, s, err);
	if (!tmp) return cudaErrorMemoryAllocation;
	UpTail tail;
	tail.c = control_at((uint32_t *)tmp, 1);
	tail.clear = (uint4 *)(tmp + off_st0);
	tail.clear_n = status_words / 4;
	tail.n = n;
	tail.in_place = false;
	{
		KernelTimer t("satradix_upsweep", s, (double)n * sizeof(K));
		e = launch_upsweep<K>(1, s, keys_in, n, ctx->sm_count, tail, shift);
		t.stop();
	}
	if (e == cudaSuccess) {
		// One populated group: the plan makes the pass a copy.
		PassArgs<K, uint32_t> pa = {};
		pa.keys[0] = const_cast<K *>(keys_in);
		pa.keys[1] = keys_out;
		pa.plan = tail.c.plan;
		pa.base = tail.c.base;
		pa.status[0] = (uint32_t *)(tmp + off_st0);
		pa.status[1] = (uint32_t *)(tmp + off_st1);
		pa.tile_counter = tail.c.counter;
		pa.dev_status = ctx->d_status;
		pa.n = n;
		pa.shift = shift;
		KernelTimer t("satradix_onesweep", s, 2.0 * (double)n * sizeof(K));
		e = launch_chained(kern, grid, TC::kThreads, smem, s, 1, pa, (uint32_t)ctiles);
		t.stop();
	}
	if (e == cudaSuccess)
		e = cudaMemcpyAsync(counts, tail.c.hist, kRadix * 4, cudaMemcpyDeviceToHost, s);
	if (e == cudaSuccess) e = cudaStreamSynchronize(s);
	count_launches(3);
	tmp_free(tmp, s);
	if (e != cudaSuccess) cuda_ok(e, err, "satradix partition");
	return e;
}

template <typename K>
cudaError_t sort_keys_vals(const void *src, void *dst, void *vals, size_t n, int val_bytes,
	int sort_bits, CCLContext *ctx, cudaStream_t s, GError **err) {
	switch (val_bytes) {
	case 0: return sort_typed<K, uint32_t, false>(src, dst, nullptr, n, sort_bits, ctx, s, err);
	case 4: return sort_typed<K, uint32_t, true>(src, dst, vals, n, sort_bits, ctx, s, err);
	case 8: return sort_typed<K, uint64_t, true>(src, dst, vals, n, sort_bits, ctx, s, err);
	}
	set_error(err, CLO_ERROR_ARGS, "Unsupported value width %d", val_bytes);
	return cudaErrorInvalidValue;
}

}  // namespace

template <typename K>
cudaError_t sort(const void *src, void *dst, void *vals, size_t n, int val_bytes, int sort_bits,
	CCLContext *ctx, cudaStream_t s, GError **err) {
	return sort_keys_vals<K>(src, dst, vals, n, val_bytes, sort_bits, ctx, s, err);
}

template <typename K>
cudaError_t msd_partition(const void *keys_in, void *keys_out, size_t n, int sort_bits,
	uint32_t *counts, CCLContext *ctx, cudaStream_t s, GError **err) {
	return msd_partition_typed<K>((const K *)keys_in, (K *)keys_out, n, sort_bits, counts, ctx, s,
		err);
}

}  // namespace radix
}  // namespace clo
