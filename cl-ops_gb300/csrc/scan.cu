// Exclusive prefix sum ("blelloch" scanner) as one single-pass kernel with
// decoupled lookback.
//
// Semantics follow src/cl_ops/scan/clo_scan_blelloch.cl:49-211: out[0] = 0
// and out[i] = sum_{j<i} (SUM_TYPE) in[j], with the element converted to
// the sum type by C rules and the sum wrapping modulo 2^(8*sizeof(SUM)).
// Integer addition is associative, so the result is bit-identical to the
// reference's work-group Blelloch trees whatever the summation order.
//
// Layout (scan_rows.cuh): tiles of 4096 to 16384 elements by type and size
// (ScanBig and the ones after it), held in registers as rows of whole vectors per lane; a row's scan is a warp scan of
// the lanes' run sums. Tiles take ids from an atomic counter (so a tile only
// ever waits on tiles already running), publish their aggregate, then warp 0
// looks back over a 64-tile window per round trip until it meets an
// inclusive prefix. Status words carry their own ready bits, so neither side
// needs a memory fence. Every wait is bounded. Staging the tile in shared
// memory (scan_staged.cuh: a lane scans 16 consecutive elements, seven shared
// wavefronts per 32 elements for uint -> ulong) takes 589 us at 2^28 against
// 517; it stays for the types and alignments the rows are slow at
// (staged_scan).
//
// HBM roofline: sizeof(in) + sizeof(out) bytes per element (12 B for
// uint -> ulong), plus 32 B of tile status per tile.
#include <algorithm>
#include <atomic>
#include <mutex>
#include <type_traits>

#include "clo_internal.h"
#include "dev_common.cuh"
#include "launch.h"
#include "scan_rows.cuh"
#include "scan_staged.cuh"
#include "scan_status.cuh"
#include "timing.h"

namespace clo {
namespace {

using scanrows::Rows;

using lb::Slots;
using lb::TileStatus;
using lb::publish;
using lb::read_status;
using lb::warp_sum;

template <typename Acc>
__device__ __forceinline__ Acc shfl_up(Acc v, int d) {
	return __shfl_up_sync(0xffffffffu, v, d);
}

// Persistent CTAs (one per resident slot) take tiles in order from an
// atomic counter. Per tile: the sums of the tile already in registers and
// publication of its aggregate; then, while warp 0 looks back, every
// warp issues the loads of the CTA's next tile (claimed at the top of the
// iteration) into registers and sums them, so the next tile's aggregate is
// published as soon as the lookback ends -- before this tile's outputs are
// written -- and no later tile waits on it longer than on a freshly
// launched one; after the outputs the prefetched tile becomes the current
// one. Every wait is on a lower tile id (down to tile 0, which
// publishes its prefix at once), so the waits cannot form a cycle.
template <typename InT, typename OutT, int THREADS, int TILE, int MINB, bool KEEP = false>
struct ScanCfg {
	static constexpr int kThreads = THREADS, kTile = TILE, kMinBlocks = MINB;
	static constexpr bool kKeepShared = KEEP, kStaged = false;
	using R = Rows<InT, OutT, THREADS, TILE>;
};
// The staged kernel's shape.
template <typename InT, typename OutT>
struct ScanStaged {
	static constexpr int kThreads = scantile::kThreads, kTile = scantile::kTile;
	static constexpr bool kStaged = true;
};
// Sums of one or two bytes, or narrower than the input: one shape for all.
template <typename InT, typename OutT>
constexpr bool kOneShape = sizeof(OutT) <= 2 || (sizeof(InT) > sizeof(OutT));
template <bool C, typename A, typename B>
using If = typename std::conditional<C, A, B>::type;

// Threads, tile and resident CTAs per SM (registers: 65536 / (CTAs x
// threads)), and whether the current tile waits in shared memory while the
// next one is loaded (KEEP: each thread parks its own vectors, conflict-free;
// two tiles' registers leave one CTA fewer an SM or spill more).
// The tile rate is bounded by the lookback (a window of 64 tiles a round trip,
// about 80 tiles a microsecond), so narrow types take tiles twice as long.
// Measured at 2^28 (us): uint -> ulong two CTAs 559, three with KEEP 517, four
// 547; ulong -> ulong 804 / 694 (two CTAs) / 1023 (three); uint -> uint
// 16384-element tiles 380 / 356 (two) / 498 (three), 8192 406; uchar -> uint
// 16384 256 (three) / 275 (two), 8192 404; ushort -> uint 310 (three, with 168
// bytes of spills a thread) / 293 (two, none), 2^24 30.5 / 24.4. Spills that
// remain, a thread: uchar -> uint 84 bytes, ulong -> ulong 60, uint -> uint
// 48, uint -> ulong in 4096-element tiles 20. Windows of 96 and 128 tiles and
// 512-thread CTAs were slower.
template <typename InT, typename OutT>
using ScanBig = If<kOneShape<InT, OutT>, ScanCfg<InT, OutT, 256, 8192, 1>,
	If<sizeof(OutT) == 8, If<sizeof(InT) == 8, ScanCfg<InT, OutT, 256, 8192, 2, true>,
		If<sizeof(InT) == 4, ScanCfg<InT, OutT, 256, 8192, 3, true>, ScanCfg<InT, OutT, 256, 8192, 2>>>,
	If<sizeof(InT) == 4, ScanCfg<InT, OutT, 256, 16384, 2, true>,
		ScanCfg<InT, OutT, 256, 16384, sizeof(InT) == 2 ? 2 : 3>>>>;
// From kSmallMax to kMidMax elements uint -> ulong tiles stay in registers: with
// about one tile a CTA nothing is prefetched (2^22 16.2 us against 17.9).
constexpr size_t kMidMax = (size_t)1 << 23;
template <typename InT, typename OutT>
using ScanMid = If<sizeof(InT) == 4 && sizeof(OutT) == 8, ScanCfg<InT, OutT, 256, 8192, 2>,
	ScanBig<InT, OutT>>;
// Up to kSmallMax elements, 4096-element tiles: twice the CTAs, each with
// half the rows to scan (2^18 uint -> ulong 6.3 us against 8.0, 2^20 8.3
// against 9.1; 2^22 20.8 against 17.5).
constexpr size_t kSmallMax = (size_t)1 << 20;
template <typename InT, typename OutT>
using ScanSmall = If<kOneShape<InT, OutT>, ScanBig<InT, OutT>,
	If<sizeof(InT) == 8, ScanCfg<InT, OutT, 512, 4096, 2>, ScanCfg<InT, OutT, 256, 4096, 4>>>;
// One tile of 1024 threads, in one launch without statuses (5003 uint ->
// ulong: 8.8 us with a memset and a 256-thread tile, 3.9 so).
template <typename InT, typename OutT>
using ScanOne = If<kOneShape<InT, OutT>, ScanBig<InT, OutT>, ScanCfg<InT, OutT, 1024, 8192, 1>>;

// Scans that take the staged kernel (scan_staged.cuh), which moves whole lines
// whatever the types and the alignment. A row's lanes are kE elements apart:
// with sums narrower than the input that is 64 to 256 bytes, and arrays that
// are not 16-byte aligned are taken element by element at that distance. us,
// rows / staged (the staged kernel before the rows came, unchained, in brackets):
//   sums of 1 or 2 bytes or narrower than the input: uint -> uchar 2^20 8.3 / 8.2
//   (12.9), 2^22 15.2 / 13.2, 2^28 627 / 322 (333); ushort -> ushort 2^22 10.9 /
//   13.3, 2^23 18.7 / 17.9, 2^28 467 / 351 (361); ulong -> uint 2^22 16.8 / 16.0,
//   6 x 10^6 21.4 / 22.5, 2^24 55 / 46, 2^28 787 / 614 (619);
//   inputs of 1 or 2 bytes, sums of 8 (too few bytes in flight with two CTAs an
//   SM): uchar 12 x 10^6 29.2 / 30.0, 2^24 36.5 / 36.2, 2^28 486 / 440 (447);
//   unaligned: uint -> uint 2^18 6.5 / 7.5, 2^19 7.1 / 8.3, 2^20 11.9 / 10.7, 2^26
//   360 / 204 (213); uchar -> ulong 2^26 666 / 201 (209); sums of the first kind
//   at every size (ulong -> uint 20000 9.6 / 7.1).
template <typename InT, typename OutT>
bool staged_scan(size_t n, int vec) {
	constexpr size_t kM = (size_t)1 << 20;
	if (!(vec & 1)) return kOneShape<InT, OutT> || n > kM / 2;
	if (kOneShape<InT, OutT>) return n > (sizeof(InT) == 4 ? kM : 8 * kM);
	return sizeof(OutT) == 8 && sizeof(InT) <= 2 && n > 16 * kM;
}

template <typename InT, typename OutT, typename CFG>
__global__ void __launch_bounds__(CFG::kThreads, CFG::kMinBlocks)
scan_lookback(const InT *in, OutT *out, size_t n, TileStatus ts,
	int *dev_status, int vec, long long debug_skip_tile,
	const void *carry_in, void *carry_out) {
	using Acc = typename std::conditional<(sizeof(OutT) <= 4), uint32_t,
		uint64_t>::type;
	using R = typename CFG::R;
	constexpr int kTile = R::kTile;
	constexpr int kWarps = R::kWarps, kE = R::kE, kRows = R::kRows;
	__shared__ Acc s_warp_tot[kWarps];
	__shared__ Acc s_next_tot[kWarps];
	__shared__ Acc s_excl;
	__shared__ uint32_t s_tile, s_next;
	static_assert(!CFG::kKeepShared || R::kWords % 4 == 0, "parked in 16-byte vectors");
	constexpr int KR = CFG::kKeepShared ? R::kRows * R::kWords / 4 : 1;
	extern __shared__ uint4 s_cur[];  // [KR][kThreads] with KEEP

	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const uint32_t num_tiles = (uint32_t)((n + kTile - 1) / kTile);
	const bool solo = num_tiles == 1;  // one tile: no statuses, no counter
	const bool in_wide = vec & 2, out_wide = vec & 4;
	auto full_tile = [&](uint32_t t) { return (vec & 1) && (size_t)(t + 1) * kTile <= n; };
	// A warp's elements of a partial tile may still be whole.
	auto full_seg = [&](size_t seg) { return (vec & 1) && seg + R::kWarpElems <= n; };
	auto load_seg = [&](R &r, size_t seg) {
		if (full_seg(seg)) r.load(in + seg, lane, in_wide);
		else r.load_some(in + (seg < n ? seg : 0), lane, seg < n ? n - seg : 0);
	};
	auto seg_of = [&](uint32_t t) { return (size_t)t * kTile + (size_t)warp * R::kWarpElems; };
	dev::pdl_wait();
	if (tid == 0) s_tile = solo ? 0u : atomicAdd(ts.counter, 1u);
	__syncthreads();
	uint32_t tile = s_tile;
	if (tile >= num_tiles) return;
	R cur;
	load_seg(cur, seg_of(tile));
	bool agg_published = false;  // the current tile's aggregate is out

	for (;;) {
		if (tid == 0) s_next = solo ? 1u : atomicAdd(ts.counter, 1u);

		// ---- run sums, row scans, the warp's total ----------------------
		Acc ex[kRows], inc[kRows];
#pragma unroll
		for (int r = 0; r < kRows; ++r) {
			Acc run = 0;
#pragma unroll
			for (int e = 0; e < kE; ++e) run += (Acc)(OutT)cur.at(r, e);
			ex[r] = run;
			inc[r] = run;
		}
#pragma unroll
		for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
			for (int r = 0; r < kRows; ++r) {
				const Acc t = shfl_up(inc[r], d);
				if (lane >= d) inc[r] += t;
			}
		}
		Acc wsum = 0;
#pragma unroll
		for (int r = 0; r < kRows; ++r) {
			ex[r] = inc[r] - ex[r] + wsum;
			wsum += __shfl_sync(0xffffffffu, inc[r], 31);
		}
		// The tile waits here while the next one takes the registers.
		if constexpr (CFG::kKeepShared) {
			const uint32_t *w = &cur.w[0][0];
#pragma unroll
			for (int i = 0; i < KR; ++i)
				s_cur[i * CFG::kThreads + tid] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
		}
		if (lane == 0) s_warp_tot[warp] = wsum;
		__syncthreads();
		const uint32_t next = s_next;
		const bool have_next = next < num_tiles;
		const bool next_full = have_next && full_tile(next);

		// ---- prefetch of the next tile (all warps) ----------------------
		R nxt;
		if (next_full) nxt.load(in + seg_of(next), lane, in_wide);
		const bool next_publish = next_full && (long long)next != debug_skip_tile;

		// ---- tile aggregate, publication and lookback (warp 0) ----------
		if (warp == 0) {
			Acc wt = lane < kWarps ? s_warp_tot[lane] : (Acc)0;
			Acc winc = wt;
#pragma unroll
			for (int d = 1; d < kWarps; d <<= 1) {
				Acc t = shfl_up(winc, d);
				if (lane >= d) winc += t;
			}
			const Acc aggregate = __shfl_sync(0xffffffffu, winc, kWarps - 1);
			if (lane < kWarps) s_warp_tot[lane] = winc - wt;  // warp exclusive
			const bool do_publish = (long long)tile != debug_skip_tile && !solo;
			constexpr int PT = Slots<Acc>::kPerTile;
			Acc excl = 0;
			if (tile == 0) {
				// A scan continuing an earlier one starts from its carry.
				if (carry_in) excl = *reinterpret_cast<const Acc *>(carry_in);
				if (lane == 0 && do_publish)
					publish<Acc>(ts.words + Slots<Acc>::kWords, excl + aggregate);
			} else {
				if (lane == 0 && do_publish && !agg_published)
					publish<Acc>(ts.words + (size_t)tile * PT, aggregate);
				excl = lb::lookback_warp<Acc>(ts.words, tile, dev_status);
				if (lane == 0 && do_publish)
					publish<Acc>(ts.words + (size_t)tile * PT + Slots<Acc>::kWords,
						excl + aggregate);
			}
			if (lane == 0) {
				s_excl = excl;
				if (carry_out && (size_t)(tile + 1) * kTile >= n)
					*reinterpret_cast<Acc *>(carry_out) = excl + aggregate;
			}
		}
		// The next tile's sum from the prefetched registers.
		if (next_full) {
			Acc part = 0;
#pragma unroll
			for (int r = 0; r < kRows; ++r)
#pragma unroll
				for (int e = 0; e < kE; ++e) part += (Acc)(OutT)nxt.at(r, e);
			part = warp_sum<Acc>(part);
			if (lane == 0) s_next_tot[warp] = part;
		}
		__syncthreads();
		if (next_publish && tid == 0) {
			Acc agg = 0;
#pragma unroll
			for (int w = 0; w < kWarps; ++w) agg += s_next_tot[w];
			publish<Acc>(ts.words + (size_t)next * Slots<Acc>::kPerTile, agg);
		}

		// ---- outputs, straight from the registers ------------------------
		const Acc base = s_excl + s_warp_tot[warp];
		const size_t seg = seg_of(tile);
		const bool full = full_seg(seg);
#pragma unroll
		for (int r = 0; r < kRows; ++r) {
			if constexpr (CFG::kKeepShared) {
#pragma unroll
				for (int i = 0; i < R::kWords / 4; ++i) {
					uint32_t a, b, c, d;
					asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(a), "=r"(b), "=r"(c), "=r"(d)
						: "r"(dev::smem_u32(&s_cur[(r * R::kWords / 4 + i) * CFG::kThreads + tid])) : "memory");
					cur.w[r][4 * i] = a;
					cur.w[r][4 * i + 1] = b;
					cur.w[r][4 * i + 2] = c;
					cur.w[r][4 * i + 3] = d;
				}
			}
			Acc run = base + ex[r];
			const size_t i0 = seg + (size_t)(32 * r + lane) * kE;
			if (full) {
				uint32_t o[8];
#pragma unroll
				for (int e = 0; e < kE; ++e) {
					scanrows::pack<OutT>(o, e, (OutT)run);
					run += (Acc)(OutT)cur.at(r, e);
				}
				scanrows::store_run(out + i0, o, out_wide);
			} else {
#pragma unroll
				for (int e = 0; e < kE; ++e) {
					if (i0 + e < n) out[i0 + e] = (OutT)run;
					run += (Acc)(OutT)cur.at(r, e);
				}
			}
		}
		if (!have_next) break;

		// ---- on to the next tile ------------------------------------------
		if (next_full) {
			cur = nxt;
		} else {
			load_seg(cur, seg_of(next));
		}
		agg_published = next_full;
		tile = next;
	}
}

__global__ void __launch_bounds__(256) clear_words(uint4 *words, size_t count) {
	dev::pdl_wait();
	for (size_t i = blockIdx.x * (size_t)256 + threadIdx.x; i < count; i += (size_t)gridDim.x * 256)
		words[i] = make_uint4(0, 0, 0, 0);
}

// 16-byte vectors where both addresses allow them (tail and otherwise bytes).
__global__ void __launch_bounds__(256) copy_words(char *dst, const char *src, size_t bytes) {
	dev::pdl_wait();
	const size_t vecs = (((uintptr_t)dst | (uintptr_t)src) % 16) == 0 ? bytes / 16 : 0;
	const size_t first = blockIdx.x * (size_t)256 + threadIdx.x, stride = (size_t)gridDim.x * 256;
#pragma unroll 4
	for (size_t i = first; i < vecs; i += stride)
		reinterpret_cast<uint4 *>(dst)[i] = reinterpret_cast<const uint4 *>(src)[i];
	for (size_t i = vecs * 16 + first; i < bytes; i += stride) dst[i] = src[i];
}

template <typename InT, typename OutT, typename CFG>
constexpr auto scan_kernel() {
	if constexpr (CFG::kStaged) return &scanstaged::scan_staged<InT, OutT>;
	else return &scan_lookback<InT, OutT, CFG>;
}
template <typename InT, typename OutT, typename CFG>
constexpr size_t scan_shared() {
	if constexpr (CFG::kStaged) return scantile::scan_smem<InT, OutT>();
	else return CFG::kKeepShared ? (size_t)CFG::kThreads * CFG::R::kRows * CFG::R::kWords * 4 : 0;
}

// Per device and type pair, once: records the kernel's resident CTAs per SM.
// Later calls (possibly while a graph is being captured) only read
// the cached count.
template <typename InT, typename OutT, typename CFG>
cudaError_t scan_prepare(int *per_sm) {
	static std::atomic<int> cached[64];
	static std::mutex mu;
	int dev = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if (e != cudaSuccess) return e;
	if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
	int v = cached[dev].load(std::memory_order_acquire);
	if (v == 0) {
		std::lock_guard<std::mutex> lk(mu);
		v = cached[dev].load(std::memory_order_relaxed);
		if (v == 0) {
			if (scan_shared<InT, OutT, CFG>() > 48 * 1024)
				e = cudaFuncSetAttribute(scan_kernel<InT, OutT, CFG>(),
					cudaFuncAttributeMaxDynamicSharedMemorySize, (int)scan_shared<InT, OutT, CFG>());
			if (e == cudaSuccess)
				e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, scan_kernel<InT, OutT, CFG>(),
					CFG::kThreads, scan_shared<InT, OutT, CFG>());
			if (e != cudaSuccess) return e;
			if (v < 1) v = 1;
			cached[dev].store(v, std::memory_order_release);
		}
	}
	*per_sm = v;
	return cudaSuccess;
}

// Persistent grid: one CTA per resident slot, at most one per tile.
inline unsigned scan_grid(size_t tiles, int per_sm, int sm_count) {
	const size_t g = std::min<size_t>(tiles, (size_t)per_sm * (size_t)sm_count);
	return (unsigned)std::max<size_t>(g, 1);
}

// The kernel's vector flags: 1 both arrays 16-byte aligned, 2 and 4 the input
// and the output 32-byte aligned.
inline int scan_vec(const void *in, const void *out) {
	const uintptr_t a = (uintptr_t)in, b = (uintptr_t)out;
	return ((a | b) % 16 == 0 ? 1 : 0) | (a % 32 == 0 ? 2 : 0) | (b % 32 == 0 ? 4 : 0);
}

template <typename InT, typename OutT, typename CFG>
cudaError_t launch_scan_cfg(const void *in, void *out, size_t n, CCLContext *ctx,
	cudaStream_t s, GError **err, long long debug_skip_tile,
	const void *carry_in = nullptr, void *carry_out = nullptr) {
	using Acc = typename std::conditional<(sizeof(OutT) <= 4), uint32_t,
		uint64_t>::type;
	const size_t tiles = (n + CFG::kTile - 1) / CFG::kTile;
	if (tiles >= (1ull << 31)) {
		set_error(err, CLO_ERROR_ARGS, "Scan of %zu elements is too large", n);
		return cudaErrorInvalidValue;
	}
	// One tile of rows needs no statuses.
	const size_t status_bytes = tiles * Slots<Acc>::kPerTile * sizeof(uint64_t);
	const size_t bytes = status_bytes + 16;
	char *tmp = nullptr;
	TileStatus ts = {nullptr, nullptr};
	cudaError_t e = cudaSuccess;
	if (tiles > 1 || CFG::kStaged) {
		tmp = (char *)tmp_alloc(ctx, bytes, s, err);
		if (!tmp) return cudaErrorMemoryAllocation;
		ts.words = (uint64_t *)tmp;
		ts.counter = (uint32_t *)(tmp + status_bytes);
		e = clear_chained(tmp, bytes, s);
	}
	int per_sm = 1;
	if (e == cudaSuccess) e = scan_prepare<InT, OutT, CFG>(&per_sm);
	if (e == cudaSuccess) {
		KernelTimer t("scan_lookback", s, (double)n * (sizeof(InT) + sizeof(OutT)));
		e = launch_chained(scan_kernel<InT, OutT, CFG>(), scan_grid(tiles, per_sm, ctx->sm_count),
			CFG::kThreads, scan_shared<InT, OutT, CFG>(), s, 1, (const InT *)in, (OutT *)out, n, ts,
			ctx->d_status, scan_vec(in, out), debug_skip_tile, carry_in, carry_out);
		t.stop();
		count_launches(1);
	}
	tmp_free(tmp, s);
	if (e != cudaSuccess) cuda_ok(e, err, "scan_lookback");
	return e;
}

template <typename InT, typename OutT>
cudaError_t launch_scan(const void *in, void *out, size_t n, CCLContext *ctx,
	cudaStream_t s, GError **err, long long debug_skip_tile, const void *ci, void *co) {
	auto go = [&](auto cfg) {
		return launch_scan_cfg<InT, OutT, decltype(cfg)>(in, out, n, ctx, s, err, debug_skip_tile, ci,
			co);
	};
	if (staged_scan<InT, OutT>(n, scan_vec(in, out))) return go(ScanStaged<InT, OutT>());
	if (n <= ScanOne<InT, OutT>::kTile) return go(ScanOne<InT, OutT>());
	if (n <= kSmallMax) return go(ScanSmall<InT, OutT>());
	if (n <= kMidMax) return go(ScanMid<InT, OutT>());
	return go(ScanBig<InT, OutT>());
}

template <typename InT>
cudaError_t dispatch_out(const void *in, void *out, size_t n, int out_bytes,
	CCLContext *ctx, cudaStream_t s, GError **err, long long dbg,
	const void *ci = nullptr, void *co = nullptr) {
	switch (out_bytes) {
	case 1: return launch_scan<InT, uint8_t>(in, out, n, ctx, s, err, dbg, ci, co);
	case 2: return launch_scan<InT, uint16_t>(in, out, n, ctx, s, err, dbg, ci, co);
	case 4: return launch_scan<InT, uint32_t>(in, out, n, ctx, s, err, dbg, ci, co);
	case 8: return launch_scan<InT, uint64_t>(in, out, n, ctx, s, err, dbg, ci, co);
	}
	set_error(err, CLO_ERROR_ARGS, "Unsupported sum width %d", out_bytes);
	return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t clear_chained(void *p, size_t bytes, cudaStream_t s) {
	const size_t vecs = bytes / 16;
	count_launches(1);
	return launch_chained(clear_words, (unsigned)std::min<size_t>((vecs + 1023) / 1024, 608), 256, 0,
		s, 1, (uint4 *)p, vecs);
}

cudaError_t copy_chained(void *dst, const void *src, size_t bytes, cudaStream_t s) {
	count_launches(1);
	return launch_chained(copy_words, (unsigned)std::min<size_t>((bytes + 4095) / 4096, 608), 256, 0,
		s, 1, (char *)dst, (const char *)src, bytes);
}

// Tile whose publication is withheld (-1: none). Only the watchdog test
// sets it, through clo_gb300_debug_scan_withhold().
static long long g_debug_skip_tile = -1;

cudaError_t scan_exclusive(const void *in, void *out, size_t n,
	CloType in_type, int out_bytes, CCLContext *ctx, cudaStream_t s,
	GError **err) {
	return scan_exclusive_carry(in, out, n, in_type, out_bytes, nullptr, nullptr, ctx, s, err);
}

cudaError_t scan_exclusive_carry(const void *in, void *out, size_t n,
	CloType in_type, int out_bytes, const void *ci, void *co, CCLContext *ctx,
	cudaStream_t s, GError **err) {
	if (n == 0) return cudaSuccess;
	long long dbg = g_debug_skip_tile;
	switch (in_type) {
	case CLO_CHAR: return dispatch_out<int8_t>(in, out, n, out_bytes, ctx, s, err, dbg, ci, co);
	case CLO_UCHAR: return dispatch_out<uint8_t>(in, out, n, out_bytes, ctx, s, err, dbg, ci, co);
	case CLO_SHORT: return dispatch_out<int16_t>(in, out, n, out_bytes, ctx, s, err, dbg, ci, co);
	case CLO_USHORT: return dispatch_out<uint16_t>(in, out, n, out_bytes, ctx, s, err, dbg, ci, co);
	case CLO_INT: return dispatch_out<int32_t>(in, out, n, out_bytes, ctx, s, err, dbg, ci, co);
	case CLO_UINT: return dispatch_out<uint32_t>(in, out, n, out_bytes, ctx, s, err, dbg, ci, co);
	case CLO_LONG: return dispatch_out<int64_t>(in, out, n, out_bytes, ctx, s, err, dbg, ci, co);
	case CLO_ULONG: return dispatch_out<uint64_t>(in, out, n, out_bytes, ctx, s, err, dbg, ci, co);
	default: break;
	}
	set_error(err, CLO_ERROR_ARGS, "Unsupported scan element type %d", (int)in_type);
	return cudaErrorInvalidValue;
}

}  // namespace clo

// Test hook for the lookback watchdog: the given tile of the next scans
// never publishes its status, so its successor's bounded wait runs out
// and reports through the context status word. -1 restores normal
// operation.
extern "C" void clo_gb300_debug_scan_withhold(long long tile) {
	clo::g_debug_skip_tile = tile;
}

// ---------------------------------------------------------------------
// Scan that allocates nothing (clo_scan_blelloch_noalloc).
//
// Same kernel as above; its tile statuses and tile counter live in the
// file-scope device array below instead of a pool temporary. The array is
// part of the library's device image: every GPU that loads the library
// holds it (1 MiB + 16 B) until the process exits. Host code cannot use
// the array's name as a device address (on the host it names a stand-in),
// so the device address is looked up once per device with
// cudaGetSymbolAddress and cached.
// ---------------------------------------------------------------------

// Largest no-allocation scan: 2^15 tiles of 8192 elements (the smallest its
// shapes take) = 2^28 elements.
#define CLO_NOALLOC_MAX_TILES (1u << 15)
// Four status words per tile (64-bit sums) and one word for the counter.
#define CLO_NOALLOC_WORDS (CLO_NOALLOC_MAX_TILES * 4u + 2u)

static __device__ __align__(256) uint64_t g_scan_noalloc_scratch[CLO_NOALLOC_WORDS];

namespace clo {
namespace {

constexpr size_t kNoAllocMaxElems = (size_t)CLO_NOALLOC_MAX_TILES * 8192;
static_assert(kNoAllocMaxElems == ((size_t)1 << 28), "no-allocation scan limit");

std::mutex g_noalloc_mu;
uint64_t *g_noalloc_addr[64] = {};

// Makes `ordinal` the calling thread's current device for the guard's
// lifetime and restores the previous one afterwards.
struct CurrentDevice {
	int prev = -1;
	cudaError_t status;
	explicit CurrentDevice(int ordinal) {
		if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
		status = cudaSetDevice(ordinal);
	}
	~CurrentDevice() {
		if (prev >= 0) cudaSetDevice(prev);
	}
};

// Opts every (element, sum) instantiation of the scan kernel into its
// shared memory and caches its occupancy, so that no later call does any
// set-up work, whatever its type pair.
template <typename InT, typename OutT>
cudaError_t noalloc_prepare() {
	int v = 0;
	cudaError_t e = scan_prepare<InT, OutT, ScanBig<InT, OutT>>(&v);
	return e == cudaSuccess ? scan_prepare<InT, OutT, ScanStaged<InT, OutT>>(&v) : e;
}
template <typename InT>
cudaError_t noalloc_prepare_in() {
	cudaError_t e = noalloc_prepare<InT, uint8_t>();
	if (e == cudaSuccess) e = noalloc_prepare<InT, uint16_t>();
	if (e == cudaSuccess) e = noalloc_prepare<InT, uint32_t>();
	if (e == cudaSuccess) e = noalloc_prepare<InT, uint64_t>();
	return e;
}

cudaError_t noalloc_prepare_all() {
	cudaError_t e = noalloc_prepare_in<int8_t>();
	if (e == cudaSuccess) e = noalloc_prepare_in<uint8_t>();
	if (e == cudaSuccess) e = noalloc_prepare_in<int16_t>();
	if (e == cudaSuccess) e = noalloc_prepare_in<uint16_t>();
	if (e == cudaSuccess) e = noalloc_prepare_in<int32_t>();
	if (e == cudaSuccess) e = noalloc_prepare_in<uint32_t>();
	if (e == cudaSuccess) e = noalloc_prepare_in<int64_t>();
	if (e == cudaSuccess) e = noalloc_prepare_in<uint64_t>();
	return e;
}

// Device address of the scratch array on device `ordinal` (which must be
// current), looked up on the first call for that device, together with
// the set-up of every scan instantiation.
uint64_t *noalloc_scratch(int ordinal, GError **err) {
	std::lock_guard<std::mutex> lk(g_noalloc_mu);
	if (g_noalloc_addr[ordinal] == nullptr) {
		void *p = nullptr;
		cudaError_t e = cudaGetSymbolAddress(&p, g_scan_noalloc_scratch);
		if (e != cudaSuccess || p == nullptr) {
			cudaGetLastError();
			set_error(err, CLO_ERROR_LIBRARY,
				"cudaGetSymbolAddress of the no-allocation scan scratch failed on "
				"device %d: %s", ordinal, cudaGetErrorString(e));
			return nullptr;
		}
		e = noalloc_prepare_all();
		if (e != cudaSuccess) {
			cudaGetLastError();
			set_error(err, CLO_ERROR_LIBRARY,
				"No-allocation scan set-up failed on device %d: %s", ordinal,
				cudaGetErrorString(e));
			return nullptr;
		}
		g_noalloc_addr[ordinal] = (uint64_t *)p;
	}
	return g_noalloc_addr[ordinal];
}

template <typename InT, typename OutT, typename CFG>
cudaError_t launch_scan_noalloc_cfg(const void *in, void *out, size_t n,
	uint64_t *scratch, int *dev_status, int sm_count, cudaStream_t s) {
	using Acc = typename std::conditional<(sizeof(OutT) <= 4), uint32_t,
		uint64_t>::type;
	const size_t tiles = (n + CFG::kTile - 1) / CFG::kTile;
	TileStatus ts;
	ts.words = scratch;
	ts.counter = (uint32_t *)(scratch + (size_t)CLO_NOALLOC_MAX_TILES * 4);
	// The array keeps the previous call's statuses: clear the words this
	// call reads before writing (its tiles' slots and the tile counter).
	cudaError_t e = cudaMemsetAsync(ts.words, 0,
		tiles * Slots<Acc>::kPerTile * sizeof(uint64_t), s);
	if (e == cudaSuccess) e = cudaMemsetAsync(ts.counter, 0, sizeof(uint64_t), s);
	if (e != cudaSuccess) return e;
	int per_sm = 1;
	e = scan_prepare<InT, OutT, CFG>(&per_sm);
	if (e != cudaSuccess) return e;
	scan_kernel<InT, OutT, CFG>()<<<scan_grid(tiles, per_sm, sm_count), CFG::kThreads,
		scan_shared<InT, OutT, CFG>(), s>>>((const InT *)in, (OutT *)out, n, ts, dev_status,
		scan_vec(in, out), -1, nullptr, nullptr);
	count_launches(1);
	return cudaGetLastError();
}

template <typename InT, typename OutT>
cudaError_t launch_scan_noalloc(const void *in, void *out, size_t n,
	uint64_t *scratch, int *dev_status, int sm_count, cudaStream_t s) {
	return staged_scan<InT, OutT>(n, scan_vec(in, out))
		? launch_scan_noalloc_cfg<InT, OutT, ScanStaged<InT, OutT>>(in, out, n, scratch, dev_status,
			sm_count, s)
		: launch_scan_noalloc_cfg<InT, OutT, ScanBig<InT, OutT>>(in, out, n, scratch, dev_status,
			sm_count, s);
}

template <typename InT>
cudaError_t noalloc_out(const void *in, void *out, size_t n, int out_bytes,
	uint64_t *scratch, int *st, int sms, cudaStream_t s) {
	switch (out_bytes) {
	case 1: return launch_scan_noalloc<InT, uint8_t>(in, out, n, scratch, st, sms, s);
	case 2: return launch_scan_noalloc<InT, uint16_t>(in, out, n, scratch, st, sms, s);
	case 4: return launch_scan_noalloc<InT, uint32_t>(in, out, n, scratch, st, sms, s);
	default: return launch_scan_noalloc<InT, uint64_t>(in, out, n, scratch, st, sms, s);
	}
}

}  // namespace
}  // namespace clo

extern "C" cl_bool clo_scan_blelloch_noalloc(CCLQueue *cq, CloType elem_type,
	CloType sum_type, const void *d_in, void *d_out, size_t numel,
	GError **err) {
	using namespace clo;
	if (err && *err) return CL_FALSE;
	if (!cq) {
		set_error(err, CLO_ERROR_ARGS, "NULL queue");
		return CL_FALSE;
	}
	if (!type_is_integer(elem_type) || !type_is_integer(sum_type)) {
		set_error(err, CLO_ERROR_ARGS,
			"No-allocation scan: integer element and sum types only");
		return CL_FALSE;
	}
	if (numel > kNoAllocMaxElems) {
		set_error(err, CLO_ERROR_ARGS,
			"No-allocation scan of %zu elements exceeds its limit of %zu elements "
			"(the size of its static device scratch); use clo_scan_with_device_data",
			numel, kNoAllocMaxElems);
		return CL_FALSE;
	}
	if (numel == 0) return CL_TRUE;
	if (!d_in || !d_out) {
		set_error(err, CLO_ERROR_ARGS, "NULL input or output pointer");
		return CL_FALSE;
	}
	const int ordinal = cq->ctx->ordinal;
	if (ordinal < 0 || ordinal >= 64) {
		set_error(err, CLO_ERROR_ARGS, "Device ordinal %d out of range", ordinal);
		return CL_FALSE;
	}
	CurrentDevice dev(ordinal);
	if (!cuda_ok(dev.status, err, "clo_scan_blelloch_noalloc: cudaSetDevice")) return CL_FALSE;
	uint64_t *scratch = noalloc_scratch(ordinal, err);
	if (!scratch) return CL_FALSE;
	const int ob = (int)clo_type_sizeof(sum_type);
	int *st = cq->ctx->d_status;
	const int sms = cq->ctx->sm_count;
	cudaStream_t s = cq->stream;
	cudaError_t e;
	switch (elem_type) {
	case CLO_CHAR: e = noalloc_out<int8_t>(d_in, d_out, numel, ob, scratch, st, sms, s); break;
	case CLO_UCHAR: e = noalloc_out<uint8_t>(d_in, d_out, numel, ob, scratch, st, sms, s); break;
	case CLO_SHORT: e = noalloc_out<int16_t>(d_in, d_out, numel, ob, scratch, st, sms, s); break;
	case CLO_USHORT: e = noalloc_out<uint16_t>(d_in, d_out, numel, ob, scratch, st, sms, s); break;
	case CLO_INT: e = noalloc_out<int32_t>(d_in, d_out, numel, ob, scratch, st, sms, s); break;
	case CLO_UINT: e = noalloc_out<uint32_t>(d_in, d_out, numel, ob, scratch, st, sms, s); break;
	case CLO_LONG: e = noalloc_out<int64_t>(d_in, d_out, numel, ob, scratch, st, sms, s); break;
	default: e = noalloc_out<uint64_t>(d_in, d_out, numel, ob, scratch, st, sms, s); break;
	}
	return cuda_ok(e, err, "clo_scan_blelloch_noalloc") ? CL_TRUE : CL_FALSE;
}
