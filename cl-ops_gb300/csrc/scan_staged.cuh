// The plain scan's kernel for what the register rows (scan_rows.cuh) are slow
// at (staged_scan in scan.cu): tiles of 8192 elements staged in shared memory
// (scan_tile.cuh), read and written in whole lines whatever the types and the
// alignment; a lane scans 16 consecutive elements there. Bound by the shared
// memory's pipe, 70% busy, and the barriers around the lookback (uint -> uchar
// 2^28: 322 us, 61% of the copy rate).
#pragma once

#include <stddef.h>
#include <stdint.h>

#include <type_traits>

#include "dev_common.cuh"
#include "scan_status.cuh"
#include "scan_tile.cuh"

namespace clo {
namespace scanstaged {

using namespace scantile;
using lb::Slots;
using lb::TileStatus;
using lb::publish;
using lb::warp_sum;

// Persistent CTAs take tiles in order as in scan_lookback (scan.cu), whose
// arguments it shares: while warp 0 looks back, the next tile's vectors are
// loaded into registers and summed; they reach shared memory after this
// tile's outputs are out.
template <typename InT, typename OutT>
__global__ void __launch_bounds__(kThreads, (scan_min_blocks<InT, OutT>()))
scan_staged(const InT *in, OutT *out, size_t n, TileStatus ts, int *dev_status, int vec,
	long long debug_skip_tile, const void *carry_in, void *carry_out) {
	using Acc = typename std::conditional<(sizeof(OutT) <= 4), uint32_t,
		uint64_t>::type;
	extern __shared__ __align__(16) unsigned char s_dyn[];
	__shared__ Acc s_warp_tot[kWarps];
	__shared__ Acc s_next_tot[kWarps];
	__shared__ Acc s_excl;
	__shared__ uint32_t s_tile, s_next;

	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const uint32_t num_tiles = (uint32_t)((n + kTile - 1) / kTile);
	InT *s_in = reinterpret_cast<InT *>(s_dyn + (size_t)warp *
		(kBlocks * padded<InT>() * sizeof(InT) + padded<OutT>() * sizeof(OutT)));
	OutT *s_out = reinterpret_cast<OutT *>(s_in + kBlocks * padded<InT>());
	const bool vec_ok = vec & 1;
	auto full_tile = [&](uint32_t t) {
		return vec_ok && (size_t)(t + 1) * kTile <= n;
	};
	dev::pdl_wait();
	if (tid == 0) s_tile = atomicAdd(ts.counter, 1u);
	__syncthreads();
	uint32_t tile = s_tile;
	if (tile >= num_tiles) return;
	{
		const size_t wseg = (size_t)tile * kTile + (size_t)warp * kWarpElems;
		if (full_tile(tile)) {
			BlockRegs<InT> r;
			issue_loads<InT>(r, in, wseg, lane);
			store_loads<InT>(r, s_in, lane);
		} else {
#pragma unroll
			for (int b = 0; b < kBlocks; ++b)
				load_block_scalar<InT>(in, n, wseg + (size_t)b * kBlock, s_in + b * padded<InT>(), lane);
		}
	}
	__syncwarp();
	bool agg_published = false;  // the current tile's aggregate is out

	for (;;) {
		if (tid == 0) s_next = atomicAdd(ts.counter, 1u);
		const size_t wseg = (size_t)tile * kTile + (size_t)warp * kWarpElems;

		// ---- lane run sums and their warp scans, per block --------------
		Acc lane_excl[kBlocks], block_tot[kBlocks];
#pragma unroll
		for (int b = 0; b < kBlocks; ++b) {
			const InT *sin = s_in + b * padded<InT>();
			Acc run = 0;
#pragma unroll
			for (int j = 0; j < kItems; ++j) run += (Acc)(OutT)sin[pidx<InT>(lane * kItems + j)];
			Acc inc = run;
#pragma unroll
			for (int d = 1; d < 32; d <<= 1) {
				Acc t = __shfl_up_sync(0xffffffffu, inc, d);
				if (lane >= d) inc += t;
			}
			lane_excl[b] = inc - run;
			block_tot[b] = __shfl_sync(0xffffffffu, inc, 31);
		}
		if (lane == 0) {
			Acc wsum = 0;
#pragma unroll
			for (int b = 0; b < kBlocks; ++b) wsum += block_tot[b];
			s_warp_tot[warp] = wsum;
		}
		__syncthreads();
		const uint32_t next = s_next;
		const bool have_next = next < num_tiles;
		const bool next_full = have_next && full_tile(next);
		const size_t nseg = (size_t)next * kTile + (size_t)warp * kWarpElems;

		// ---- prefetch of the next tile (all warps) ----------------------
		BlockRegs<InT> r;
		if (next_full) issue_loads<InT>(r, in, nseg, lane);
		const bool next_publish = next_full && (long long)next != debug_skip_tile;

		// ---- tile aggregate, publication and lookback (warp 0) ----------
		if (warp == 0) {
			Acc wt = lane < kWarps ? s_warp_tot[lane] : (Acc)0;
			Acc winc = wt;
#pragma unroll
			for (int d = 1; d < kWarps; d <<= 1) {
				Acc t = __shfl_up_sync(0xffffffffu, winc, d);
				if (lane >= d) winc += t;
			}
			const Acc aggregate = __shfl_sync(0xffffffffu, winc, kWarps - 1);
			if (lane < kWarps) s_warp_tot[lane] = winc - wt;  // warp exclusive
			const bool do_publish = (long long)tile != debug_skip_tile;
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
			constexpr int EPC = BlockRegs<InT>::kEpc;
			Acc part = 0;
#pragma unroll
			for (int b = 0; b < kBlocks; ++b)
#pragma unroll
				for (int k = 0; k < BlockRegs<InT>::kPerLane; ++k) {
					const InT *e = reinterpret_cast<const InT *>(&r.v[b][k]);
#pragma unroll
					for (int q = 0; q < EPC; ++q) part += (Acc)(OutT)e[q];
				}
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

		// ---- outputs per block: second read, staged, coalesced stores ----
		Acc base = s_excl + s_warp_tot[warp];
#pragma unroll
		for (int b = 0; b < kBlocks; ++b) {
			const InT *sin = s_in + b * padded<InT>();
			Acc run = base + lane_excl[b];
#pragma unroll
			for (int j = 0; j < kItems; ++j) {
				const int q = lane * kItems + j;
				const Acc v = (Acc)(OutT)sin[pidx<InT>(q)];
				s_out[pidx<OutT>(q)] = (OutT)run;
				run += v;
			}
			base += block_tot[b];
			__syncwarp();
			const size_t seg = wseg + (size_t)b * kBlock;
			if (seg + kBlock <= n && vec_ok) {
				constexpr int EPC = 16 / sizeof(OutT);
				constexpr int CHUNKS = kBlock / EPC;
				uint4 *dst = reinterpret_cast<uint4 *>(out + seg);
#pragma unroll
				for (int c = lane; c < CHUNKS; c += 32) {
					uint4 v;
					OutT *e = reinterpret_cast<OutT *>(&v);
#pragma unroll
					for (int k = 0; k < EPC; ++k) e[k] = s_out[pidx<OutT>(c * EPC + k)];
					dev::st_stream_v4(dst + c, v);
				}
			} else {
				for (int i = lane; i < kBlock; i += 32)
					if (seg + i < n) out[seg + i] = s_out[pidx<OutT>(i)];
			}
			__syncwarp();
		}
		if (!have_next) break;

		// ---- the next tile into shared memory ---------------------------
		if (next_full) {
			store_loads<InT>(r, s_in, lane);
		} else {
#pragma unroll
			for (int b = 0; b < kBlocks; ++b)
				load_block_scalar<InT>(in, n, nseg + (size_t)b * kBlock, s_in + b * padded<InT>(), lane);
		}
		__syncwarp();
		agg_published = next_full;
		tile = next;
	}
}

}  // namespace scanstaged
}  // namespace clo
