// RNG kernels: DEV_GID seed initialisation and the batched draw ("fill").
//
// Seed init (src/cl_ops/rng/clo_rng_init.cl:47-60): state[gid] =
// convert(hash(gid + main_seed)) where `hash` is a compiled stack program
// (rng.cpp) and `convert` is the generator's clo_ulong2statetype:
// identity for lcg/xorshift64, (s, s>>16, s>>32, s>>46) masked to 32 bits
// for xorshift128 (clo_rng_xorshift128.cl:30), (low, high) words for
// mwc64x (clo_rng_mwc64x.cl:32), the low word as int for parkmiller
// (clo_rng_parkmiller.cl:31) and as_uint4((ulong2)(s, s)) for tauslcg
// (clo_rng_tauslcg.cl:35).
//
// Fill (the draw loop of src/benchmarks/clo_rng_bench.c:302-324 with the
// kernel of clo_rng_bench.cl:23-37, moved on device): out[r * count + i]
// = next(state i) >> (32 - bits), or % maxint, for r = 0..draws-1. Each
// thread keeps one state, or four consecutive ones, in registers for all
// draws, so the states are read and written once.
//
// HBM roofline: 4 B per draw + 2 x state size per state.
#include "clo_internal.h"
#include "clo_rng_device.cuh"
#include "dev_common.cuh"
#include "launch.h"
#include "timing.h"

namespace clo {
namespace {

__device__ __forceinline__ uint64_t run_hash(const HashProgram &hp, uint64_t x) {
	uint64_t st[16];
	int sp = 0;
	for (int i = 0; i < hp.n_ops; ++i) {
		uint8_t op = hp.op[i];
		uint64_t a = 0, b = 0;
		if (op >= 4 && op != 14 && op != 15 && op != 16 && sp >= 2) {
			b = st[--sp];
			a = st[--sp];
		}
		switch (op) {
		case 0: if (sp < 16) st[sp++] = hp.imm[i]; break;     // IMM
		case 1: if (sp < 16) st[sp++] = x; break;             // X
		case 2: if (sp > 0) x = st[--sp]; break;              // STORE
		case 3: if (sp > 0) --sp; break;                      // POP
		case 4: st[sp++] = a + b; break;
		case 5: st[sp++] = a - b; break;
		case 6: st[sp++] = a * b; break;
		case 7: st[sp++] = b ? a / b : 0; break;
		case 8: st[sp++] = b ? a % b : 0; break;
		case 9: st[sp++] = a & b; break;
		case 10: st[sp++] = a | b; break;
		case 11: st[sp++] = a ^ b; break;
		case 12: st[sp++] = a << (b & 63); break;
		case 13: st[sp++] = a >> (b & 63); break;
		case 14: if (sp > 0) st[sp - 1] = 0 - st[sp - 1]; break;  // NEG
		case 15: if (sp > 0) st[sp - 1] = ~st[sp - 1]; break;     // NOT
		case 16: if (sp > 0) st[sp - 1] = !st[sp - 1]; break;     // LNOT
		case 17: st[sp++] = a == b; break;
		case 18: st[sp++] = a != b; break;
		case 19: st[sp++] = a < b; break;
		case 20: st[sp++] = a > b; break;
		case 21: st[sp++] = a <= b; break;
		case 22: st[sp++] = a >= b; break;
		case 23: st[sp++] = a && b; break;
		case 24: st[sp++] = a || b; break;
		}
	}
	return x;
}

__global__ void rng_init_kernel(void *states, size_t count, int gen,
	uint64_t main_seed, HashProgram hp) {
	size_t gid = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
	if (gid >= count) return;
	// The reference adds the work-item id (a size_t) to the ulong seed.
	uint64_t seed = run_hash(hp, (uint64_t)gid + main_seed);
	switch (gen) {
	case RNG_LCG:
	case RNG_XS64:
		((uint64_t *)states)[gid] = seed;
		break;
	case RNG_XS128:
		((uint4 *)states)[gid] = make_uint4((uint32_t)seed, (uint32_t)(seed >> 16),
			(uint32_t)(seed >> 32), (uint32_t)(seed >> 46));
		break;
	case RNG_MWC64X:
		((uint2 *)states)[gid] = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
		break;
	case RNG_PARKMILLER:
		((int32_t *)states)[gid] = (int32_t)(uint32_t)seed;
		break;
	case RNG_TAUSLCG:
		((uint4 *)states)[gid] = make_uint4((uint32_t)seed, (uint32_t)(seed >> 32),
			(uint32_t)seed, (uint32_t)(seed >> 32));
		break;
	}
}

template <int GEN>
struct Gen;
template <>
struct Gen<RNG_LCG> {
	using S = uint64_t;
	__device__ __forceinline__ static uint32_t next(S &s) { return clo_rng_step_lcg(&s); }
};
template <>
struct Gen<RNG_XS64> {
	using S = uint64_t;
	__device__ __forceinline__ static uint32_t next(S &s) { return clo_rng_step_xorshift64(&s); }
};
template <>
struct Gen<RNG_XS128> {
	using S = uint4;
	__device__ __forceinline__ static uint32_t next(S &s) { return clo_rng_step_xorshift128(&s); }
};
template <>
struct Gen<RNG_MWC64X> {
	using S = uint2;
	__device__ __forceinline__ static uint32_t next(S &s) { return clo_rng_step_mwc64x(&s); }
};
template <>
struct Gen<RNG_PARKMILLER> {
	using S = int32_t;
	__device__ __forceinline__ static uint32_t next(S &s) { return clo_rng_step_parkmiller(&s); }
};
template <>
struct Gen<RNG_TAUSLCG> {
	using S = uint4;
	__device__ __forceinline__ static uint32_t next(S &s) { return clo_rng_step_tauslcg(&s); }
};

constexpr int kFillThreads = 256;

// V consecutive states per thread (4: one 16-byte store per draw; 1: coalesced
// 4-byte stores, any count and alignment).
template <int GEN, bool MAXINT, int V>
__global__ void __launch_bounds__(kFillThreads)
rng_fill_kernel(typename Gen<GEN>::S *states, size_t count,
	uint32_t *out, size_t draws, uint32_t shift, uint32_t maxint) {
	using S = typename Gen<GEN>::S;
	const size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
	const size_t i0 = q * V;
	dev::pdl_wait();
	if (i0 >= count) return;
	auto emit = [&](uint32_t v) -> uint32_t {
		return MAXINT ? v % maxint : (v >> shift);
	};
	S s[V];
#pragma unroll
	for (int k = 0; k < V; ++k) s[k] = states[i0 + k];
	uint32_t *o = out + i0;
#pragma unroll 4
	for (size_t r = 0; r < draws; ++r, o += count) {
		uint32_t v[V];
#pragma unroll
		for (int k = 0; k < V; ++k) v[k] = emit(Gen<GEN>::next(s[k]));
		if constexpr (V == 4)
			dev::st_stream_v4(reinterpret_cast<uint4 *>(o), make_uint4(v[0], v[1], v[2], v[3]));
		else
			__stcs(o, v[0]);
	}
#pragma unroll
	for (int k = 0; k < V; ++k) states[i0 + k] = s[k];
}

template <int GEN, bool MAXINT, int V>
cudaError_t launch_fill(void *states, size_t count, uint32_t *out, size_t draws, uint32_t shift,
	unsigned maxint, cudaStream_t s) {
	using S = typename Gen<GEN>::S;
	const size_t threads = (count + V - 1) / V;
	return launch_chained(rng_fill_kernel<GEN, MAXINT, V>,
		(unsigned)((threads + kFillThreads - 1) / kFillThreads), kFillThreads, 0, s, 1, (S *)states,
		count, out, draws, shift, maxint);
}

// Counts from which a thread takes four states (whole rows of 16-byte stores
// need count % 4 == 0 and an aligned output too); below, one state a thread
// keeps the SMs fuller. us, four / one, states x draws: mwc64x 65536 x 64 5.8 /
// 4.0, 2^20 x 32 20.9 / 19.5, 2^22 x 8 26.4 / 23.6, 2^22 x 64 157 / 157, 2^23 x
// 32 174 / 179 (lcg and xorshift64 alike); 16-byte states: xorshift128 2^20 x
// 32 22.8 / 19.5, 2^21 x 8 18.2 / 13.4, 2^22 x 8 34.1 / 32.0, 2^22 x 32 92.6 /
// 96.5, tauslcg 2^21 x 8 18.2 / 14.9, x 32 42.7 / 47.0; parkmiller 262144 x 32
// 6.6 / 6.8, 2^20 x 32 20.1 / 22.8, 2^22 x 8 20.6 / 26.3. Counts that are no
// multiple of four (2^22 - 1 mwc64x x 32): 138 us, whose rows' stores meet the
// 32-byte sectors unaligned; 524 with four states a thread one after the other.
template <int GEN>
size_t vec_min(size_t draws) {
	if (GEN == RNG_PARKMILLER) return (size_t)1 << 18;
	return sizeof(typename Gen<GEN>::S) == 16 && draws >= 32 ? (size_t)1 << 21 : (size_t)1 << 23;
}

template <int GEN>
cudaError_t fill_gen(void *states, size_t count, uint32_t *out, size_t draws,
	unsigned bits, unsigned maxint, cudaStream_t s) {
	using S = typename Gen<GEN>::S;
	const uint32_t shift = 32u - bits;
	const bool vec = (count % 4) == 0 && ((uintptr_t)out % 16) == 0 &&
		count >= vec_min<GEN>(draws);
	KernelTimer t("rng_fill", s, (double)count * (4.0 * draws + 2.0 * sizeof(S)));
	const cudaError_t e = maxint
		? (vec ? launch_fill<GEN, true, 4>(states, count, out, draws, shift, maxint, s)
			   : launch_fill<GEN, true, 1>(states, count, out, draws, shift, maxint, s))
		: (vec ? launch_fill<GEN, false, 4>(states, count, out, draws, shift, maxint, s)
			   : launch_fill<GEN, false, 1>(states, count, out, draws, shift, maxint, s));
	t.stop();
	count_launches(1);
	return e;
}

}  // namespace

cudaError_t rng_init_gid(void *states, size_t count, int gen,
	uint64_t main_seed, const HashProgram &hp, cudaStream_t s) {
	if (count == 0) return cudaSuccess;
	rng_init_kernel<<<(unsigned)((count + 255) / 256), 256, 0, s>>>(states, count,
		gen, main_seed, hp);
	count_launches(1);
	return cudaGetLastError();
}

cudaError_t rng_fill(void *states, size_t count, int gen, uint32_t *out,
	size_t draws, unsigned bits, unsigned maxint, cudaStream_t s) {
	if (count == 0 || draws == 0) return cudaSuccess;
	switch (gen) {
	case RNG_LCG: return fill_gen<RNG_LCG>(states, count, out, draws, bits, maxint, s);
	case RNG_XS64: return fill_gen<RNG_XS64>(states, count, out, draws, bits, maxint, s);
	case RNG_XS128: return fill_gen<RNG_XS128>(states, count, out, draws, bits, maxint, s);
	case RNG_MWC64X: return fill_gen<RNG_MWC64X>(states, count, out, draws, bits, maxint, s);
	case RNG_PARKMILLER: return fill_gen<RNG_PARKMILLER>(states, count, out, draws, bits, maxint, s);
	case RNG_TAUSLCG: return fill_gen<RNG_TAUSLCG>(states, count, out, draws, bits, maxint, s);
	}
	return cudaErrorInvalidValue;
}

}  // namespace clo
