// Kernel launches with the attributes the library's launch chains use.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace clo {

// Launches `kern` with programmatic stream serialisation, in clusters of
// `cluster` CTAs when that is above 1. The kernel is set up while the
// stream's previous one runs and holds its CTAs in dev::pdl_wait until that
// one has ended; a launch in a chain costs 2-3 us less than a plain one (a
// bitonic sort of 2^20 ints, 11 launches: 87 -> 60 us). No kernel asks for
// its successor early (griddepcontrol.launch_dependents): CTAs that wait
// take SM slots from the running kernels and spread the next one's unevenly
// (the same sort: 88 us with the request at the start of the work, 99 us
// before the stores, 128 us at the top of the kernel).
template <typename... P, typename... A>
cudaError_t launch_chained(void (*kern)(P...), unsigned grid, unsigned threads, size_t smem,
	cudaStream_t s, unsigned cluster, A &&...args) {
	cudaLaunchConfig_t c = {};
	c.gridDim = dim3(grid);
	c.blockDim = dim3(threads);
	c.dynamicSmemBytes = smem;
	c.stream = s;
	cudaLaunchAttribute at[2];
	c.attrs = at;
	at[c.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at[c.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
	if (cluster > 1) {
		at[c.numAttrs].id = cudaLaunchAttributeClusterDimension;
		at[c.numAttrs].val.clusterDim.x = cluster;
		at[c.numAttrs].val.clusterDim.y = 1;
		at[c.numAttrs++].val.clusterDim.z = 1;
	}
	return cudaLaunchKernelEx(&c, kern, P(std::forward<A>(args))...);
}

}  // namespace clo
