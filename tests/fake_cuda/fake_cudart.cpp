// A CUDA runtime without a GPU for tests of the library's host code: memory
// is host memory, kernels do not run, and every launch is recorded with its
// kernel's name, its grid and the device that was current. Two devices.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {

struct Launch {
	std::string name;
	unsigned grid;
	int device, stream_device;
};
struct Stream {
	int device;
};
std::map<const void *, std::string> &names() {
	static std::map<const void *, std::string> m;
	return m;
}
std::vector<Launch> g_launches;
std::map<const void *, void *> g_symbols;
int g_device = 0, g_sms = 152;
dim3 g_grid, g_block;
size_t g_shared;
cudaStream_t g_stream;

void record(const void *f, dim3 grid, cudaStream_t s) {
	g_launches.push_back({names()[f], grid.x, g_device, s ? ((Stream *)s)->device : g_device});
}

}  // namespace

extern "C" {

// ------------------------------------------------------- what tests read
void fake_reset(int device) {
	g_launches.clear();
	g_device = device;
}
void fake_set_sms(int sms) { g_sms = sms; }
int fake_launches(void) { return (int)g_launches.size(); }
const char *fake_name(int i) { return g_launches[i].name.c_str(); }
unsigned fake_grid(int i) { return g_launches[i].grid; }
int fake_device(int i) { return g_launches[i].device; }
int fake_stream_device(int i) { return g_launches[i].stream_device; }

// ---------------------------------------------------- what compiled code calls
void **__cudaRegisterFatBinary(void *) {
	static void *handle;
	return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *,
	dim3 *, dim3 *, int *) {
	names()[host] = name;
}
void __cudaRegisterVar(void **, char *host, char *, const char *, int, size_t size, int, int) {
	g_symbols[host] = calloc(1, size);
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shared, cudaStream_t s) {
	g_grid = grid;
	g_block = block;
	g_shared = shared;
	g_stream = s;
	return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *shared, void *s) {
	*grid = g_grid;
	*block = g_block;
	*shared = g_shared;
	*(cudaStream_t *)s = g_stream;
	return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) {
	*k = (cudaKernel_t)f;
	return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3, void **, size_t, cudaStream_t s) {
	record(k, grid, s);
	return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 grid, dim3, void **, size_t, cudaStream_t s) {
	record(f, grid, s);
	return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) {
	record(f, c->gridDim, c->stream);
	return cudaSuccess;
}

// -------------------------------------------------------------- the runtime
cudaError_t cudaGetDeviceCount(int *n) {
	*n = 2;
	return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
	g_device = d;
	return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
	*d = g_device;
	return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
	*v = a == cudaDevAttrMultiProcessorCount ? g_sms
		: a == cudaDevAttrComputeCapabilityMajor ? 10
		: a == cudaDevAttrComputeCapabilityMinor ? 3
		: a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 227 * 1024 : 1;
	return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t,
	unsigned) {
	*n = 2;
	return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }

cudaError_t cudaMalloc(void **p, size_t n) {
	*p = aligned_alloc(256, (n + 255) / 256 * 256 + 256);
	return cudaSuccess;
}
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaMallocHost(void **p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void *p) {
	free(p);
	return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaFreeHost(void *p) { return cudaFree(p); }
cudaError_t cudaMemset(void *, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *, size_t n, cudaMemcpyKind k) {
	if (k == cudaMemcpyDeviceToHost) memset(d, 0, n);
	return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) {
	return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaGetSymbolAddress(void **p, const void *symbol) {
	*p = g_symbols[symbol];
	return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *p, int) {
	*p = nullptr;
	return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
	*s = (cudaStream_t) new Stream{g_device};
	return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
	delete (Stream *)s;
	return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *st) {
	*st = cudaStreamCaptureStatusNone;
	return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) {
	*e = nullptr;
	return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
	*ms = 0.f;
	return cudaSuccess;
}

// Graphs and run-time compiled libraries: not served here.
#define FAKE_UNSERVED(name, ...) \
	cudaError_t name(__VA_ARGS__) { return cudaErrorNotSupported; }
FAKE_UNSERVED(cudaStreamBeginCapture, cudaStream_t, cudaStreamCaptureMode)
FAKE_UNSERVED(cudaStreamEndCapture, cudaStream_t, cudaGraph_t *)
FAKE_UNSERVED(cudaGraphInstantiate, cudaGraphExec_t *, cudaGraph_t, unsigned long long)
FAKE_UNSERVED(cudaGraphLaunch, cudaGraphExec_t, cudaStream_t)
FAKE_UNSERVED(cudaGraphDestroy, cudaGraph_t)
FAKE_UNSERVED(cudaGraphExecDestroy, cudaGraphExec_t)
FAKE_UNSERVED(cudaGraphGetNodes, cudaGraph_t, cudaGraphNode_t *, size_t *)
FAKE_UNSERVED(cudaLibraryLoadData, cudaLibrary_t *, const void *, enum cudaJitOption *, void **, unsigned,
	enum cudaLibraryOption *, void **, unsigned)
FAKE_UNSERVED(cudaLibraryGetKernel, cudaKernel_t *, cudaLibrary_t, const char *)
FAKE_UNSERVED(cudaLibraryUnload, cudaLibrary_t)
FAKE_UNSERVED(cudaKernelSetAttributeForDevice, cudaKernel_t, cudaFuncAttribute, int, int)

}  // extern "C"
