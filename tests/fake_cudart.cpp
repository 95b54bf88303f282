// A CUDA runtime without a GPU, for the CPU tests of the host code: two devices, device memory on the heap, kernels that do
// nothing.  A launch is refused, as on a GPU, when it asks for more shared memory than its kernel may use on the current
// device: 48 KB, static and dynamic together, until cudaFuncSetAttribute raises the kernel's limit there.  Every launch is
// written to the file named by FAKE_CUDART_LOG: device, kernel.  FAKE_CUDART_MEMORY: bytes of device memory, read at every
// allocation.
#include <cuda_runtime_api.h>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

namespace {
constexpr int kDevices = 2, kOptin = 232448, kStatic = 4096;
std::mutex mu;
std::map<const void *, std::string> names;
std::map<std::pair<int, const void *>, size_t> limits;
std::map<char *, size_t> blocks;
size_t used = 0, most = 0;
thread_local int device = 0;
thread_local cudaError_t last = cudaSuccess;
struct Config { dim3 g, b; size_t smem; cudaStream_t s; };
thread_local std::vector<Config> configs;

cudaError_t ret(cudaError_t e) { if (e != cudaSuccess) last = e; return e; }

size_t limit_of(const void *f)
{
	auto it = limits.find({device, f});
	return it == limits.end() ? (size_t) 48 * 1024 - kStatic : it->second;
}

cudaError_t launch(const void *f, size_t smem)
{
	std::lock_guard<std::mutex> g(mu);
	const bool ok = smem <= limit_of(f);
	if (const char *path = std::getenv("FAKE_CUDART_LOG"))
		if (FILE *o = std::fopen(path, "a")) {
			std::fprintf(o, "%d %s%s\n", device, names[f].c_str(), ok ? "" : " refused");
			std::fclose(o);
		}
	return ret(ok ? cudaSuccess : cudaErrorInvalidValue);
}

cudaError_t alloc(void **p, size_t n)
{
	std::lock_guard<std::mutex> g(mu);
	const char *cap = std::getenv("FAKE_CUDART_MEMORY");
	*p = cap && used + n > (size_t) std::atoll(cap) ? nullptr : std::calloc(1, n ? n : 1);
	if (!*p) return ret(cudaErrorMemoryAllocation);
	blocks[(char *) *p] = n;
	used += n;
	if (used > most) most = used;
	return cudaSuccess;
}

cudaError_t release(void *p)
{
	if (!p) return cudaSuccess;
	std::lock_guard<std::mutex> g(mu);
	used -= blocks[(char *) p];
	blocks.erase((char *) p);
	std::free(p);
	return cudaSuccess;
}
char symbol[1 << 20];
}  // namespace

extern "C" {
// most device memory in use at once since the last call
size_t fake_cudart_most() { const size_t m = most; most = used; return m; }

void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *)
{
	std::lock_guard<std::mutex> g(mu);
	names[f] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) { *k = (cudaKernel_t) f; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void **, size_t smem, cudaStream_t) { return launch((const void *) k, smem); }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) { configs.push_back({g, b, smem, s}); return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *s)
{
	const Config c = configs.back();
	configs.pop_back();
	*g = c.g; *b = c.b; *smem = c.smem; *(cudaStream_t *) s = c.s;
	return cudaSuccess;
}
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3, dim3, void **, size_t smem, cudaStream_t) { return launch(f, smem); }

cudaError_t cudaGetDeviceCount(int *n) { *n = kDevices; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int)
{
	*v = a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? kOptin : a == cudaDevAttrMultiProcessorCount ? 152 : 1;
	return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int)
{
	std::memset(p, 0, sizeof *p);
	std::strcpy(p->name, "fake");
	p->multiProcessorCount = 152;
	return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *m, int) { *m = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *)
{
	std::memset(a, 0, sizeof *a);
	a->sharedSizeBytes = kStatic;
	return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v)
{
	if (a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
	if (v < 0 || v + kStatic > kOptin) return ret(cudaErrorInvalidValue);
	std::lock_guard<std::mutex> g(mu);
	limits[{device, f}] = (size_t) v;
	return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *f, int, size_t smem)
{
	std::lock_guard<std::mutex> g(mu);
	*n = smem <= limit_of(f) ? 1 : 0;
	return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int b, size_t smem, unsigned)
{
	return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, f, b, smem);
}

cudaError_t cudaMalloc(void **p, size_t n) { return alloc(p, n); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return alloc(p, n); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaFree(void *p) { return release(p); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return release(p); }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { *f = *t = (size_t) 8 << 30; return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) { *p = symbol; return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p)
{
	std::memset(a, 0, sizeof *a);
	std::lock_guard<std::mutex> g(mu);
	auto it = blocks.upper_bound((char *) p);
	if (it != blocks.begin()) {
		--it;
		if ((char *) p < it->first + it->second) { a->type = cudaMemoryTypeDevice; a->devicePointer = (void *) p; }
	}
	return cudaSuccess;
}

cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t) 1; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t) 1; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t) 1; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorInvalidValue ? "invalid argument" : "error"; }
}
