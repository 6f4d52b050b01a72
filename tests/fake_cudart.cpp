// A CUDA runtime without a GPU for the library's host code: device memory is host
// memory, copies are done at once, kernel launches are counted and not run.  Built
// and preloaded ahead of libcudart by tests/test_host_paths.py, which sets the
// fake_* switches through ctypes.
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <string>

#include <cuda_runtime_api.h>

namespace {

std::mutex mutex;
std::map<void*, size_t> device_memory;
std::map<const void*, std::string> kernel_names;
std::map<std::string, long long> counts;
std::string trace;	// kernels launched since fake_reset, one a line
size_t in_use = 0, limit = 0;
long long launch_to_fail = 0, news_armed = 0;
bool no_pinned = false, busy = false;
const char *pinned_first = nullptr, *pinned_last = nullptr;
const void* last_copy_to = nullptr;
thread_local cudaError_t last_error = cudaSuccess;
thread_local long long news_left = 0;

cudaError_t give(cudaError_t e)
{
	if (e != cudaSuccess)
		last_error = e;
	return e;
}

struct Call
{
	dim3 grid, block;
	size_t shared;
	cudaStream_t stream;
};
thread_local Call call;
thread_local int captured = -1;

cudaError_t launch(const void* func)
{
	std::lock_guard<std::mutex> lock(mutex);
	if (launch_to_fail > 0 && --launch_to_fail == 0)
		return give(cudaErrorLaunchOutOfResources);
	counts[captured < 0 ? "launches" : "nodes"]++;
	if (captured >= 0)
		captured++;
	trace += kernel_names[func] + "\n";
	return cudaSuccess;
}

}  // namespace

void* operator new(size_t n)
{
	if (news_left > 0 && --news_left == 0) {
		counts["thrown"]++;
		throw std::bad_alloc();
	}
	if (void* p = std::malloc(n ? n : 1))
		return p;
	throw std::bad_alloc();
}
void operator delete(void* p) noexcept
{
	std::free(p);
}
void operator delete(void* p, size_t) noexcept
{
	std::free(p);
}

extern "C" {

void fake_reset()
{
	counts.clear();
	trace.clear();
}
long long fake_count(const char* what)
{
	return counts[what];
}
const char* fake_trace()
{
	return trace.c_str();
}
size_t fake_in_use()
{
	return in_use;
}
void fake_limit(size_t bytes)  // of device memory, 0: none
{
	limit = bytes;
}
void fake_fail_launch(long long n)	// the n-th launch from here fails
{
	launch_to_fail = n;
}
void fake_busy(int on)	// streams are at work when asked
{
	busy = on;
}
void fake_no_pinned(int on)
{
	no_pinned = on;
}
void fake_pinned(const char* p, size_t bytes)  // host memory that counts as pinned by the caller
{
	pinned_first = p;
	pinned_last = p + bytes;
}
const void* fake_last_copy_to()
{
	return last_copy_to;
}
// the n-th operator new of the thread after its next synchronisation throws (the
// names of counts are short and there already: this file allocates nothing there)
void fake_fail_new(long long n)
{
	counts["host copies"] = counts["thrown"] = 0;
	news_armed = n;
}

void** __cudaRegisterFatBinary(void*)
{
	static void* handle;
	return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*)
{
	std::lock_guard<std::mutex> lock(mutex);
	kernel_names[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shared, void* stream)
{
	call = Call{grid, block, shared, (cudaStream_t) stream};
	return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* shared, void* stream)
{
	*grid = call.grid;
	*block = call.block;
	*shared = call.shared;
	*(cudaStream_t*) stream = call.stream;
	return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t)
{
	return launch(f);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* f, void**)
{
	return launch(f);
}

cudaError_t cudaGetLastError()
{
	const cudaError_t e = last_error;
	last_error = cudaSuccess;
	return e;
}
const char* cudaGetErrorString(cudaError_t)
{
	return "error of the fake runtime";
}

cudaError_t cudaGetDevice(int* d)
{
	*d = 0;
	return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n)
{
	*n = 1;
	return cudaSuccess;
}
cudaError_t cudaSetDevice(int)
{
	return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int)
{
	*v = a == cudaDevAttrMultiProcessorCount ? 148 : 1 << 16;
	return cudaSuccess;
}
cudaError_t cudaDeviceCanAccessPeer(int* v, int, int)
{
	*v = 0;
	return cudaSuccess;
}
cudaError_t cudaDeviceEnablePeerAccess(int, unsigned)
{
	return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* low, int* high)
{
	if (low)
		*low = 0;
	if (high)
		*high = 0;
	return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*)
{
	std::memset(a, 0, sizeof *a);
	return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int)
{
	return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned)
{
	*n = 4;
	return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void* s)
{
	*p = const_cast<void*>(s);
	return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t n)
{
	std::lock_guard<std::mutex> lock(mutex);
	*p = nullptr;
	if ((limit && in_use + n > limit) || !(*p = std::calloc(n ? n : 1, 1)))
		return give(cudaErrorMemoryAllocation);
	device_memory[*p] = n;
	in_use += n;
	counts["allocations"]++;
	return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
	std::lock_guard<std::mutex> lock(mutex);
	const auto it = device_memory.find(p);
	if (it != device_memory.end()) {
		in_use -= it->second;
		device_memory.erase(it);
	}
	std::free(p);
	return cudaSuccess;
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t)
{
	return cudaMalloc(p, n);
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t)
{
	return cudaFree(p);
}
cudaError_t cudaMallocHost(void** p, size_t n)
{
	*p = nullptr;
	if (no_pinned)
		return give(cudaErrorMemoryAllocation);
	*p = std::calloc(n, 1);
	counts["pinned"]++;
	return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned)
{
	*p = std::calloc(n, 1);
	return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p)
{
	std::free(p);
	return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned)
{
	*d = h;
	return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p)
{
	std::memset(a, 0, sizeof *a);
	a->type = p >= pinned_first && p < pinned_last ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
	return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, cudaMemcpyKind kind, cudaStream_t)
{
	std::memcpy(to, from, n);
	std::lock_guard<std::mutex> lock(mutex);
	if (kind == cudaMemcpyDeviceToHost) {
		counts["host copies"]++;
		last_copy_to = to;
	}
	return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t)
{
	return cudaSuccess;	 // the memory is cleared when it is allocated
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned)
{
	*s = (cudaStream_t) std::calloc(1, 1);
	return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int)
{
	return cudaStreamCreateWithFlags(s, f);
}
cudaError_t cudaStreamDestroy(cudaStream_t s)
{
	std::free(s);
	return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t)
{
	if (news_armed > 0) {
		news_left = news_armed;
		news_armed = 0;
	}
	return cudaSuccess;
}
cudaError_t cudaStreamQuery(cudaStream_t)
{
	return busy ? give(cudaErrorNotReady) : cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned)
{
	return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode)
{
	captured = 0;
	return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g)
{
	*g = (cudaGraph_t) std::calloc(1, 1);
	captured = -1;
	return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g)
{
	std::free(g);
	return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long)
{
	*e = (cudaGraphExec_t) std::calloc(1, 1);
	counts["graphs"]++;
	return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e)
{
	std::free(e);
	return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t)
{
	counts["graph launches"]++;
	return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e)
{
	*e = (cudaEvent_t) std::calloc(1, 1);
	return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned)
{
	return cudaEventCreate(e);
}
cudaError_t cudaEventDestroy(cudaEvent_t e)
{
	std::free(e);
	return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t)
{
	return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t)
{
	return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t)
{
	*ms = 1;
	return cudaSuccess;
}

}  // extern "C"
