// Device-to-host copies of fields into the caller's memory (host_copy.h).
#include "host_copy.h"

#include <atomic>
#include <cstring>
#include <exception>
#include <functional>
#include <thread>

namespace lbm {

namespace {

struct Job
{
	HostCopy* c;
	int device;
	cudaStream_t stream;
	const unsigned char* dev;
	unsigned char* host;
	int dev_size, host_size;
	long long n, per_chunk, nchunks;
	int threads;
	std::atomic<int> error{cudaSuccess};
};

void deliver(const unsigned char* from, int dev_size, unsigned char* host, int host_size, long long first, long long count)
{
	unsigned char* to = host + first * host_size;
	if (dev_size == host_size) {
		std::memcpy(to, from, (size_t) (count * dev_size));
		return;
	}
	const float* f = reinterpret_cast<const float*>(from);
	double* d = reinterpret_cast<double*>(to);
	for (long long i = 0; i < count; i++)
		d[i] = f[i];
}

// thread k takes chunks k, k + threads, ... through its two pinned chunks
void work(Job& j, int k)
{
	cudaError_t e = cudaSetDevice(j.device);
	auto issue = [&](long long chunk, int slot)
	{
		const long long first = chunk * j.per_chunk, count = j.n - first < j.per_chunk ? j.n - first : j.per_chunk;
		e = cudaMemcpyAsync(j.c->pinned + (size_t) (2 * k + slot) * HostCopy::CHUNK, j.dev + first * j.dev_size,
							(size_t) (count * j.dev_size), cudaMemcpyDeviceToHost, j.stream);
		if (e == cudaSuccess)
			e = cudaEventRecord(j.c->landed[2 * k + slot], j.stream);
	};
	int slot = 0;
	if (e == cudaSuccess && k < j.nchunks)
		issue(k, 0);
	for (long long chunk = k; e == cudaSuccess && chunk < j.nchunks; chunk += j.threads) {
		if (chunk + j.threads < j.nchunks)
			issue(chunk + j.threads, slot ^ 1);
		const cudaError_t s = cudaEventSynchronize(j.c->landed[2 * k + slot]);
		if (e == cudaSuccess)
			e = s;
		if (e != cudaSuccess)
			break;
		const long long first = chunk * j.per_chunk;
		deliver(j.c->pinned + (size_t) (2 * k + slot) * HostCopy::CHUNK, j.dev_size, j.host, j.host_size, first,
				j.n - first < j.per_chunk ? j.n - first : j.per_chunk);
		slot ^= 1;
	}
	if (e != cudaSuccess) {
		cudaStreamSynchronize(j.stream);  // nothing of ours is in flight into the pinned chunks
		j.error = (int) e;
	}
}

// memory that the runtime knows (pinned, registered, managed): the device copies into it itself
bool reached_by_device(const void* host)
{
	cudaPointerAttributes a;
	if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
		cudaGetLastError();
		return false;
	}
	return a.type != cudaMemoryTypeUnregistered;
}

bool at_work(cudaStream_t stream)
{
	const cudaError_t e = cudaStreamQuery(stream);
	if (e != cudaSuccess)
		cudaGetLastError();	 // not ready, or an error that the copy reports
	return e == cudaErrorNotReady;
}

cudaError_t direct_copy(cudaStream_t stream, const void* dev, void* host, size_t bytes)
{
	const cudaError_t e = cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, stream);
	return e == cudaSuccess ? cudaStreamSynchronize(stream) : e;
}

// floats widened to doubles without staging: one copy into the upper half of the
// caller's memory, widened there from the front.  Value i ends at byte 8 i + 8, and
// the next one still waits from 4 n + 4 (i + 1) on: not before that for any i < n.
cudaError_t widen_in_place(cudaStream_t stream, const void* dev, void* host, long long n)
{
	unsigned char* const floats = (unsigned char*) host + 4 * (size_t) n;
	const cudaError_t e = direct_copy(stream, dev, floats, 4 * (size_t) n);
	if (e != cudaSuccess)
		return e;
	float part[1024];
	for (long long first = 0; first < n; first += 1024) {
		const long long count = n - first < 1024 ? n - first : 1024;
		std::memcpy(part, floats + 4 * first, 4 * (size_t) count);
		deliver(reinterpret_cast<const unsigned char*>(part), 4, (unsigned char*) host, 8, first, count);
	}
	return cudaSuccess;
}

}  // namespace

void host_copy_free(HostCopy& c)
{
	if (c.pinned)
		cudaFreeHost(c.pinned);
	c.pinned = nullptr;
	for (cudaEvent_t& ev : c.landed) {
		if (ev)
			cudaEventDestroy(ev);
		ev = nullptr;
	}
}

cudaError_t host_copy(HostCopy& c, int device, cudaStream_t stream, const void* dev, int dev_size, void* host, int host_size,
					  long long n)
{
	if (n < 1)
		return cudaStreamSynchronize(stream);
	const bool widen = dev_size != host_size;
	const size_t bytes = (size_t) n * host_size;
	if (!widen && (bytes < HostCopy::STAGE_COPIES || reached_by_device(host)))
		return direct_copy(stream, dev, host, bytes);
	if (!c.pinned && widen && (c.unstaged += bytes) < HostCopy::STAGE_WIDENED
		&& (bytes < HostCopy::STAGE_BUSY || !at_work(stream)))
		return widen_in_place(stream, dev, host, n);
	if (!c.pinned) {
		cudaError_t e = cudaMallocHost((void**) &c.pinned, 2 * HostCopy::THREADS * HostCopy::CHUNK);
		for (cudaEvent_t& ev : c.landed)
			if (e == cudaSuccess)
				e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
		if (e != cudaSuccess) {
			// no pinned memory to be had
			host_copy_free(c);
			cudaGetLastError();
			return widen ? widen_in_place(stream, dev, host, n) : direct_copy(stream, dev, host, bytes);
		}
	}
	Job j;
	j.c = &c;
	j.device = device;
	j.stream = stream;
	j.dev = (const unsigned char*) dev;
	j.host = (unsigned char*) host;
	j.dev_size = dev_size;
	j.host_size = host_size;
	j.n = n;
	j.per_chunk = (long long) HostCopy::CHUNK / dev_size;
	j.nchunks = (n + j.per_chunk - 1) / j.per_chunk;
	// a thread is worth starting for a few chunks
	j.threads = j.nchunks >= 4 * HostCopy::THREADS ? HostCopy::THREADS : 1;
	std::thread helpers[HostCopy::THREADS - 1];
	int started = 0;
	if (j.threads > 1) {
		// the stream's work first: the helpers start when there is something to move
		const cudaError_t e = cudaStreamSynchronize(stream);
		if (e != cudaSuccess)
			return e;
		try {
			for (; started < HostCopy::THREADS - 1; started++)
				helpers[started] = std::thread(work, std::ref(j), started + 1);
		}
		catch (const std::exception&) {
			// no more threads to be had, or no memory for one: this one takes the
			// others' shares below
		}
	}
	for (int k = 0; k < j.threads; k++)
		if (k == 0 || k > started)
			work(j, k);
	for (int k = 0; k < started; k++)
		helpers[k].join();
	return (cudaError_t) j.error.load();
}

}  // namespace lbm
