// Device-to-host copies of fields into the caller's memory.
#pragma once

#include <cuda_runtime.h>

namespace lbm {

// What a lattice keeps for them: pinned staging of THREADS x 2 chunks and
// an event for each, made on the first copy that needs them
struct HostCopy
{
	static constexpr int THREADS = 4;
	static constexpr size_t CHUNK = 1 << 18;  // bytes
	unsigned char* pinned = nullptr;
	cudaEvent_t landed[2 * THREADS] = {};
};
void host_copy_free(HostCopy&);

// Copies n values of dev_size bytes at dev into host, after the work on
// `stream`, and returns when they are there: as they are (host_size ==
// dev_size), or floats widened to doubles (4 and 8).  Memory that the device
// reaches itself takes values that go as they are in one copy.  Otherwise up to
// THREADS threads, the caller among them, each move their share through two
// pinned chunks, the copy of one chunk under the conversion of the other: the
// caller's memory is usually fresh, so most of the time is the operating system
// mapping its pages, and that goes in parallel.  100 steps of a 192x64x64 duct
// with a scalar and its two fields copied out: 10.9-12.1 ms through a pageable
// float copy widened by one thread, 5.2 ms here (the steps alone take 3.7).
cudaError_t host_copy(HostCopy& c, int device, cudaStream_t stream, const void* dev, int dev_size, void* host, int host_size,
					  long long n);

}  // namespace lbm
