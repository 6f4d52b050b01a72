// Device-to-host copies of fields into the caller's memory.
#pragma once

#include <cuda_runtime.h>

namespace lbm {

// What a lattice keeps for them: pinned staging of THREADS x 2 chunks and an event
// for each, made by the first copy that they pay for
struct HostCopy
{
	static constexpr int THREADS = 4;
	static constexpr size_t CHUNK = 1 << 18;  // bytes
	// when staging is made and used (host_copy): bytes handed out widened without
	// it; bytes to be widened while the stream is at work; bytes of a copy that goes
	// as it is
	static constexpr size_t STAGE_WIDENED = 16 << 20, STAGE_BUSY = 4 << 20, STAGE_COPIES = 32 << 20;
	unsigned char* pinned = nullptr;
	cudaEvent_t landed[2 * THREADS] = {};
	size_t unstaged = 0;  // bytes handed out widened without it
};
void host_copy_free(HostCopy&);

// Copies n values of dev_size bytes at dev into host, after the work on
// `stream`, and returns when they are there: as they are (host_size ==
// dev_size), or floats widened to doubles (4 and 8).  Either in one pageable copy
// (widened where it lands), or staged: up to THREADS threads, the caller among
// them, each move their share through two pinned chunks, the copy of one chunk
// under the conversion of the other.
//
// Staging pays where the operating system has yet to map the caller's memory,
// which then goes in parallel, and for the conversion; making it costs 1-2.6 ms and
// 0.4 with the lattice's end.  B200 box, 16 cores, one copy / staged, us, into
// memory that is mapped (and fresh): as doubles 3.4 MB 306 / 331 (1282 / 1252), 24
// MB 2520 / 1459 (10168 / 3269); widened 1 MB 142 / 44 (362 / 219), 8 MB 958 / 494
// (3327 / 1106), 24 MB 2789 / 888 (10296 / 2553).  Arrays of numpy below 32 MB are
// mostly mapped (the allocator's limit) and in huge pages, where one copy is the
// faster up to that size (8 MB 529 / 800, 28 MB 1685 / 1714): values that go as they
// are are staged from 32 MB on, unless the device reaches the caller's memory
// itself.  Values to be widened are staged once 16 MB have been handed out without,
// which is about where the time saved repays the making; smaller read-outs of a new
// lattice would wait for it longer than they take (32^3 lattice 2.9 ms with it, 0.16
// without).  Ahead of work of the stream the making costs less or nothing, so there
// 4 MB suffice.  100 steps of a 192x64x64 duct with a scalar and its two fields
// copied out: 10.9-12.1 ms with one copy of floats, widened by one thread, 5.2 ms
// staged (the steps alone take 3.7); the first pass of a new lattice 11.8 and 6.9.
cudaError_t host_copy(HostCopy& c, int device, cudaStream_t stream, const void* dev, int dev_size, void* host, int host_size,
					  long long n);

}  // namespace lbm
