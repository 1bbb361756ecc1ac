// Copies between device memory and ordinary host memory, for the calls that hand out or take in whole arrays (weights, data
// sets, outputs).
//
// cudaMemcpy on pageable memory goes through the driver's staging buffer on one thread.  What bounds it is that thread: it copies
// at about 10 GB/s, and where the destination is fresh memory -- an array just allocated for the result -- it takes the
// page faults as well (101 MB of weights: 21 ms, 4.8 GB/s, against the 55 GB/s of the link).  Here a few threads share the array
// in chunks; each has a stream and a pinned slot of its own, so one thread's DMA runs under the others' memory copies and
// page faults.  Chunks of 2 MB: long enough for the link (40 us), short enough that twelve threads find work in a few tens of
// MB, and the size of a huge page.  Up to SMALL bytes one plain copy is quicker than waking threads (2.6 MB: 0.3 ms, 0.4 on two threads).
#include "host_copy.h"

#include <errno.h>
#include <stdint.h>
#include <string.h>
#include <sys/mman.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <thread>

namespace glb {
namespace {

constexpr size_t CHUNK = (size_t)2 << 20;
constexpr size_t SMALL = (size_t)4 << 20;
constexpr int MAX_THREADS = 12;
constexpr int MAX_DEVICES = 64;
constexpr size_t PREFAULT = (size_t)256 << 10;
#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23
#endif

// One per device: MAX_THREADS pinned slots (24 MB in all) and streams, made by the first large copy, freed with the last handle.
// One copy uses them at a time.
struct Lanes
{
	std::mutex mutex;
	int handles = 0;
	int lanes = 0;
	char* slot[MAX_THREADS] = {};
	cudaStream_t stream[MAX_THREADS] = {};

	void drop()
	{
		for (int i = 0; i < MAX_THREADS; ++i)
		{
			if (slot[i]) cudaFreeHost(slot[i]);
			if (stream[i]) cudaStreamDestroy(stream[i]);
			slot[i] = nullptr;
			stream[i] = nullptr;
		}
		lanes = 0;
	}
	// Makes up to `want` lanes; how many there are (fewer where pinned memory or streams run out).
	int make(int want)
	{
		for (; lanes < want; ++lanes)
		{
			cudaError_t e = cudaMallocHost(reinterpret_cast<void**>(&slot[lanes]), CHUNK);
			if (e != cudaSuccess) slot[lanes] = nullptr;
			if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&stream[lanes], cudaStreamNonBlocking);
			if (e != cudaSuccess)
			{
				if (slot[lanes]) cudaFreeHost(slot[lanes]);
				slot[lanes] = nullptr;
				stream[lanes] = nullptr;
				cudaGetLastError();
				break;
			}
		}
		return std::min(lanes, want);
	}
};
Lanes g_lanes[MAX_DEVICES];

cudaError_t plain_to_device(void* d_dst, const void* src, size_t bytes)
{
	const cudaError_t e = cudaMemcpy(d_dst, src, bytes, cudaMemcpyHostToDevice);
	return e == cudaSuccess ? cudaStreamSynchronize(0) : e;
}

cudaError_t copy_chunks(char* host, char* dev, size_t bytes, int device, bool to_host)
{
	const size_t chunks = (bytes + CHUNK - 1) / CHUNK;
	int threads = (int)std::thread::hardware_concurrency();
	threads = std::max(1, std::min(std::min(threads, MAX_THREADS), (int)std::min<size_t>(chunks, MAX_THREADS)));
	Lanes& L = g_lanes[device];
	std::lock_guard<std::mutex> lock(L.mutex);
	// Whatever cannot be had -- pinned slots here, threads below -- the copy goes on with less, down to one plain copy: it sits
	// behind a C interface, through which no exception may leave, and needed neither to succeed.
	threads = L.make(threads);
	if (threads == 0)
		return to_host ? cudaMemcpy(host, dev, bytes, cudaMemcpyDeviceToHost) : plain_to_device(dev, host, bytes);
	std::atomic<size_t> next(0);
	std::atomic<int> failed(cudaSuccess);
	auto work = [&](int lane) {
		cudaError_t e = cudaSetDevice(device);
		for (size_t c = next++; e == cudaSuccess && c < chunks && failed == cudaSuccess; c = next++)
		{
			const size_t off = c * CHUNK, n = std::min(CHUNK, bytes - off);
			if (to_host)
			{
				e = cudaMemcpyAsync(L.slot[lane], dev + off, n, cudaMemcpyDeviceToHost, L.stream[lane]);
				if (e == cudaSuccess) e = cudaStreamSynchronize(L.stream[lane]);
				if (e == cudaSuccess) memcpy(host + off, L.slot[lane], n);
			}
			else
			{
				memcpy(L.slot[lane], host + off, n);
				e = cudaMemcpyAsync(dev + off, L.slot[lane], n, cudaMemcpyHostToDevice, L.stream[lane]);
				if (e == cudaSuccess) e = cudaStreamSynchronize(L.stream[lane]);
			}
		}
		if (e != cudaSuccess) failed = e;
	};
	std::thread pool[MAX_THREADS];
	try
	{
		for (int i = 1; i < threads; ++i) pool[i] = std::thread(work, i);
	}
	catch (...)  // the system starts no more of them: those that run, and this one, take the chunks
	{
	}
	work(0);
	for (std::thread& t : pool)
		if (t.joinable()) t.join();
	return (cudaError_t)failed.load();
}

}  // namespace

cudaError_t copy_to_host(void* dst, const void* d_src, size_t bytes, int device)
{
	if (bytes <= SMALL || device < 0 || device >= MAX_DEVICES) return cudaMemcpy(dst, d_src, bytes, cudaMemcpyDeviceToHost);
	return copy_chunks(static_cast<char*>(dst), const_cast<char*>(static_cast<const char*>(d_src)), bytes, device, true);
}

cudaError_t copy_to_device(void* d_dst, const void* src, size_t bytes, int device)
{
	if (bytes <= SMALL || device < 0 || device >= MAX_DEVICES) return plain_to_device(d_dst, src, bytes);
	return copy_chunks(const_cast<char*>(static_cast<const char*>(src)), static_cast<char*>(d_dst), bytes, device, false);
}

void host_prefault(void* p, size_t bytes)
{
	if (bytes < PREFAULT) return;
	const uintptr_t page = 4096, first = ((uintptr_t)p + page - 1) & ~(page - 1), last = ((uintptr_t)p + bytes) & ~(page - 1);
	const int saved = errno;
	madvise(reinterpret_cast<void*>(first), last - first, MADV_POPULATE_WRITE);  // (contents unchanged; a kernel that does not know it says so)
	errno = saved;
}

void host_copy_retain(int device)
{
	if (device < 0 || device >= MAX_DEVICES) return;
	std::lock_guard<std::mutex> lock(g_lanes[device].mutex);
	++g_lanes[device].handles;
}

void host_copy_release(int device)
{
	if (device < 0 || device >= MAX_DEVICES) return;
	std::lock_guard<std::mutex> lock(g_lanes[device].mutex);
	if (--g_lanes[device].handles == 0) g_lanes[device].drop();
}

}  // namespace glb
