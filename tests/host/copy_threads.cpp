// Runs the large host copies of host_copy.cu on a CPU, with stand-ins for the CUDA calls and for pthread_create, where threads
// or pinned slots run out at a given number.  Exit code 0: every copy arrived whole and every thread was joined.
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <stdio.h>
#include <stdlib.h>

#include <string>

#include "host_copy.cu"

static std::atomic<int> g_threads_left(0), g_slots_left(0), g_slots_out(0), g_threads_started(0);

extern "C" {
int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* arg)
{
	typedef int (*Create)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
	static Create real = (Create)dlsym(RTLD_NEXT, "pthread_create");
	if (g_threads_left-- <= 0) return EAGAIN;
	++g_threads_started;
	return real(t, a, f, arg);
}
cudaError_t cudaMallocHost(void** p, size_t n)
{
	if (g_slots_left-- <= 0) return cudaErrorMemoryAllocation;
	++g_slots_out;
	*p = malloc(n);
	return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p)
{
	--g_slots_out;
	free(p);
	return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned)
{
	*s = nullptr;
	return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind)
{
	memcpy(d, s, n);
	return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t)
{
	memcpy(d, s, n);
	return cudaSuccess;
}
}

int main(int argc, char** argv)
{
	if (argc != 3) return 2;
	const int threads = atoi(argv[1]), slots = atoi(argv[2]);
	const size_t bytes = ((size_t)45 << 20) + 12345;  // a last chunk that is not whole
	std::string from(bytes, 0), to(bytes, 0);
	for (size_t i = 0; i < bytes; ++i) from[i] = (char)(i * 2654435761u >> 13);
	glb::host_copy_retain(0);
	for (int way = 0; way < 2; ++way)
	{
		g_threads_left = threads;
		g_slots_left = slots;
		std::fill(to.begin(), to.end(), 0);
		const cudaError_t e = way ? glb::copy_to_device(&to[0], from.data(), bytes, 0) : glb::copy_to_host(&to[0], from.data(), bytes, 0);
		if (e != cudaSuccess || to != from)
		{
			printf("way %d: error %d, data %s\n", way, (int)e, to == from ? "whole" : "wrong");
			return 1;
		}
	}
	glb::host_copy_release(0);
	if (g_slots_out != 0)
	{
		printf("%d slots not given back\n", (int)g_slots_out);
		return 1;
	}
	printf("%d threads started\n", (int)g_threads_started);
	return 0;
}
