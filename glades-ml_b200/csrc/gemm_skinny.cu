// Skinny products (N <= 16 output nodes, e.g. a 10-class or single-node output layer): the whole B
// operand sits in shared memory, one warp per row of A, lanes stride over k with 16-byte loads, the
// N partial sums are combined by warp shuffles.  Bound by reading A once from HBM.
#include "common.cuh"
#include "internal.h"

namespace glb {

// This file is compiled once for every four widths (SKINNY_WIDTHS = 0..3: 1 to 4, 5 to 8, ...), and once more for the host side: a process
// loads the code of the widths that it runs, not of all 64 kernels (first call of a process, beside the other fp32 products in one object and now: one
// row of 300-500-300-10 12.5 and 0.6 ms, 1000 rows of it 16.2 and 4.0, of 301-501-303-40 14.4 and 2.1, a window of 784-1000-500-10 20 and 8.4).
#ifdef SKINNY_WIDTHS
// N = the layer's width as a compile-time constant: the accumulators are registers and the inner loops carry
// no per-column predicates (the first version's 16-way predicated body stalled on instruction fetch).
template <int EPI, int N, int SK_ROWS>
__global__ void __launch_bounds__(256) gemm_skinny_kernel(const GemmArgs g)
{
	extern __shared__ __align__(16) float sW[];  // [N][K]
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
	asm volatile("griddepcontrol.wait;" ::: "memory");
	const int K = g.K;
	const uint32_t w_addr = (uint32_t)__cvta_generic_to_shared(sW);
#pragma unroll
	for (int n = 0; n < N; ++n)
		for (int k = threadIdx.x; k < K; k += blockDim.x) cp_async4(w_addr + (uint32_t)(n * K + k) * 4, g.B + n * g.b_sn + k, true);
	cp_async_commit();
	cp_async_wait<0>();
	__syncthreads();
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
	const float bias = (EPI == EPI_FORWARD && g.bias_ptr) ? *g.bias_ptr : 0.0f;
	const int K4 = K >> 2;
	// a warp takes SK_ROWS consecutive rows at a time: every weight chunk read from shared memory serves
	// all of them, and the rows' independent 16-byte loads keep HBM busy; one row where four would leave SMs idle
	const long long groups = (g.M + SK_ROWS - 1) / SK_ROWS;
	for (long long gi = (long long)blockIdx.x * wpb + warp; gi < groups; gi += (long long)gridDim.x * wpb)
	{
		const long long m0 = gi * SK_ROWS;
		const float4* arow[SK_ROWS];
#pragma unroll
		for (int r = 0; r < SK_ROWS; ++r)
		{
			const long long m = (m0 + r < g.M) ? m0 + r : g.M - 1;  // the tail repeats the last row (not stored)
			arow[r] = reinterpret_cast<const float4*>(g.A + m * g.a_sm);
		}
		float acc[SK_ROWS][N];
#pragma unroll
		for (int r = 0; r < SK_ROWS; ++r)
#pragma unroll
			for (int n = 0; n < N; ++n) acc[r][n] = 0.0f;
		// Two 16-byte chunks per row and lane, rotated: while one set of four loads is consumed the other set is in
		// flight, so the warp always has loads outstanding.  (Measured the same 2.7 TB/s as loading both sets and
		// then computing on both: with 16 warps per SM the kernel is bound by the latency of the bytes it can keep
		// in flight -- 123 registers, 80 KB of weights in shared memory per block -- not by instruction issue.)
		auto consume = [&](const float4 (&v)[SK_ROWS], int kq) {
#pragma unroll
			for (int n = 0; n < N; ++n)
			{
				const float4 w = reinterpret_cast<const float4*>(sW + n * K)[kq];
#pragma unroll
				for (int r = 0; r < SK_ROWS; ++r)
					acc[r][n] = fmaf(v[r].x, w.x, fmaf(v[r].y, w.y, fmaf(v[r].z, w.z, fmaf(v[r].w, w.w, acc[r][n]))));
			}
		};
		float4 a[SK_ROWS], b[SK_ROWS];
		if (lane < K4)
		{
#pragma unroll
			for (int r = 0; r < SK_ROWS; ++r) a[r] = arow[r][lane];
		}
		for (int k4 = lane; k4 < K4; k4 += 64)
		{
			const int k4b = k4 + 32, k4n = k4 + 64;
			const bool two = k4b < K4;
			if (two)
			{
#pragma unroll
				for (int r = 0; r < SK_ROWS; ++r) b[r] = arow[r][k4b];
			}
			consume(a, k4);
			if (k4n < K4)
			{
#pragma unroll
				for (int r = 0; r < SK_ROWS; ++r) a[r] = arow[r][k4n];
			}
			if (two) consume(b, k4b);
		}
#pragma unroll
		for (int r = 0; r < SK_ROWS; ++r)
#pragma unroll
			for (int n = 0; n < N; ++n) acc[r][n] = warp_sum(acc[r][n]);
		if (lane == 0)
		{
#pragma unroll
			for (int r = 0; r < SK_ROWS; ++r)
			{
				if (m0 + r >= g.M) break;
#pragma unroll
				for (int n = 0; n < N; ++n)
				{
					float v = acc[r][n];
					if (EPI == EPI_FORWARD) v = squash_b(v + bias, g.act, g.par);
					g.C[(m0 + r) * g.ldc + n] = v;
				}
			}
		}
	}
}

template <int EPI, int NN, int ROWS>
static cudaError_t launch_skinny(const GemmArgs& g, long long blocks, size_t bytes, cudaStream_t s)
{
	const cudaError_t e = cudaFuncSetAttribute(gemm_skinny_kernel<EPI, NN, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
	if (e != cudaSuccess) return e;
	ChainedLaunch c(dim3((unsigned)blocks), 256, bytes, true, s);
	return cudaLaunchKernelEx(&c.config, gemm_skinny_kernel<EPI, NN, ROWS>, g);
}

template <int NN>
static cudaError_t launch_width(const GemmArgs& g, cudaStream_t s)
{
	const size_t bytes = (size_t)g.N * g.K * sizeof(float);
	const bool few = g.M < 148 * 32;
	long long blocks = few ? (g.M + 7) / 8 : (g.M + 31) / 32;  // 8 warps x 1 or 4 rows per CTA pass
	if (blocks > 148 * 4) blocks = 148 * 4;
	if (blocks < 1) blocks = 1;
	if (g.epi == EPI_FORWARD) return few ? launch_skinny<EPI_FORWARD, NN, 1>(g, blocks, bytes, s) : launch_skinny<EPI_FORWARD, NN, 4>(g, blocks, bytes, s);
	return few ? launch_skinny<EPI_NONE, NN, 1>(g, blocks, bytes, s) : launch_skinny<EPI_NONE, NN, 4>(g, blocks, bytes, s);
}

cudaError_t GL_CAT(launch_gemm_skinny_, SKINNY_WIDTHS)(const GemmArgs& g, cudaStream_t s)
{
	switch (g.N - 4 * SKINNY_WIDTHS)
	{
	case 1: return launch_width<4 * SKINNY_WIDTHS + 1>(g, s);
	case 2: return launch_width<4 * SKINNY_WIDTHS + 2>(g, s);
	case 3: return launch_width<4 * SKINNY_WIDTHS + 3>(g, s);
	case 4: return launch_width<4 * SKINNY_WIDTHS + 4>(g, s);
	default: return cudaErrorInvalidValue;
	}
}
#else
constexpr int SK_NMAX = 16;

bool gemm_skinny_ok(const GemmArgs& g)
{
	return (g.epi == EPI_FORWARD || g.epi == EPI_NONE) && g.N <= SK_NMAX && g.a_sk == 1 && g.b_sk == 1 && !g.kscale &&
	       g.K % 4 == 0 && g.a_sm % 4 == 0 && (((uintptr_t)g.A) & 15) == 0 && (size_t)g.N * g.K * 4 <= 160 * 1024 && g.M >= 64;
}

cudaError_t launch_gemm_skinny_0(const GemmArgs& g, cudaStream_t s);
cudaError_t launch_gemm_skinny_1(const GemmArgs& g, cudaStream_t s);
cudaError_t launch_gemm_skinny_2(const GemmArgs& g, cudaStream_t s);
cudaError_t launch_gemm_skinny_3(const GemmArgs& g, cudaStream_t s);

cudaError_t launch_gemm_skinny(const GemmArgs& g, cudaStream_t s)
{
	switch ((g.N - 1) / 4)
	{
	case 0: return launch_gemm_skinny_0(g, s);
	case 1: return launch_gemm_skinny_1(g, s);
	case 2: return launch_gemm_skinny_2(g, s);
	default: return launch_gemm_skinny_3(g, s);
	}
}
#endif  // SKINNY_WIDTHS

}  // namespace glb
