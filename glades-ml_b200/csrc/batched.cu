// Batched-mode kernels that are not a tiled product: fp32 products of few rows, gradients of few output nodes, the
// output-layer head (delta + metrics + confusion counts, optional softmax), the scalar-bias reduction, the weight-decay column
// term and the fused update.
//
// One window step of batched mode is, per weight layer l (reference arithmetic of
// Networks/network.cpp:457-668 with aligned windows, frozen weights and a plain error sum):
//   forward   A_{l+1} = squash(A_l W_l^T + b_l)                       (EPI_FORWARD)
//   head      D_{H+1} = cost'(Y, A_{H+1})  or  softmax(Z) - Y;  metrics; confusion counts
//   errprop   D_l     = (D_{l+1} W_l) * act'(A_l)                     (EPI_ERRPROP)
//   gradient  G_l     = lr_l * D_{l+1}^T diag(c) A_l + decay          (EPI_GRAD)
//   update    W -= G / mb ;  b_l -= scale_l * lr_l * sum(D_{l+1})
#include "common.cuh"
#include "internal.h"
#include "tc_gemm.h"

namespace glb {

// ---------------------------------------------------------------------------------------------
// Forward products of few rows (single requests, small batches): the sums of 16 output nodes and MB (at most 32) rows per
// CTA, every sum one fmaf chain with k ascending like the tiles above, so that a row's result does not depend on the rows that
// come with it.  One row of a 2048-wide layer is 16 MB of weights and 2048 dependent multiply-adds, 4 clocks each: both want all
// SMs, which 64 x 64 tiles leave idle (32 CTAs).  TN x TM outputs per thread: for one row the chain is the bound (4.3 us at 2048),
// with more rows the words that shared memory delivers, (TN + TM) / (TN * TM) per multiply-add.  The first warps compute, the
// others copy RW_ST stages of KT inputs and weights ahead by cp.async.  Measured, one row, 784-2048-2048-10, the three products:
// tiles 207 us, this kernel 35 us, a whole request 281 and 72 us.
constexpr int RW_N = 16, RW_T = 128, RW_K = 128, RW_P = RW_K + 4;  // pitch: an odd number of quads
__host__ __device__ constexpr int rw_stages(int mb) { return mb <= 16 ? 5 : 3; }
__host__ __device__ constexpr size_t rw_smem(int mb) { return (size_t)rw_stages(mb) * (RW_N + mb) * RW_P * sizeof(float); }

template <int TN, int TM, int MB>
__global__ void __launch_bounds__(RW_T) gemm_rows_kernel(const GemmArgs g, bool a16, bool b16)
{
	constexpr int ST = rw_stages(MB);
	constexpr int NG = RW_N / TN, CT = NG * (MB / TM);       // threads that compute
	constexpr int CW = (CT + 31) / 32, LW = RW_T / 32 - CW;  // warps that compute, warps that copy
	constexpr int STAGE = (RW_N + MB) * RW_P;
	constexpr int G = TM * TN == 1 ? 4 : (TM * TN == 4 ? 2 : 1);  // quads of k per step: read one step ahead of their use
	extern __shared__ __align__(16) float sm[];
	const int t = threadIdx.x, lane = t & 31, loader = (t >> 5) - CW;
	const int n0 = blockIdx.x * RW_N, m0 = blockIdx.y * MB;
	const int stages = (g.K + RW_K - 1) / RW_K;
	const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm);
	// a warp copies whole rows: 128 k of a weight row or of an input row (what lies outside the matrices is filled with zeros)
	auto part = [&](int st, const float* src, long long pitch, int left, int count, int at, bool vec) {
		if (loader < 0 || st >= stages) return;
		const uint32_t dst = base + (uint32_t)((st % ST) * STAGE) * 4;
		const int k0 = st * RW_K;
		for (int r = loader; r < count; r += LW)
		{
			const float* row = src + (r < left ? r : 0) * pitch;
			const uint32_t d = dst + (uint32_t)((at + r) * RW_P) * 4;
			if (vec)
			{
				const int k = k0 + lane * 4, n = r < left ? (g.K - k < 4 ? g.K - k : 4) : 0;
				cp_async16(d + lane * 16, n > 0 ? row + k : row, n > 0 ? n : 0);
			}
			else
#pragma unroll
				for (int q = 0; q < 4; ++q)
				{
					const int k = k0 + lane + 32 * q;
					const bool ok = r < left && k < g.K;
					cp_async4(d + (lane + 32 * q) * 4, ok ? row + k : row, ok);
				}
		}
	};
	auto weights = [&](int st) { part(st, g.B + n0 * g.b_sn, g.b_sn, g.N - n0, RW_N, 0, b16); };
	auto inputs = [&](int st) { part(st, g.A + m0 * g.a_sm, g.a_sm, g.M - m0, MB, RW_N, a16); };
	// In a chain of these products the next one starts early: its first weights travel while this one runs, and only then does
	// it wait for the inputs (everything before the chain's first product has ended when that one starts).
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#pragma unroll
	for (int st = 0; st < ST - 1; ++st) weights(st);
	asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
	for (int st = 0; st < ST - 1; ++st)
	{
		inputs(st);
		cp_async_commit();  // (the first group holds all the weights so far)
	}
	const int tn = t % NG, tm = t / NG;
	float acc[TM][TN] = {};
	for (int st = 0; st < stages; ++st)
	{
		cp_async_wait<ST - 2>();
		__syncthreads();  // the stage has landed, and the one before it has been consumed
		weights(st + ST - 1);
		inputs(st + ST - 1);
		cp_async_commit();
		if (t < CT)
		{
			const float* w = sm + (st % ST) * STAGE + tn * RW_P;
			const float* x = sm + (st % ST) * STAGE + (RW_N + tm) * RW_P;
			float4 b[2][G][TN], a[2][G][TM];
			auto read = [&](int buf, int k) {
#pragma unroll
				for (int q = 0; q < G; ++q)
				{
#pragma unroll
					for (int j = 0; j < TN; ++j) b[buf][q][j] = *reinterpret_cast<const float4*>(w + j * NG * RW_P + k + 4 * q);
#pragma unroll
					for (int i = 0; i < TM; ++i) a[buf][q][i] = *reinterpret_cast<const float4*>(x + i * (MB / TM) * RW_P + k + 4 * q);
				}
			};
			auto use = [&](int buf) {
#pragma unroll
				for (int q = 0; q < G; ++q)
				{
#pragma unroll
					for (int i = 0; i < TM; ++i)
#pragma unroll
						for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[buf][q][i].x, b[buf][q][j].x, acc[i][j]);
#pragma unroll
					for (int i = 0; i < TM; ++i)
#pragma unroll
						for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[buf][q][i].y, b[buf][q][j].y, acc[i][j]);
#pragma unroll
					for (int i = 0; i < TM; ++i)
#pragma unroll
						for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[buf][q][i].z, b[buf][q][j].z, acc[i][j]);
#pragma unroll
					for (int i = 0; i < TM; ++i)
#pragma unroll
						for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[buf][q][i].w, b[buf][q][j].w, acc[i][j]);
				}
			};
			read(0, 0);
#pragma unroll 1
			for (int k = 0; k < RW_K; k += 8 * G)
			{
				read(1, k + 4 * G);
				use(0);
				if (k + 8 * G < RW_K) read(0, k + 8 * G);
				use(1);
			}
		}
	}
	cp_async_wait<0>();
	if (t >= CT) return;
	const float bias = g.bias_ptr ? *g.bias_ptr : 0.0f;
#pragma unroll
	for (int i = 0; i < TM; ++i)
#pragma unroll
		for (int j = 0; j < TN; ++j)
		{
			const int m = m0 + tm + i * (MB / TM), n = n0 + tn + j * NG;
			if (m < g.M && n < g.N) g.C[(long long)m * g.ldc + n] = squash_b(acc[i][j] + bias, g.act, g.par);
		}
}

template <int TN, int TM, int MB>
static cudaError_t launch_rows(const GemmArgs& g, cudaStream_t s)
{
	const bool a16 = ((g.a_sm & 3) == 0 || g.M == 1) && (((uintptr_t)g.A) & 15) == 0, b16 = ((g.b_sn & 3) == 0 || g.N == 1) && (((uintptr_t)g.B) & 15) == 0;
	if (rw_smem(MB) > 48 * 1024)
	{
		const cudaError_t e = cudaFuncSetAttribute(gemm_rows_kernel<TN, TM, MB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rw_smem(MB));
		if (e != cudaSuccess) return e;
	}
	ChainedLaunch c(dim3((g.N + RW_N - 1) / RW_N, (g.M + MB - 1) / MB), RW_T, rw_smem(MB), g.chained, s);
	return cudaLaunchKernelEx(&c.config, gemm_rows_kernel<TN, TM, MB>, g, a16, b16);
}

// By rows or by tiles: the smaller of the two in clocks.  Measured, K = 256, 1000 and 2048, N = 50 to 2048: one row 5.2 / 9.3 / 14.4 us
// against 10.3 / 26.7 / 48.6 us by 32-row tiles, 8 rows 6.3 / 14.4 / 20.6, 16 rows 8.3 / 20.6 / 32.9, 32 rows 10.3 / 20.6 / 34.9 against
// 10.3 / 28.8 / 53.4.  (64 rows per CTA: 16.5 / 32.9 / 53.4, nowhere better than the tiles, and a wave of its CTAs ends sooner.)
static int rows_block(int M) { return M <= 1 ? 1 : (M <= 8 ? 8 : (M <= 16 ? 16 : 32)); }
static bool rows_ok(const GemmArgs& g)
{
	if (g.epi != EPI_FORWARD || g.a_sk != 1 || g.b_sk != 1 || g.kscale || g.M > 32) return false;
	const int mb = rows_block(g.M);
	const long long per_k = mb == 1 ? 11 : (mb == 8 ? 16 : (mb == 16 ? 27 : 28)), ends = mb == 1 ? 2000 : 5000;
	return ((g.N + RW_N - 1) / RW_N + 147) / 148 * (per_k * g.K + ends) < ffma_tile_clocks(g.M, g.N, g.K);
}

// Gradients of layers with at most 16 outputs (M <= 16): the sums over the window's rows have to stay one chain each, and
// 64-wide tiles would run them on a handful of SMs with most of each tile empty (10 x 500 over 1000 rows: 50 us on eight CTAs).
// A CTA takes 16 inputs: two warps hold 4 x 1 sums per thread, four warps copy TG_ST stages of 64 rows ahead; bound by the chain and
// the three shared-memory reads per row.  (10 x 500 over 1000 rows: 18.8 us with two copying warps that made every address anew, and
// a branch per row on the momentum weights.)
constexpr int TG_M = 16, TG_N = 16, TG_K = 64, TG_ST = 5, TG_C = 64, TG_T = TG_C + 128;

template <bool SCALED>
__global__ void __launch_bounds__(TG_T) gemm_thin_gradient_kernel(const GemmArgs g, bool vec_b)
{
	__shared__ __align__(16) float sA[TG_ST][TG_K][TG_M], sB[TG_ST][TG_K][TG_N];
	__shared__ float sC[TG_ST][TG_K];
	const int t = threadIdx.x, c = t - TG_C, n0 = blockIdx.x * TG_N;
	const int stages = (g.K + TG_K - 1) / TG_K;
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
	asm volatile("griddepcontrol.wait;" ::: "memory");
	// copying thread c: column c % 16 of rows c / 16, c / 16 + 8, ...; inputs by quads (vec_b) of rows c / 4, c / 4 + 32
	const bool in_a = (c & 15) < g.M, in_b = n0 + (c & 15) < g.N;
	const float* pa = g.A + (in_a ? c & 15 : 0) + (long long)(c >> 4) * g.a_sk;
	const float* pb = vec_b ? g.B + n0 + 4 * (c & 3) + (long long)(c >> 2) * g.b_sk : g.B + (in_b ? n0 + (c & 15) : 0) + (long long)(c >> 4) * g.b_sk;
	const int quad = g.N - n0 - 4 * (c & 3);
	auto fill = [&](int st) {
		if (c >= 0 && st < stages)
		{
			const int b = st % TG_ST, left = g.K - st * TG_K;
			const uint32_t da = (uint32_t)__cvta_generic_to_shared(&sA[b][0][0]) + c * 4, db = (uint32_t)__cvta_generic_to_shared(&sB[b][0][0]);
			const float* p = pa;
#pragma unroll
			for (int q = 0; q < TG_K / 8; ++q, p += 8 * g.a_sk)
			{
				const bool in = in_a && (c >> 4) + 8 * q < left;
				cp_async4(da + q * 8 * TG_M * 4, in ? p : g.A, in);
			}
			p = pb;
			if (vec_b)
			{
#pragma unroll
				for (int q = 0; q < 2; ++q, p += 32 * g.b_sk)
				{
					const int n = (c >> 2) + 32 * q < left ? quad : 0;
					cp_async16(db + (c + 128 * q) * 16, n > 0 ? p : g.B, n);
				}
			}
			else
#pragma unroll
				for (int q = 0; q < TG_K / 8; ++q, p += 8 * g.b_sk)
				{
					const bool in = in_b && (c >> 4) + 8 * q < left;
					cp_async4(db + c * 4 + q * 8 * TG_N * 4, in ? p : g.B, in);
				}
			if (SCALED && c < TG_K)
				cp_async4((uint32_t)__cvta_generic_to_shared(&sC[b][c]), c < left ? g.kscale + st * TG_K + c : g.kscale, c < left);
			pa += TG_K * g.a_sk;
			pb += TG_K * g.b_sk;
		}
		cp_async_commit();
	};
#pragma unroll
	for (int st = 0; st < TG_ST - 1; ++st) fill(st);
	const int n = t & 15, m = ((t >> 4) & 3) * 4;
	float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
	for (int st = 0; st < stages; ++st)
	{
		cp_async_wait<TG_ST - 2>();
		__syncthreads();  // the stage has landed, and the one before it has been consumed
		fill(st + TG_ST - 1);
		if (t < TG_C)
		{
			const int b = st % TG_ST;
#pragma unroll 32
			for (int k = 0; k < TG_K; ++k)
			{
				float4 a = *reinterpret_cast<const float4*>(&sA[b][k][m]);
				const float x = sB[b][k][n];
				if (SCALED)
				{
					const float c = sC[b][k];
					a.x *= c; a.y *= c; a.z *= c; a.w *= c;
				}
				acc[0] = fmaf(a.x, x, acc[0]);
				acc[1] = fmaf(a.y, x, acc[1]);
				acc[2] = fmaf(a.z, x, acc[2]);
				acc[3] = fmaf(a.w, x, acc[3]);
			}
		}
	}
	cp_async_wait<0>();
	if (t >= TG_C || n0 + n >= g.N) return;
	bool bad = false;
#pragma unroll
	for (int i = 0; i < 4; ++i)
	{
		if (m + i >= g.M) continue;
		const float x = g.alpha * acc[i] + (g.colterm ? g.colterm[n0 + n] : 0.0f);
		if (g.W)
		{
			float* wp = g.W + (long long)(m + i) * g.N + n0 + n;
			const float w = *wp - x * g.inv_mb;
			bad = bad || !isfinite(w);
			*wp = w;
		}
		else g.C[(long long)(m + i) * g.ldc + n0 + n] = x;
	}
	if (bad) atomicOr(g.bad_flag, 1);
}

bool gemm_ffma_by_rows(const GemmArgs& g) { return !gemm_skinny_ok(g) && rows_ok(g); }
static bool thin_ok(const GemmArgs& g) { return g.epi == EPI_GRAD && g.a_sm == 1 && g.b_sn == 1 && g.M <= TG_M; }

int ffma_route(int epi, int M, int N, int K, int* rows)
{
	GemmArgs g;
	memset(&g, 0, sizeof g);
	g.epi = epi;
	g.M = M;
	g.N = N;
	g.K = K;
	// (as the layers' operands lie: pitches of the activations padded to whole quads, so that none of the strides rules a kernel out)
	const bool forward = epi == EPI_FORWARD || epi == EPI_NONE;
	(forward || epi == EPI_ERRPROP ? g.a_sk : g.a_sm) = 1;
	(forward ? g.b_sk : g.b_sn) = 1;
	*rows = 0;
	if (gemm_skinny_ok(g) || thin_ok(g)) return 0;
	const bool by_rows = rows_ok(g);
	*rows = by_rows ? rows_block(M) : ffma_tile_rows(M, N, K);
	return by_rows ? 1 : 2;
}

cudaError_t launch_gemm_ffma(const GemmArgs& g, cudaStream_t s)
{
	if (gemm_skinny_ok(g)) return launch_gemm_skinny(g, s);
	if (thin_ok(g))
	{
		ChainedLaunch c(dim3((g.N + TG_N - 1) / TG_N), TG_T, 0, true, s);
		const bool vec_b = (g.b_sk & 3) == 0 && (((uintptr_t)g.B) & 15) == 0;
		return g.kscale ? cudaLaunchKernelEx(&c.config, gemm_thin_gradient_kernel<true>, g, vec_b) : cudaLaunchKernelEx(&c.config, gemm_thin_gradient_kernel<false>, g, vec_b);
	}
	if (rows_ok(g))
		switch (rows_block(g.M))
		{
		case 1: return launch_rows<1, 1, 1>(g, s);
		case 8: return launch_rows<1, 4, 8>(g, s);
		case 16: return launch_rows<2, 4, 16>(g, s);
		default: return launch_rows<2, 4, 32>(g, s);
		}
	return launch_ffma_tiles(g, s);
}

// ---------------------------------------------------------------------------------------------
// Output-layer head: one warp per row.  Metrics follow network.cpp:519-547 (cost / (rows*n_out),
// |p-e| accuracy) and CMatrix::addResult (GMath/cmatrix.cpp:57-98: strict > from 0, first maximum
// wins); the output delta is the bare cost derivative (network.cpp:599-612: the output activation's
// derivative is dropped), or p - y behind the softmax extension.
__global__ void __launch_bounds__(256) head_kernel(const HeadArgs h)
{
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
	asm volatile("griddepcontrol.wait;" ::: "memory");
	const int lane = threadIdx.x & 31;
	const int warp = threadIdx.x >> 5;
	const int wpb = blockDim.x >> 5;
	double cost_acc = 0.0, acc_acc = 0.0, d_acc = 0.0;
	float d_max = 0.0f;  // largest finite |D|
	auto put_delta = [&](long long at, float d) {
		h.D[at] = d;
		d_acc += (double)d;
		const float m = fabsf(d);
		if (m <= 3.402823466e38f) d_max = fmaxf(d_max, m);
	};
	for (long long r = (long long)blockIdx.x * wpb + warp; r < h.rows; r += (long long)gridDim.x * wpb)
	{
		float* p = h.P + r * h.n;
		const float* y = h.Y + r * h.n;
		float mx = -INFINITY, inv_den = 1.0f;
		if (h.softmax)
		{
			// (unrolled: the row's loads are independent, and one warp per row leaves few warps to hide their latency)
#pragma unroll 8
			for (int o = lane; o < h.n; o += 32) mx = fmaxf(mx, p[o]);
			mx = warp_max(mx);
			float den = 0.0f;
#pragma unroll 8
			for (int o = lane; o < h.n; o += 32) den += expf(p[o] - mx);
			den = warp_sum(den);
			inv_den = 1.0f / den;
		}
		// running first-maximum argmax of expected and predicted (value, index) per lane
		float be = 0.0f, bp = 0.0f;
		int ie = -1, ip = -1;
#pragma unroll 4
		for (int o = lane; o < h.n; o += 32)
		{
			float pv = p[o];
			const float e = y[o];
			float cost;
			if (h.softmax)
			{
				pv = expf(pv - mx) * inv_den;
				p[o] = pv;
				cost = (e != 0.0f) ? -(e * logf(pv)) / h.data_size : 0.0f;
				if (h.D) put_delta(r * h.n + o, pv - e);
			}
			else
			{
				if (h.out_type == GL_OUT_REGRESSION) { const float t = e - pv; cost = t * t / h.data_size; }
				else if (h.out_type == GL_OUT_CLASSIFICATION)
					cost = -((e * logf(pv)) + ((1.0f - e) * logf(1.0f - pv))) / h.data_size;
				else cost = logf(e / pv) / h.data_size;
				if (h.D)
				{
					float d;
					if (h.out_type == GL_OUT_REGRESSION) d = 2.0f * (pv - e);
					else if (h.out_type == GL_OUT_CLASSIFICATION) d = (pv - e) / ((1.0f - pv) * pv);
					else d = -(e / pv);
					put_delta(r * h.n + o, d);
				}
			}
			if (h.P_host) h.P_host[r * h.n + o] = pv;
			cost_acc += (double)cost;
			float pe = fabsf(pv - e);
			pe = fminf(pe, 1.0f);
			acc_acc += (double)fmaxf((1.0f - pe) * 100.0f, 0.0f);
			if (e > be) { be = e; ie = o; }
			if (pv > bp) { bp = pv; ip = o; }
		}
		// warp argmax: larger value wins, ties go to the smaller index (first maximum wins)
#pragma unroll
		for (int off = 16; off > 0; off >>= 1)
		{
			const float oe = __shfl_xor_sync(0xffffffffu, be, off);
			const int oie = __shfl_xor_sync(0xffffffffu, ie, off);
			if (oie >= 0 && (ie < 0 || oe > be || (oe == be && oie < ie))) { be = oe; ie = oie; }
			const float op = __shfl_xor_sync(0xffffffffu, bp, off);
			const int oip = __shfl_xor_sync(0xffffffffu, ip, off);
			if (oip >= 0 && (ip < 0 || op > bp || (op == bp && oip < ip))) { bp = op; ip = oip; }
		}
		if (h.last_out && r == h.rows - 1)
			for (int o = lane; o < h.n; o += 32) h.last_out[o] = p[o];
		if (lane == 0)
		{
			if (h.argmax) h.argmax[r] = ip;
			if (h.confusion && h.out_type != GL_OUT_REGRESSION && ie >= 0 && ip >= 0)
				atomicAdd(&h.confusion[ie * h.n + ip], 1);
		}
	}
	cost_acc = warp_sum_d(cost_acc);
	acc_acc = warp_sum_d(acc_acc);
	__shared__ double s_c[8], s_a[8], s_d[8];
	__shared__ unsigned s_m;
	if (threadIdx.x == 0) s_m = 0u;
	d_acc = warp_sum_d(d_acc);
	const unsigned d_bits = __reduce_max_sync(0xffffffffu, __float_as_uint(d_max));
	if (lane == 0) { s_c[warp] = cost_acc; s_a[warp] = acc_acc; s_d[warp] = d_acc; }
	__syncthreads();
	if (lane == 0 && h.dsc) atomicMax(&s_m, d_bits);
	__syncthreads();
	if (threadIdx.x == 0)
	{
		double c = 0.0, a = 0.0, d = 0.0;
		for (int w = 0; w < wpb; ++w) { c += s_c[w]; a += s_a[w]; d += s_d[w]; }
		if (h.sums2)
		{
			atomicAdd(&h.sums2[0], c);
			atomicAdd(&h.sums2[1], a);
		}
		if (h.dsum) h.dsum[blockIdx.x] = d;
		if (h.dsc && s_m) atomicMax(&h.dsc->amax, s_m);
	}
}

int head_blocks(long long rows)
{
	long long blocks = (rows + 7) / 8;
	if (blocks > 148 * 8) blocks = 148 * 8;
	return (int)(blocks < 1 ? 1 : blocks);
}

cudaError_t launch_head(const HeadArgs& h, cudaStream_t s)
{
	ChainedLaunch c(dim3(head_blocks(h.rows)), 256, 0, true, s);
	return cudaLaunchKernelEx(&c.config, head_kernel, h);
}

// ---------------------------------------------------------------------------------------------
// *out += alpha * sum(D[0..count)), reproducibly: every block sums a fixed set of elements in double and leaves its
// partial in `part`; the block that arrives last (a ticket counter) adds the partials in a fixed order and is the only
// one to touch *out.  (A float atomic per block would make the scalar bias depend on the order the blocks finish in.)
// part: gridDim.x doubles; ticket: one word, zero before the launch and zero again after it.
__global__ void __launch_bounds__(256) sum_scaled_kernel(const float* __restrict__ D, long long count, float alpha, float* out,
                                                         double* part, unsigned* ticket)
{
	double acc = 0.0;
	const long long stride = (long long)gridDim.x * blockDim.x;
	const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if ((reinterpret_cast<uintptr_t>(D) & 15) == 0)
	{
		const long long n4 = count >> 2;
		const float4* D4 = reinterpret_cast<const float4*>(D);
#pragma unroll 4
		for (long long i = i0; i < n4; i += stride)
		{
			const float4 v = D4[i];
			acc += ((double)v.x + (double)v.y) + ((double)v.z + (double)v.w);
		}
		for (long long i = (n4 << 2) + i0; i < count; i += stride) acc += (double)D[i];
	}
	else
		for (long long i = i0; i < count; i += stride) acc += (double)D[i];
	acc = warp_sum_d(acc);
	__shared__ double sw[8];
	__shared__ bool last;
	if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = acc;
	__syncthreads();
	if (threadIdx.x == 0)
	{
		double t = 0.0;
		for (int w = 0; w < 8; ++w) t += sw[w];
		part[blockIdx.x] = t;
		__threadfence();
		last = atomicAdd(ticket, 1u) == gridDim.x - 1;
	}
	__syncthreads();
	if (last && threadIdx.x < 32)
	{
		__threadfence();
		double t = 0.0;
		for (unsigned b = threadIdx.x; b < gridDim.x; b += 32) t += __ldcg(part + b);
		t = warp_sum_d(t);
		if (threadIdx.x == 0)
		{
			*out += (float)(t * (double)alpha);
			*ticket = 0u;
		}
	}
}

cudaError_t launch_sum_scaled(const float* D, long long count, float alpha, float* out, double* part, unsigned* ticket, cudaStream_t s)
{
	long long blocks = (count + 256 * 16 - 1) / (256 * 16);
	if (blocks > SUM_SCALED_MAX_BLOCKS) blocks = SUM_SCALED_MAX_BLOCKS;
	if (blocks < 1) blocks = 1;
	sum_scaled_kernel<<<(unsigned)blocks, 256, 0, s>>>(D, count, alpha, out, part, ticket);
	return cudaGetLastError();
}

// colterm[i] = lr * sum_j c_j * (wd1*|A[j][i]| + wd2*A[j][i])   (decay terms of Node::getDelta,
// State/node.cpp:284-289: they use the INPUT activation, not the weight)
__global__ void decay_colterm_kernel(const float* A, int rows, int n, long long ld, const float* c, float lr, float wd1, float wd2,
                                     float* colterm)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	double s = 0.0;
	for (int j = 0; j < rows; ++j)
	{
		const float a = A[(long long)j * ld + i];
		const float cj = c ? c[j] : 1.0f;
		s += (double)cj * ((double)wd1 * fabs((double)a) + (double)wd2 * (double)a);
	}
	colterm[i] = (float)((double)lr * s);
}

cudaError_t launch_decay_colterm(const float* A, int rows, int n, long long ld, const float* c, float lr, float wd1, float wd2,
                                 float* colterm, cudaStream_t s)
{
	decay_colterm_kernel<<<(n + 127) / 128, 128, 0, s>>>(A, rows, n, ld, c, lr, wd1, wd2, colterm);
	return cudaGetLastError();
}

// W -= G * inv_mb (Node::applyDeltas, State/node.cpp:294-307: the window sum is always divided by
// the minibatch size); scalar biases; non-finite flag.
__global__ void __launch_bounds__(256) update_kernel(float* W, const float* G, long long count, float inv_mb,
                                                      float* bias, const float* gb, const float* bscale, int H, int* flags)
{
	int bad = 0;
	const long long stride = (long long)gridDim.x * blockDim.x;
	const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	const long long n4 = count / 4;
	float4* W4 = reinterpret_cast<float4*>(W);
	const float4* G4 = reinterpret_cast<const float4*>(G);
	for (long long i = i0; i < n4; i += stride)
	{
		float4 w = W4[i];
		const float4 g = G4[i];
		w.x -= g.x * inv_mb; w.y -= g.y * inv_mb; w.z -= g.z * inv_mb; w.w -= g.w * inv_mb;
		if (!(isfinite(w.x) && isfinite(w.y) && isfinite(w.z) && isfinite(w.w))) bad = 1;
		W4[i] = w;
	}
	for (long long i = n4 * 4 + i0; i < count; i += stride)
	{
		const float w = W[i] - G[i] * inv_mb;
		if (!isfinite(w)) bad = 1;
		W[i] = w;
	}
	if (blockIdx.x == 0 && threadIdx.x >= 1 && threadIdx.x <= H)
	{
		const float b = bias[threadIdx.x] - gb[threadIdx.x] * bscale[threadIdx.x];
		if (!isfinite(b)) bad = 1;
		bias[threadIdx.x] = b;
	}
	if (bad) atomicOr(flags, 1);
}

cudaError_t launch_update(float* W, const float* G, long long count, float inv_mb, float* bias, const float* gb,
                          const float* bscale, int H, int* flags, cudaStream_t s)
{
	long long blocks = (count / 4 + 255) / 256;
	if (blocks > 148 * 8) blocks = 148 * 8;
	if (blocks < 1) blocks = 1;
	update_kernel<<<(unsigned)blocks, 256, 0, s>>>(W, G, count, inv_mb, bias, gb, bscale, H, flags);
	return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) zero_ranges_kernel(const ZeroRanges z)
{
	for (int k = 0; k < 4; ++k)
		for (int i = threadIdx.x; i < z.n[k]; i += blockDim.x) z.p[k][i] = 0u;
}

cudaError_t launch_zero_ranges(const ZeroRanges& z, cudaStream_t s)
{
	zero_ranges_kernel<<<1, 256, 0, s>>>(z);
	return cudaGetLastError();
}

// One block per hidden layer; every thread adds a fixed set of the partial sums and the block adds the threads' sums in a
// fixed order, so the scalar biases are reproducible.
__global__ void __launch_bounds__(256) bias_finish_kernel(const BiasSums b, float* gb, int apply, float* bias, const float* bscale, int* flags)
{
	asm volatile("griddepcontrol.wait;" ::: "memory");
	const int l = blockIdx.x + 1;
	double t = 0.0;
	for (int i = threadIdx.x; i < b.count[l]; i += blockDim.x) t += b.part[l][i];
	t = warp_sum_d(t);
	__shared__ double sw[8];
	if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = t;
	__syncthreads();
	if (threadIdx.x != 0) return;
	t = 0.0;
	for (int w = 0; w < 8; ++w) t += sw[w];
	const float g = b.part[l] ? (float)(t * (double)b.lr[l]) : gb[l];  // (no partial sums: gb holds the whole one)
	gb[l] = g;
	if (!apply) return;
	const float v = bias[l] - g * bscale[l];
	if (!isfinite(v)) atomicOr(flags, 1);
	bias[l] = v;
}

cudaError_t launch_bias_finish(const BiasSums& b, int H, float* gb, int apply, float* bias, const float* bscale, int* flags, cudaStream_t s)
{
	ChainedLaunch c(dim3(H), 256, 0, true, s);
	return cudaLaunchKernelEx(&c.config, bias_finish_kernel, b, gb, apply, bias, bscale, flags);
}

}  // namespace glb
