// fp32 tile GEMM in a fixed order of operations: C[m][n] is ONE chain of fused multiply-adds over k = 0, 1, ..., K-1, whatever
// the tile.  (The reference's ReLU jumps from 0 to 0.046 at its threshold, so sums taken in another order would move single
// activations by that much; the order is part of what this kernel computes.)
//
// Bound: fp32 multiply-adds, 128 per clock and SM.  The products here are small and cannot be split along k without changing the
// order (1000 x 1000 is 128 tiles of 128 x 64 for 148 SMs), so one warp per scheduler has to come near that rate alone:
//   * two chains per instruction (fma.rn.f32x2: neighbouring rows; the column's value is repeated in both halves), which leaves
//     every second issue slot to loads and moves.  In registers alone 8 x 8 outputs per thread run at 119 multiply-adds per
//     clock this way;
//   * operands lie in shared memory with m or n running fastest, so that a 16-byte load brings two pairs, and are read one k ahead
//     of their use (8 x 8 outputs per thread, four warps on an SM: 93 per clock without that, 108 with it);
//   * lanes 2q and 2q + 1 read the same columns, lanes that differ by 16 or 1 other rows: a 16-byte shared-memory load costs two
//     clocks where neighbouring lanes share addresses, and four where eight in a row differ;
//   * four other warps fill a ring of FB_ST stages of 32 k: by cp.async where m or n is contiguous in memory, through registers
//     (whole 128-byte lines along k, stored transposed) or by 4-byte copies where k is.  Stages change hands through named barriers.
// Measured, one product after the other (the tiles of 64 x 64 and 32 x 64 with 8 x 4 scalar outputs per thread, copies by the computing
// warps, in brackets): forward 1000 x 1000 x 784 47 us (62), 1000 x 500 x 1000 35 (49), error propagation 1000 x 1000 x 500 34 (46),
// gradients 1000 x 784 x 1000 43 (76), 500 x 1000 x 1000 33 (60).  At K = 8176 a tile of 128 x 64 per SM runs at 82 multiply-adds per
// clock; the same loop without copies at 93, without barriers too at 99.
#include "common.cuh"
#include "internal.h"

namespace glb {

constexpr int FB_N = 64;  // columns of a tile

#ifdef FFMA_EPI
constexpr int FB_C = 128, FB_T = 256;      // threads that compute (4 warps), threads of a CTA
constexpr int FB_K = 32;                   // depth of a stage
constexpr int FB_ST = 4, FB_LAG = 2;       // stages of the ring, stages whose copies may be in flight when one is handed over
// A stage: A [32][8 TI], B [32][64], per-k factors.  Where k is contiguous in memory the columns of row k are permuted by
// x ^ 4 (k / 4): eight quads of k x 4 rows of a transposed store then lie in 32 banks.
__host__ __device__ constexpr int fb_stage(int ti) { return FB_K * (8 * ti + FB_N + 1); }
__host__ __device__ constexpr size_t fb_smem(int ti) { return (size_t)FB_ST * fb_stage(ti) * sizeof(float); }

// Named barriers 1..FB_ST: stage filled; FB_ST + 1..2 FB_ST: stage read.  Every use has FB_T participants.
__device__ __forceinline__ void bar_sync(int id) { asm volatile("barrier.cta.sync %0, %1;" ::"r"(id), "n"(FB_T) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id) { asm volatile("barrier.cta.arrive %0, %1;" ::"r"(id), "n"(FB_T) : "memory"); }

// A producer thread's part of filling one operand's R x 32 tile, which lies in shared memory as [k][R] (permuted, see above).
// Element (r, k) of the operand lies at src[r * sr + k * sk]; KC: k is contiguous (sk == 1), else r (sr == 1) or, with ANY, neither.
// vec: 16-byte accesses along the contiguous index are aligned.  What lies outside the operand is filled with zeros.
template <bool KC, int R, bool ANY>
struct FfmaFill
{
	static constexpr int NV = R * FB_K / 4 / 128, NS = R * FB_K / 128;
	const float* src;
	long long sr, sk;
	int left, K, t, k0;   // rows from this tile's first one to the operand's end; k of the stage that is issued next
	bool vec;
	float4 hold[KC ? NV : 1];
	__device__ FfmaFill(const float* s, long long sr_, long long sk_, int r0, int end, int K_, bool v)
	    : src(s + (long long)r0 * sr_), sr(sr_), sk(sk_), left(end - r0), K(K_), t(threadIdx.x - FB_C), k0(0), vec(v)
	{
	}
	// k contiguous: a warp takes 4 rows (4 (4 i + warp) + lane / 8), whole 128-byte lines of them; lane & 7 is the quad of k
	__device__ __forceinline__ int row(int i) const { return 16 * i + 4 * (t >> 5) + ((t & 31) >> 3); }
	__device__ __forceinline__ void load()
	{
		if (!KC || !vec) return;
		const int k = k0 + 4 * (t & 7);
#pragma unroll
		for (int i = 0; i < NV; ++i)
		{
			float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
			if (row(i) < left && k < K)
			{
				const float* p = src + (long long)row(i) * sr + k;
				if (k + 4 <= K) v = __ldg(reinterpret_cast<const float4*>(p));
				else
				{
					v.x = p[0];
					if (k + 1 < K) v.y = p[1];
					if (k + 2 < K) v.z = p[2];
				}
			}
			hold[KC ? i : 0] = v;
		}
	}
	__device__ __forceinline__ void store(float* dst, uint32_t dst_addr)
	{
		if (KC && vec)
		{
			const int q = t & 7;
#pragma unroll
			for (int i = 0; i < NV; ++i)
			{
				float* d = dst + 4 * q * R + (row(i) ^ (4 * q));
				const float4 v = hold[KC ? i : 0];
				d[0] = v.x;
				d[R] = v.y;
				d[2 * R] = v.z;
				d[3 * R] = v.w;
			}
		}
		else if (KC)
		{
			const int q = t & 7;
#pragma unroll
			for (int i = 0; i < NS / 4; ++i)
			{
				const float* p = src + (long long)row(i) * sr + k0 + 4 * q;
#pragma unroll
				for (int j = 0; j < 4; ++j)
				{
					const bool ok = row(i) < left && k0 + 4 * q + j < K;
					cp_async4(dst_addr + (uint32_t)((4 * q + j) * R + (row(i) ^ (4 * q))) * 4, ok ? p + j : src, ok);
				}
			}
		}
		else if (vec)
		{
#pragma unroll
			for (int i = 0; i < NV; ++i)
			{
				const int e = t + i * 128, k = e / (R / 4), r = (e % (R / 4)) * 4;
				const int n = k0 + k < K ? left - r : 0;
				cp_async16(dst_addr + (uint32_t)(k * R + r) * 4, n > 0 ? src + (long long)(k0 + k) * sk + r : src, n);
			}
		}
		else
		{
#pragma unroll
			for (int i = 0; i < NS; ++i)
			{
				const int e = t + i * 128, k = e / R, r = e % R;
				const bool ok = r < left && k0 + k < K;
				cp_async4(dst_addr + (uint32_t)(k * R + r) * 4, ok ? src + (long long)(k0 + k) * sk + (ANY ? r * sr : r) : src, ok);
			}
		}
		k0 += FB_K;
	}
};

// The sums of one compute thread: rows 32 h + 4 ty + {0..3}, h = 0..TI/4-1, in pairs; columns 4 tx + {0..3}.
template <int TI, bool AK, bool BK, bool SCALED>
__device__ __forceinline__ void ffma_sums(const float* sm, int K, int tx, int ty, f32x2 (&acc)[TI / 2][4])
{
	constexpr int R = 8 * TI, STAGE = fb_stage(TI), HALF = FB_K / 2;
	const int halves = (K + HALF - 1) / HALF, steps = (K + FB_K - 1) / FB_K;  // (the last stage's second half may lie beyond K)
	float4 a[2][TI / 4], b[2];
	float c[2] = {1.0f, 1.0f};
	// k: of the half stage at st, whose rows start at row h0 of the stage
	auto read = [&](int buf, const float* st, int h0, int k) {
		const int x = h0 + (k & ~3);
		const float* pa = st + k * R + (AK ? (4 * ty) ^ x : 4 * ty);
		const float* pb = st + FB_K * R - h0 * R + (h0 + k) * FB_N + (BK ? (4 * tx) ^ x : 4 * tx);
#pragma unroll
		for (int h = 0; h < TI / 4; ++h) a[buf][h] = *reinterpret_cast<const float4*>(pa + 32 * h);
		b[buf] = *reinterpret_cast<const float4*>(pb);
		if (SCALED) c[buf] = st[FB_K * (R + FB_N) - h0 * R + h0 + k];
	};
	bar_sync(1);
	read(0, sm, 0, 0);
	for (int u = 0; u < halves; ++u)
	{
		const int s = u >> 1, h0 = (u & 1) * HALF;
		const float* st = sm + (s % FB_ST) * STAGE + h0 * R;
#pragma unroll
		for (int k = 0; k < HALF; ++k)
		{
			const int buf = k & 1;
			if (k + 1 < HALF) read(buf ^ 1, st, h0, k + 1);
			else if (u + 1 < halves)
			{
				const int b1 = ((u + 1) >> 1) % FB_ST, h1 = HALF - h0;
				if (h1 == 0) bar_sync(1 + b1);
				read(buf ^ 1, sm + b1 * STAGE + h1 * R, h1, 0);
			}
			const f32x2 b2[4] = {pair2(b[buf].x, b[buf].x), pair2(b[buf].y, b[buf].y), pair2(b[buf].z, b[buf].z), pair2(b[buf].w, b[buf].w)};
#pragma unroll
			for (int h = 0; h < TI / 4; ++h)
			{
				f32x2 a0 = pair2(a[buf][h].x, a[buf][h].y), a1 = pair2(a[buf][h].z, a[buf][h].w);
				if (SCALED)
				{
					const f32x2 c2 = pair2(c[buf], c[buf]);
					a0 = mul2(a0, c2);
					a1 = mul2(a1, c2);
				}
#pragma unroll
				for (int j = 0; j < 4; ++j) acc[2 * h][j] = fma2(a0, b2[j], acc[2 * h][j]);
#pragma unroll
				for (int j = 0; j < 4; ++j) acc[2 * h + 1][j] = fma2(a1, b2[j], acc[2 * h + 1][j]);
			}
		}
		if (h0 != 0 && s + FB_ST < steps) bar_arrive(FB_ST + 1 + s % FB_ST);
	}
}

// Four neighbouring results of an activation: one switch for all of them, so that one case's code is fetched.
__device__ __forceinline__ void squash4(float (&v)[4], float bias, int act, float par)
{
#define GL_EACH(a)                                                     \
	case a:                                                            \
		for (int j = 0; j < 4; ++j) v[j] = squash_b(v[j] + bias, a, par); \
		break;
	switch (act)
	{
		GL_EACH(GL_ACT_TANH) GL_EACH(GL_ACT_TANHP) GL_EACH(GL_ACT_SIGMOID) GL_EACH(GL_ACT_SIGMOIDP) GL_EACH(GL_ACT_RELU)
		GL_EACH(GL_ACT_LEAKY) GL_EACH(GL_ACT_LINEAR) GL_EACH(GL_ACT_STEP) GL_EACH(GL_ACT_SOFTMAX)
	default: v[0] = v[1] = v[2] = v[3] = 0.0f; break;
	}
#undef GL_EACH
}

// TI x 4 outputs per thread, tiles of 8 TI x 64.
template <int EPI, bool AK, bool BK, int TI>
__global__ void __launch_bounds__(FB_T, TI >= 12 ? 1 : (TI == 8 ? 2 : 3)) gemm_ffma_kernel(const GemmArgs g, bool vec_a, bool vec_b)
{
	constexpr int TM = 8 * TI, STAGE = fb_stage(TI);
	constexpr int PO = FB_N + 4;  // the epilogue's pitch
	extern __shared__ __align__(16) float sm[];
	const int t = threadIdx.x;
	const int m0 = blockIdx.y * TM, n0 = blockIdx.x * FB_N;
	const int steps = (g.K + FB_K - 1) / FB_K;
	const bool scaled = EPI == EPI_GRAD && g.kscale != nullptr;
	if (t >= FB_C)
	{
		FfmaFill<AK, TM, EPI == EPI_NONE> fill_a(g.A, g.a_sm, g.a_sk, m0, g.M, g.K, vec_a);
		FfmaFill<BK, FB_N, EPI == EPI_NONE> fill_b(g.B, g.b_sn, g.b_sk, n0, g.N, g.K, vec_b);
		const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm);
		fill_a.load();
		fill_b.load();
		for (int s = 0; s < steps + FB_LAG; ++s)
		{
			const int b = s % FB_ST;
			if (s < steps)
			{
				if (s >= FB_ST) bar_sync(FB_ST + 1 + b);  // the stage that lay here has been read
				float* st = sm + b * STAGE;
				const uint32_t sa = base + (uint32_t)(b * STAGE) * 4;
				fill_a.store(st, sa);
				fill_b.store(st + FB_K * TM, sa + FB_K * TM * 4);
				if (scaled && t < FB_C + FB_K)
				{
					const int k = s * FB_K + t - FB_C;
					cp_async4(sa + (uint32_t)(FB_K * (TM + FB_N) + t - FB_C) * 4, k < g.K ? g.kscale + k : g.kscale, k < g.K);
				}
			}
			cp_async_commit();  // one group per step, empty ones included: the wait counts groups
			if (s + 1 < steps)
			{
				fill_a.load();
				fill_b.load();
			}
			cp_async_wait<FB_LAG>();
			if (s >= FB_LAG) bar_arrive(1 + (s - FB_LAG) % FB_ST);
		}
	}
	else
	{
		const int lane = t & 31;
		const int tx = ((lane >> 1) & 7) + 8 * ((t >> 5) & 1), ty = ((lane >> 3) & 2) + (lane & 1) + 4 * (t >> 6);
		f32x2 acc[TI / 2][4];
#pragma unroll
		for (int i = 0; i < TI / 2; ++i)
#pragma unroll
			for (int j = 0; j < 4; ++j) acc[i][j] = pair2(0.0f, 0.0f);
		// (the momentum weights' variant is a loop of its own: a branch per k would end the overlap of loads and multiply-adds)
		if (scaled) ffma_sums<TI, AK, BK, true>(sm, g.K, tx, ty, acc);
		else ffma_sums<TI, AK, BK, false>(sm, g.K, tx, ty, acc);
		// The results go through shared memory, so that the epilogue is one short loop over quads of a row and not 4 TI copies of the
		// activation's code (which took 20 us to fetch at TI = 16), and the copying warps share it.
		asm volatile("barrier.cta.sync %0, %1;" ::"n"(2 * FB_ST + 1), "n"(FB_C) : "memory");  // the stages are no longer read
#pragma unroll
		for (int i = 0; i < TI / 2; ++i)
		{
			const int r = 32 * (i >> 1) + 4 * ty + 2 * (i & 1);
			float4 lo, hi;
			unpair2(acc[i][0], lo.x, hi.x);
			unpair2(acc[i][1], lo.y, hi.y);
			unpair2(acc[i][2], lo.z, hi.z);
			unpair2(acc[i][3], lo.w, hi.w);
			*reinterpret_cast<float4*>(sm + r * PO + 4 * tx) = lo;
			*reinterpret_cast<float4*>(sm + (r + 1) * PO + 4 * tx) = hi;
		}
	}
	__syncthreads();
	const int q = 4 * (t & 15), n = n0 + q;
	const float bias = (EPI == EPI_FORWARD && g.bias_ptr) ? *g.bias_ptr : 0.0f;
	const bool update = EPI == EPI_GRAD && g.W != nullptr;
	float* const C = update ? g.W : g.C;
	const long long ldc = update ? g.N : g.ldc;
	const int width = g.N - n < 4 ? g.N - n : 4;  // (none: this thread's columns lie outside)
	const bool vec_c = width == 4 && (ldc & 3) == 0 && (((uintptr_t)C) & 15) == 0;
	const bool vec_s = vec_c && (((uintptr_t)g.C_scaled) & 15) == 0;
	const bool vec_x = width == 4 && (g.ld_aux & 3) == 0 && (((uintptr_t)g.aux) & 15) == 0;
	auto put = [&](float* p, const float (&v)[4], bool vec) {
		if (vec) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
		else
#pragma unroll
			for (int j = 0; j < 4; ++j)
				if (j < width) p[j] = v[j];
	};
	auto get = [&](const float* p, float (&v)[4], bool vec) {
		if (vec)
		{
			const float4 x = *reinterpret_cast<const float4*>(p);
			v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
		}
		else
#pragma unroll
			for (int j = 0; j < 4; ++j) v[j] = j < width ? p[j] : 0.0f;
	};
	float ct[4] = {0.0f, 0.0f, 0.0f, 0.0f};
	if (EPI == EPI_GRAD && g.colterm) get(g.colterm + n, ct, false);
	bool bad = false;
	double dsum = 0.0;
	// EB rows of a thread at a time: what they read from memory is on its way together
	constexpr int RS = FB_T / 16, EB = TI % 8 ? 2 : 4;
	static_assert(TM % (EB * RS) == 0, "whole passes over the tile's rows");
	const bool reads = EPI == EPI_ERRPROP || update;
	for (int r0 = t >> 4; r0 < TM && m0 + r0 < g.M && width > 0; r0 += EB * RS)
	{
		float v[EB][4], o[EB][4], rs[EB];
#pragma unroll
		for (int e = 0; e < EB; ++e)
		{
			const int r = r0 + e * RS, m = m0 + r;
			if (m >= g.M) continue;
			if (reads) get(EPI == EPI_ERRPROP ? g.aux + (long long)m * g.ld_aux + n : C + (long long)m * ldc + n, o[e], EPI == EPI_ERRPROP ? vec_x : vec_c);
			rs[e] = EPI == EPI_ERRPROP && g.C_scaled ? g.row_scale[m] : 0.0f;
			get(sm + r * PO + q, v[e], true);
		}
#pragma unroll
		for (int e = 0; e < EB; ++e)
		{
			const int m = m0 + r0 + e * RS;
			if (m >= g.M) continue;
			if (EPI == EPI_FORWARD) squash4(v[e], bias, g.act, g.par);
			else if (EPI == EPI_ERRPROP)
			{
#pragma unroll
				for (int j = 0; j < 4; ++j) v[e][j] = v[e][j] * act_der_b(o[e][j], g.act, g.par);
				if (g.dsum)
#pragma unroll
					for (int j = 0; j < 4; ++j) dsum += j < width ? (double)v[e][j] : 0.0;
			}
			else if (EPI == EPI_GRAD)
			{
#pragma unroll
				for (int j = 0; j < 4; ++j) v[e][j] = g.alpha * v[e][j] + ct[j];
				if (update)
				{
#pragma unroll
					for (int j = 0; j < 4; ++j)
					{
						v[e][j] = o[e][j] - v[e][j] * g.inv_mb;
						bad = bad || (j < width && !isfinite(v[e][j]));
					}
				}
			}
			put(C + (long long)m * ldc + n, v[e], vec_c);
			if (EPI == EPI_ERRPROP && g.C_scaled)
			{
#pragma unroll
				for (int j = 0; j < 4; ++j) o[e][j] = v[e][j] * rs[e];
				put(g.C_scaled + (long long)m * g.ldc + n, o[e], vec_s);
			}
		}
	}
	if (bad) atomicOr(g.bad_flag, 1);
	if (EPI == EPI_ERRPROP && g.dsum)
	{
		// the tile's sum, in a fixed order
		__shared__ double part[FB_T / 32];
		dsum = warp_sum_d(dsum);
		if ((t & 31) == 0) part[t >> 5] = dsum;
		__syncthreads();
		if (t == 0)
		{
			double x = 0.0;
			for (int w = 0; w < FB_T / 32; ++w) x += part[w];
			g.dsum[blockIdx.y * gridDim.x + blockIdx.x] = x;
		}
	}
}

#else
// Which tile.  An SM's time is what its tiles hold of outputs over the rate that TI x 4 outputs per thread reach with that many
// CTAs side by side (multiply-adds per clock and SM, measured at K = 8176), plus each tile's ends (600 clocks per TI, measured at
// K = 17); the tile with the smallest time wins, the larger one of equals.
static long long ffma_time(int M, int N, int K, int ti)  // clocks
{
	const long long tiles = (long long)((M + 8 * ti - 1) / (8 * ti)) * ((N + FB_N - 1) / FB_N), per_sm = (tiles + 147) / 148;
	const int rate = ti == 16 ? 82 : (ti == 12 ? 84 : (ti == 8 ? (per_sm == 1 ? 74 : 76) : (per_sm == 1 ? 40 : 60)));
	return per_sm * ti * (8ll * FB_N * K / rate + (ti == 4 ? 500 : 600));
}
static int ffma_tile(int M, int N, int K)
{
	int best = 16;
	for (int ti = 12; ti >= 4; ti -= 4)
		if (ffma_time(M, N, K, ti) < ffma_time(M, N, K, best)) best = ti;
	while (best < 16 && (M + 8 * best - 1) / (8 * best) > 65535) best += 4;
	return best;
}
int ffma_dsum_parts(int M, int N, int K)
{
	const int ti = ffma_tile(M, N, K);
	return (M + 8 * ti - 1) / (8 * ti) * ((N + FB_N - 1) / FB_N);
}
int ffma_tile_rows(int M, int N, int K) { return 8 * ffma_tile(M, N, K); }
long long ffma_tile_clocks(int M, int N, int K) { return ffma_time(M, N, K, ffma_tile(M, N, K)); }

#endif  // FFMA_EPI

// This file is compiled once per kind of product (FFMA_EPI), and once more for the choice of a tile: a process loads the code of the products
// that it runs (first call of a process, 1000 rows of 301-501-303-40: 16.3 ms with one object, 14.4 ms now).
#ifdef FFMA_EPI
template <int EPI, bool AK, bool BK, int TI>
static cudaError_t launch_tile(const GemmArgs& g, bool va, bool vb, cudaStream_t s)
{
	const cudaError_t e = cudaFuncSetAttribute(gemm_ffma_kernel<EPI, AK, BK, TI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fb_smem(TI));
	if (e != cudaSuccess) return e;
	const dim3 grid((g.N + FB_N - 1) / FB_N, (g.M + 8 * TI - 1) / (8 * TI));
	// (not an early launch: CTAs that arrive while the kernel in front still holds most SMs pile up on the others)
	gemm_ffma_kernel<EPI, AK, BK, TI><<<grid, FB_T, fb_smem(TI), s>>>(g, va, vb);
	return cudaGetLastError();
}

template <int EPI, bool AK, bool BK>
static cudaError_t launch_layout(const GemmArgs& g, int tile, cudaStream_t s)
{
	// 16-byte copies of an operand where each of its rows starts on a 16-byte boundary
	auto vec = [](const float* p, bool kc, long long sr, long long sk) { return (kc ? sk : sr) == 1 && ((kc ? sr : sk) & 3) == 0 && (((uintptr_t)p) & 15) == 0; };
	const bool va = vec(g.A, AK, g.a_sm, g.a_sk), vb = vec(g.B, BK, g.b_sn, g.b_sk);
	switch (tile)
	{
	case 4: return launch_tile<EPI, AK, BK, 4>(g, va, vb, s);
	case 8: return launch_tile<EPI, AK, BK, 8>(g, va, vb, s);
	case 12: return launch_tile<EPI, AK, BK, 12>(g, va, vb, s);
	default: return launch_tile<EPI, AK, BK, 16>(g, va, vb, s);
	}
}

static_assert(EPI_NONE == 0 && EPI_FORWARD == 1 && EPI_ERRPROP == 2 && EPI_GRAD == 3, "FFMA_EPI below");
cudaError_t GL_CAT(launch_ffma_tiles_, FFMA_EPI)(const GemmArgs& g, int tile, cudaStream_t s)
{
#if FFMA_EPI == 1
	return launch_layout<EPI_FORWARD, true, true>(g, tile, s);
#elif FFMA_EPI == 2
	return launch_layout<EPI_ERRPROP, true, false>(g, tile, s);
#elif FFMA_EPI == 3
	return launch_layout<EPI_GRAD, false, false>(g, tile, s);
#else
	// (a matrix of one row or column is contiguous both ways: along k, then)
	const bool ak = g.a_sk == 1, bk = g.b_sk == 1;
	if (ak && bk) return launch_layout<EPI_NONE, true, true>(g, tile, s);
	if (ak) return launch_layout<EPI_NONE, true, false>(g, tile, s);
	if (bk) return launch_layout<EPI_NONE, false, true>(g, tile, s);
	return launch_layout<EPI_NONE, false, false>(g, tile, s);
#endif
}
#else
cudaError_t launch_ffma_tiles_0(const GemmArgs& g, int tile, cudaStream_t s);
cudaError_t launch_ffma_tiles_1(const GemmArgs& g, int tile, cudaStream_t s);
cudaError_t launch_ffma_tiles_2(const GemmArgs& g, int tile, cudaStream_t s);
cudaError_t launch_ffma_tiles_3(const GemmArgs& g, int tile, cudaStream_t s);

cudaError_t launch_ffma_tiles(const GemmArgs& g, cudaStream_t s)
{
	const int tile = ffma_tile(g.M, g.N, g.K);
	switch (g.epi)
	{
	case EPI_FORWARD: return launch_ffma_tiles_1(g, tile, s);
	case EPI_ERRPROP: return launch_ffma_tiles_2(g, tile, s);
	case EPI_GRAD: return launch_ffma_tiles_3(g, tile, s);
	default: return launch_ffma_tiles_0(g, tile, s);
	}
}
#endif  // FFMA_EPI

}  // namespace glb
