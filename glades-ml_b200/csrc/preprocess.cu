// Input standardisation on the device: the step in front of the training loop,
// NumberInput::standardizeInputTable (DataObjects/NumberInput.cpp:43-285) with the one-hot vectors of
// OHE::operator[] (GMath/OHE.cpp:159-198), on a raw table that already lies in HBM as a row-major
// [rows][cols] fp32 matrix (a categorical column holds each cell's category index, in order of first
// appearance -- the strings themselves stay on the host).
//
// Everything is bound by HBM: rows * cols * 4 bytes read twice (extrema, then transform), rows * (nx + ny) * 4 bytes
// written once.  The launches follow one another without the host in between: the layout of the results depends on the
// extrema (a min-max column of range 0 moves to the input matrix), so a small kernel makes it on the device,
// and the transform writes nothing if it is not the one that the caller has room for.
//
// Pass 1, column statistics.  Minimum and maximum do not depend on the order of the rows, so they are reduced in
// parallel.  The reference starts the running minimum and maximum from the first cell only for raw column 0 and from
// 0.0 for every other column (NumberInput.cpp:105-109): columns other than 0 therefore start their reduction at 0.
// The mean and the standard deviation (z-score mode only) are sequential fp32 sums in row order in the reference
// (:118-121,236-249): one chain of rounded additions per column, whose length times four clocks is the floor; one
// warp runs the chains of 32 columns from shared memory while the other warps of its block keep the rows coming.
// Pass 2, transform, from the results' side: separately rounded fp32 operations in the reference's order,
// ((x - min) / range) * 0.98 + 0.01 (any categorical column in the table) or (x - min) / range, or (x - mean) / stdev,
// or the 0.99 / 0.01 one-hot group of a categorical cell.
#include <string.h>

#include "copy_ring.h"
#include "internal.h"
#include "tc_device.cuh"

namespace glb {
namespace {

__device__ __forceinline__ int float_order(float f)
{
	// monotone map float -> int (so that integer atomicMin / atomicMax order floats)
	const int i = __float_as_int(f);
	return i >= 0 ? i : i ^ 0x7FFFFFFF;
}
__device__ __forceinline__ float order_float(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7FFFFFFF); }

// The reference starts the running minimum and maximum from the first cell only for raw column 0 and from 0.0 for every other
// column (NumberInput.cpp:105-109).  A neutral start gives column 0 the same extrema unless its first cell is not a number: no
// cell then compares, and both stay that (minmax_kernel sees to it).  No zero replaces the 0.0 that the other columns start
// from, so a negative zero counts as a positive one there.  (Column 0 takes the sign of its first zero, here that of a negative
// one wherever there is any; the difference is the sign of results that are zero.)
__host__ __device__ __forceinline__ int start_of(int word)
{
	if (word == 0) return 0x7FFFFFFF;
	return word == 1 ? (int)0x80000000 : 0;
}

// One column of a result, and what it needs.
enum OutMode
{
	OC_ONEHOT,
	OC_COPY,
	OC_SCALE,
	OC_SCALE_SAFE  // the divisor lies outside the range of quotient()
};
struct OutColumn
{
	int src, mode, k;  // raw column; k: category of a one-hot column
	float a, d, r;     // (x - a) / d, r = 1 / d
};

// The accumulators live in `acc` between calls, at their start values; the last kernel moves them out and puts these back.
struct TableJob
{
	int cols, flag, want_nx, want_ny;
	const int* host_spec;  // pinned host memory: kind | classes | to_output, [cols] each
	int* spec;         // device: the same, fetched by the first kernel under its work
	int* acc;          // [cols][4]: minimum image, maximum image, mean, deviation
	OutColumn* table;  // the results' columns: those of X followed by those of Y
	int* shape;        // device: {nx, ny, 1 if that is what the caller has room for}
	int* host;         // pinned host memory: statistics [cols][4], then nx, ny
};

// The layout of the results: columns keep their raw order inside each destination; a numeric column whose min-max range is
// 0 is copied unscaled and lands in the input matrix whatever its output mark (NumberInput.cpp:166-171).
// Executed by one whole block; `at` is shared memory for 2 * cols words.
__device__ void make_layout(const TableJob& j, int* at)
{
	const int cols = j.cols;
	__shared__ int total[2];
	for (int c = threadIdx.x; c < cols; c += blockDim.x)
	{
		const int mn = j.acc[4 * c], mx = j.acc[4 * c + 1];
		const int kind = j.spec[c], classes = j.spec[cols + c], output = j.spec[2 * cols + c];
		const bool flat = kind == 0 && j.flag == 0 && __fsub_rn(order_float(mx), order_float(mn)) == 0.0f;
		at[c] = (output && !flat) ? 1 << 30 : 0;
		at[cols + c] = kind == 1 ? classes : -1;
	}
	__syncthreads();
	if (threadIdx.x == 0)
	{
		int n[2] = {0, 0};
		for (int c = 0; c < cols; ++c)
		{
			const int y = at[c] >> 30;
			at[c] |= n[y];
			n[y] += at[cols + c] < 0 ? 1 : at[cols + c];
		}
		for (int k = 0; k < 2; ++k) total[k] = j.shape[k] = n[k];
		j.shape[2] = n[0] == j.want_nx && n[1] == j.want_ny;
	}
	__syncthreads();
	for (int c = threadIdx.x; c < cols; c += blockDim.x)
	{
		OutColumn* o = j.table + ((at[c] >> 30) ? total[0] : 0) + (at[c] & ~(1 << 30));
		OutColumn e;
		memset(&e, 0, sizeof e);
		e.src = c;
		if (at[cols + c] >= 0)
		{
			e.mode = OC_ONEHOT;
			for (int k = 0; k < at[cols + c]; ++k)
			{
				e.k = k;
				o[k] = e;
			}
		}
		else
		{
			const float mn = order_float(j.acc[4 * c]), range = __fsub_rn(order_float(j.acc[4 * c + 1]), mn);
			e.a = j.flag == 0 ? mn : __int_as_float(j.acc[4 * c + 2]);
			e.d = j.flag == 0 ? range : __int_as_float(j.acc[4 * c + 3]);
			e.r = __fdiv_rn(1.0f, e.d);
			const float m = fabsf(e.d);
			e.mode = (j.flag == 0 && e.d == 0.0f) ? OC_COPY : ((m >= 1e-18f && m <= 1e18f) ? OC_SCALE : OC_SCALE_SAFE);
			*o = e;
		}
	}
}

__global__ void __launch_bounds__(256) layout_kernel(const TableJob job)
{
	extern __shared__ int at[];
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
	asm volatile("griddepcontrol.wait;" ::: "memory");
	make_layout(job, at);
}

// The grid's threads stride over the row-major cells, 16 bytes at a time where V (the table is 16-byte
// aligned); the stride is a multiple of the column count, so a thread stays on its columns and keeps their extrema in
// registers, and consecutive threads read consecutive addresses.  A block merges its threads' extrema in shared memory and
// issues one global atomic per column it touched.
// Measured, 1 Mi x 33: one cell per load 42 us (3.3 TB/s); four cells per load, four loads in flight: 28 us.
template <bool V>
__global__ void __launch_bounds__(256) minmax_kernel(const float* __restrict__ raw, long long rows, const TableJob job)
{
	const int cols = job.cols;
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
	int* stats = job.acc;
	constexpr int W = V ? 4 : 1;
	extern __shared__ int sext[];  // [2][cols]: images of the block's minimum and maximum per column
	for (int c = threadIdx.x; c < cols; c += blockDim.x)
	{
		sext[c] = 0x7FFFFFFF;
		sext[cols + c] = (int)0x80000000;
	}
	if (blockIdx.x == 0)
		for (int k = threadIdx.x; k < 3 * cols; k += blockDim.x) job.spec[k] = job.host_spec[k];
	if (blockIdx.x == 0 && threadIdx.x == 0)
	{
		const float first = raw[0];
		if (first != first)  // (see start_of)
		{
			atomicMin(stats, (int)0x80000000);  // both decode to a NaN
			atomicMax(stats + 1, 0x7FFFFFFF);
		}
	}
	__syncthreads();
	const long long total = rows * (long long)cols;
	const long long stride = (long long)gridDim.x * blockDim.x * W;
	const long long start = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * W;
	float mn[W], mx[W];
#pragma unroll
	for (int k = 0; k < W; ++k)
	{
		mn[k] = __int_as_float(0x7F800000);
		mx[k] = __int_as_float(0xFF800000);
	}
	auto take = [&](const float (&v)[W]) {
#pragma unroll
		for (int k = 0; k < W; ++k)
		{
			mn[k] = fminf(mn[k], v[k]);
			mx[k] = fmaxf(mx[k], v[k]);
		}
	};
	auto load = [&](long long i, float (&v)[W]) {
		if (V) *reinterpret_cast<float4*>(v) = __ldg(reinterpret_cast<const float4*>(raw + i));
		else v[0] = raw[i];
	};
	long long i = start;
	for (; i + 3 * stride + W <= total; i += 4 * stride)
	{
		float a[W], b[W], c[W], d[W];
		load(i, a);
		load(i + stride, b);
		load(i + 2 * stride, c);
		load(i + 3 * stride, d);
		take(a);
		take(b);
		take(c);
		take(d);
	}
	for (; i + W <= total; i += stride)
	{
		float a[W];
		load(i, a);
		take(a);
	}
	int c = (int)(start % cols);
	const bool tail = V && i < total;  // up to three cells at the very end of the table
#pragma unroll
	for (int k = 0; k < W; ++k)
	{
		if (tail && i + k < total)
		{
			mn[k] = fminf(mn[k], raw[i + k]);
			mx[k] = fmaxf(mx[k], raw[i + k]);
		}
		if (start + k < total)
		{
			const float zero = c == 0 ? -0.0f : 0.0f;  // (see start_of; adding -0.0 changes nothing)
			atomicMin(sext + c, float_order(mn[k] + zero));
			atomicMax(sext + cols + c, float_order(mx[k] + zero));
		}
		if (++c == cols) c = 0;
	}
	__syncthreads();
	for (int k = threadIdx.x; k < cols; k += blockDim.x)
	{
		if (sext[k] != 0x7FFFFFFF) atomicMin(stats + 4 * k, sext[k]);
		if (sext[cols + k] != (int)0x80000000) atomicMax(stats + 4 * k + 1, sext[cols + k]);
	}
}

// Sequential fp32 sums in row order, as the reference accumulates them: mean, then standard deviation.
// One block per 32 columns.  Lane c of warp 0 adds column c's cells one after the other from a ring of tiles in shared memory,
// the next 16 loaded under the additions of the current ones; the warps of the other three schedulers keep the tiles coming
// by asynchronous copies.  The tiles' pitch is a constant, so a row is one load with an immediate offset and one addition
// (four instructions in the second pass), which fit in the four clocks of the dependent addition.  100,003 x 24: 0.80 ms,
// against 4.1 ms for one thread per column reading global memory.
constexpr int MS_ROWS = 256, MS_RING = 4, MS_LOADERS = 6;
constexpr size_t MS_SMEM = ((size_t)MS_RING * MS_ROWS + 32) * 32 * sizeof(float);  // (the loads ahead may run past the last tile)

template <int PASS>
__device__ __forceinline__ float ms_chain(float acc, const float* s, int n, float mean)
{
	constexpr int pitch = 32;
	auto add = [&](float x) {
		if (PASS == 0) acc = __fadd_rn(acc, x);
		else
		{
			const float d = __fsub_rn(x, mean);
			acc = __fadd_rn(acc, __fmul_rn(d, d));
		}
	};
	int r = 0;
	if (n >= 32)
	{
		float v[16], w[16];
#pragma unroll
		for (int k = 0; k < 16; ++k) v[k] = s[k * pitch];
#pragma unroll 1
		for (; r + 32 <= n; r += 32)
		{
			const float* q = s + (r + 16) * pitch;
#pragma unroll
			for (int k = 0; k < 16; ++k) w[k] = q[k * pitch];
#pragma unroll
			for (int k = 0; k < 16; ++k) add(v[k]);
			q += 16 * pitch;
#pragma unroll
			for (int k = 0; k < 16; ++k) v[k] = q[k * pitch];
#pragma unroll
			for (int k = 0; k < 16; ++k) add(w[k]);
		}
	}
	for (; r < n; ++r) add(s[r * pitch]);
	return acc;
}

__global__ void __launch_bounds__(256) mean_stdev_kernel(const float* __restrict__ raw, long long rows, const TableJob job)
{
	const int cols = job.cols;
	extern __shared__ __align__(16) float ring[];  // [MS_RING][MS_ROWS][32]
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int c0 = blockIdx.x * 32, c = c0 + lane;
	const bool mine = c < cols && job.spec[c] == 0;
	constexpr int tile_rows = MS_ROWS;
	const uint32_t ring_addr = (uint32_t)__cvta_generic_to_shared(ring);
	const long long tiles = (rows + tile_rows - 1) / tile_rows;
	const int loader = (warp & 3) ? warp - 1 - (warp >> 2) : -1;  // 0..5; the chain's scheduler has none
	float mean = 0.0f, sd = 0.0f;
	for (int pass = 0; pass < 2; ++pass)
	{
		auto fill = [&](long long tile) {
			if (tile < tiles && loader >= 0)
			{
				const long long r0 = tile * tile_rows;
				const int n = (int)(rows - r0 < tile_rows ? rows - r0 : tile_rows);
				const uint32_t dst = ring_addr + (uint32_t)((tile % MS_RING) * MS_ROWS * 32 + loader * 32 + lane) * 4;
				const float* src = raw + (r0 + loader) * cols + c;
				if (mine)
#pragma unroll 4
					for (int r = loader; r < n; r += MS_LOADERS, src += MS_LOADERS * (long long)cols) cp_async4(dst + (uint32_t)(r - loader) * 128, src, true);
			}
			cp_async_commit();
		};
		float acc = 0.0f;
		for (int k = 0; k < MS_RING - 1; ++k) fill(k);
		for (long long tile = 0; tile < tiles; ++tile)
		{
			cp_async_wait<MS_RING - 2>();
			__syncthreads();  // the tile has landed, and the one before it has been consumed
			fill(tile + MS_RING - 1);
			if (warp == 0 && mine)
			{
				const float* s = ring + (tile % MS_RING) * (MS_ROWS * 32) + lane;
				const int n = (int)(rows - tile * tile_rows < tile_rows ? rows - tile * tile_rows : tile_rows);
				acc = pass == 0 ? ms_chain<0>(acc, s, n, 0.0f) : ms_chain<1>(acc, s, n, mean);
			}
		}
		cp_async_wait<0>();
		__syncthreads();
		if (pass == 0) mean = __fdiv_rn(acc, (float)(unsigned int)rows);
		else sd = __fsqrt_rn(__fdiv_rn(acc, (float)((unsigned int)rows - 1u)));
	}
	if (warp == 0 && mine)
	{
		job.acc[4 * c + 2] = __float_as_int(mean);
		job.acc[4 * c + 3] = __float_as_int(sd);
	}
}

// x / d for one d and many x: y = RN(1/d) once, then two corrections of q = x y by the exact remainder (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990: with y the correctly
// rounded reciprocal, RN(q + y (x - q d)) is the correctly rounded quotient once q is within an ulp of it, which the first
// correction makes sure of).  Holds while no remainder underflows: d and x between 1e-18 and 1e18 in magnitude; everything
// else, zero among it, takes the division.
__device__ __forceinline__ float quotient(float x, float d, float y)
{
	const float ax = fabsf(x);
	if (!(ax >= 1e-18f && ax <= 1e18f)) return __fdiv_rn(x, d);
	float q = __fmul_rn(x, y);
	q = __fmaf_rn(__fmaf_rn(-q, d, x), y, q);
	return __fmaf_rn(__fmaf_rn(-q, d, x), y, q);
}

// The statistics and widths to the host, and the accumulators back at their start values.
__device__ __forceinline__ void hand_over(const TableJob& job, int nx, int ny)
{
	const int cols = job.cols;
	for (int k = threadIdx.x; k < 4 * cols; k += blockDim.x)
	{
		job.host[k] = job.acc[k];
		job.acc[k] = start_of(k);
	}
	if (threadIdx.x < 2) job.host[4 * cols + threadIdx.x] = threadIdx.x ? ny : nx;
}

// A cell of the results.
__device__ __forceinline__ float scaled_cell(float v, const OutColumn& o, bool slow, int squeeze)
{
	const float x = __fsub_rn(v, o.a);
	const float q = slow ? __fdiv_rn(x, o.d) : quotient(x, o.d, o.r);
	return squeeze ? __fadd_rn(__fmul_rn(q, 0.98f), 0.01f) : q;
}

// (The kernel behind this one takes the tables that it can; this one the others: bases off 16-byte boundaries, very wide tables.)
// A thread stays on one column of the results, so its constants are in registers, and takes every (256 / width)-th row of the
// block's piece of the table: neighbouring threads read neighbouring cells of a row and write neighbouring ones.  TX_ROWS
// cells are loaded before the first is used.  The last pieces come first: they are what the pass over the extrema has left in
// L2; the results are stored past it.  Block 0 also hands the statistics to the host, under the others' work.
// Bound by the loads in flight: six blocks per SM (40 registers) with 8 loads a thread 76 us for 1 Mi x 33 behind the pass over the
// extrema, four blocks 80 us, 4 loads 88 us; a tile of rows in shared memory 81 us, threads on raw columns that write wherever
// their column went 100 us.  A copy without arithmetic takes 72 us in the same place.
constexpr int TX_ROWS = 8;
__global__ void __launch_bounds__(256, 6) transform_kernel(const float* __restrict__ raw, long long rows, const TableJob job, int squeeze,
                                                         float* __restrict__ X, float* __restrict__ Y)
{
	asm volatile("griddepcontrol.wait;" ::: "memory");
	const int cols = job.cols, nx = job.shape[0], ny = job.shape[1], width = nx + ny;
	if (blockIdx.x == 0) hand_over(job, nx, ny);
	if (!job.shape[2]) return;
	const int wide = width < 256 ? width : 256;       // columns taken at a time
	const int rstep = max(1, (int)blockDim.x / wide);  // rows taken at a time
	const int jt = threadIdx.x % wide, rt = threadIdx.x / wide;
	if (rt >= rstep) return;
	const long long piece = (long long)rstep * TX_ROWS, pieces = (rows + piece - 1) / piece;
	for (int j = jt; j < width; j += wide)
	{
		const OutColumn o = job.table[j];
		const int pitch = j < nx ? nx : ny;
		float* out = j < nx ? X + j : Y + (j - nx);
		const bool slow = o.mode == OC_SCALE_SAFE;
		for (long long p = pieces - 1 - blockIdx.x; p >= 0; p -= gridDim.x)
		{
			const long long r0 = p * piece + rt;
			const float* q = raw + r0 * cols + o.src;
			float* w = out + r0 * pitch;
			const long long left = (rows - r0 + rstep - 1) / rstep;
			const int n = left < TX_ROWS ? (int)left : TX_ROWS;
			float v[TX_ROWS];
#pragma unroll
			for (int k = 0; k < TX_ROWS; ++k) v[k] = k < n ? __ldg(q + (long long)k * rstep * cols) : 0.0f;
			// (columns of several kinds meet in a warp: only the arithmetic diverges, the loads and stores are common)
			if (o.mode == OC_ONEHOT)
			{
#pragma unroll
				for (int k = 0; k < TX_ROWS; ++k) v[k] = (int)v[k] == o.k ? 0.99f : 0.01f;
			}
			else if (o.mode != OC_COPY)
			{
#pragma unroll
				for (int k = 0; k < TX_ROWS; ++k) v[k] = scaled_cell(v[k], o, slow, squeeze);
			}
#pragma unroll
			for (int k = 0; k < TX_ROWS; ++k)
				if (k < n) __stcs(w + (long long)k * rstep * pitch, v[k]);
		}
	}
}

// The same from tiles of whole rows: rows of the table, of X and of Y are contiguous, so a tile of them is one bulk copy each way, and what
// is left for the threads is a load from shared memory, the arithmetic and a store to shared memory.  Two tiles on their way in and
// up to two on their way out per block, three blocks per SM; one thread asks for the copies.  The last tiles come first: they are what
// the pass over the extrema has left in L2; the results are marked to leave it first.  rows_tile: a multiple of 4, so that every tile of
// every width starts on a 16-byte boundary; the rows behind the last whole tile go cell by cell.
// 1 Mi x 33, behind the pass over the extrema: 53 us, 64 % of the SMs' issue and 0.80 of the copy bandwidth; transform_kernel 78 us.
__global__ void __launch_bounds__(256, 3) transform_tiles_kernel(const float* __restrict__ raw, long long rows, const TableJob job, int squeeze, int rows_tile,
                                                                 float* __restrict__ X, float* __restrict__ Y)
{
	extern __shared__ __align__(128) uint8_t tiles_sm[];
	__shared__ uint64_t full[2];
	__shared__ int abort_flag;
	const int t = threadIdx.x, cols = job.cols;
	if (t == 0)
	{
		tc::mbar_init(tc::smem_u32(&full[0]), 1);
		tc::mbar_init(tc::smem_u32(&full[1]), 1);
		abort_flag = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	asm volatile("griddepcontrol.wait;" ::: "memory");
	__syncthreads();
	const int nx = job.shape[0], ny = job.shape[1], width = nx + ny;
	if (blockIdx.x == 0) hand_over(job, nx, ny);
	if (!job.shape[2]) return;
	const uint32_t in_bytes = (uint32_t)(rows_tile * cols) * 4, x_bytes = (uint32_t)(rows_tile * nx) * 4, y_bytes = (uint32_t)(rows_tile * ny) * 4;
	const uint32_t in_pitch = (in_bytes + 127) & ~127u, x_pitch = (x_bytes + 127) & ~127u, out_pitch = x_pitch + ((y_bytes + 127) & ~127u);
	uint8_t* const out_sm = tiles_sm + 2 * in_pitch;
	const long long tiles = rows / rows_tile;
	const int mine = tiles > blockIdx.x ? (int)((tiles - 1 - blockIdx.x) / gridDim.x + 1) : 0;
	auto tile_at = [&](int k) { return tiles - 1 - blockIdx.x - (long long)k * gridDim.x; };
	uint64_t first_out;  // results leave L2 first
	asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(first_out));
	CopyRing<2> ring;
	auto fetch = [&](int k, unsigned stage) {
		const uint32_t bar = tc::smem_u32(&full[stage]);
		tc::mbar_expect_tx(bar, in_bytes);
		asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(tc::smem_u32(tiles_sm + stage * in_pitch)),
		             "l"(raw + tile_at(k) * rows_tile * cols), "r"(in_bytes), "r"(bar)
		             : "memory");
	};
	auto store = [&](float* to, const uint8_t* from, uint32_t bytes) {
		asm volatile("cp.async.bulk.global.shared::cta.bulk_group.L2::cache_hint [%0], [%1], %2, %3;" ::"l"(to), "r"(tc::smem_u32(from)), "r"(bytes), "l"(first_out)
		             : "memory");
	};
	ring.begin(mine);
	if (t == 0) ring.start(2, fetch);
	const int wide = width < 256 ? width : 256, rstep = 256 / wide;  // columns and rows taken at a time
	const int jt = t % wide, rt = t / wide;
	OutColumn o = job.table[jt < width ? jt : 0];
	for (int k = 0; k < mine; ++k)
	{
		if (t == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");  // the results of the tile before the last have been read
		ring.await(
		    k, 2, [&](unsigned stage, unsigned parity) { return tc::mbar_wait(tc::smem_u32(&full[stage]), parity, &abort_flag, job.host + 4 * cols + 3, 1); },
		    [&](unsigned lo, unsigned hi) { tc::mbar_drain<2>(tc::smem_u32(full), lo, hi); });
		__syncthreads();
		const float* in = reinterpret_cast<const float*>(tiles_sm + (k & 1) * in_pitch);
		uint8_t* const ob = out_sm + (k & 1) * out_pitch;
		if (rt < rstep)
			for (int j = jt; j < width; j += wide)
			{
				if (width > wide) o = job.table[j];
				const bool slow = o.mode == OC_SCALE_SAFE;
				const int pitch = j < nx ? nx : ny;
				const float* q = in + rt * cols + o.src;
				float* w = reinterpret_cast<float*>(ob + (j < nx ? 0 : x_pitch)) + rt * pitch + (j < nx ? j : j - nx);
				const int dq = rstep * cols, dw = rstep * pitch;
				int left = (rows_tile - rt + rstep - 1) / rstep;
				// (columns of several kinds meet in a warp: only the arithmetic diverges, the loads and stores are common)
				for (; left > 0; left -= 4, q += 4 * dq, w += 4 * dw)
				{
					float v[4];
#pragma unroll
					for (int r = 0; r < 4; ++r) v[r] = r < left ? q[r * dq] : 0.0f;
					if (o.mode == OC_ONEHOT)
					{
#pragma unroll
						for (int r = 0; r < 4; ++r) v[r] = (int)v[r] == o.k ? 0.99f : 0.01f;
					}
					else if (o.mode != OC_COPY)
					{
#pragma unroll
						for (int r = 0; r < 4; ++r) v[r] = scaled_cell(v[r], o, slow, squeeze);
					}
#pragma unroll
					for (int r = 0; r < 4; ++r)
						if (r < left) w[r * dw] = v[r];
				}
			}
		asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // (the stores read through the asynchronous proxy)
		__syncthreads();
		if (t == 0)
		{
			const long long r0 = tile_at(k) * rows_tile;
			if (nx) store(X + r0 * nx, ob, x_bytes);
			if (ny) store(Y + r0 * ny, ob + x_pitch, y_bytes);
			asm volatile("cp.async.bulk.commit_group;" ::: "memory");
			ring.refill(k, 2, fetch);
		}
	}
	// the rows behind the last whole tile
	if (blockIdx.x == gridDim.x - 1 && rt < rstep)
		for (int j = jt; j < width; j += wide)
		{
			if (width > wide) o = job.table[j];
			for (long long r = tiles * rows_tile + rt; r < rows; r += rstep)
			{
				const float v = raw[r * cols + o.src];
				float* w = j < nx ? X + r * nx + j : Y + r * ny + (j - nx);
				*w = o.mode == OC_ONEHOT ? ((int)v == o.k ? 0.99f : 0.01f) : (o.mode == OC_COPY ? v : scaled_cell(v, o, o.mode == OC_SCALE_SAFE, squeeze));
			}
		}
	if (t == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // (shared memory is read until then)
}

}  // namespace

size_t standardize_acc_words(int cols) { return (size_t)cols * 7; }
void standardize_acc_start(int* acc, int cols)
{
	for (int k = 0; k < 7 * cols; ++k) acc[k] = start_of(k);
}
size_t standardize_table_bytes(int width) { return (size_t)width * sizeof(OutColumn); }

cudaError_t launch_standardize(const StandardizeArgs& a, cudaStream_t s)
{
	if (a.cols > 6000) return cudaErrorInvalidValue;  // a block's extrema live in shared memory
	TableJob job;
	job.cols = a.cols;
	job.flag = a.flag;
	job.want_nx = a.write ? a.want_nx : -1;
	job.want_ny = a.write ? a.want_ny : -1;
	job.host_spec = a.spec;
	job.spec = a.acc + (size_t)4 * a.cols;
	job.acc = a.acc;
	job.table = static_cast<OutColumn*>(a.table);
	job.shape = a.shape;
	job.host = a.host;
	const long long total = a.rows * (long long)a.cols;
	// about 32 cells per thread, at most four blocks per SM (every block ends with two atomics per column on the same 2 * cols
	// words), and a multiple of cols, so that the grid's stride is one (a thread then stays on its columns)
	const bool vec = (((uintptr_t)a.raw) & 15) == 0;
	long long blocks = (total / 32 + 255) / 256;
	const long long cap = 148ll * (vec ? 4 : 6);
	if (blocks > cap) blocks = cap;
	if (blocks < 1) blocks = 1;
	blocks = ((blocks + a.cols - 1) / a.cols) * a.cols;
	const size_t smem = (size_t)2 * a.cols * sizeof(int);
	if (vec) minmax_kernel<true><<<(unsigned)blocks, 256, smem, s>>>(a.raw, a.rows, job);
	else minmax_kernel<false><<<(unsigned)blocks, 256, smem, s>>>(a.raw, a.rows, job);
	cudaError_t e = cudaGetLastError();
	if (e == cudaSuccess && a.flag == 1)
	{
		e = cudaFuncSetAttribute(mean_stdev_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MS_SMEM);
		if (e != cudaSuccess) return e;
		mean_stdev_kernel<<<(a.cols + 31) / 32, 256, MS_SMEM, s>>>(a.raw, a.rows, job);
		e = cudaGetLastError();
	}
	if (e != cudaSuccess) return e;
	ChainedLaunch layout(dim3(1), 256, smem, true, s);
	e = cudaLaunchKernelEx(&layout.config, layout_kernel, job);
	if (e != cudaSuccess) return e;
	const int squeeze = a.flag == 0 && a.classification;
	// By tiles: a third of an SM's shared memory holds two tiles of the table and two of the results, of at least 16 rows each
	// (cols + width up to 560 columns), and all three start on 16-byte boundaries.
	int tile = (int)((72 * 1024 - 1024) / (2ll * 4 * (a.cols + a.width)) / 4 * 4);
	if (tile > 128) tile = 128;
	if (a.write && tile >= 16 && a.rows >= tile && ((((uintptr_t)a.raw) | ((uintptr_t)a.x) | ((uintptr_t)a.y)) & 15) == 0)
	{
		const size_t bytes = 2 * ((size_t)tile * 4 * (a.cols + a.width) + 3 * 128);
		e = cudaFuncSetAttribute(transform_tiles_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
		if (e != cudaSuccess) return e;
		const long long tiles = a.rows / tile;
		ChainedLaunch c(dim3((unsigned)(tiles < 148 * 3 ? tiles : 148 * 3)), 256, bytes, true, s);
		return cudaLaunchKernelEx(&c.config, transform_tiles_kernel, a.raw, (long long)a.rows, job, squeeze, tile, a.x, a.y);
	}
	// blocks of as many whole rows as 256 threads hold, so that few threads have no column; as many as fill the SMs 16 blocks of
	// 256 deep (without that, 150 columns left 106 of 256 threads idle: 357 us a call for 487,596 x 60 with 15 categorical ones, 217 now)
	const int wide = a.width < 256 ? a.width : 256, threads = (256 / wide * wide + 31) / 32 * 32;
	ChainedLaunch c(dim3(a.write ? 148 * 16 * 256 / threads : 1), threads, 0, true, s);
	return cudaLaunchKernelEx(&c.config, transform_kernel, a.raw, (long long)a.rows, job, squeeze, a.x, a.y);
}

float order_float_host(int i)
{
	i = i >= 0 ? i : i ^ 0x7FFFFFFF;
	float f;
	memcpy(&f, &i, sizeof f);
	return f;
}

}  // namespace glb
