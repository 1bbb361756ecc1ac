// Device-side building blocks of the tensor-core layer-product kernel: mbarrier waits with a bound, TMA tile loads,
// shared-memory matrix descriptors, the tcgen05 MMA / commit / tensor-memory load wrappers, and the epilogue.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>
#include <stdlib.h>

#include "common.cuh"
#include "tc_gemm.h"

namespace glb {
namespace tc {

constexpr int TC_BM = 128;
constexpr int TC_BK = 32;         // k per pipeline stage: 64-byte rows of fp16
// The tensor core adds into its fp32 accumulator with truncation, not round-to-nearest: a chain of n accumulations
// drifts by up to n * 2^-24 of the running sum, towards zero.  One accumulator therefore holds at most 24 additions
// (16 k each) of the hi*hi products before the epilogue warps drain it into fp32 registers with round-to-nearest adds.  The
// cross products hi*lo + lo*hi go to an accumulator of their own that is 2^-11 of the result, so its chain may be longer.
constexpr int TC_CHUNK_KB = 12;       // stages per hi*hi chunk: 384 k, 24 additions
constexpr int TC_XCHUNK_KB = 96;      // stages per cross chunk: 3072 k, 384 additions of terms 2^-11 as large
constexpr long long TC_WAIT_CYCLES = 2000000000ll;  // about a second

// Low TF32 part of an fp32 value for the 3xTF32 products: v - trunc_tf32(v), rounded to TF32 (the tensor core itself reads
// trunc_tf32(v) from the unmodified fp32 word).
__device__ __forceinline__ float tf32_lo(float v)
{
	const float hi = __uint_as_float(__float_as_uint(v) & 0xFFFFE000u);
	uint32_t t;
	asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(t) : "f"(v - hi));
	return __uint_as_float(t);
}

struct TcParams
{
	float* C;
	long long ldc;
	int M, N, K;
	int a_mn, b_mn;  // 1: operand is M/N-contiguous (MN-major), 0: K-contiguous (K-major)
	const TensorScale* sca;
	const TensorScale* scb;
	int epi;
	int c_mode;      // 0: no fp32 output, 1: rows are 16-byte aligned, 2: they are not
	TensorScale* csc;  // split output: record (or NULL) and parts
	__half* Chi;
	__half* Clo;
	long long ldch;
	float* Clo32;      // low TF32 parts of the output (pitch ldc; of the new weights: pitch N), or NULL
	const float* bias_ptr;
	int act;
	float par;
	const float* aux;
	long long ld_aux;
	float alpha;
	const float* colterm;
	int* err_flag;
	unsigned* relu_mask_out;
	const unsigned* relu_mask_in;
	int mask_ld;
	double* dsum;
	float* W;        // fused update
	const TensorScale* wsc;
	float inv_mb;
	float decay_bound;
	int* bad_flag;
	int tiles_m, tiles_n;  // the CTAs walk the tiles_m * tiles_n output tiles persistently
	// Split of the last, partial wave of tiles along k ("stream-K", see TcWork): the first sk_full_tiles tiles
	// are whole-tile work items; the k-blocks of the remaining tiles are dealt out evenly over the CTAs.
	// sk_work == NULL: every tile is a whole-tile item.
	float* sk_work;        // [grid][128 x BN] fp32: a CTA's partial tile, if it has one
	unsigned* sk_flags;    // [grid][8]: launch number, per epilogue warp, once that warp's part of the partial is stored
	unsigned sk_epoch;     // this launch's number (flags only ever grow)
	int sk_full_tiles;
};

// The work items of one CTA, the same sequence for the producer, the MMA lane and the epilogue warps.
// First the whole tiles t = cta, cta + grid, ... below sk_full_tiles.  Then the CTA's share of the remaining
// tiles' k-blocks: with R tiles of KB k-blocks left, CTA c owns the units [c * R * KB / grid, (c + 1) * R * KB / grid)
// of the sequence (tile 0 k-block 0, tile 0 k-block 1, ..., tile R - 1 k-block KB - 1) -- at most the tail of one tile
// (a PARTIAL: its accumulators go to the CTA's workspace slot), whole tiles, and the head of one more tile (the
// tile's FINISHER: it adds the partials of the CTAs that hold the rest of the tile, in CTA order, and runs the
// epilogue).  A CTA computes its partial first and finishes a tile last, so a finisher rarely waits.  The split
// depends only on the shape and the grid, and the partials are added in a fixed order: results are reproducible.
struct TcWork
{
	// (ints: the launch only splits when grid * units fits 31 bits)
	int grid, KB, full, units;
	int u, u1;  // units of the split region still to do: [u, u1)
	int t;      // next whole tile of the first phase
	__device__ TcWork(int cta, int grid_, int KB_, int total, int full_)
	    : grid(grid_), KB(KB_), full(full_), units((total - full_) * KB_), t(cta)
	{
		u = share_begin(cta);
		u1 = share_begin(cta + 1);
	}
	// tile, k-block range [kb0, kb1) of the next item; false when the CTA is done
	__device__ bool next(int& tile, int& kb0, int& kb1)
	{
		if (t < full)
		{
			tile = t;
			kb0 = 0;
			kb1 = KB;
			t += grid;
			return true;
		}
		if (u >= u1) return false;
		const int tr = u / KB;
		tile = full + tr;
		kb0 = u - tr * KB;
		kb1 = min(KB, kb0 + (u1 - u));
		u += kb1 - kb0;
		return true;
	}
	// first unit of CTA j's share
	__device__ int share_begin(int j) const { return (int)(((unsigned)j * (unsigned)units) / (unsigned)grid); }
};

// Data-parallel weight gradient: rows [o * band_rows, (o + 1) * band_rows) of C belong to rank o and
// are stored straight into that rank's memory (maps[o] describes the band as a [band_rows][N] matrix
// there) instead of into C.
struct TcPeer
{
	const CUtensorMap* maps;  // device array, one map per owner
	int band_rows;
	int self;                 // this rank: its CTAs walk the owners' bands starting with owner self + 1
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
	asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
	asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity)
{
	uint32_t ok;
	asm volatile(
	    "{\n\t.reg .pred p;\n\t"
	    "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
	    "selp.b32 %0, 1, 0, p;\n\t}"
	    : "=r"(ok)
	    : "r"(bar), "r"(parity)
	    : "memory");
	return ok != 0;
}
// Bounded wait: false when the limit ran out or another role already gave up.  The first try is inline -- it usually
// succeeds, and the issuing threads' own instructions are what bounds a short stage.
__device__ __noinline__ static bool mbar_wait_slow(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* err_flag, int code)
{
	const long long t0 = clock64();
	for (;;)
	{
		if (mbar_try(bar, parity)) return true;
		if (*abort_flag) return false;
		if (clock64() - t0 > TC_WAIT_CYCLES)
		{
			*abort_flag = 1;
			atomicExch(err_flag, code);
			return false;
		}
	}
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* err_flag, int code)
{
	return mbar_try(bar, parity) || mbar_wait_slow(bar, parity, abort_flag, err_flag, code);
}
// Where a kernel has given up: the copies lo .. hi - 1 of a ring of n barriers, which may still be in flight, waited for within the limit
// (out of line: it must not lengthen the code that runs)
template <unsigned n>
__device__ __noinline__ void mbar_drain(uint32_t bars, unsigned lo, unsigned hi)
{
#pragma unroll 1
	for (unsigned k = lo; k < hi; ++k)
	{
		const long long t0 = clock64();
		while (!mbar_try(bars + 8 * (k % n), (k / n) & 1u) && clock64() - t0 < TC_WAIT_CYCLES) {}
	}
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1)
{
	asm volatile(
	    "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
	    "l"(map), "r"(bar), "r"(c0), "r"(c1)
	    : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2)
{
	asm volatile(
	    "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
	    "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
	    : "memory");
}

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3)
{
	asm volatile(
	    "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(dst),
	    "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
	    : "memory");
}

// Shared-memory matrix descriptor (descriptor version 1).  layout_type 4 = 64-byte swizzle (K-major tiles of 32 fp16
// per row), layout_type 2 = 128-byte swizzle (MN-major tiles of 64 fp16 per row).
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes, uint32_t layout_type)
{
	uint64_t d = 0;
	d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
	d |= (uint64_t)(lbo_bytes >> 4) << 16;
	d |= (uint64_t)(sbo_bytes >> 4) << 32;
	d |= 1ull << 46;
	d |= (uint64_t)layout_type << 61;
	return d;
}

__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate)
{
	asm volatile(
	    "{\n\t.reg .pred p;\n\t"
	    "setp.ne.b32 p, %4, 0;\n\t"
	    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
	    "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
	    : "memory");
}
__device__ __forceinline__ void umma_tf32(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate)
{
	asm volatile(
	    "{\n\t.reg .pred p;\n\t"
	    "setp.ne.b32 p, %4, 0;\n\t"
	    "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
	    "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
	    : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar)
{
	asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Where the issuing lane has given up: the MMAs that it has issued read shared memory and write tensor memory until they are done, and
// both are about to be given back.  bar: a barrier of one arrival, not used before.
__device__ __noinline__ static void mma_drain(uint32_t bar)
{
	umma_commit(bar);
	const long long t0 = clock64();
	while (!mbar_try(bar, 0) && clock64() - t0 < TC_WAIT_CYCLES) {}
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16])
{
	asm volatile(
	    "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
	    "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
	    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
	      "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
	    : "r"(taddr)
	    : "memory");
}

// ---- scales --------------------------------------------------------------------------------------------------
__device__ __forceinline__ float pow2f(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }  // -126 <= e <= 127
// The exponent under which values up to b in magnitude stay below 2^15 (fp16's range ends at 65504 = 2^16 - 32).
__device__ __forceinline__ int scale_for(float b)
{
	const uint32_t u = __float_as_uint(b) & 0x7FFFFFFFu;
	if (u == 0u) return 0;
	int e = 14 - ((int)(u >> 23) - 127);  // infinity and NaN count as 2^128
	return e < -110 ? -110 : (e > 110 ? 110 : e);
}
// x -> its two fp16 parts under the factor s = 2^e
__device__ __forceinline__ void split_f16(float x, float s, __half& hi, __half& lo)
{
	const float xs = x * s;
	hi = __float2half_rn(xs);
	lo = __float2half_rn((xs - __half2float(hi)) * 2048.0f);
}
__device__ __forceinline__ float join_f16(__half hi, __half lo, float inv_s)
{
	return fmaf(__half2float(lo), 1.0f / 2048.0f, __half2float(hi)) * inv_s;
}
// two values' high (low) parts in one word
__device__ __forceinline__ uint32_t hi_pair(float x, float y, float s)
{
	const __half2 h = __floats2half2_rn(x * s, y * s);
	return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t lo_pair(float x, float y, float s)
{
	const float xs = x * s, ys = y * s;
	const float2 h = __half22float2(__floats2half2_rn(xs, ys));
	const __half2 l = __floats2half2_rn((xs - h.x) * 2048.0f, (ys - h.y) * 2048.0f);
	return *reinterpret_cast<const uint32_t*>(&l);
}
__device__ __forceinline__ uint32_t pack_f16(__half a, __half b) { return (uint32_t)__half_as_ushort(a) | ((uint32_t)__half_as_ushort(b) << 16); }

// A bound on the magnitude of what the epilogue computes, from the operands' largest elements: every product is at most
// amax(A) * amax(B).  The bound lies about sqrt(K) above the values that appear, which costs as many of the 29 binades
// that a split matrix resolves in full; what is left is still far below the rounding of the sum itself.
__device__ __forceinline__ float epilogue_bound(const TcParams& p)
{
	const float b = (float)p.K * __uint_as_float(p.sca->amax) * __uint_as_float(p.scb->amax);
	if (p.epi == EPI_FORWARD)
	{
		const float z = b + (p.bias_ptr ? fabsf(*p.bias_ptr) : 0.0f);
		switch (p.act)
		{
		case GL_ACT_RELU:
		case GL_ACT_SOFTMAX: return z;
		case GL_ACT_LEAKY: return z * fmaxf(1.0f, fabsf(p.par));
		case GL_ACT_LINEAR: return z * fabsf(p.par);
		default: return 1.0f;
		}
	}
	if (p.epi == EPI_ERRPROP) return b * fmaxf(1.0f, fabsf(p.par));
	if (p.epi == EPI_GRAD && p.W)
		return __uint_as_float(p.wsc->amax) +
		       p.inv_mb * (fabsf(p.alpha) * b + (p.colterm ? p.decay_bound * __uint_as_float(p.scb->amax) : 0.0f));
	return b;
}

// ---- epilogue --------------------------------------------------------------------------------------------------
struct EpiWarp
{
	uint32_t stage;  // shared-memory address of the warp's staging areas (32 x 32 floats), 4 KB apart
	int nbuf;        // 1 or 2 of them
	int turn;        // running count of bulk-stored pieces, to alternate between the areas
	int lane;
	int row0, col0;  // first row and column of the warp's block
};

// Four consecutive values of this lane's row, 16-byte chunk v of the piece, in the order of a 128-byte-swizzled tensor map
// (which also keeps both the row-per-lane writes and the eight-lanes-per-row reads free of bank conflicts).
__device__ __forceinline__ void piece_put(const EpiWarp& k, uint32_t area, int v, float o0, float o1, float o2, float o3)
{
	asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(area + (uint32_t)k.lane * 128u + (uint32_t)((v ^ (k.lane & 7)) << 4)),
	             "f"(o0), "f"(o1), "f"(o2), "f"(o3)
	             : "memory");
}
// Start of a piece that leaves as a bulk store: pick the staging area and make sure no earlier store still reads it.
__device__ __forceinline__ uint32_t piece_begin(EpiWarp& k)
{
	const uint32_t area = k.stage + (uint32_t)(k.turn % k.nbuf) * 4096u;
	++k.turn;
	if (k.lane == 0)
	{
		if (k.nbuf == 2) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
		else asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
	}
	__syncwarp();
	return area;
}
// End of the piece: hand it to the copy engine.
__device__ __forceinline__ void piece_store(const EpiWarp& k, uint32_t area, const CUtensorMap* map, int x, int y)
{
	asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
	__syncwarp();
	if (k.lane == 0)
	{
		asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map), "r"(area), "r"(x), "r"(y)
		             : "memory");
		asm volatile("cp.async.bulk.commit_group;" ::: "memory");
	}
}

}  // namespace tc
}  // namespace glb
