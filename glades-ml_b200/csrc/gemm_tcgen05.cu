// Batched-mode matrix product on the 5th-generation tensor cores (sm_100a): TMA-fed tcgen05.mma kind::f16 with fp32
// accumulators in tensor memory, made fp32-faithful by splitting every operand into two fp16 parts,
//     x * 2^e = hi + lo * 2^-11,     hi = fp16(x * 2^e),  lo = fp16((x * 2^e - hi) * 2^11),
//     A*B  ~=  (A_hi*B_hi + 2^-11 (A_hi*B_lo + A_lo*B_hi)) * 2^-(eA + eB),
// with one power-of-two scale per matrix.  fp16 has the 11 significant bits of TF32 but runs at twice its rate and half its
// bytes.  Precision: hi and lo together keep an element to 2^-23 of itself (22 bits and the sign of lo; the two TF32 parts that
// this kernel used before kept 2^-22 and dropped a lo*lo term four times as large) for every element down to 2^-29 of
// the matrix's largest, and to 2^-51 of the largest below that.  lo carries its own factor 2^11 so that it does not
// become a subnormal 11 binades before hi does; the cross products therefore have an accumulator of their own and meet
// the hi*hi sum in fp32 registers.
//
// One CTA computes one 128 x BN tile of C at a time (BN = 256, 128, 64 or 32):
//   warp 0, one lane   TMA producer: per 32-deep k-block, four tiled bulk copies (A_hi, A_lo, B_hi, B_lo) into a swizzled
//                      shared-memory stage, completion on an mbarrier;
//   warp 1             allocates 2*BN tensor-memory columns (hi*hi | cross); one lane issues per stage the four cross
//                      MMAs, then the two hi*hi MMAs, and commits the stage's "empty" barrier;
//   warps 2..          epilogue, one warp per (32-lane quarter, 128-column half): drains finished chunks of the
//                      accumulations into fp32 registers, then applies the layer's epilogue (bias + activation, or times
//                      activation derivative, or the weight update itself) and stores fp32 and / or the split parts
//                      that the next product reads.
// Neither accumulator is double-buffered (2 * 256 columns are all there are): while one is drained the MMAs of the other
// run -- the cross MMAs of the next stage cover the drain of hi*hi, the last hi*hi MMAs of a tile the drain of its
// cross sums.
// Both operand layouts of the layer products are consumed as they lie in memory: K-contiguous rows (forward: activations
// and weights) through K-major descriptors, and M/N-contiguous rows (error propagation reads W_l as [k][n]; the weight
// gradient reads deltas and activations as [batch][node]) through MN-major descriptors, so no transposed copies exist.
// Any M, N and K: the copies fill what lies outside a matrix with zeros and the stores leave it out.
// Every wait on an mbarrier is bounded: when it runs out the kernel raises *err_flag, leaves its
// loops, waits (bounded) for the copies it still has in flight, frees its tensor memory and returns.
#include <atomic>

#include <string.h>

#include <mutex>
#include <vector>

#include "tc_epilogue.cuh"

namespace glb {
using namespace tc;
namespace {

// launches per tile variant since the library was loaded (diagnostics for the tests: which instantiation
// a shape ran on): [0] tiles up to 128 columns wide, [1] 256-wide tiles, [2] launches whose CTAs walked more than one
// tile each, [3] launches of the data-parallel variant that stores into the owners' memory, [4] launches
// that split their last wave of tiles along k
std::atomic<long long> g_variant_counts[5];
std::atomic<long long> g_engine_counts[2];  // launches of the 3xFP16 kernel, of the 3xTF32 kernel

template <int BN>
struct TcSmem
{
	static constexpr int STAGES = BN == 256 ? 4 : (BN == 128 ? 6 : 8);
	static constexpr int SBUF = BN == 256 ? 1 : 2;           // staging areas per epilogue warp (two help the bulk stores of PEER)
	static constexpr int EC = BN < 128 ? BN : 128;           // columns per epilogue warp
	static constexpr int A_BYTES = TC_BM * TC_BK * 2;
	static constexpr int B_BYTES = BN * TC_BK * 2;
	static constexpr int STAGE_BYTES = 2 * A_BYTES + 2 * B_BYTES;
	static constexpr int TILES_BYTES = STAGES * STAGE_BYTES;
	static constexpr int EPI_WARPS = 4 * (BN / EC);          // one warp per (lane quarter, EC-column part)
	static constexpr int STAGING_BYTES = EPI_WARPS * 4096 * SBUF;
	static constexpr int TOTAL = TILES_BYTES + STAGING_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/;
	static constexpr int THREADS = 64 + 32 * EPI_WARPS;
};

struct TcMaps
{
	CUtensorMap a_hi, a_lo, b_hi, b_lo;
};

// PEER: the data-parallel weight-gradient variant, whose epilogue (learning rate, decay term) stores
// each tile into the memory of the rank that owns its row band; a separate instantiation so that the
// register allocation of the plain kernel stays as it was tuned.
template <int BN, int MODE, bool PEER>
__global__ void __launch_bounds__(TcSmem<BN>::THREADS, 1)
    gemm_tc_kernel(const __grid_constant__ TcMaps maps, const __grid_constant__ TcParams p, const TcPeer peer)
{
	using S = TcSmem<BN>;
	constexpr int STAGES = S::STAGES, EC = S::EC;
	extern __shared__ uint8_t smem_raw[];
	// the swizzled tiles need a 1024-byte aligned base
	const uint32_t raw = smem_u32(smem_raw);
	const uint32_t base = (raw + 1023u) & ~1023u;
	uint8_t* gen_base = smem_raw + (base - raw);
	const uint32_t staging0 = base + S::TILES_BYTES;  // 1024-byte aligned, as the swizzled stores need
	uint64_t* bars = reinterpret_cast<uint64_t*>(gen_base + S::TILES_BYTES + S::STAGING_BYTES);
	const uint32_t bar0 = base + S::TILES_BYTES + S::STAGING_BYTES;
	// barrier slots: full[s] = s, empty[s] = STAGES + s, then hh_full, hh_empty, x_full, x_empty, given_up
	constexpr int NBARS = 2 * STAGES + 5;
	const uint32_t bar_hh_full = bar0 + 8 * (2 * STAGES), bar_hh_empty = bar_hh_full + 8;
	const uint32_t bar_x_full = bar_hh_full + 16, bar_x_empty = bar_hh_full + 24, bar_given_up = bar_hh_full + 32;
	uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + NBARS);
	volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

	const int warp = threadIdx.x >> 5;
	const int lane = threadIdx.x & 31;
	const int KB = (p.K + TC_BK - 1) / TC_BK;
	// Persistent CTAs: tile t of this CTA is blockIdx.x + i * gridDim.x.  Tiles are numbered m-fastest
	// inside bands of TC_BAND m-tiles, so that the CTAs running at one time share a band of A rows
	// and a few B column blocks in L2.  All three roles walk the same sequence; the stage and
	// accumulator barriers simply keep counting across tiles, which lets the producer and the MMA lane
	// run ahead into the next tile while the epilogue warps still store the previous one.
	const int total_tiles = p.tiles_m * p.tiles_n;
	constexpr int TC_BAND = 16;
	auto tile_origin = [&](int t, int& m0, int& n0) {
		if (PEER)
		{
			peer_tile_origin(peer, p, BN, t, m0, n0);
			return;
		}
		const int band_tiles = TC_BAND * p.tiles_n;
		const int band = t / band_tiles;
		const int in_band = t - band * band_tiles;
		const int band_m = min(TC_BAND, p.tiles_m - band * TC_BAND);
		const int mt = band * TC_BAND + in_band % band_m;
		const int nt = in_band / band_m;
		m0 = mt * TC_BM;
		n0 = nt * BN;
	};

	if (threadIdx.x == 0)
	{
		for (int s = 0; s < STAGES; ++s)
		{
			mbar_init(bar0 + 8 * s, 1);
			mbar_init(bar0 + 8 * (STAGES + s), 1);
		}
		mbar_init(bar_hh_full, 1);
		mbar_init(bar_hh_empty, S::EPI_WARPS);
		mbar_init(bar_x_full, 1);
		mbar_init(bar_x_empty, S::EPI_WARPS);
		mbar_init(bar_given_up, 1);
		*abort_flag = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (warp == 1)
	{
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
		             "r"(2 * BN)
		             : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
	const uint32_t tmem_base = *tmem_slot;

	if (warp == 0 && lane == 0)
	{
		// ------------------------------------------------ TMA producer
		int issued = 0;       // k-blocks issued so far, over all work items
		int s = 0;            // the next one's stage, and how often (mod 2) the ring has been walked
		uint32_t ph = 0;
		bool ok = true;
		TcWork work(blockIdx.x, gridDim.x, KB, total_tiles, p.sk_work ? p.sk_full_tiles : total_tiles);
		int t, kb0, kb1;
		while (ok && work.next(t, kb0, kb1))
		{
			int m0, n0;
			tile_origin(t, m0, n0);
			const int am = p.a_mn ? m0 / 64 : m0, bn = p.b_mn ? n0 / 64 : n0;
			int k0 = kb0 * TC_BK;
			for (int kb = kb0; kb < kb1; ++kb, k0 += TC_BK)
			{
				const uint32_t full = bar0 + 8 * s;
				if (!mbar_wait(full + 8 * STAGES, ph ^ 1u, abort_flag, p.err_flag, 1))
				{
					ok = false;
					break;
				}
				mbar_expect_tx(full, S::STAGE_BYTES);
				const uint32_t sa = base + s * S::STAGE_BYTES;
				const uint32_t sb = sa + 2 * S::A_BYTES;
				if (p.a_mn)
				{
					tma_load_3d(sa, &maps.a_hi, full, 0, k0, am);
					tma_load_3d(sa + S::A_BYTES, &maps.a_lo, full, 0, k0, am);
				}
				else
				{
					tma_load_2d(sa, &maps.a_hi, full, k0, am);
					tma_load_2d(sa + S::A_BYTES, &maps.a_lo, full, k0, am);
				}
				if (p.b_mn)
				{
					tma_load_3d(sb, &maps.b_hi, full, 0, k0, bn);
					tma_load_3d(sb + S::B_BYTES, &maps.b_lo, full, 0, k0, bn);
				}
				else
				{
					tma_load_2d(sb, &maps.b_hi, full, k0, bn);
					tma_load_2d(sb + S::B_BYTES, &maps.b_lo, full, k0, bn);
				}
				++issued;
				if (++s == STAGES)
				{
					s = 0;
					ph ^= 1u;
				}
			}
		}
		if (*abort_flag)
		{
			// give copies that are still in flight a bounded time to land before the CTA ends
			const int lo = issued > STAGES ? issued - STAGES : 0;
			for (int kb = lo; kb < issued; ++kb)
			{
				const long long t0 = clock64();
				while (!mbar_try(bar0 + 8 * (kb % STAGES), (uint32_t)(kb / STAGES) & 1u) && clock64() - t0 < TC_WAIT_CYCLES) {}
			}
		}
	}
	else if (warp == 1 && lane == 0)
	{
		// ------------------------------------------------ MMA issuer
		// kind::f16: fp32 accumulator, A and B fp16
		const uint32_t idesc = (1u << 4) | ((uint32_t)p.a_mn << 15) | ((uint32_t)p.b_mn << 16) | ((uint32_t)(BN >> 3) << 17) |
		                       ((uint32_t)(TC_BM >> 4) << 24);
		// K-major: rows of 64 bytes (64-byte swizzle), 8-row groups 512 bytes apart; a k-step of 16 is 32 bytes along the row.
		// MN-major: 64-element (128-byte) runs, one k per 128-byte row, 128-byte swizzle, groups of 8 k-rows 1024 bytes
		// apart, so a k-step of 16 is 2048 bytes; the next 64-element chunk of M/N lies a whole 64 x 32 box (4096
		// bytes) further.
		// Descriptors differ in their address only: each is stage 0's plus (bytes >> 4).  One thread issues everything, and at
		// 64 to 128 cycles per MMA its own instructions are what bounds a stage if they are not few.
		constexpr uint32_t MN_LBO = 128u * TC_BK;
		const uint64_t desc_a = make_smem_desc(base, p.a_mn ? MN_LBO : 0u, p.a_mn ? 1024u : 512u, p.a_mn ? 2u : 4u);
		const uint64_t desc_b = make_smem_desc(base + 2 * S::A_BYTES, p.b_mn ? MN_LBO : 0u, p.b_mn ? 1024u : 512u, p.b_mn ? 2u : 4u);
		const uint32_t a_step = p.a_mn ? 2048u >> 4 : 32u >> 4, b_step = p.b_mn ? 2048u >> 4 : 32u >> 4;
		constexpr uint32_t A_LO = S::A_BYTES >> 4, B_LO = S::B_BYTES >> 4;
		const uint32_t tmem_hh = tmem_base, tmem_x = tmem_base + BN;
		static_assert(TC_BK == 32, "two k-steps per stage below");
		bool ok = true;
		int s = 0;                       // the next k-block's stage, and how often (mod 2) the ring has been walked
		uint32_t ph = 0;
		uint32_t hh_ph = 1, x_ph = 1;    // parities of the next waits for drained accumulators
		TcWork work(blockIdx.x, gridDim.x, KB, total_tiles, p.sk_work ? p.sk_full_tiles : total_tiles);
		int t, kb0, kb1;
		while (ok && work.next(t, kb0, kb1))
		{
			int hin = 0, xin = 0;  // k-blocks of the running chunks so far (chunks count from the item's first k-block)
			for (int left = kb1 - kb0; left > 0; --left)
			{
				// an accumulator's first MMA of a chunk waits until the previous chunk has been drained
				if (xin == 0)
				{
					if (!mbar_wait(bar_x_empty, x_ph, abort_flag, p.err_flag, 4)) { ok = false; break; }
					x_ph ^= 1u;
				}
				const uint32_t full = bar0 + 8 * s;
				if (!mbar_wait(full, ph, abort_flag, p.err_flag, 2)) { ok = false; break; }
				asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
				const uint32_t off = (uint32_t)s * (S::STAGE_BYTES >> 4);
				const uint64_t a0 = desc_a + off, b0 = desc_b + off;
				const uint64_t a1 = a0 + a_step, b1 = b0 + b_step;
				umma_f16(tmem_x, a0, b0 + B_LO, idesc, (uint32_t)xin);
				umma_f16(tmem_x, a0 + A_LO, b0, idesc, 1u);
				umma_f16(tmem_x, a1, b1 + B_LO, idesc, 1u);
				umma_f16(tmem_x, a1 + A_LO, b1, idesc, 1u);
				if (++xin == TC_XCHUNK_KB || left == 1)
				{
					umma_commit(bar_x_full);
					xin = 0;
				}
				if (hin == 0)
				{
					if (!mbar_wait(bar_hh_empty, hh_ph, abort_flag, p.err_flag, 4)) { ok = false; break; }
					hh_ph ^= 1u;
					asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
				}
				umma_f16(tmem_hh, a0, b0, idesc, (uint32_t)hin);
				umma_f16(tmem_hh, a1, b1, idesc, 1u);
				umma_commit(full + 8 * STAGES);  // frees the stage once these MMAs have read it
				if (++hin == TC_CHUNK_KB || left == 1)
				{
					umma_commit(bar_hh_full);
					hin = 0;
				}
				if (++s == STAGES)
				{
					s = 0;
					ph ^= 1u;
				}
			}
		}
		if (!ok) mma_drain(bar_given_up);
	}
	else if (warp >= 2)
	{
		// ------------------------------------------------ epilogue: drain chunks, then the layer epilogue
		const int q = warp & 3;            // the tensor-memory lane quarter this warp may read
		const int half = (warp - 2) >> 2;  // which EC columns of the tile
		bool ok = true;
		uint32_t hh = 0, x = 0;            // chunks drained so far
		EpiWarp ew;
		ew.stage = staging0 + (uint32_t)(warp - 2) * (4096u * S::SBUF);
		ew.nbuf = S::SBUF;
		ew.turn = 0;
		ew.lane = lane;
		// 2^-(eA + eB) as two factors, so that neither leaves the range of a float
		const int es = -(p.sca->e + p.scb->e);
		const float inv1 = pow2f(es / 2), inv2 = pow2f(es - es / 2);
		int eo = 0;
		if (p.Chi)
		{
			eo = scale_for(epilogue_bound(p));
			if (blockIdx.x == 0 && warp == 2 && lane == 0) p.csc->e = eo;
		}
		const float so = pow2f(eo);
		const uint32_t lane_base = (uint32_t)(q * 32) << 16;
		TcWork work(blockIdx.x, gridDim.x, KB, total_tiles, p.sk_work ? p.sk_full_tiles : total_tiles);
		int t, kb0, kb1;
		while (ok && work.next(t, kb0, kb1))
		{
			int m0, n0;
			tile_origin(t, m0, n0);
			float acc[EC];
#pragma unroll
			for (int i = 0; i < EC; ++i) acc[i] = 0.0f;
			auto drain = [&](uint32_t bar_full, uint32_t bar_empty, uint32_t& use, uint32_t column, float f) {
				if (!mbar_wait(bar_full, use & 1u, abort_flag, p.err_flag, 3)) return false;
				asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
				const uint32_t taddr = tmem_base + lane_base + column + (uint32_t)(half * EC);
#pragma unroll
				for (int c = 0; c < EC / 16; ++c)
				{
					uint32_t r[16];
					tmem_ld16(taddr + (uint32_t)(c * 16), r);
					asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
					for (int e = 0; e < 16; ++e) acc[c * 16 + e] = fmaf(__uint_as_float(r[e]), f, acc[c * 16 + e]);
				}
				asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
				__syncwarp();
				if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_empty) : "memory");
				++use;
				return true;
			};
			const int nkb = kb1 - kb0;
			for (int done = 0; done < nkb && ok;)
			{
				done = min(done + TC_CHUNK_KB, nkb);
				// (the cross chunk that ends with this stage was committed before the hi*hi chunk)
				if (done == nkb || done % TC_XCHUNK_KB == 0) ok = drain(bar_x_full, bar_x_empty, x, BN, 1.0f / 2048.0f);
				if (ok) ok = drain(bar_hh_full, bar_hh_empty, hh, 0, 1.0f);
			}
			if (ok && kb0 != 0)
			{
				send_partial<BN, EC>(acc, p, warp - 2, lane);  // the tile's finisher (an earlier CTA) adds it
				continue;
			}
			if (ok && kb1 != KB) ok = add_partials<BN, EC>(acc, p, work, t, KB, warp - 2, lane, abort_flag);
			if (ok)
			{
				ew.row0 = m0 + q * 32;
				ew.col0 = n0 + half * EC;
				if (PEER)
					send_block<EC>(acc, ew, p, inv1, inv2, peer, m0);
				else
					finish_block<EC, MODE>(acc, ew, p, inv1, inv2, so, (long long)((m0 / TC_BM) * p.tiles_n + n0 / BN) * S::EPI_WARPS + (warp - 2));
			}
		}
		// every bulk store of this warp must have completed before the CTA may exit
		if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
	}
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	if (warp == 1)
	{
		asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * BN) : "memory");
	}
}

// ---- host side: tensor maps ---------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn()
{
	static EncodeTiledFn fn = nullptr;
	if (!fn)
	{
		void* p = nullptr;
		cudaDriverEntryPointQueryResult qr;
		if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) == cudaSuccess &&
		    qr == cudaDriverEntryPointSuccess)
			fn = (EncodeTiledFn)p;
	}
	return fn;
}

// row-major [rows][cols] matrix of pitch ld elements, boxes of box_rows x box_cols
bool make_map_2d(CUtensorMap* m, CUtensorMapDataType type, int elem, const void* ptr, long long rows, long long cols, long long ld,
                 int box_cols, int box_rows, CUtensorMapSwizzle swizzle)
{
	EncodeTiledFn fn = encode_fn();
	if (!fn) return false;
	cuuint64_t dim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
	cuuint64_t str[1] = {(cuuint64_t)ld * elem};
	cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
	cuuint32_t es[2] = {1, 1};
	return fn(m, type, 2, const_cast<void*>(ptr), dim, str, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
	          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Operand X(r, k), r in [0, R): mn == 0: X[r*ld + k] (K-contiguous), box = 32 k x box_r rows; mn == 1: X[k*ld + r]
// (contiguous in r), viewed as [r/64][k][r%64], box = 64 x 32 k x box_r/64.
bool make_operand_map(CUtensorMap* m, const __half* ptr, int mn, long long R, long long K, long long ld, int box_r)
{
	if (!mn) return make_map_2d(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, ptr, R, K, ld, TC_BK, box_r, CU_TENSOR_MAP_SWIZZLE_64B);
	EncodeTiledFn fn = encode_fn();
	if (!fn) return false;
	cuuint64_t dim[3] = {64, (cuuint64_t)K, (cuuint64_t)((R + 63) / 64)};
	cuuint64_t str[2] = {(cuuint64_t)ld * 2, 128};
	cuuint32_t box[3] = {64, TC_BK, (cuuint32_t)(box_r / 64)};
	cuuint32_t es[3] = {1, 1, 1};
	return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<__half*>(ptr), dim, str, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
	          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, int MODE, bool PEER>
cudaError_t launch_cfg(const TcMaps& maps, const TcParams& p, int sm_reserve, cudaStream_t s, const TcPeer& peer, const TcSplitK* sk,
                       int* dsum_count = nullptr)
{
	using S = TcSmem<BN>;
	int sm_count = 0;
	if (cudaError_t e = prepare_tc_launch(reinterpret_cast<const void*>(&gemm_tc_kernel<BN, MODE, PEER>), S::TOTAL, &sm_count)) return e;
	TcParams q = p;
	q.tiles_m = (p.M + TC_BM - 1) / TC_BM;
	q.tiles_n = (p.N + BN - 1) / BN;
	const int total = q.tiles_m * q.tiles_n;
	if (dsum_count) *dsum_count = total * S::EPI_WARPS;
	int avail = sm_count - sm_reserve;
	if (avail < 1) avail = 1;
	int grid = total < avail ? total : avail;
	// Split the last, partial wave of tiles along k over all CTAs where that wave would leave a quarter or more of
	// the SMs idle (32 tiles of a narrow layer; 68 tiles after three whole waves) and the caller gave a workspace.
	// Not below that: CTAs that share a tile's operands then sit at different k offsets, the operands stop being
	// fetched once and shared through L2, and 128 tiles on 148 SMs measured 17-30 % slower split than whole.
	// The data-parallel variant (epilogue stores into peers' memory) is never split: with the SMs it leaves to the
	// exchange its tile counts are whole waves, and the combination has no parity test.
	q.sk_full_tiles = total;
	const int KB = (p.K + TC_BK - 1) / TC_BK;
	if (q.sk_work && sk && KB >= 4 && !PEER)
	{
		const int g2 = avail;
		const int full = (total / g2) * g2;
		const int rem = total - full;
		if (rem > 0 && (g2 - rem) * 100 >= g2 * sk->min_idle_pct && (long long)rem * KB >= 2ll * g2 && (size_t)g2 <= sk->slots &&
		    (long long)(g2 + 1) * rem * KB < (1ll << 31))
		{
			grid = g2;
			q.sk_full_tiles = full;
			q.sk_epoch = ++*sk->epoch;
		}
	}
	if (q.sk_full_tiles == total) q.sk_work = nullptr;
	tc_count_launch(0, BN == 256, total > grid, PEER, q.sk_work != nullptr);
	gemm_tc_kernel<BN, MODE, PEER><<<grid, S::THREADS, S::TOTAL, s>>>(maps, q, peer);
	return cudaGetLastError();
}

// 256-wide tiles unless they would leave more than half of the SMs without a tile (with a split-k workspace a few wide
// tiles still fill the GPU: their k-blocks are dealt out over all CTAs) or their last column of tiles would be mostly
// outside the matrix; narrow outputs take the narrowest tile that holds them (their products are bound by reading A).
int tile_width(int M, int N, bool can_split, bool narrow_ok)
{
	const long long wide = (long long)((M + TC_BM - 1) / TC_BM) * ((N + 255) / 256);
	const long long w256 = (long long)((N + 255) / 256) * 256, w128 = (long long)((N + 127) / 128) * 128;
	if (N > 128 && w256 * 20 <= w128 * 23 && (wide >= 74 || (can_split && wide >= 16))) return 256;
	if (N > 64) return 128;
	return (N > 32 || !narrow_ok) ? 64 : 32;
}

// ---- fp32 -> split parts -------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) amax_kernel(const float* __restrict__ src, long long rows, int cols, long long ld, TensorScale* sc)
{
	float m = 0.0f;
	const long long stride = (long long)gridDim.x * blockDim.x;
	const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (ld == cols)
	{
		const long long n = rows * cols;
		long long head = (4 - (((uintptr_t)src >> 2) & 3)) & 3;  // elements before the first 16-byte boundary
		if (head > n) head = n;
		const long long n4 = (n - head) >> 2;
		const float4* s4 = reinterpret_cast<const float4*>(src + head);
#pragma unroll 4
		for (long long i = i0; i < n4; i += stride)
		{
			const float4 v = s4[i];
			m = fmaxf(fmaxf(m, fmaxf(finite_abs(v.x), finite_abs(v.y))), fmaxf(finite_abs(v.z), finite_abs(v.w)));
		}
		for (long long i = i0; i < head; i += stride) m = fmaxf(m, finite_abs(src[i]));
		for (long long i = head + 4 * n4 + i0; i < n; i += stride) m = fmaxf(m, finite_abs(src[i]));
	}
	else
		for (long long r = blockIdx.x; r < rows; r += gridDim.x)
			for (int c = threadIdx.x; c < cols; c += blockDim.x) m = fmaxf(m, finite_abs(src[r * ld + c]));
	__shared__ float sw[8];
	const unsigned b = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
	if ((threadIdx.x & 31) == 0) sw[threadIdx.x >> 5] = __uint_as_float(b);
	__syncthreads();
	if (threadIdx.x < 32) merge_amax(&sc->amax, threadIdx.x < 8 ? sw[threadIdx.x] : 0.0f);
}

// Thread = 8 consecutive columns of a row (one 16-byte store of each part).
template <class LOAD>
__device__ __forceinline__ void split_rows(long long rows, float s, __half* hi, __half* lo, long long ldo, LOAD load)
{
	const int w8 = (int)(ldo >> 3);
	const long long n8 = rows * w8;
	const long long stride = (long long)gridDim.x * blockDim.x;
#pragma unroll 2
	for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += stride)
	{
		const long long r = n8 < (1ll << 31) ? (long long)((unsigned)i / (unsigned)w8) : i / w8;
		const int c = (int)(i - r * w8) * 8;
		float v[8];
		load(r, c, v);
		__half h[8], l[8];
#pragma unroll
		for (int k = 0; k < 8; ++k) split_f16(v[k], s, h[k], l[k]);
		*reinterpret_cast<uint4*>(hi + r * ldo + c) = make_uint4(pack_f16(h[0], h[1]), pack_f16(h[2], h[3]), pack_f16(h[4], h[5]), pack_f16(h[6], h[7]));
		*reinterpret_cast<uint4*>(lo + r * ldo + c) = make_uint4(pack_f16(l[0], l[1]), pack_f16(l[2], l[3]), pack_f16(l[4], l[5]), pack_f16(l[6], l[7]));
	}
}

__global__ void __launch_bounds__(256) split_kernel(const float* __restrict__ src, long long rows, int cols, long long ld,
                                                     TensorScale* sc, __half* __restrict__ hi, __half* __restrict__ lo, long long ldo)
{
	const int e = scale_for(__uint_as_float(sc->amax));
	if (blockIdx.x == 0 && threadIdx.x == 0) sc->e = e;
	const bool vec = ((ld & 3) | (((uintptr_t)src >> 2) & 3)) == 0;
	split_rows(rows, pow2f(e), hi, lo, ldo, [&](long long r, int c, float (&v)[8]) {
		const float* q = src + r * ld + c;
		if (vec && c + 8 <= cols)
		{
			const float4 a = *reinterpret_cast<const float4*>(q), b = *reinterpret_cast<const float4*>(q + 4);
			v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
			v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
		}
		else
		{
#pragma unroll
			for (int k = 0; k < 8; ++k) v[k] = c + k < cols ? q[k] : 0.0f;
		}
	});
}

__global__ void __launch_bounds__(256) rescale_split_kernel(const __half* __restrict__ shi, const __half* __restrict__ slo, const TensorScale* ssc,
                                                             long long rows, int cols, long long lds, const float* __restrict__ rowscale,
                                                             float rowscale_max, TensorScale* sc, __half* __restrict__ hi,
                                                             __half* __restrict__ lo, long long ldo)
{
	const float bound = __uint_as_float(ssc->amax) * rowscale_max;
	const int e = scale_for(bound);
	if (blockIdx.x == 0 && threadIdx.x == 0)
	{
		sc->e = e;
		sc->amax = __float_as_uint(bound);
	}
	const float inv = pow2f(-ssc->e);
	split_rows(rows, pow2f(e), hi, lo, ldo, [&](long long r, int c, float (&v)[8]) {
		const float f = rowscale[r];
		const uint4 a = *reinterpret_cast<const uint4*>(shi + r * lds + c), b = *reinterpret_cast<const uint4*>(slo + r * lds + c);
		const __half* ah = reinterpret_cast<const __half*>(&a);
		const __half* bh = reinterpret_cast<const __half*>(&b);
#pragma unroll
		for (int k = 0; k < 8; ++k) v[k] = c + k < cols ? join_f16(ah[k], bh[k], inv) * f : 0.0f;
	});
}

unsigned stream_blocks(long long items)
{
	long long blocks = (items + 255) / 256;
	if (blocks > 148 * 8) blocks = 148 * 8;
	return (unsigned)(blocks < 1 ? 1 : blocks);
}

}  // namespace

int tc_splitk_min_idle_pct()
{
	const char* e = getenv("GLADES_TC_SPLITK_IDLE");
	const int v = e ? atoi(e) : 25;
	return v < 1 ? 1 : (v > 100 ? 100 : v);
}
void tc_count_launch(int engine, bool wide, bool several_tiles, bool peer, bool split)
{
	g_engine_counts[engine].fetch_add(1, std::memory_order_relaxed);
	const bool is[5] = {!wide, wide, several_tiles, peer, split};
	for (int i = 0; i < 5; ++i)
		if (is[i]) g_variant_counts[i].fetch_add(1, std::memory_order_relaxed);
}
void tc_engine_counts(long long out2[2])
{
	for (int i = 0; i < 2; ++i) out2[i] = g_engine_counts[i].load(std::memory_order_relaxed);
}
void tc_variant_counts(long long out5[5])
{
	for (int i = 0; i < 5; ++i) out5[i] = g_variant_counts[i].load(std::memory_order_relaxed);
}

bool tc_make_store_map(void* out128, const float* base, long long rows, long long cols, long long ld)
{
	return make_map_2d(reinterpret_cast<CUtensorMap*>(out128), CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, rows, cols, ld, 32, 32,
	                   CU_TENSOR_MAP_SWIZZLE_128B);
}

bool tc_make_map2d(void* out128, const float* base, long long rows, long long cols, long long ld, int box_cols, int box_rows,
                   int swizzle128)
{
	return make_map_2d(reinterpret_cast<CUtensorMap*>(out128), CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, rows, cols, ld, box_cols, box_rows,
	                   swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE);
}

bool tc_make_rows_map(void* out128, const float* base, long long stages, long long ld, int box_cols, int box_groups, int box_stages)
{
	EncodeTiledFn fn = encode_fn();
	if (!fn) return false;
	cuuint64_t dim[4] = {(cuuint64_t)ld, 8, 8, (cuuint64_t)stages};
	cuuint64_t str[3] = {(cuuint64_t)ld * 4, (cuuint64_t)ld * 32, (cuuint64_t)ld * 256};
	cuuint32_t box[4] = {(cuuint32_t)box_cols, 8, (cuuint32_t)box_groups, (cuuint32_t)box_stages};
	cuuint32_t es[4] = {1, 1, 1, 1};
	return fn(reinterpret_cast<CUtensorMap*>(out128), CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(base), dim, str, box, es,
	          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool tc_make_operand_map_f32(void* out128, const float* ptr, int mn, long long R, long long K, long long ld, int box_r)
{
	CUtensorMap* m = reinterpret_cast<CUtensorMap*>(out128);
	if (!mn) return make_map_2d(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, ptr, R, K, ld, 16, box_r, CU_TENSOR_MAP_SWIZZLE_64B);
	EncodeTiledFn fn = encode_fn();
	if (!fn) return false;
	cuuint64_t dim[3] = {32, (cuuint64_t)K, (cuuint64_t)(R / 32)};
	cuuint64_t str[2] = {(cuuint64_t)ld * 4, 128};
	cuuint32_t box[3] = {32, 16, (cuuint32_t)(box_r / 32)};
	cuuint32_t es[3] = {1, 1, 1};
	return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(ptr), dim, str, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
	          CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The shared-memory opt-in of a kernel and the SM count of the current device (both belong to a device, not to the process; kept
// per kernel and device).
cudaError_t prepare_tc_launch(const void* kernel, int smem_bytes, int* sm_count)
{
	constexpr int kMaxDev = 64;
	struct Done { const void* kernel; bool dev[kMaxDev]; };
	static std::mutex mutex;
	static std::vector<Done> done;
	static int sms[kMaxDev] = {};
	int dev = 0;
	if (cudaError_t e = cudaGetDevice(&dev)) return e;
	if (dev < 0 || dev >= kMaxDev) return cudaErrorInvalidDevice;
	std::lock_guard<std::mutex> lock(mutex);
	Done* d = nullptr;
	for (Done& x : done)
		if (x.kernel == kernel) d = &x;
	if (!d)
	{
		done.push_back(Done());
		d = &done.back();
		memset(d, 0, sizeof *d);
		d->kernel = kernel;
	}
	if (!d->dev[dev])
	{
		if (cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes)) return e;
		d->dev[dev] = true;
	}
	if (!sms[dev])
		if (cudaError_t e = cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev)) return e;
	*sm_count = sms[dev];
	return cudaSuccess;
}

bool tc_gemm_available() { return encode_fn() != nullptr; }

static int width_of(const TcGemmArgs& g)
{
	const bool can_split = g.sk && g.sk->work && g.K >= 128;
	// 32-wide tiles for forward products only (an MN-major B comes in chunks of 64 columns)
	return tile_width(g.M, g.N, can_split, g.epi == EPI_FORWARD && !g.B.mn);
}

long long tc_dsum_parts(int M, int N)
{
	// one per tile and epilogue warp, whatever the tile width: at most one per 128 x 32 block and lane quarter
	return (long long)((M + TC_BM - 1) / TC_BM) * ((N + 31) / 32) * 4;
}

int tc::tc_mode(const TcGemmArgs& g)
{
	if (g.epi == EPI_FORWARD) return g.act == GL_ACT_RELU ? TC_RELU : TC_ACT;
	if (g.epi == EPI_ERRPROP) return g.act == GL_ACT_RELU && g.relu_mask_in ? TC_ERR_MASK : TC_ERR_ACT;
	return g.W ? TC_UPDATE : TC_STORE;
}
void tc::tc_fill_params(TcParams& p, const TcGemmArgs& g)
{
	memset(&p, 0, sizeof p);
	p.C = g.C;
	p.ldc = g.ldc;
	p.M = g.M;
	p.N = g.N;
	p.K = g.K;
	p.sca = g.A.sc;
	p.scb = g.B.sc;
	p.epi = g.epi;
	// 16-byte stores of C where its rows allow them, else one column at a time
	if (g.C && !g.peer_maps) p.c_mode = (g.ldc % 4 == 0 && ((uintptr_t)g.C & 15) == 0) ? 1 : 2;
	p.csc = g.csc;
	p.Chi = g.Chi;
	p.Clo = g.Clo;
	p.ldch = g.ldch;
	p.Clo32 = g.Clo32;
	p.bias_ptr = g.bias_ptr;
	p.act = g.act;
	p.par = g.par;
	p.aux = g.aux;
	p.ld_aux = g.ld_aux;
	p.alpha = g.epi == EPI_GRAD ? g.alpha : 1.0f;
	p.colterm = g.colterm;
	p.relu_mask_out = g.relu_mask_out;
	p.relu_mask_in = g.relu_mask_in;
	p.mask_ld = g.mask_ld;
	p.dsum = g.dsum;
	p.W = g.W;
	p.wsc = g.wsc;
	p.inv_mb = g.inv_mb;
	p.decay_bound = g.decay_bound;
	p.bad_flag = g.bad_flag;
}

bool tc::tc_fill_peer(TcPeer& peer, const TcGemmArgs& g)
{
	peer.maps = reinterpret_cast<const CUtensorMap*>(g.peer_maps);
	peer.band_rows = g.band_rows;
	peer.self = g.peer_self;
	// (bands are whole tiles of rows, columns whole 32 x 32 pieces)
	return g.epi == EPI_GRAD && g.band_rows >= TC_BM && g.band_rows % TC_BM == 0 && g.M % TC_BM == 0 && g.N % 32 == 0 && !g.csc;
}

template <int MODE>
static cudaError_t launch_width(int BN, const TcMaps& maps, const TcParams& p, const TcGemmArgs& g, cudaStream_t s, const TcSplitK* sk)
{
	const TcPeer none = TcPeer();
	int* const count = g.dsum ? g.dsum_count : nullptr;
	if (BN == 256) return launch_cfg<256, MODE, false>(maps, p, g.sm_reserve, s, none, sk, count);
	if (BN == 128) return launch_cfg<128, MODE, false>(maps, p, g.sm_reserve, s, none, sk, count);
	if (BN == 32 && (MODE == TC_RELU || MODE == TC_ACT)) return launch_cfg<32, MODE <= TC_ACT && MODE >= TC_RELU ? MODE : TC_ACT, false>(maps, p, g.sm_reserve, s, none, sk, count);
	return launch_cfg<64, MODE, false>(maps, p, g.sm_reserve, s, none, sk, count);
}

cudaError_t launch_gemm_tc(const TcGemmArgs& g, int* err_flag, cudaStream_t s)
{
	const SplitOperand &A = g.A, &B = g.B;
	if (g.M < 1 || g.N < 1 || g.K < 1 || !A.hi || !A.lo || !B.hi || !B.lo || A.ld % 8 || B.ld % 8) return cudaErrorInvalidValue;
	const int BN = width_of(g);
	TcMaps maps;
	if (!make_operand_map(&maps.a_hi, A.hi, A.mn, g.M, g.K, A.ld, TC_BM) || !make_operand_map(&maps.a_lo, A.lo, A.mn, g.M, g.K, A.ld, TC_BM) ||
	    !make_operand_map(&maps.b_hi, B.hi, B.mn, g.N, g.K, B.ld, BN) || !make_operand_map(&maps.b_lo, B.lo, B.mn, g.N, g.K, B.ld, BN))
		return cudaErrorInvalidValue;
	if (g.Chi && (!g.csc || !g.Clo || g.ldch % 4)) return cudaErrorInvalidValue;
	TcParams p;
	tc_fill_params(p, g);
	p.a_mn = A.mn;
	p.b_mn = B.mn;
	p.err_flag = err_flag;
	const TcSplitK* sk = (g.sk && g.sk->work && g.K >= 128) ? g.sk : nullptr;
	p.sk_work = sk ? sk->work : nullptr;
	p.sk_flags = sk ? sk->flags : nullptr;
	if (g.peer_maps)
	{
		TcPeer peer;
		if (!tc_fill_peer(peer, g)) return cudaErrorInvalidValue;
		return BN == 256 ? launch_cfg<256, TC_STORE, true>(maps, p, g.sm_reserve, s, peer, sk)
		                 : launch_cfg<128, TC_STORE, true>(maps, p, g.sm_reserve, s, peer, sk);  // (never narrower: bands are multiples of 128)
	}
	switch (tc_mode(g))
	{
	case TC_STORE: return launch_width<TC_STORE>(BN, maps, p, g, s, sk);
	case TC_RELU: return launch_width<TC_RELU>(BN, maps, p, g, s, sk);
	case TC_ACT: return launch_width<TC_ACT>(BN, maps, p, g, s, sk);
	case TC_ERR_MASK: return launch_width<TC_ERR_MASK>(BN, maps, p, g, s, sk);
	case TC_ERR_ACT: return launch_width<TC_ERR_ACT>(BN, maps, p, g, s, sk);
	default: return launch_width<TC_UPDATE>(BN, maps, p, g, s, sk);
	}
}

cudaError_t launch_amax(const float* src, long long rows, int cols, long long ld, TensorScale* sc, cudaStream_t s)
{
	amax_kernel<<<stream_blocks(rows * cols / 16), 256, 0, s>>>(src, rows, cols, ld, sc);
	return cudaGetLastError();
}

cudaError_t launch_split(const float* src, long long rows, int cols, long long ld, TensorScale* sc, __half* hi, __half* lo, long long ldo,
                         cudaStream_t s)
{
	if (ldo % 8 || ldo < cols || (((uintptr_t)hi | (uintptr_t)lo) & 15)) return cudaErrorInvalidValue;
	split_kernel<<<stream_blocks(rows * (ldo / 8)), 256, 0, s>>>(src, rows, cols, ld, sc, hi, lo, ldo);
	return cudaGetLastError();
}

cudaError_t launch_rescale_split(const __half* shi, const __half* slo, const TensorScale* ssc, long long rows, int cols, long long lds,
                                 const float* rowscale, float rowscale_max, TensorScale* sc, __half* hi, __half* lo, long long ldo,
                                 cudaStream_t s)
{
	if (ldo % 8 || ldo < cols || lds < ldo) return cudaErrorInvalidValue;
	rescale_split_kernel<<<stream_blocks(rows * (ldo / 8)), 256, 0, s>>>(shi, slo, ssc, rows, cols, lds, rowscale, rowscale_max, sc, hi, lo, ldo);
	return cudaGetLastError();
}

bool tc_matmul_shape_ok(const GemmArgs& g)
{
	if (g.M < TC_BM || g.N < 128 || g.K < 16 || g.M % TC_BM || g.N % 128 || g.K % 16) return false;
	const bool a_k = (g.a_sk == 1), a_mn = (g.a_sm == 1);
	const bool b_k = (g.b_sk == 1), b_mn = (g.b_sn == 1);
	if (!(a_k || a_mn) || !(b_k || b_mn)) return false;
	const long long lda = a_k ? g.a_sm : g.a_sk, ldb = b_k ? g.b_sn : g.b_sk;
	if (lda % 4 || ldb % 4 || g.ldc % 4) return false;
	if (((uintptr_t)g.A | (uintptr_t)g.B | (uintptr_t)g.C) & 15) return false;
	return encode_fn() != nullptr;
}

size_t tc_matmul_operand_bytes(long long r, long long k) { return (size_t)(r * k) * 2 * sizeof(__half); }

cudaError_t tc_matmul(const GemmArgs& g, void* header, void* a_scratch, void* b_scratch, const TcSplitK* sk, int* err_flag, cudaStream_t s,
                      const TcGemmArgs* bands)
{
	if (!tc_matmul_shape_ok(g)) return cudaErrorInvalidValue;
	TensorScale* sc = static_cast<TensorScale*>(header);
	TcGemmArgs t;
	if (bands) t = *bands;
	else
	{
		memset(&t, 0, sizeof t);
		t.epi = EPI_NONE;
	}
	auto operand = [&](SplitOperand& o, const float* src, long long sr, long long sk1, int R, TensorScale* rec, void* scratch) {
		o.mn = sk1 == 1 ? 0 : 1;
		const long long rows = o.mn ? g.K : R;
		const int cols = o.mn ? R : g.K;
		__half* hi = static_cast<__half*>(scratch);
		o.hi = hi;
		o.lo = hi + rows * cols;
		o.ld = cols;
		o.sc = rec;
		const long long ld = o.mn ? sk1 : sr;
		cudaError_t e = launch_amax(src, rows, cols, ld, rec, s);
		return e == cudaSuccess ? launch_split(src, rows, cols, ld, rec, hi, hi + rows * cols, cols, s) : e;
	};
	cudaError_t e = operand(t.A, g.A, g.a_sm, g.a_sk, g.M, sc, a_scratch);
	if (e == cudaSuccess) e = operand(t.B, g.B, g.b_sn, g.b_sk, g.N, sc + 1, b_scratch);
	if (e != cudaSuccess) return e;
	t.M = g.M;
	t.N = g.N;
	t.K = g.K;
	t.C = g.C;
	t.ldc = g.ldc;
	t.sk = sk;
	return launch_gemm_tc(t, err_flag, s);
}

}  // namespace glb
