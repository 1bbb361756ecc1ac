// Layer product on the tensor cores in the 3xTF32 arithmetic,
//     A*B  ~=  A_hi*B_lo + A_lo*B_hi + A_hi*B_hi,      X_hi = trunc_tf32(X),  X_lo = tf32(X - X_hi).
// The tensor core reads only the upper 19 bits of an fp32 word, so the unmodified fp32 matrix serves as X_hi and only the
// X_lo matrices are materialised.
//
// What this kernel is for, next to the twice as fast 3xFP16 product of gemm_tcgen05.cu: networks whose activations JUMP.  The
// reference's ReLU is 0 below 0.046 and the identity above it, so a sum taken in another order -- which is all that two
// correct fp32 products differ by -- moves single activations by 0.046 and, through training, whole runs apart.  The order
// of operations is therefore kept: k ascending in steps of 8, the three products of a step in the order above, an
// accumulator drained into fp32 registers (round to nearest) every 128 k because the tensor core itself adds with
// truncation, and the last partial wave of tiles split along k exactly as the tile counts say.
//
// Structure, waits and epilogue are those of gemm_tcgen05.cu: warp 0 TMA producer (16-deep k-blocks of fp32, four copies per
// stage), warp 1 MMA issuer (six kind::tf32 MMAs per stage; two accumulators of BN columns, one drained while the other
// fills), warps 2.. epilogue.  Measured on the wide network's 8192 x 4096 x 4096 forward product: 1.03 ms = 266 TFLOP/s, the
// tensor pipe active in 85 % of the cycles (a third of what cuBLAS reaches in plain TF32 would be 248); 8192 x 4096 x 1024:
// 0.34 ms, 61 %.
#include <string.h>

#include "tc_epilogue.cuh"

namespace glb {
using namespace tc;
namespace {

constexpr int TF_BK = 16;
constexpr int TF_CHUNK_KB = 8;  // stages per accumulator chunk: 128 k, 48 additions

template <int BN>
struct TfSmem
{
	static constexpr int STAGES = BN == 256 ? 4 : 6;
	static constexpr int EC = 128;
	static constexpr int A_BYTES = TC_BM * TF_BK * 4;
	static constexpr int B_BYTES = BN * TF_BK * 4;
	static constexpr int STAGE_BYTES = 2 * A_BYTES + 2 * B_BYTES;
	static constexpr int TILES_BYTES = STAGES * STAGE_BYTES;
	static constexpr int EPI_WARPS = 4 * (BN / EC);
	static constexpr int STAGING_BYTES = EPI_WARPS * 4096;
	static constexpr int TOTAL = TILES_BYTES + STAGING_BYTES + 1024 + 256;
	static constexpr int THREADS = 64 + 32 * EPI_WARPS;
};

struct TfMaps
{
	CUtensorMap a, a_lo, b, b_lo;
};

// PEER: the data-parallel weight gradient, whose epilogue stores each tile into the memory of the rank that owns its rows.
template <int BN, int MODE, bool PEER>
__global__ void __launch_bounds__(TfSmem<BN>::THREADS, 1)
    gemm_tf32_kernel(const __grid_constant__ TfMaps maps, const __grid_constant__ TcParams p, const TcPeer peer)
{
	using S = TfSmem<BN>;
	constexpr int STAGES = S::STAGES, EC = S::EC;
	extern __shared__ uint8_t smem_raw[];
	const uint32_t raw = smem_u32(smem_raw);
	const uint32_t base = (raw + 1023u) & ~1023u;
	uint8_t* gen_base = smem_raw + (base - raw);
	const uint32_t staging0 = base + S::TILES_BYTES;
	uint64_t* bars = reinterpret_cast<uint64_t*>(gen_base + S::TILES_BYTES + S::STAGING_BYTES);
	const uint32_t bar0 = base + S::TILES_BYTES + S::STAGING_BYTES;
	// barrier slots: full[s] = s, empty[s] = STAGES + s, acc_full[b] = 2*STAGES + b, acc_empty[b] = 2*STAGES + 2 + b, then given_up
	constexpr int NBARS = 2 * STAGES + 5;
	const uint32_t bar_acc_full = bar0 + 8 * (2 * STAGES), bar_acc_empty = bar_acc_full + 16, bar_given_up = bar_acc_full + 32;
	uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + NBARS);
	volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int KB = p.K / TF_BK;
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
		m0 = (band * TC_BAND + in_band % band_m) * TC_BM;
		n0 = (in_band / band_m) * BN;
	};
	if (threadIdx.x == 0)
	{
		for (int s = 0; s < 2 * STAGES; ++s) mbar_init(bar0 + 8 * s, 1);
		for (int b = 0; b < 2; ++b)
		{
			mbar_init(bar_acc_full + 8 * b, 1);
			mbar_init(bar_acc_empty + 8 * b, S::EPI_WARPS);
		}
		mbar_init(bar_given_up, 1);
		*abort_flag = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if (warp == 1)
	{
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * BN) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
	const uint32_t tmem_base = *tmem_slot;
	TcWork work(blockIdx.x, gridDim.x, KB, total_tiles, p.sk_work ? p.sk_full_tiles : total_tiles);
	int t, kb0, kb1;

	if (warp == 0 && lane == 0)
	{
		int issued = 0, s = 0;
		uint32_t ph = 0;
		bool ok = true;
		while (ok && work.next(t, kb0, kb1))
		{
			int m0, n0;
			tile_origin(t, m0, n0);
			int k0 = kb0 * TF_BK;
			for (int kb = kb0; kb < kb1; ++kb, k0 += TF_BK)
			{
				const uint32_t full = bar0 + 8 * s;
				if (!mbar_wait(full + 8 * STAGES, ph ^ 1u, abort_flag, p.err_flag, 1))
				{
					ok = false;
					break;
				}
				mbar_expect_tx(full, S::STAGE_BYTES);
				const uint32_t sa = base + s * S::STAGE_BYTES, sb = sa + 2 * S::A_BYTES;
				if (p.a_mn)
				{
					tma_load_3d(sa, &maps.a, full, 0, k0, m0 / 32);
					tma_load_3d(sa + S::A_BYTES, &maps.a_lo, full, 0, k0, m0 / 32);
				}
				else
				{
					tma_load_2d(sa, &maps.a, full, k0, m0);
					tma_load_2d(sa + S::A_BYTES, &maps.a_lo, full, k0, m0);
				}
				if (p.b_mn)
				{
					tma_load_3d(sb, &maps.b, full, 0, k0, n0 / 32);
					tma_load_3d(sb + S::B_BYTES, &maps.b_lo, full, 0, k0, n0 / 32);
				}
				else
				{
					tma_load_2d(sb, &maps.b, full, k0, n0);
					tma_load_2d(sb + S::B_BYTES, &maps.b_lo, full, k0, n0);
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
		// kind::tf32: fp32 accumulator.  K-major: 64-byte rows (64-byte swizzle), a k-step of 8 is 32 bytes along the row.
		// MN-major: 32-element (128-byte) runs, one k per row, the 128-byte swizzle of 32-byte atoms that 32-bit operands need
		// (4 k-rows, 512 bytes), so a k-step is 1024 bytes; the next 32-element chunk lies a 32 x 16 box (2048 bytes) on.
		const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)p.a_mn << 15) | ((uint32_t)p.b_mn << 16) |
		                       ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
		const uint64_t desc_a = make_smem_desc(base, p.a_mn ? 128u * TF_BK : 0u, 512u, p.a_mn ? 1u : 4u);
		const uint64_t desc_b = make_smem_desc(base + 2 * S::A_BYTES, p.b_mn ? 128u * TF_BK : 0u, 512u, p.b_mn ? 1u : 4u);
		const uint32_t a_step = p.a_mn ? 1024u >> 4 : 32u >> 4, b_step = p.b_mn ? 1024u >> 4 : 32u >> 4;
		constexpr uint32_t A_LO = S::A_BYTES >> 4, B_LO = S::B_BYTES >> 4;
		bool ok = true;
		int s = 0;
		uint32_t ph = 0, chunk = 0;
		while (ok && work.next(t, kb0, kb1))
		{
			int kin = 0;  // k-blocks of the running chunk so far (chunks count from the item's first k-block)
			for (int left = kb1 - kb0; left > 0; --left)
			{
				const uint32_t buf = chunk & 1u;
				const uint32_t d = tmem_base + buf * BN;
				if (kin == 0)
				{
					// this accumulator must have been drained by the epilogue (two chunks ago)
					if (!mbar_wait(bar_acc_empty + 8 * buf, ((chunk >> 1) & 1u) ^ 1u, abort_flag, p.err_flag, 4)) { ok = false; break; }
					asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
				}
				const uint32_t full = bar0 + 8 * s;
				if (!mbar_wait(full, ph, abort_flag, p.err_flag, 2)) { ok = false; break; }
				asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
				const uint32_t off = (uint32_t)s * (S::STAGE_BYTES >> 4);
				const uint64_t a0 = desc_a + off, b0 = desc_b + off;
				umma_tf32(d, a0, b0 + B_LO, idesc, (uint32_t)kin);
				umma_tf32(d, a0 + A_LO, b0, idesc, 1u);
				umma_tf32(d, a0, b0, idesc, 1u);
				umma_tf32(d, a0 + a_step, b0 + B_LO + b_step, idesc, 1u);
				umma_tf32(d, a0 + A_LO + a_step, b0 + b_step, idesc, 1u);
				umma_tf32(d, a0 + a_step, b0 + b_step, idesc, 1u);
				umma_commit(full + 8 * STAGES);
				if (++kin == TF_CHUNK_KB || left == 1)
				{
					umma_commit(bar_acc_full + 8 * buf);
					++chunk;
					kin = 0;
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
		const int q = warp & 3;            // the tensor-memory lane quarter this warp may read
		const int half = (warp - 2) >> 2;  // which 128 columns of the tile
		bool ok = true;
		uint32_t chunk = 0;
		EpiWarp ew;
		ew.stage = staging0 + (uint32_t)(warp - 2) * 4096u;
		ew.nbuf = 1;
		ew.turn = 0;
		ew.lane = lane;
		int eo = 0;
		if (p.Chi)
		{
			eo = scale_for(epilogue_bound(p));
			if (blockIdx.x == 0 && warp == 2 && lane == 0) p.csc->e = eo;
		}
		const float so = pow2f(eo);
		const uint32_t lane_base = (uint32_t)(q * 32) << 16;
		while (ok && work.next(t, kb0, kb1))
		{
			int m0, n0;
			tile_origin(t, m0, n0);
			float acc[EC];
#pragma unroll
			for (int i = 0; i < EC; ++i) acc[i] = 0.0f;
			const int nchunk = (kb1 - kb0 + TF_CHUNK_KB - 1) / TF_CHUNK_KB;
			for (int c_in = 0; c_in < nchunk && ok; ++c_in, ++chunk)
			{
				const uint32_t buf = chunk & 1u;
				if (!mbar_wait(bar_acc_full + 8 * buf, (chunk >> 1) & 1u, abort_flag, p.err_flag, 3))
				{
					ok = false;
					break;
				}
				asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
				const uint32_t taddr = tmem_base + lane_base + buf * BN + (uint32_t)(half * EC);
#pragma unroll
				for (int c = 0; c < EC / 16; ++c)
				{
					uint32_t r[16];
					tmem_ld16(taddr + (uint32_t)(c * 16), r);
					asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
					for (int e = 0; e < 16; ++e) acc[c * 16 + e] += __uint_as_float(r[e]);
				}
				asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
				__syncwarp();
				if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_acc_empty + 8 * buf) : "memory");
			}
			if (ok && kb0 != 0)
			{
				// a partial: the tile's finisher (an earlier CTA) adds it (see gemm_tcgen05.cu)
				send_partial<BN, EC>(acc, p, warp - 2, lane);
				continue;
			}
			if (ok && kb1 != KB) ok = add_partials<BN, EC>(acc, p, work, t, KB, warp - 2, lane, abort_flag);
			if (ok)
			{
				ew.row0 = m0 + q * 32;
				ew.col0 = n0 + half * EC;
				if (PEER)
					send_block<EC>(acc, ew, p, 1.0f, 1.0f, peer, m0);
				else
					finish_block<EC, MODE>(acc, ew, p, 1.0f, 1.0f, so, (long long)((m0 / TC_BM) * p.tiles_n + n0 / BN) * S::EPI_WARPS + (warp - 2));
			}
		}
		// every bulk store of this warp must have completed before the CTA may exit
		if (PEER && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
	}
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	if (warp == 1)
	{
		asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * BN) : "memory");
	}
}

template <int BN, int MODE, bool PEER = false>
cudaError_t launch_tf(const TfMaps& maps, const TcParams& p, const TcGemmArgs& g, const TcSplitK* sk, cudaStream_t s, const TcPeer& peer = TcPeer())
{
	using S = TfSmem<BN>;
	int sm_count = 0;
	if (cudaError_t e = prepare_tc_launch(reinterpret_cast<const void*>(&gemm_tf32_kernel<BN, MODE, PEER>), S::TOTAL, &sm_count)) return e;
	TcParams q = p;
	q.tiles_m = p.M / TC_BM;
	q.tiles_n = p.N / BN;
	const int total = q.tiles_m * q.tiles_n;
	if (g.dsum && g.dsum_count) *g.dsum_count = total * S::EPI_WARPS;
	int avail = sm_count - g.sm_reserve;
	if (avail < 1) avail = 1;
	int grid = total < avail ? total : avail;
	// (the split rule is part of the order of operations: a quarter of the SMs idle in the last wave, enough k-blocks to deal out)
	q.sk_full_tiles = total;
	const int KB = p.K / TF_BK;
	if (q.sk_work && sk && KB >= 8)
	{
		const int full = (total / avail) * avail, rem = total - full;
		if (rem > 0 && (avail - rem) * 100 >= avail * sk->min_idle_pct && (long long)rem * KB >= 4ll * avail && (size_t)avail <= sk->slots &&
		    (long long)(avail + 1) * rem * KB < (1ll << 31))
		{
			grid = avail;
			q.sk_full_tiles = full;
			q.sk_epoch = ++*sk->epoch;
		}
	}
	if (q.sk_full_tiles == total) q.sk_work = nullptr;
	tc_count_launch(1, BN == 256, total > grid, PEER, q.sk_work != nullptr);
	gemm_tf32_kernel<BN, MODE, PEER><<<grid, S::THREADS, S::TOTAL, s>>>(maps, q, peer);
	return cudaGetLastError();
}

template <int MODE>
cudaError_t launch_tf_width(int BN, const TfMaps& maps, const TcParams& p, const TcGemmArgs& g, const TcSplitK* sk, cudaStream_t s)
{
	return BN == 256 ? launch_tf<256, MODE>(maps, p, g, sk, s) : launch_tf<128, MODE>(maps, p, g, sk, s);
}

__global__ void __launch_bounds__(256) split_lo_kernel(const float4* __restrict__ src, float4* __restrict__ lo, long long n4)
{
	const long long stride = (long long)gridDim.x * blockDim.x;
	for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += stride)
	{
		const float4 a = src[i];
		lo[i] = make_float4(tf32_lo(a.x), tf32_lo(a.y), tf32_lo(a.z), tf32_lo(a.w));
	}
}

// dst = src * rowscale (per row) and lo = the low TF32 parts of dst; n4 float4, ld4 of them per row
__global__ void __launch_bounds__(256) scale_split_lo_kernel(const float4* __restrict__ src, const float* __restrict__ rowscale, int ld4,
                                                              float4* __restrict__ dst, float4* __restrict__ lo, long long n4)
{
	const long long stride = (long long)gridDim.x * blockDim.x;
	for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += stride)
	{
		float4 a = src[i];
		const float c = rowscale[i / ld4];
		a.x *= c; a.y *= c; a.z *= c; a.w *= c;
		dst[i] = a;
		lo[i] = make_float4(tf32_lo(a.x), tf32_lo(a.y), tf32_lo(a.z), tf32_lo(a.w));
	}
}

unsigned lo_blocks(long long n4)
{
	long long blocks = (n4 + 255) / 256;
	if (blocks > 148 * 8) blocks = 148 * 8;
	return (unsigned)(blocks < 1 ? 1 : blocks);
}

}  // namespace

bool tf32_gemm_fits(const Tf32Operand& A, const Tf32Operand& B, int M, int N, int K)
{
	if (M < TC_BM || N < 128 || K < 16 || M % TC_BM || N % 128 || K % 16) return false;
	if (A.ld % 4 || B.ld % 4 || (((uintptr_t)A.x | (uintptr_t)B.x) & 15)) return false;
	return tc_gemm_available();
}

cudaError_t launch_gemm_tf32(const TcGemmArgs& g, const Tf32Operand& A, const Tf32Operand& B, int* err_flag, cudaStream_t s)
{
	if (!tf32_gemm_fits(A, B, g.M, g.N, g.K) || (g.Chi && (!g.csc || !g.Clo || !g.A.sc || !g.B.sc || g.ldch % 4))) return cudaErrorInvalidValue;
	const long long wide = (long long)(g.M / TC_BM) * (g.N / 256);
	// (the data-parallel variant is never split along k, for the reasons given at launch_cfg in gemm_tcgen05.cu)
	const TcSplitK* sk = (g.sk && g.sk->work && g.K / TF_BK >= 8 && !g.peer_maps) ? g.sk : nullptr;
	const int BN = (g.N % 256 == 0 && (wide >= 74 || (sk && wide >= 16))) ? 256 : 128;
	TfMaps maps;
	if (!tc_make_operand_map_f32(&maps.a, A.x, A.mn, g.M, g.K, A.ld, TC_BM) || !tc_make_operand_map_f32(&maps.a_lo, A.lo, A.mn, g.M, g.K, A.ld, TC_BM) ||
	    !tc_make_operand_map_f32(&maps.b, B.x, B.mn, g.N, g.K, B.ld, BN) || !tc_make_operand_map_f32(&maps.b_lo, B.lo, B.mn, g.N, g.K, B.ld, BN))
		return cudaErrorInvalidValue;
	TcParams p;
	tc_fill_params(p, g);
	p.a_mn = A.mn;
	p.b_mn = B.mn;
	p.err_flag = err_flag;
	p.sk_work = sk ? sk->work : nullptr;
	p.sk_flags = sk ? sk->flags : nullptr;
	if (g.peer_maps)
	{
		TcPeer peer;
		if (!tc_fill_peer(peer, g)) return cudaErrorInvalidValue;
		return BN == 256 ? launch_tf<256, TC_STORE, true>(maps, p, g, sk, s, peer) : launch_tf<128, TC_STORE, true>(maps, p, g, sk, s, peer);
	}
	switch (tc_mode(g))
	{
	case TC_STORE: return launch_tf_width<TC_STORE>(BN, maps, p, g, sk, s);
	case TC_RELU: return launch_tf_width<TC_RELU>(BN, maps, p, g, sk, s);
	case TC_ACT: return launch_tf_width<TC_ACT>(BN, maps, p, g, sk, s);
	case TC_ERR_MASK: return launch_tf_width<TC_ERR_MASK>(BN, maps, p, g, sk, s);
	case TC_ERR_ACT: return launch_tf_width<TC_ERR_ACT>(BN, maps, p, g, sk, s);
	default: return launch_tf_width<TC_UPDATE>(BN, maps, p, g, sk, s);
	}
}

cudaError_t launch_split_lo(const float* src, float* lo, long long count, cudaStream_t s)
{
	if (count % 4 || (((uintptr_t)src | (uintptr_t)lo) & 15)) return cudaErrorInvalidValue;
	split_lo_kernel<<<lo_blocks(count / 4), 256, 0, s>>>(reinterpret_cast<const float4*>(src), reinterpret_cast<float4*>(lo), count / 4);
	return cudaGetLastError();
}

cudaError_t launch_scale_split_lo(const float* src, const float* rowscale, int ld, float* dst, float* lo, long long count, cudaStream_t s)
{
	if (count % 4 || ld % 4 || (((uintptr_t)src | (uintptr_t)dst | (uintptr_t)lo) & 15)) return cudaErrorInvalidValue;
	scale_split_lo_kernel<<<lo_blocks(count / 4), 256, 0, s>>>(reinterpret_cast<const float4*>(src), rowscale, ld / 4, reinterpret_cast<float4*>(dst),
	                                                           reinterpret_cast<float4*>(lo), count / 4);
	return cudaGetLastError();
}

}  // namespace glb
