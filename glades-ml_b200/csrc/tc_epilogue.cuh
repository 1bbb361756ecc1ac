// Epilogue of the tensor-core layer products: what happens to a finished block of accumulators.
#pragma once
#include "tc_device.cuh"

namespace glb {
namespace tc {

// Largest finite magnitude of the warp's values into *amax (uint order is float order for magnitudes).
__device__ __forceinline__ void merge_amax(unsigned* amax, float m)
{
	const unsigned b = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
	if ((threadIdx.x & 31) == 0 && b > *reinterpret_cast<volatile unsigned*>(amax)) atomicMax(amax, b);
}
__device__ __forceinline__ float finite_abs(float v)
{
	const float a = fabsf(v);
	return a <= 3.402823466e38f ? a : 0.0f;
}

// What the epilogue of a launch does, as a template parameter: the row loop below is short, and a run-time choice among
// all of them would spread it over so much code that the warps wait for instructions (2.5 us per 32 x 32 piece).
enum
{
	TC_STORE = 0,     // C (EPI_NONE, EPI_GRAD without update)
	TC_RELU = 1,      // forward, ReLU; with or without the bits for the backward pass
	TC_ACT = 2,       // forward, any other activation
	TC_ERR_MASK = 3,  // error propagation through ReLU bits
	TC_ERR_ACT = 4,   // error propagation from the activations themselves
	TC_UPDATE = 5     // weight gradient applied to the weights
};

// Everything that happens to a finished 32 x EC block of C: the layer's arithmetic f on four neighbouring columns of a row, the
// statistics that later launches need (largest magnitude, sum), and the stores.  The accumulators lie one row per lane;
// each 32 x 32 piece is turned through the warp's 4 KB staging area so that eight lanes share a row: memory then sees whole
// 128-byte rows, whatever the pitch, and the arithmetic is a short loop instead of EC unrolled copies of it.
template <int EC, int MODE, class F>
__device__ __forceinline__ void block_rows(float (&acc)[EC], const EpiWarp& ew, const TcParams& p, float inv1, float inv2, float so,
                                           long long block_index, F f)
{
	const int cols = min(EC, p.N - ew.col0);  // valid columns and rows of the block (may be <= 0)
	const int rows = min(32, p.M - ew.row0);
	const int ch = ew.lane & 7, rr = ew.lane >> 3;  // this lane's four columns of a piece and its row of four
	const bool c16 = p.c_mode == 1;
	const bool w16 = ((p.N & 3) | (int)((uintptr_t)p.W & 15)) == 0;
	const bool stats = MODE != TC_STORE && p.csc != nullptr, split = MODE != TC_STORE && p.Chi != nullptr;
	float m = 0.0f;
	double d = 0.0;
	bool bad = false;
	// one copy of the loop's code for all pieces: the accumulators move down by 32 after each
#pragma unroll 1
	for (int c0 = 0; c0 < EC; c0 += 32)
	{
		if (c0 >= cols || rows <= 0) break;
#pragma unroll
		for (int v = 0; v < 8; ++v)
			piece_put(ew, ew.stage, v, acc[4 * v] * inv1 * inv2, acc[4 * v + 1] * inv1 * inv2, acc[4 * v + 2] * inv1 * inv2, acc[4 * v + 3] * inv1 * inv2);
#pragma unroll
		for (int c = 32; c < EC; ++c) acc[c - 32] = acc[c];
		__syncwarp();
		const int col = ew.col0 + c0 + ch * 4;
		const int left = p.N - col;  // columns from this lane's first one on
		float ct[4] = {0.0f, 0.0f, 0.0f, 0.0f};
		if ((MODE == TC_STORE || MODE == TC_UPDATE) && p.colterm)
#pragma unroll
			for (int k = 0; k < 4; ++k)
				if (k < left) ct[k] = p.colterm[col + k];
#pragma unroll 1
		for (int i0 = 0; i0 < 8; i0 += 4)
		{
			// what the four rows need from memory, all loads in flight at once: old weights, activations or ReLU bits
			float4 side[4];
			float v[4][4];
#pragma unroll
			for (int i = 0; i < 4; ++i)
			{
				const int r = (i0 + i) * 4 + rr;
				const long long row = ew.row0 + r;
				const bool on = r < rows && left > 0;
				side[i] = make_float4(0.f, 0.f, 0.f, 0.f);
				if (MODE == TC_UPDATE && on)
				{
					const float* wp = p.W + row * p.N + col;
					if (w16) side[i] = *reinterpret_cast<const float4*>(wp);
					else
					{
						side[i].x = wp[0];
						if (left > 1) side[i].y = wp[1];
						if (left > 2) side[i].z = wp[2];
						if (left > 3) side[i].w = wp[3];
					}
				}
				if (MODE == TC_ERR_MASK && on) side[i].x = __uint_as_float(p.relu_mask_in[row * p.mask_ld + (col >> 5)] >> (ch * 4));
				if (MODE == TC_ERR_ACT && on) side[i] = *reinterpret_cast<const float4*>(p.aux + row * p.ld_aux + col);  // (rows padded to multiples of four)
				asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
				             : "=f"(v[i][0]), "=f"(v[i][1]), "=f"(v[i][2]), "=f"(v[i][3])
				             : "r"(ew.stage + (uint32_t)r * 128u + (uint32_t)((ch ^ (r & 7)) << 4)));
			}
#pragma unroll
			for (int i = 0; i < 4; ++i)
			{
				const int r = (i0 + i) * 4 + rr;
				const int row = ew.row0 + r;
				const bool on = r < rows && left > 0;
				if (MODE == TC_RELU && p.relu_mask_out)
				{
					// one bit per output: what the error propagation needs of this layer's activations
					unsigned bits = 0u;
#pragma unroll
					for (int k = 0; k < 4; ++k)
						if (f(v[i][k], 0.0f) != 0.0f) bits |= 1u << (ch * 4 + k);
					bits |= __shfl_xor_sync(0xffffffffu, bits, 1);
					bits |= __shfl_xor_sync(0xffffffffu, bits, 2);
					bits |= __shfl_xor_sync(0xffffffffu, bits, 4);
					if (ch == 0 && on) p.relu_mask_out[(long long)row * p.mask_ld + (col >> 5)] = bits;
				}
				if (MODE == TC_ERR_MASK)
				{
					const unsigned bits = __float_as_uint(side[i].x);
#pragma unroll
					for (int k = 0; k < 4; ++k) v[i][k] = (bits >> k) & 1u ? v[i][k] : 0.0f;
				}
				else if (MODE == TC_STORE || MODE == TC_UPDATE)
				{
#pragma unroll
					for (int k = 0; k < 4; ++k) v[i][k] = f(v[i][k], ct[k]);
				}
				else
				{
					v[i][0] = f(v[i][0], side[i].x);
					v[i][1] = f(v[i][1], side[i].y);
					v[i][2] = f(v[i][2], side[i].z);
					v[i][3] = f(v[i][3], side[i].w);
				}
				if (!on) continue;
				if (MODE == TC_UPDATE)
				{
					// the update itself: W -= C * inv_mb, and the new weights' two parts for the next products
					float* wp = p.W + (long long)row * p.N + col;
					v[i][0] = side[i].x - v[i][0] * p.inv_mb; v[i][1] = side[i].y - v[i][1] * p.inv_mb;
					v[i][2] = side[i].z - v[i][2] * p.inv_mb; v[i][3] = side[i].w - v[i][3] * p.inv_mb;
					if (w16) *reinterpret_cast<float4*>(wp) = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
					else
#pragma unroll
						for (int k = 0; k < 4; ++k)
							if (k < left) wp[k] = v[i][k];
#pragma unroll
					for (int k = 0; k < 4; ++k)
						if (k < left && !isfinite(v[i][k])) bad = true;
				}
				if (left < 4)
#pragma unroll
					for (int k = 1; k < 4; ++k)
						if (k >= left) v[i][k] = 0.0f;  // padding columns of the split output stay zero
				if (MODE != TC_STORE && MODE != TC_UPDATE && p.Clo32)
					*reinterpret_cast<float4*>(p.Clo32 + (long long)row * p.ldc + col) =
					    make_float4(tf32_lo(v[i][0]), tf32_lo(v[i][1]), tf32_lo(v[i][2]), tf32_lo(v[i][3]));
				if (MODE == TC_UPDATE && p.Clo32)
				{
					if (w16)
						*reinterpret_cast<float4*>(p.Clo32 + (long long)row * p.N + col) =
						    make_float4(tf32_lo(v[i][0]), tf32_lo(v[i][1]), tf32_lo(v[i][2]), tf32_lo(v[i][3]));
					else
#pragma unroll
						for (int k = 0; k < 4; ++k)
							if (k < left) p.Clo32[(long long)row * p.N + col + k] = tf32_lo(v[i][k]);
				}
				if (stats) m = fmaxf(fmaxf(m, fmaxf(finite_abs(v[i][0]), finite_abs(v[i][1]))), fmaxf(finite_abs(v[i][2]), finite_abs(v[i][3])));
				if (split)
				{
					const long long at = (long long)row * p.ldch + col;
					*reinterpret_cast<uint2*>(p.Chi + at) = make_uint2(hi_pair(v[i][0], v[i][1], so), hi_pair(v[i][2], v[i][3], so));
					*reinterpret_cast<uint2*>(p.Clo + at) = make_uint2(lo_pair(v[i][0], v[i][1], so), lo_pair(v[i][2], v[i][3], so));
				}
				if ((MODE == TC_ERR_MASK || MODE == TC_ERR_ACT) && p.dsum) d += ((double)v[i][0] + (double)v[i][1]) + ((double)v[i][2] + (double)v[i][3]);
				if (MODE != TC_UPDATE && p.c_mode)
				{
					float* cp = p.C + (long long)row * p.ldc + col;
					if (c16 && left >= 4)
						*reinterpret_cast<float4*>(cp) = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
					else
#pragma unroll
						for (int k = 0; k < 4; ++k)
							if (k < left) cp[k] = v[i][k];
				}
			}
		}
		__syncwarp();  // the area is rewritten by the next piece
	}
	if (stats) merge_amax(&p.csc->amax, m);
	if ((MODE == TC_ERR_MASK || MODE == TC_ERR_ACT) && p.dsum)
	{
		d = warp_sum_d(d);
		if (ew.lane == 0) p.dsum[block_index] = d;
	}
	if (MODE == TC_UPDATE && bad) atomicOr(p.bad_flag, 1);
}

template <int EC, int MODE>
__device__ __forceinline__ void finish_block(float (&acc)[EC], const EpiWarp& ew, const TcParams& p, float inv1, float inv2, float so,
                                             long long block_index)
{
	const float par = p.par;
	const int act = p.act;
	if (MODE == TC_STORE || MODE == TC_UPDATE)
	{
		const float alpha = p.alpha;  // 1 for a plain product
		block_rows<EC, MODE>(acc, ew, p, inv1, inv2, so, block_index, [=](float g, float ct) { return alpha * g + ct; });
	}
	else if (MODE == TC_ERR_MASK)
		block_rows<EC, MODE>(acc, ew, p, inv1, inv2, so, block_index, [](float e, float) { return e; });
	else if (MODE == TC_ERR_ACT)
	{
		if (act == GL_ACT_TANH || act == GL_ACT_TANHP)
			block_rows<EC, MODE>(acc, ew, p, inv1, inv2, so, block_index, [](float e, float a) { return e * (1.0f - a * a); });
		else
			block_rows<EC, MODE>(acc, ew, p, inv1, inv2, so, block_index, [=](float e, float a) { return e * act_der_b(a, act, par); });
	}
	else
	{
		const float bias = p.bias_ptr ? *p.bias_ptr : 0.0f;
		if (MODE == TC_RELU)
			block_rows<EC, MODE>(acc, ew, p, inv1, inv2, so, block_index, [=](float z, float) { z += bias; return z < GL_OUTLIER ? 0.0f : z; });
		else if (act == GL_ACT_TANH)
			block_rows<EC, MODE>(acc, ew, p, inv1, inv2, so, block_index, [=](float z, float) { return tanhf(z + bias); });
		else if (act == GL_ACT_SIGMOID)
			block_rows<EC, MODE>(acc, ew, p, inv1, inv2, so, block_index, [=](float z, float) { return 1.0f / (1.0f + expf(-(z + bias))); });
		else if (act == GL_ACT_SOFTMAX)
			block_rows<EC, MODE>(acc, ew, p, inv1, inv2, so, block_index, [=](float z, float) { return z + bias; });
		else
			block_rows<EC, MODE>(acc, ew, p, inv1, inv2, so, block_index, [=](float z, float) { return squash_b(z + bias, act, par); });
	}
}

// ---- the split of a partial wave of tiles along k (TcWork) ---------------------------------------------------------
// A partial goes to the CTA's workspace slot: of a warp's 32 x EC block, piece v = columns 4v..4v+3 of the 32 rows (one float4
// per lane), so every store instruction of the warp writes 512 contiguous bytes.
template <int BN, int EC>
__device__ __forceinline__ void send_partial(const float (&acc)[EC], const TcParams& p, int w, int lane)
{
	float4* ws = reinterpret_cast<float4*>(p.sk_work + (size_t)blockIdx.x * (TC_BM * BN) + (size_t)w * (32 * EC));
#pragma unroll
	for (int v = 0; v < EC / 4; ++v) ws[v * 32 + lane] = make_float4(acc[4 * v], acc[4 * v + 1], acc[4 * v + 2], acc[4 * v + 3]);
	__threadfence();
	__syncwarp();
	if (lane == 0)
		asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p.sk_flags + (size_t)blockIdx.x * 8 + w), "r"(p.sk_epoch) : "memory");
}
// The tile's finisher: the rest of tile t's k-blocks were computed by the next CTAs as their first items; their partials
// are added in CTA order.  False when a (bounded) wait for one ran out.
template <int BN, int EC>
__device__ __forceinline__ bool add_partials(float (&acc)[EC], const TcParams& p, const TcWork& work, int t, int KB, int w, int lane,
                                             volatile int* abort_flag)
{
	const int tile_end = (t - work.full + 1) * KB;
	for (int j = blockIdx.x + 1; j < (int)gridDim.x && work.share_begin(j) < tile_end; ++j)
	{
		if (work.share_begin(j + 1) <= work.share_begin(j)) continue;  // an empty share
		const unsigned* flag = p.sk_flags + (size_t)j * 8 + w;
		unsigned seen;
		const long long t0 = clock64();
		for (;;)
		{
			asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(flag) : "memory");
			if (seen == p.sk_epoch) break;
			if (*abort_flag || clock64() - t0 > TC_WAIT_CYCLES)
			{
				*abort_flag = 1;
				atomicExch(p.err_flag, 5);
				return false;
			}
		}
		const float4* ws = reinterpret_cast<const float4*>(p.sk_work + (size_t)j * (TC_BM * BN) + (size_t)w * (32 * EC));
#pragma unroll
		for (int v = 0; v < EC / 4; ++v)
		{
			const float4 w4 = __ldcg(ws + v * 32 + lane);
			acc[4 * v] += w4.x;
			acc[4 * v + 1] += w4.y;
			acc[4 * v + 2] += w4.z;
			acc[4 * v + 3] += w4.w;
		}
	}
	return true;
}

// ---- data-parallel weight gradient (TcPeer) ------------------------------------------------------------------------
// Origin of tile t.  The tiles are walked owner band by owner band, m-fastest inside a band, and every rank starts with
// the band of the rank after it.  At any moment the ranks of the group therefore store into different owners, so no owner's
// NVLink ingress carries more than one sender's stream (all ranks walking the bands in the same order would aim all their
// stores at the same owner at once).  This rank's own band comes last: its stores are local.
__device__ __forceinline__ void peer_tile_origin(const TcPeer& peer, const TcParams& p, int bn, int t, int& m0, int& n0)
{
	const int band_mt = peer.band_rows / TC_BM;
	const int nbands = (p.tiles_m + band_mt - 1) / band_mt;
	for (int s = 0; s < nbands; ++s)
	{
		const int band = (peer.self + 1 + s) % nbands;
		const int mt_in = min(band_mt, p.tiles_m - band * band_mt);
		const int cnt = mt_in * p.tiles_n;
		if (t < cnt)
		{
			m0 = (band * band_mt + t % mt_in) * TC_BM;
			n0 = (t / mt_in) * bn;
			return;
		}
		t -= cnt;
	}
	m0 = 0;  // not reached: t < tiles_m * tiles_n
	n0 = 0;
}

// A finished block: its rows lie inside one owner's band (bands are whole tiles) and leave as bulk tensor stores into the
// owner's memory, so the warp does not wait for NVLink.
template <int EC>
__device__ __forceinline__ void send_block(const float (&acc)[EC], EpiWarp& ew, const TcParams& p, float inv1, float inv2, const TcPeer& peer, int m0)
{
	const int owner = m0 / peer.band_rows;
	const int y = ew.row0 - owner * peer.band_rows;
	const float alpha = p.alpha;
	if (ew.row0 >= p.M) return;
#pragma unroll
	for (int piece = 0; piece < EC / 32; ++piece)
	{
		const int col = ew.col0 + piece * 32;
		if (col >= p.N) break;
		const uint32_t area = piece_begin(ew);
#pragma unroll
		for (int v = 0; v < 8; ++v)
		{
			float o[4];
#pragma unroll
			for (int k = 0; k < 4; ++k)
			{
				const int c = col + v * 4 + k;
				o[k] = alpha * (acc[piece * 32 + v * 4 + k] * inv1 * inv2) + (p.colterm && c < p.N ? p.colterm[c] : 0.0f);
			}
			piece_put(ew, area, v, o[0], o[1], o[2], o[3]);
		}
		piece_store(ew, area, peer.maps + owner, col, y);
	}
}

// ---- host side, shared by the launches of both products ----
int tc_mode(const TcGemmArgs& g);
void tc_fill_params(TcParams& p, const TcGemmArgs& g);
bool tc_fill_peer(TcPeer& peer, const TcGemmArgs& g);  // false: not a product that can be stored in bands

}  // namespace tc
}  // namespace glb
