// Batched mode for mid-size networks (weights of a few hundred KB: too large for one SM's shared
// memory, far too small to fill the GPU one layer product at a time): ONE cooperative launch trains
// n_epochs * windows, every SM working on every window, with two grid-wide barriers per window.
//
// Per window (aligned, `mb` rows, weights frozen inside it):
//   phase 1  a CTA takes groups of R = 2, 4, 8, 12 or 16 samples through the whole network: per layer a
//            [256 outputs] x [32 inputs] weight tile is staged in shared memory (a ring of bulk tensor copies, or of
//            4-byte asynchronous copies where rows do not start on 16-byte boundaries; from L2, the weights change every
//            window) and four warps accumulate up to four output nodes x R/2 rows per thread, k ascending; head (optional softmax,
//            output delta, cost / accuracy / argmax, one warp per sample); then the hidden deltas the same way with
//            neighbouring input nodes per thread over [32 outputs] x [256 inputs] tiles.  Activations and deltas of
//            the group go to a window-sized scratch in global memory (it stays in L2), the deltas times learning rate and c_j.
//   phase 2  the weights are cut into 16 x 32 tiles, one per CTA at a time: c_j * (lr * d_jo * a_ji + decay terms) is
//            summed over the window's samples, 8 of every 64 rows per warp, from rings of bulk tensor copies that every warp has to
//            itself; the warps' sums are added in warp order (deterministic), and W -= G / len applied in place; one CTA (the last one,
//            which has the fewest tiles) adds the CTAs' partial sums (cost, accuracy, scalar-bias deltas) in CTA order, a warp for each:
//            one warp for cost and accuracy took 8.4 k clocks of loads, longer than the tiles of a small network.
// What bounds it (32-256-256-1, windows of 1024 rows, clocks of 1.96 GHz per window): 17 tile steps of 900 clocks in phase 1 -- the loads of
// weights and activations from shared memory take 512 of them, the multiply-adds as many, and they do not overlap fully with one warp per
// scheduler; two per scheduler would double the loads -- head, activations, stores and latencies at the layers' ends 16 k, phase 2 13 k, two
// grid barriers 7 k.  55 k clocks, 81 k when a step ended in a block barrier, the block copied phase 2's stages by 16-byte
// asynchronous copies and every element's activation was a copy of its own of the code.
// Arithmetic = the batched mode of batched.cu / small_fused.cu (reference loop
// Networks/network.cpp:457-668 with aligned windows, frozen weights and a plain error sum); c_j is
// the closed form of the reference's intra-window momentum history (State/node.cpp:278-292).
#pragma nv_diag_suppress 177  // (this file is compiled in parts, see its end: each leaves functions of the others unused)
#include <cooperative_groups.h>
#include <type_traits>

#include "copy_ring.h"
#include "tc_device.cuh"

namespace cg = cooperative_groups;

namespace glb {
using namespace tc;
namespace {

constexpr int GF_THREADS = 256;
constexpr int GF_ROWS = 16;     // samples a CTA carries through the network together, at most
constexpr int GF_TILE = 256;    // weight tile: 256 output nodes x 32 inputs (forward), 32 output nodes x 256 inputs (deltas)
constexpr int GF_TO = 16, GF_TJ = 64;  // phase 2: weight tile 16 outputs x 32 inputs, 64 rows per stage
constexpr int GF_NS = 3;                // stages of the weight-tile ring (bulk tensor copies, 32 KB each)
constexpr int GF_STAGE = 32768;
constexpr int GF_SEQ_MAX = 704;         // weight tiles one sample group walks through, at most: 8 layers of at most 1024 nodes and 2^19 weights
                                        // have less than 64 + 8 * 37 forward and 64 + 7 * 37 back
static_assert(GF_TILE * 32 * 4 == GF_STAGE, "a stage holds one weight tile");
constexpr int GF_PART = 2 + GL_MAX_WEIGHT_LAYERS;  // doubles per CTA: cost, accuracy, bias-delta sums per layer

// ---- phase 2, asynchronous fill ------------------------------------------------------------------
// (For the cluster variant; grid_fused_kernel's own follows below.)
// One 16 x 32 tile of layer l's weights.  The window's deltas and activations reach shared memory through a ring
// of GF_P2_STAGES 64-row stages filled by 16-byte cp.async copies (zero-filled outside the window or the layer):
// all stages but one are in flight while that one is consumed, so a step no longer waits one L2 round trip (the former
// global -> registers -> shared memory fill with one step of prefetch did: 16 steps x 1.2 us per tile).
// Lane = 4 outputs x 4 inputs (four output groups x eight input groups: 16 multiply-adds per two 16-byte loads),
// warp w takes rows 8w..8w+7 of every stage; the eight warps' partial sums are added in warp order and the update
// is applied in place.  Deterministic; the sum is no longer one chain in row order.
constexpr int GF_P2_TI = 32;
constexpr int GF_P2_STAGES = 6;   // tile path: five stages in flight while one is consumed
constexpr int GF_P2N_STAGES = 4;  // narrow-layer path (its stages are larger)
constexpr int GF_P2_STAGE_FLOATS = GF_TJ * GF_TO + GF_TJ * GF_P2_TI + GF_TJ;          // deltas, activations, momentum weights
constexpr int GF_P2_FLOATS = GF_P2_STAGES * GF_P2_STAGE_FLOATS + 8 * GF_TO * GF_P2_TI;  // + the warps' partial sums
static_assert(GF_P2_FLOATS * 4 <= GF_NS * GF_STAGE, "the phase-2 stages live inside the weight-tile ring");
static_assert((GF_P2_STAGE_FLOATS * 4) % 16 == 0, "stages keep the 16-byte alignment of the vector loads");

__device__ __forceinline__ void gf_grad_tile_async(const GridFusedArgs& a, int l, int o0, int i0, int len, int pitch, int off_in,
                                                   int off_out, float* stages, const float* ckl, float inv_len, int& bad)
{
	const NetView& n = a.net;
	const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
	const int ni = n.sizes[l], no = n.sizes[l + 1];
	const float lr = n.lr[l], w1 = n.wd1[l] * lr, w2 = n.wd2[l] * lr;
	const bool decay = w1 != 0.0f || w2 != 0.0f;
	const int og = lane >> 3, ig = lane & 7;
	float* red = stages + GF_P2_STAGES * GF_P2_STAGE_FLOATS;
	const uint32_t st_addr = smem_u32(stages);
	float g[4][4];
#pragma unroll
	for (int x = 0; x < 4; ++x)
#pragma unroll
		for (int y = 0; y < 4; ++y) g[x][y] = 0.0f;
	const int steps = (len + GF_TJ - 1) / GF_TJ;
	// one 16-byte copy of deltas and two of activations per thread and stage (the scratch rows and the layers'
	// first columns are 16-byte aligned), one 4-byte copy of a momentum weight for the first 64 threads
	const int d_jj = t >> 2, d_x = (t & 3) << 2;
	auto issue = [&](int s) {
		if (s < steps)
		{
			const int jb = s * GF_TJ;
			const int jn = (len - jb) < GF_TJ ? (len - jb) : GF_TJ;
			const uint32_t base = st_addr + (uint32_t)((s % GF_P2_STAGES) * GF_P2_STAGE_FLOATS * 4);
			{
				const int left = (d_jj < jn) ? no - (o0 + d_x) : 0;
				cp_async16(base + (uint32_t)t * 16, left > 0 ? a.delbuf + (size_t)(jb + d_jj) * pitch + off_out + o0 + d_x : a.delbuf, left);
			}
#pragma unroll
			for (int k = 0; k < 2; ++k)
			{
				const int e = t + k * GF_THREADS, jj = e >> 3, x = (e & 7) << 2;
				const int left = (jj < jn) ? ni - (i0 + x) : 0;
				cp_async16(base + (uint32_t)(GF_TJ * GF_TO * 4) + (uint32_t)e * 16,
				           left > 0 ? a.actbuf + (size_t)(jb + jj) * pitch + off_in + i0 + x : a.actbuf, left);
			}
			if (t < GF_TJ)
			{
				const bool ok = t < jn;
				cp_async4(base + (uint32_t)(GF_TJ * GF_TO + GF_TJ * GF_P2_TI + t) * 4, ok ? ckl + (len - (jb + t)) : ckl, ok);
			}
		}
		cp_async_commit();  // one group per step, empty ones included: the wait counts groups
	};
	__syncthreads();  // the previous work item no longer reads the stages
#pragma unroll
	for (int s = 0; s < GF_P2_STAGES - 1; ++s) issue(s);
	for (int s = 0; s < steps; ++s)
	{
		cp_async_wait<GF_P2_STAGES - 2>();  // this thread's copies of stage s have landed
		__syncthreads();                    // everybody's have; and stage s - 1 is no longer read
		issue(s + GF_P2_STAGES - 1);        // refills the stage consumed in the previous step
		const float* Dt = stages + (s % GF_P2_STAGES) * GF_P2_STAGE_FLOATS;
		const float* At = Dt + GF_TJ * GF_TO;
		const float* Ct = At + GF_TJ * GF_P2_TI;
#pragma unroll 4
		for (int q = 0; q < 8; ++q)
		{
			const int jj = warp * 8 + q;  // rows beyond the window hold zeros
			const float4 dv = *reinterpret_cast<const float4*>(Dt + jj * GF_TO + og * 4);
			const float4 av = *reinterpret_cast<const float4*>(At + jj * GF_P2_TI + ig * 4);
			const float c = Ct[jj];
			const float d4[4] = {dv.x, dv.y, dv.z, dv.w};
			const float a4[4] = {av.x, av.y, av.z, av.w};
			if (!decay)
			{
				// c_j * lr * d_jo first (rounded as the staged fill used to round it), then one multiply-add per weight
#pragma unroll
				for (int x = 0; x < 4; ++x)
				{
					const float dx = d4[x] * lr * c;
#pragma unroll
					for (int y = 0; y < 4; ++y) g[x][y] = fmaf(dx, a4[y], g[x][y]);
				}
			}
			else
			{
				float dec[4];
#pragma unroll
				for (int y = 0; y < 4; ++y) dec[y] = fmaf(w1, fabsf(a4[y]), w2 * a4[y]);
#pragma unroll
				for (int x = 0; x < 4; ++x)
#pragma unroll
					for (int y = 0; y < 4; ++y) g[x][y] = fmaf(c, fmaf(lr * d4[x], a4[y], dec[y]), g[x][y]);
			}
		}
	}
	cp_async_wait<0>();
	// the warps' partial sums: red[warp][output 0..15][input 0..31] (not part of the stages)
#pragma unroll
	for (int x = 0; x < 4; ++x)
		*reinterpret_cast<float4*>(red + warp * (GF_TO * GF_P2_TI) + (og * 4 + x) * GF_P2_TI + ig * 4) = make_float4(g[x][0], g[x][1], g[x][2], g[x][3]);
	__syncthreads();
#pragma unroll
	for (int k = 0; k < GF_TO * GF_P2_TI / GF_THREADS; ++k)
	{
		const int e = t + k * GF_THREADS;
		const int o = o0 + e / GF_P2_TI, i = i0 + (e & (GF_P2_TI - 1));
		float sum = red[e];
#pragma unroll
		for (int w = 1; w < 8; ++w) sum += red[w * (GF_TO * GF_P2_TI) + e];
		if (o < no && i < ni)
		{
			float* wp = n.W[l] + (size_t)o * ni + i;
			const float wv = __ldcg(wp) - sum * inv_len;
			if (!isfinite(wv)) bad = 1;
			*wp = wv;
		}
	}
}


// The same for a layer with at most GF_NARROW output nodes (the usual regression head): one work item per GF_NCOLS
// input columns, the same ring of 64-row stages (activations [64][64], deltas [64][4], momentum weights [64]);
// thread = one column and the rows 16p..16p+15 of every stage (p = thread / 64); the four parts are added in fixed
// order through shared memory.
constexpr int GF_NARROW = 4;
constexpr int GF_NCOLS = 64;
constexpr int GF_P2N_STAGE_FLOATS = GF_TJ * GF_NCOLS + GF_TJ * GF_NARROW + GF_TJ;
constexpr int GF_P2N_FLOATS = GF_P2N_STAGES * GF_P2N_STAGE_FLOATS + GF_THREADS * GF_NARROW;
static_assert(GF_P2N_FLOATS * 4 <= GF_NS * GF_STAGE, "the narrow-layer stages live inside the weight-tile ring");
constexpr int GF_P2_MAX_FLOATS = GF_P2N_FLOATS > GF_P2_FLOATS ? GF_P2N_FLOATS : GF_P2_FLOATS;
__device__ __forceinline__ void gf_grad_narrow(const GridFusedArgs& a, int l, int i0, int len, int pitch, int off_in, int off_out,
                                               const float* ckl, float inv_len, float* stages, int& bad)
{
	const NetView& n = a.net;
	const int t = threadIdx.x;
	const int ni = n.sizes[l], no = n.sizes[l + 1];
	const int col = t & (GF_NCOLS - 1), part = t / GF_NCOLS;  // 4 parts
	const int i = i0 + col;
	const float lr = n.lr[l], w1 = n.wd1[l] * lr, w2 = n.wd2[l] * lr;
	float* red = stages + GF_P2N_STAGES * GF_P2N_STAGE_FLOATS;
	const uint32_t st_addr = smem_u32(stages);
	float g[GF_NARROW];
#pragma unroll
	for (int o = 0; o < GF_NARROW; ++o) g[o] = 0.0f;
	const int steps = (len + GF_TJ - 1) / GF_TJ;
	auto issue = [&](int s) {
		if (s < steps)
		{
			const int jb = s * GF_TJ;
			const int jn = (len - jb) < GF_TJ ? (len - jb) : GF_TJ;
			const uint32_t base = st_addr + (uint32_t)((s % GF_P2N_STAGES) * GF_P2N_STAGE_FLOATS * 4);
#pragma unroll
			for (int k = 0; k < 4; ++k)
			{
				const int e = t + k * GF_THREADS, jj = e >> 4, x = (e & 15) << 2;
				const int left = (jj < jn) ? ni - (i0 + x) : 0;
				cp_async16(base + (uint32_t)e * 16, left > 0 ? a.actbuf + (size_t)(jb + jj) * pitch + off_in + i0 + x : a.actbuf, left);
			}
			if (t < GF_TJ)
			{
				const int left = (t < jn) ? no : 0;
				cp_async16(base + (uint32_t)(GF_TJ * GF_NCOLS * 4) + (uint32_t)t * 16, left > 0 ? a.delbuf + (size_t)(jb + t) * pitch + off_out : a.delbuf,
				           left);
			}
			else if (t < 2 * GF_TJ)
			{
				const int r = t - GF_TJ;
				const bool ok = r < jn;
				cp_async4(base + (uint32_t)(GF_TJ * GF_NCOLS + GF_TJ * GF_NARROW + r) * 4, ok ? ckl + (len - (jb + r)) : ckl, ok);
			}
		}
		cp_async_commit();
	};
	__syncthreads();  // the previous work item no longer reads the stages
#pragma unroll
	for (int s = 0; s < GF_P2N_STAGES - 1; ++s) issue(s);
	for (int s = 0; s < steps; ++s)
	{
		cp_async_wait<GF_P2N_STAGES - 2>();
		__syncthreads();
		issue(s + GF_P2N_STAGES - 1);
		const float* At = stages + (s % GF_P2N_STAGES) * GF_P2N_STAGE_FLOATS;
		const float* Dt = At + GF_TJ * GF_NCOLS;
		const float* Ct = Dt + GF_TJ * GF_NARROW;
#pragma unroll 4
		for (int q = 0; q < GF_TJ / 4; ++q)
		{
			const int jj = part * (GF_TJ / 4) + q;  // rows beyond the window hold zeros (c = 0)
			const float av = At[jj * GF_NCOLS + col];
			const float4 dv = *reinterpret_cast<const float4*>(Dt + jj * GF_NARROW);
			const float c = Ct[jj];
			const float dec = fmaf(w1, fabsf(av), w2 * av);
			const float d4[4] = {dv.x, dv.y, dv.z, dv.w};
#pragma unroll
			for (int o = 0; o < GF_NARROW; ++o) g[o] = fmaf(c, fmaf(lr * d4[o], av, dec), g[o]);
		}
	}
	cp_async_wait<0>();
#pragma unroll
	for (int o = 0; o < GF_NARROW; ++o) red[(part * GF_NCOLS + col) * GF_NARROW + o] = g[o];
	__syncthreads();
	if (part == 0 && i < ni)
	{
#pragma unroll
		for (int o = 0; o < GF_NARROW; ++o)
			if (o < no)
			{
				float sum = red[col * GF_NARROW + o];
				for (int p2 = 1; p2 < GF_THREADS / GF_NCOLS; ++p2) sum += red[(p2 * GF_NCOLS + col) * GF_NARROW + o];
				float* wp = n.W[l] + (size_t)o * ni + i;
				const float w = __ldcg(wp) - sum * inv_len;
				if (!isfinite(w)) bad = 1;
				*wp = w;
			}
	}
}

// ---- phase 2 of grid_fused_kernel ------------------------------------------------------------------
// The same sums in the same order (rows 8w..8w+7 of every 64-row stage are warp w's chain, the warps' sums are added in warp order),
// but every warp fetches the rows of its own chain, by bulk tensor copies of two stages (16 rows) each into a ring of its own, so that no
// barrier of the block stands between two stages; and the factors that do not depend on the weight (learning rate and, without
// decay, the momentum weight) are multiplied into the deltas when phase 1 writes them.  18 instructions per row and warp, of which two are
// loads of two clocks each (the functions above take 27, three loads of seven clocks, three asynchronous copies per thread and stage with
// their addresses, and two barriers' worth of waits per stage).
constexpr int GF_P2S = 3;                                // copies in flight per warp; of a narrow layer's larger ones: two
constexpr int GF_P2_BYTES = 16 * (GF_P2_TI + GF_TO) * 4;   // activations [2][8][32], deltas [2][8][16]
constexpr int GF_P2N_BYTES = 32 * (32 + GF_NARROW) * 4;    // activations [2][16][32], deltas [2][16][4]
constexpr int GF_P2_RED = 8 * GF_P2S * GF_P2_BYTES, GF_P2N_RED = 8 * 2 * GF_P2N_BYTES;  // behind the stages: the warps' partial sums
static_assert(GF_P2_RED + 8 * GF_TO * GF_P2_TI * 4 <= GF_NS * GF_STAGE, "stages and the warps' sums live inside the weight-tile ring");
static_assert(GF_P2N_RED + GF_THREADS * GF_NARROW * 4 <= GF_NS * GF_STAGE, "so do a narrow layer's");

struct GfP2
{
	const CUtensorMap* maps;  // of the scratch, see GridFusedArgs::window_maps
	uint8_t* ring;
	uint64_t* bars;           // [8 warps][GF_P2S]
	int* abort_flag;
	int* err;
	CopyRing<GF_P2S> copies;  // of the warp; its lane 0 asks
	__device__ __forceinline__ uint32_t bar(unsigned stage) const { return smem_u32(bars + (threadIdx.x >> 5) * GF_P2S + stage); }
	__device__ __forceinline__ void wait(int s, int depth)
	{
		copies.await(
		    s, depth, [&](unsigned stage, unsigned parity) { return mbar_wait(bar(stage), parity, abort_flag, err, 31); },
		    [&](unsigned lo, unsigned hi) { mbar_drain<GF_P2S>(bar(0), lo, hi); });
	}
	__device__ __forceinline__ uint32_t arm(unsigned stage, uint32_t bytes)
	{
		mbar_expect_tx(bar(stage), bytes);
		return bar(stage);
	}
};

// One 16 x 32 tile of layer l's weights.  `between` runs after the first copies have been asked for.
template <typename Between>
__device__ __forceinline__ void gf_grad_tile(const GridFusedArgs& a, GfP2& q, int l, int o0, int i0, int len, int off_in, int off_out, float inv_len,
                                             int& bad, Between between)
{
	const NetView& n = a.net;
	const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
	const int ni = n.sizes[l], no = n.sizes[l + 1], steps = (len + 2 * GF_TJ - 1) / (2 * GF_TJ);
	uint8_t* const stages = q.ring + warp * (GF_P2S * GF_P2_BYTES);
	auto issue = [&](int s, unsigned stage) {
		const uint32_t dst = smem_u32(stages) + (uint32_t)(s % GF_P2S) * GF_P2_BYTES, b = q.arm(stage, GF_P2_BYTES);
		tma_load_4d(dst, q.maps, b, off_in + i0, 0, warp, 2 * s);
		tma_load_4d(dst + 16 * GF_P2_TI * 4, q.maps + 1, b, off_out + o0, 0, warp, 2 * s);
	};
	q.copies.begin(steps);
	if (lane == 0) q.copies.start(GF_P2S, issue);
	float w[2];
#pragma unroll
	for (int k = 0; k < 2; ++k)
	{
		const int e = t + k * GF_THREADS, o = o0 + e / GF_P2_TI, i = i0 + (e & (GF_P2_TI - 1));
		w[k] = o < no && i < ni ? __ldcg(n.W[l] + (size_t)o * ni + i) : 0.0f;
	}
	between();
	// lane: outputs 4 og + {0..3}, inputs 4 ig + {0..3}, neighbouring lanes with the same inputs
	const int og = ((lane >> 3) & 2) | (lane & 1), ig = (lane >> 1) & 7;
	f32x2 g[4][2];
#pragma unroll
	for (int x = 0; x < 4; ++x) g[x][0] = g[x][1] = pair2(0.0f, 0.0f);
	const float w1 = n.wd1[l] * n.lr[l], w2 = n.wd2[l] * n.lr[l];
	const bool decay = w1 != 0.0f || w2 != 0.0f;
	const float* ckl = a.ck + (size_t)l * (n.mb + 1);
	for (int s = 0; s < steps; ++s)
	{
		q.wait(s, GF_P2S);
		const float* At = reinterpret_cast<const float*>(stages + (s % GF_P2S) * GF_P2_BYTES) + ig * 4;
		const float* Dt = reinterpret_cast<const float*>(stages + (s % GF_P2S) * GF_P2_BYTES) + 16 * GF_P2_TI + og * 4;
		int left = len - s * 2 * GF_TJ - warp * 8;  // rows from this warp's first one to the window's end
		auto row = [&](int r) {
			const float4 av = *reinterpret_cast<const float4*>(At + r * GF_P2_TI), dv = *reinterpret_cast<const float4*>(Dt + r * GF_TO);
			const f32x2 a01 = pair2(av.x, av.y), a23 = pair2(av.z, av.w);
			const float d[4] = {dv.x, dv.y, dv.z, dv.w};
#pragma unroll
			for (int x = 0; x < 4; ++x)
			{
				const f32x2 d2 = pair2(d[x], d[x]);
				g[x][0] = fma2(d2, a01, g[x][0]);
				g[x][1] = fma2(d2, a23, g[x][1]);
			}
		};
		// the two stages' rows; what lies behind the window's last row is another window's
#pragma unroll
		for (int h = 0; h < 2; ++h, At += 8 * GF_P2_TI, Dt += 8 * GF_TO, left -= GF_TJ)
		{
			if (!decay && left >= 8)
			{
#pragma unroll
				for (int r = 0; r < 8; ++r) row(r);
				continue;
			}
#pragma unroll 1
			for (int r = 0; r < 8 && r < left; ++r)
			{
				if (!decay)
				{
					row(r);
					continue;
				}
				const float4 av = *reinterpret_cast<const float4*>(At + r * GF_P2_TI), dv = *reinterpret_cast<const float4*>(Dt + r * GF_TO);
				const float c = __ldg(ckl + (left - r));
				const float a4[4] = {av.x, av.y, av.z, av.w}, d4[4] = {dv.x, dv.y, dv.z, dv.w};
				float dec[4];
#pragma unroll
				for (int y = 0; y < 4; ++y) dec[y] = fmaf(w1, fabsf(a4[y]), w2 * a4[y]);
#pragma unroll
				for (int x = 0; x < 4; ++x)
#pragma unroll
					for (int y = 0; y < 2; ++y)
					{
						float lo, hi;
						unpair2(g[x][y], lo, hi);
						g[x][y] = pair2(fmaf(c, fmaf(d4[x], a4[2 * y], dec[2 * y]), lo), fmaf(c, fmaf(d4[x], a4[2 * y + 1], dec[2 * y + 1]), hi));
					}
			}
		}
		__syncwarp();
		if (lane == 0) q.copies.refill(s, GF_P2S, issue);
	}
	q.copies.end(steps);
	// the warps' partial sums: red[warp][output 0..15][input 0..31]
	float* red = reinterpret_cast<float*>(q.ring + GF_P2_RED);
	__syncthreads();  // (the previous tile's have been added)
#pragma unroll
	for (int x = 0; x < 4; ++x)
	{
		float4 v;
		unpair2(g[x][0], v.x, v.y);
		unpair2(g[x][1], v.z, v.w);
		*reinterpret_cast<float4*>(red + warp * (GF_TO * GF_P2_TI) + (og * 4 + x) * GF_P2_TI + ig * 4) = v;
	}
	__syncthreads();
#pragma unroll
	for (int k = 0; k < 2; ++k)
	{
		const int e = t + k * GF_THREADS, o = o0 + e / GF_P2_TI, i = i0 + (e & (GF_P2_TI - 1));
		float sum = red[e];
#pragma unroll
		for (int v = 1; v < 8; ++v) sum += red[v * (GF_TO * GF_P2_TI) + e];
		if (o < no && i < ni)
		{
			const float wv = w[k] - sum * inv_len;
			if (!isfinite(wv)) bad = 1;
			n.W[l][(size_t)o * ni + i] = wv;
		}
	}
}

// Layers with at most GF_NARROW output nodes: 64 input columns per work item, thread = one column and the rows 16p..16p+15 of every
// 64-row stage (p = thread / 64); the four parts are added in order.
template <int NO, typename Between>
__device__ __forceinline__ void gf_grad_columns(const GridFusedArgs& a, GfP2& q, int l, int i0, int len, int off_in, int off_out, float inv_len,
                                                int& bad, Between between)
{
	constexpr int S = 2;
	const NetView& n = a.net;
	const int t = threadIdx.x, lane = t & 31, warp = t >> 5, part = t / GF_NCOLS, col = t & (GF_NCOLS - 1), i = i0 + col;
	const int ni = n.sizes[l], steps = (len + 2 * GF_TJ - 1) / (2 * GF_TJ);
	uint8_t* const stages = q.ring + warp * (S * GF_P2N_BYTES);
	auto issue = [&](int s, unsigned stage) {
		const uint32_t dst = smem_u32(stages) + (uint32_t)(s % S) * GF_P2N_BYTES, b = q.arm(stage, GF_P2N_BYTES);
		tma_load_4d(dst, q.maps + 2, b, off_in + i0 + 32 * (warp & 1), 0, 2 * part, 2 * s);
		tma_load_4d(dst + 32 * 128, q.maps + 3, b, off_out, 0, 2 * part, 2 * s);
	};
	q.copies.begin(steps);
	if (lane == 0) q.copies.start(S, issue);
	float w[NO], g[NO];
#pragma unroll
	for (int o = 0; o < NO; ++o)
	{
		w[o] = part == 0 && i < ni ? __ldcg(n.W[l] + (size_t)o * ni + i) : 0.0f;
		g[o] = 0.0f;
	}
	between();
	const float w1 = n.wd1[l] * n.lr[l], w2 = n.wd2[l] * n.lr[l];
	const float* ckl = a.ck + (size_t)l * (n.mb + 1);
	for (int s = 0; s < steps; ++s)
	{
		int left = len - s * 2 * GF_TJ - part * 16;  // rows from this part's first one to the window's end
		// lane k: the momentum weight of row k of the 32
		const int j = (lane & 15) + (lane >> 4) * GF_TJ;
		const float ck = j < left ? __ldg(ckl + (left - j)) : 0.0f;
		q.wait(s, S);
		const float* At = reinterpret_cast<const float*>(stages + (s % S) * GF_P2N_BYTES) + lane;
		const float* Dt = reinterpret_cast<const float*>(stages + (s % S) * GF_P2N_BYTES) + 32 * 32;
#pragma unroll 1
		for (int h = 0; h < 2; ++h, At += 16 * 32, Dt += 16 * GF_NARROW, left -= GF_TJ)
		{
			const float cr = h ? __shfl_down_sync(0xffffffffu, ck, 16) : ck;  // (lanes 0..15: the momentum weights of these rows)
			auto row = [&](int r, auto decay) {
				const float c = __shfl_sync(0xffffffffu, cr, r), av = At[r * 32];
				const float dec = decltype(decay)::value ? fmaf(w1, fabsf(av), w2 * av) : 0.0f;
#pragma unroll
				for (int o = 0; o < NO; ++o) g[o] = fmaf(c, decltype(decay)::value ? fmaf(Dt[r * GF_NARROW + o], av, dec) : Dt[r * GF_NARROW + o] * av, g[o]);
			};
			if (left >= 16 && w1 == 0.0f && w2 == 0.0f)
			{
#pragma unroll
				for (int r = 0; r < 16; ++r) row(r, std::false_type());
			}
			else
#pragma unroll 1
				for (int r = 0; r < 16 && r < left; ++r) row(r, std::true_type());
		}
		__syncwarp();
		if (lane == 0) q.copies.refill(s, S, issue);
	}
	q.copies.end(steps);
	float* red = reinterpret_cast<float*>(q.ring + GF_P2N_RED);
	__syncthreads();  // (the previous item's have been added)
#pragma unroll
	for (int o = 0; o < NO; ++o) red[(part * GF_NCOLS + col) * GF_NARROW + o] = g[o];
	__syncthreads();
	if (part == 0 && i < ni)
#pragma unroll
		for (int o = 0; o < NO; ++o)
		{
			float sum = red[col * GF_NARROW + o];
#pragma unroll
			for (int p = 1; p < GF_THREADS / GF_NCOLS; ++p) sum += red[(p * GF_NCOLS + col) * GF_NARROW + o];
			const float wv = w[o] - sum * inv_len;
			if (!isfinite(wv)) bad = 1;
			n.W[l][(size_t)o * ni + i] = wv;
		}
}

// The window scratch: one row per sample, layer l's nodes from column soff[l] on; every layer starts at a multiple
// of 4 columns and the pitch is one too, so that rows and layers are 16-byte aligned for the copies of phase 2.
__host__ __device__ inline int gf_scratch_layout(const NetView& n, int* soff)
{
	int c = 0;
	for (int l = 0; l <= n.H + 1; ++l)
	{
		soff[l] = c;
		c += (n.sizes[l] + 3) & ~3;
	}
	return c;
}

// The arithmetic of phase 1.  The first four warps compute, one per scheduler: a warp takes 16, 32 or 64 neighbouring nodes of a layer
// (of 256 at a time, gf_box), lane (g, h) = (lane / 2, lane % 2) 1, 2 or 4 of them and half of the group's rows.  Neighbouring lanes read the
// same weights, so that a 16-byte load costs two clocks (32 rows of weights, one per lane, cost four), and what the next four k need is
// read ahead of the current ones' multiply-adds.  Every sum is one chain, k ascending.  The warps wait for one another at the ends of layers
// only.
constexpr int GF_COMPUTE = 128;
__host__ __device__ inline int gf_box(int nodes) { return nodes <= 64 ? 16 : (nodes <= 128 ? 32 : 64); }
template <int R>
struct GfSums
{
	static constexpr int RT = R / 2, P = RT / 2;  // rows of a thread, pairs of them (R = 2: a single row)
	f32x2 p[4][P ? P : 1];
	float s[4];
	__device__ __forceinline__ void clear()
	{
#pragma unroll
		for (int j = 0; j < 4; ++j)
		{
			s[j] = 0.0f;
#pragma unroll
			for (int i = 0; i < P; ++i) p[j][i] = pair2(0.0f, 0.0f);
		}
	}
	__device__ __forceinline__ void add(int j, float w, const float (&x)[RT])
	{
		if (P == 0) s[j] = fmaf(w, x[0], s[j]);
		else
		{
			const f32x2 w2 = pair2(w, w);
#pragma unroll
			for (int i = 0; i < P; ++i) p[j][i] = fma2(w2, pair2(x[2 * i], x[RT > 1 ? 2 * i + 1 : 0]), p[j][i]);
		}
	}
	__device__ __forceinline__ float get(int j, int r) const
	{
		if (P == 0) return s[j];
		float lo, hi;
		unpair2(p[j][r >> 1], lo, hi);
		return (r & 1) ? hi : lo;
	}
};
template <int RT>
__device__ __forceinline__ void gf_rows(float (&x)[RT], const float* p)
{
	if (RT % 4 == 0)
#pragma unroll
		for (int i = 0; i < RT / 4; ++i) reinterpret_cast<float4*>(x)[i] = reinterpret_cast<const float4*>(p)[i];
	else if (RT % 2 == 0)
#pragma unroll
		for (int i = 0; i < RT / 2; ++i) reinterpret_cast<float2*>(x)[i] = reinterpret_cast<const float2*>(p)[i];
	else x[0] = p[0];
}
__device__ __forceinline__ void gf_quad(float (&x)[4], const float* p) { *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(p); }

// Forward: the nodes g + 16 j, j < NJ, over `lim` (at most 32) inputs; w: row g of the tile (128-byte rows, quads permuted by the
// row), x: the inputs' rows of this thread.
template <int R, int NJ>
__device__ __forceinline__ void gf_forward_tile(GfSums<R>& acc, const float* w, int sw, const float* x, int lim)
{
	constexpr int RT = R / 2, NB = R <= 8 ? 3 : 2;  // four k in use, the next four, and those after them where there are registers
	float u[NB][NJ][4], v[NB][4][RT];
	auto read = [&](int b, int c) {
#pragma unroll
		for (int j = 0; j < NJ; ++j) gf_quad(u[b][j], w + j * 16 * 32 + ((c ^ sw) << 2));
#pragma unroll
		for (int q = 0; q < 4; ++q) gf_rows<RT>(v[b][q], x + (4 * c + q) * R);
	};
	auto use = [&](int b) {
#pragma unroll
		for (int q = 0; q < 4; ++q)
#pragma unroll
			for (int j = 0; j < NJ; ++j) acc.add(j, u[b][j][q], v[b][q]);
	};
	if (lim == 32)
	{
#pragma unroll
		for (int c = 0; c < NB - 1; ++c) read(c, c);
#pragma unroll
		for (int c = 0; c < 8; ++c)
		{
			if (c + NB - 1 < 8) read((c + NB - 1) % NB, c + NB - 1);
			use(c % NB);
		}
		return;
	}
	// the layer's last tile: whole quads, then single k
	const int quads = lim >> 2;
#pragma unroll 1
	for (int c = 0; c < quads; ++c)
	{
		read(0, c);
		use(0);
	}
#pragma unroll 1
	for (int k = quads * 4; k < lim; ++k)
	{
		float z[RT];
		gf_rows<RT>(z, x + k * R);
#pragma unroll
		for (int j = 0; j < NJ; ++j) acc.add(j, w[j * 16 * 32 + (((k >> 2) ^ sw) << 2) + (k & 3)], z);
	}
}

// Deltas: the nodes NJ g + {0..NJ-1} over `lim` (at most 32) nodes of the layer above; w: column NJ g of the warp's part of the tile (rows
// of PITCH NJ), x: the deltas' rows of this thread.
template <int R, int NJ, int PITCH>
__device__ __forceinline__ void gf_delta_tile(GfSums<R>& acc, const float* w, const float* x, int lim)
{
	constexpr int RT = R / 2, NB = R <= 8 ? 3 : 2;
	float u[NB][4][NJ], v[NB][4][RT];
	auto read = [&](int b, int c) {
#pragma unroll
		for (int q = 0; q < 4; ++q)
		{
			gf_rows<NJ>(u[b][q], w + (4 * c + q) * PITCH * NJ);
			gf_rows<RT>(v[b][q], x + (4 * c + q) * R);
		}
	};
	auto use = [&](int b) {
#pragma unroll
		for (int q = 0; q < 4; ++q)
#pragma unroll
			for (int j = 0; j < NJ; ++j) acc.add(j, u[b][q][j], v[b][q]);
	};
	if (lim == 32)
	{
#pragma unroll
		for (int c = 0; c < NB - 1; ++c) read(c, c);
#pragma unroll
		for (int c = 0; c < 8; ++c)
		{
			if (c + NB - 1 < 8) read((c + NB - 1) % NB, c + NB - 1);
			use(c % NB);
		}
		return;
	}
	const int quads = lim >> 2;
#pragma unroll 1
	for (int c = 0; c < quads; ++c)
	{
		read(0, c);
		use(0);
	}
#pragma unroll 1
	for (int k = quads * 4; k < lim; ++k)
	{
		float y[NJ], z[RT];
		gf_rows<NJ>(y, w + k * PITCH * NJ);
		gf_rows<RT>(z, x + k * R);
#pragma unroll
		for (int j = 0; j < NJ; ++j) acc.add(j, y[j], z);
	}
}

// USE_TMA: the weight tiles arrive in the ring by bulk tensor copies (a.tma != NULL), which the fifth warp asks for, else by 4-byte
// asynchronous ones of four more warps, one for each computing warp's nodes.  Two instantiations rather than a run-time flag: each
// carries one tile path only, which halves the body the instruction cache has to hold.
template <bool USE_TMA, int R>
__global__ void __launch_bounds__(GF_THREADS, 1) grid_fused_kernel(const __grid_constant__ GridFusedArgs a)
{
	extern __shared__ __align__(16) float sm[];
	cg::grid_group grid = cg::this_grid();
	const NetView& n = a.net;
	const int H = n.H;
	const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
	const int cw = warp & 3, tg = lane >> 1, th = lane & 1;  // the computing warp that this one is or copies for
	const bool computes = warp < 4;
	constexpr int RT = R / 2;
	const int n_out = n.sizes[H + 1];
	const int mb = n.mb;

	// layer l's nodes start at node_off[l], a multiple of 4, in shared memory and in the window scratch alike
	// (tot = the scratch's pitch); the few padding nodes are carried along and never read as values
	int node_off[GL_MAX_WEIGHT_LAYERS + 2];
	const int tot = gf_scratch_layout(n, node_off);
	// shared memory: activations [tot][R] | deltas [tot][R] | per-row metric scratch | tile list |
	// weight-tile ring (phase 2 reuses it for its stages)
	float* As = sm;
	float* Ds = As + (size_t)tot * R;
	float* rowm = Ds + (size_t)tot * R;  // [R][2]: cost, accuracy of the group's rows
	unsigned* seq = reinterpret_cast<unsigned*>(rowm + 2 * R);  // [GF_SEQ_MAX]: tensor map | x << 8 | y << 20 of a group's weight tiles
	// weight tiles: a ring of GF_NS stages (1024-byte aligned for the 128-byte swizzle) filled by bulk tensor copies, or --
	// where the weights' layout does not allow tensor maps -- in the same layout by 4-byte asynchronous copies
	// A narrow output layer (at most GF_NARROW nodes: the usual regression head) does not go through weight tiles --
	// a [256 outputs] x [32 inputs] tile would carry one useful row and leave 255 threads idle for n_in / 32
	// steps.  Its few weight rows are copied to shared memory once per window (wn); the forward product splits the
	// inputs over the threads and adds the partial sums in a fixed order, the hidden deltas read wn directly.
	const bool narrow_head = n.sizes[H + 1] <= GF_NARROW && H >= 1;
	float* wn = reinterpret_cast<float*>(seq + GF_SEQ_MAX);          // [n_out][n_H]
	float* nred = wn + (narrow_head ? ((n.sizes[H + 1] * n.sizes[H] + 3) & ~3) : 0);  // [8 warps][R][GF_NARROW]
	uint8_t* ring_gen;
	{
		uint8_t* after = reinterpret_cast<uint8_t*>(nred + (narrow_head ? 8 * R * GF_NARROW : 0));
		const uint32_t au = smem_u32(after);
		ring_gen = after + (((au + 1023u) & ~1023u) - au);
	}
	__shared__ double s_part[GF_PART];
	__shared__ uint64_t full_bars[4][GF_NS], empty_bars[4][GF_NS], p2_bars[8][GF_P2S];
	__shared__ int gf_abort;
	__shared__ float sbias[GL_MAX_WEIGHT_LAYERS];             // the window's scalar biases
	__shared__ float scale[GL_MAX_WEIGHT_LAYERS + 1][GF_ROWS];  // momentum weights of the group's rows, by the layer below the delta
	constexpr bool use_tma = USE_TMA;
	const CUtensorMap* maps = reinterpret_cast<const CUtensorMap*>(a.tma);
	if (t == 0)
	{
		for (int w = 0; w < 4; ++w)
			for (int k = 0; k < GF_NS; ++k)
			{
				mbar_init(smem_u32(&full_bars[w][k]), use_tma ? 1 : 32);
				mbar_init(smem_u32(&empty_bars[w][k]), use_tma ? 4 : 1);  // (bulk copies: the first ones serve all four warps)
			}
		for (int w = 0; w < 8; ++w)
			for (int k = 0; k < GF_P2S; ++k) mbar_init(smem_u32(&p2_bars[w][k]), 1);
		gf_abort = 0;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	// the tile order of one group: forward layer by layer (output chunk, then input tile), then the hidden deltas from the top (input
	// chunk, then output tile).  map | k / 32 << 5 | chunk << 11
	int nsteps = 0, nforward = 0;  // weight tiles per sample group, those of the forward pass
	auto list = [&](int map, int nodes, int ks) {
		for (int c = 0; c * GF_TILE < nodes; ++c)
			for (int k = 0; k * 32 < ks; ++k, ++nsteps)
				if (t == 0) seq[nsteps] = (unsigned)map | (unsigned)k << 5 | (unsigned)c << 11;
	};
	for (int l = 0; l <= H - (narrow_head ? 1 : 0); ++l) list(2 * l, n.sizes[l + 1], n.sizes[l]);
	nforward = nsteps;
	for (int L = H + 1 - (narrow_head ? 1 : 0); L >= 2; --L) list(2 * (L - 1) + 1, n.sizes[L - 1], n.sizes[L]);
	// optional phase timing (diagnostics): CTA 0, thread 0 adds up the nanoseconds of
	// [phase 1, barrier, phase 2, barrier] in a.timing[0..3]
	const bool timed = a.timing != nullptr && blockIdx.x == 0 && t == 0;
	unsigned long long tm[16] = {}, t_a = 0, t_b = 0, t_c = 0, t_d = 0;
	// tm[9..14]: inside phase 1 -- waits for weight tiles, (unused), forward, head, deltas, tail
	auto now = []() {
		unsigned long long v;
		asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(v));
		return v;
	};

	unsigned cs = 0;       // computing warps: tiles consumed so far
	CopyRing<GF_NS> tiles_asked;                // who fetches tiles (each a run of one copy)
	int p_at = 0, p_left = 0, group_left = 0;  // position in the list, tiles of the window and of the group left
	// A copying warp's tiles lie in its quarter of the stage, one behind the other in rows of its own nodes: the computing warps need not be
	// at the same tile.  A bulk copy's rows hold the nodes of all four.
	constexpr int PITCH = use_tma ? 64 : 16;
	const bool fetches = use_tma ? warp == 4 && lane == 0 : !computes;
	bool dead = false;     // a bounded wait ran out: stop waiting, finish the launch
	auto drain_tiles = [&](unsigned lo, unsigned hi) { mbar_drain<GF_NS>(smem_u32(&full_bars[0][0]), lo, hi); };
	// up to `most` more tiles of the current group; each waits for the tile three before it to be read
	auto fetch_tiles = [&](int most) {
		for (; most > 0 && group_left > 0; --most, --group_left, --p_left)
		{
			auto read = [&](unsigned stage, unsigned parity) { return mbar_wait(smem_u32(&empty_bars[use_tma ? 0 : cw][stage]), parity, &gf_abort, a.flags + 1, 32); };
			// (plain copies arm nothing: the lanes' arrivals complete a barrier's phases in whatever order they come)
			const unsigned ps = tiles_asked.base;
			if (use_tma && !tiles_asked.may_ask(read, drain_tiles)) return;
			if (!use_tma && ps >= GF_NS && !dead && !read(ps % GF_NS, (ps / GF_NS - 1) & 1u)) dead = true;
			const unsigned e = seq[p_at], st = ps % GF_NS;
			if (++p_at == nsteps) p_at = 0;
			uint64_t* const full = &full_bars[use_tma ? 0 : cw][st];
			const int l = (int)(e & 31) >> 1, ni = n.sizes[l], no = n.sizes[l + 1];
			const int k = (int)(e >> 5 & 63) * 32, chunk = (int)(e >> 11) * GF_TILE;
			const uint32_t dst = smem_u32(ring_gen) + st * GF_STAGE + (use_tma ? 0 : cw * (GF_STAGE / 4));
			if (use_tma)
			{
				mbar_expect_tx(smem_u32(full), (uint32_t)gf_box((e & 1) ? ni : no) * 512);
				tma_load_2d(dst, maps + (e & 31), smem_u32(full), (e & 1) ? chunk : k, (e & 1) ? k : chunk);
			}
			else
			{
				if ((e & 1) == 0)
				{
					// rows of 32 inputs, quads permuted by the row as the bulk copies leave them (what lies outside the matrix is not read)
					const int box = gf_box(no), node = chunk + cw * box, rows = no - node < box ? no - node : box;
					const float* src = n.W[l] + (size_t)node * ni + k + lane;
					if (k + lane < ni)
#pragma unroll 4
						for (int r = 0; r < rows; ++r, src += ni)
							cp_async4(dst + (uint32_t)r * 128 + (uint32_t)(((lane >> 2) ^ (r & 7)) << 4) + (uint32_t)(lane & 3) * 4, src, true);
				}
				else
				{
					// 32 rows of `box` nodes
					const int box = gf_box(ni), node = chunk + cw * box, rows = no - k < 32 ? no - k : 32;
					const float* src = n.W[l] + (size_t)k * ni + node;
					const int c0 = box == 16 ? lane & 15 : lane, r0 = box == 16 ? lane >> 4 : 0, dr = box == 16 ? 2 : 1;
					for (int c = c0; c < box; c += 32)
						if (node + c < ni)
#pragma unroll 4
							for (int r = r0; r < rows; r += dr) cp_async4(dst + (uint32_t)(r * box + c) * 4, src + (size_t)r * ni + c, true);
				}
				asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(full)) : "memory");
			}
			tiles_asked.end(1);
		}
	};
	auto next_group = [&]() {
		group_left = p_left < nsteps ? p_left : nsteps;
		fetch_tiles(GF_NS);
	};
	auto acquire = [&]() -> const float* {
		unsigned long long t0 = 0;
		if (timed) t0 = now();
		if (!dead && !mbar_wait(smem_u32(&full_bars[use_tma ? 0 : cw][cs % GF_NS]), (cs / GF_NS) & 1u, &gf_abort, a.flags + 1, 30)) dead = true;
		if (timed) tm[9] += now() - t0;
		return reinterpret_cast<const float*>(ring_gen + (cs % GF_NS) * GF_STAGE + (use_tma ? 0 : cw * (GF_STAGE / 4)));
	};
	auto release = [&]() {
		__syncwarp();
		// (a lane whose wait ran out has not seen the copy land, and does not give its stage back)
		if (lane == 0 && !dead) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&empty_bars[use_tma ? 0 : cw][cs % GF_NS])) : "memory");
		++cs;
	};
	auto sync_computing = [&]() { asm volatile("barrier.cta.sync 1, %0;" ::"n"(GF_COMPUTE) : "memory"); };

	// a.ck[l][k] = sum_{q<k} m_l^q: the weight of a sample with k samples of its window still to come (itself
	// included); made once on the host, [H+1][mb+1], read by phase 2 straight from global memory

	const bool classify = n.out_type != GL_OUT_REGRESSION;
	const bool softmax = n.act[H] == GL_ACT_SOFTMAX;
	const float data_size = a.data_size;

	// phase-2 tile list: layer l has ceil(no/16) * ceil(ni/32) tiles
	const int tile_i = GF_P2_TI;
	int tile_off[GL_MAX_WEIGHT_LAYERS + 1];
	int tiles = 0;
	for (int l = 0; l <= H; ++l)
	{
		tile_off[l] = tiles;
		tiles += (n.sizes[l + 1] <= GF_NARROW) ? (n.sizes[l] + GF_NCOLS - 1) / GF_NCOLS
		                                       : ((n.sizes[l + 1] + GF_TO - 1) / GF_TO) * ((n.sizes[l] + tile_i - 1) / tile_i);
	}
	tile_off[H + 1] = tiles;

	// the CTA that adds up the scalars: the last one, which has the fewest tiles; where all have as many, one whose tiles are not a narrow
	// layer's (they take a little longer, and lie at the end)
	const int acc_warp = H < GF_THREADS / 32 - 1 ? GF_THREADS / 32 - 1 : 0;  // (warps 1..H have the biases)
	const unsigned scalar_cta = tiles % (int)gridDim.x == 0 ? 0u : gridDim.x - 1;
	GfP2 p2 = {reinterpret_cast<const CUtensorMap*>(a.window_maps), ring_gen, &p2_bars[0][0], &gf_abort, a.flags + 1, {}};
	// a group's inputs, transposed to [node][row]; rows outside the window are zeros
	auto fetch_inputs = [&](long long first, int valid) {
		const uint32_t dst = smem_u32(As);
		for (int r = warp; r < R; r += GF_THREADS / 32)
		{
			const float* src = a.X + (r < valid ? (first + r) * n.sizes[0] : 0);
			for (int i = lane; i < n.sizes[0]; i += 32) cp_async4(dst + (uint32_t)(i * R + r) * 4, src + i, r < valid);
		}
		cp_async_commit();
	};
	bool fetched = false;  // the first group's inputs are on their way already

	int bad = 0;
	for (int ep = 0; ep < a.n_epochs; ++ep)
	{
		const bool last_epoch = ep == a.n_epochs - 1;
		double ecost = 0.0, eacc = 0.0;  // scalar_cta, warp 0 and acc_warp
		for (long long r0 = 0; r0 < a.rows; r0 += mb)
		{
			const int len = (int)((a.rows - r0) < mb ? (a.rows - r0) : mb);
			const int groups = (len + R - 1) / R;
			if (t < GF_PART) s_part[t] = 0.0;
			if (ep == 0 && r0 == 0) __syncthreads();  // (the list of tiles and the barriers are complete)
			{
				// this window's tiles: nsteps per group of this CTA; nobody runs ahead into the next window, whose weights do not
				// exist yet
				const int mine = (groups > (int)blockIdx.x) ? (groups - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
				p_left = mine * nsteps;
				p_at = 0;
				if (fetches)
				{
					if (use_tma) asm volatile("fence.proxy.async;" ::: "memory");  // (the weights were written through the generic proxy)
					next_group();
				}
			}
			if (t >= 1 && t <= H) sbias[t] = __ldcg(n.bias + t);  // visible after the group's first barrier
			if (narrow_head)
				for (int e = t; e < n.sizes[H + 1] * n.sizes[H]; e += GF_THREADS) wn[e] = __ldcg(n.W[H] + e);  // visible after the group's first barrier
			if (timed) t_a = now();
			// ================= phase 1: forward, head, deltas, R samples at a time
			for (int gidx = blockIdx.x; gidx < groups; gidx += gridDim.x)
			{
				const int j0 = gidx * R;
				const int valid = (len - j0) < R ? (len - j0) : R;
				if (timed) t_c = now();
				__syncthreads();
				if (!fetched) fetch_inputs(r0 + j0, valid);
				fetched = false;
				if (t < (H + 1) * R)
				{
					const int l = t / R, r = t - l * R;
					scale[l][r] = r < valid ? __ldg(a.ck + (size_t)l * (mb + 1) + (len - (j0 + r))) : 0.0f;
				}
				cp_async_wait<0>();
				__syncthreads();
				const int wide = H - (narrow_head ? 1 : 0);
				if (computes)
					for (int l = 0; l <= wide; ++l)
					{
						const int ni = n.sizes[l], no = n.sizes[l + 1], box = gf_box(no);
						const float* in = As + (size_t)node_off[l] * R + th * RT;
						const float b = (l >= 1) ? sbias[l] : 0.0f;
						const int act = n.act[l];
						const float par = n.par[l];
						for (int chunk = 0; chunk < no; chunk += GF_TILE)
						{
							const int o0 = chunk + cw * box;  // (a warp without nodes here takes part in the tiles' barriers)
							GfSums<R> acc;
							acc.clear();
							for (int i0 = 0; i0 < ni; i0 += 32)
							{
								// tile rows = this warp's output nodes, 32 inputs each, 16-byte chunks XOR-swizzled by the row
								const float* w = acquire() + (use_tma ? cw * box + tg : tg) * 32;
								unsigned long long tq = 0;
								if (timed) tq = now();
								const float* x = in + (size_t)i0 * R;
								const int lim = ni - i0 < 32 ? ni - i0 : 32;
								if (o0 >= no) ;
								else if (box == 64) gf_forward_tile<R, 4>(acc, w, tg & 7, x, lim);
								else if (box == 32) gf_forward_tile<R, 2>(acc, w, tg & 7, x, lim);
								else gf_forward_tile<R, 1>(acc, w, tg & 7, x, lim);
								if (timed) { tm[15] += now() - tq; tm[8] += 1; }
								release();
							}
							float* const out = As + (size_t)(node_off[l + 1] + o0 + tg) * R + th * RT;
							auto put = [&](auto f) {
#pragma unroll
								for (int j = 0; j < 4; ++j)
									if (16 * j < box && o0 + tg + 16 * j < no)
#pragma unroll
										for (int r = 0; r < RT; ++r) out[j * 16 * R + r] = f(acc.get(j, r) + b);
							};
							// (what costs a few instructions from registers; the others in one short loop, whose code is fetched once)
							if (act == GL_ACT_RELU) put([](float z) { return z < GL_OUTLIER ? 0.0f : z; });
							else if (act == GL_ACT_SOFTMAX) put([](float z) { return z; });
							else
							{
								put([](float z) { return z; });
#pragma unroll 4
								for (int e = 0; e < box / 16 * RT; ++e)
								{
									const int j = e / RT, r = e - j * RT;
									if (o0 + tg + 16 * j < no) out[j * 16 * R + r] = squash_b(out[j * 16 * R + r], act, par);
								}
							}
						}
						sync_computing();  // the next layer reads these outputs
					}
				else if (fetches)
					// the rest of the forward tiles, and as many of the deltas' as the ring has room for when those have been read (one more
					// would wait for the head, which waits for this warp)
					fetch_tiles(nforward + GF_NS - (nsteps - group_left));
				__syncthreads();
				if (narrow_head)
				{
					const int ni = n.sizes[H], no = n_out;
					const float* in = As + (size_t)node_off[H] * R;
					float* out = As + (size_t)node_off[H + 1] * R;
					const float b = sbias[H];
					const int act = n.act[H];
					const float par = n.par[H];
					// (row r, input class q): inputs i = q, q + 32, ...; the sums of classes 4k..4k+3 are added as (0 + 1) + (2 + 3) by
					// neighbouring lanes, the eight sums of four through shared memory in class order
					for (int u = t; u < 32 * R; u += GF_THREADS)
					{
						const int q = (u & 3) + 4 * (u / (4 * R)), r = (u >> 2) % R;
						for (int o = 0; o < no; ++o)
						{
							float s = 0.0f;
#pragma unroll 4
							for (int i = q; i < ni; i += 32) s = fmaf(wn[o * ni + i], in[(size_t)i * R + r], s);
							s += __shfl_xor_sync(0xffffffffu, s, 1);
							s += __shfl_xor_sync(0xffffffffu, s, 2);
							if ((q & 3) == 0) nred[((q >> 2) * R + r) * GF_NARROW + o] = s;
						}
					}
					__syncthreads();
					if (t < R * no)
					{
						const int rr = t % R, o = t / R;
						float z = nred[rr * GF_NARROW + o];
						for (int w = 1; w < 8; ++w) z += nred[(w * R + rr) * GF_NARROW + o];
						out[(size_t)o * R + rr] = squash_b(z + b, act, par);
					}
					__syncthreads();
				}
				if (timed) { t_d = now(); tm[11] += t_d - t_c; t_c = t_d; }
				// ---- head: a warp per sample of the group
				for (int r = warp; r < R; r += GF_THREADS / 32)
				{
					float* p = As + (size_t)node_off[H + 1] * R + r;   // stride R
					float* dout = Ds + (size_t)node_off[H + 1] * R + r;
					float c_acc = 0.0f, a_acc = 0.0f, be = 0.0f, bp = 0.0f;
					int ie = -1, ip = -1;
					if (r < valid)
					{
						const float* y = a.Y + (r0 + j0 + r) * n_out;
						float mx = -INFINITY, inv_den = 1.0f;
						if (softmax)
						{
							for (int o = lane; o < n_out; o += 32) mx = fmaxf(mx, p[(size_t)o * R]);
							mx = warp_max(mx);
							float den = 0.0f;
							for (int o = lane; o < n_out; o += 32) den += expf(p[(size_t)o * R] - mx);
							inv_den = 1.0f / warp_sum(den);
						}
						for (int o = lane; o < n_out; o += 32)
						{
							float pv = p[(size_t)o * R];
							const float e = y[o];
							float cost, d;
							if (softmax)
							{
								pv = expf(pv - mx) * inv_den;
								p[(size_t)o * R] = pv;
								cost = (e != 0.0f) ? -(e * logf(pv)) / data_size : 0.0f;
								d = pv - e;
							}
							else if (n.out_type == GL_OUT_REGRESSION)
							{
								const float tt = e - pv;
								cost = tt * tt / data_size;
								d = 2.0f * (pv - e);
							}
							else if (n.out_type == GL_OUT_CLASSIFICATION)
							{
								cost = -((e * logf(pv)) + ((1.0f - e) * logf(1.0f - pv))) / data_size;
								d = (pv - e) / ((1.0f - pv) * pv);
							}
							else
							{
								cost = logf(e / pv) / data_size;
								d = -(e / pv);
							}
							dout[(size_t)o * R] = d;
							c_acc += cost;
							a_acc += fmaxf((1.0f - fminf(fabsf(pv - e), 1.0f)) * 100.0f, 0.0f);
							if (e > be) { be = e; ie = o; }
							if (pv > bp) { bp = pv; ip = o; }
						}
						c_acc = warp_sum(c_acc);
						a_acc = warp_sum(a_acc);
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
						if (lane == 0 && classify && last_epoch && ie >= 0 && ip >= 0) atomicAdd(a.confusion + ie * n_out + ip, 1);
						if (a.last_out && last_epoch && r0 + j0 + r == a.rows - 1)
							for (int o = lane; o < n_out; o += 32) a.last_out[o] = p[(size_t)o * R];
					}
					else
					{
						for (int o = lane; o < n_out; o += 32) dout[(size_t)o * R] = 0.0f;
					}
					if (lane == 0)
					{
						rowm[2 * r] = c_acc;
						rowm[2 * r + 1] = a_acc;
					}
				}
				__syncthreads();
				if (timed) { t_d = now(); tm[12] += t_d - t_c; t_c = t_d; }
				// ---- hidden deltas: D_l = (D_{l+1} W_l) * act'(A_l)
				if (narrow_head)
				{
					// D_H = (D_out W_H) * act'(A_H) from the shared copy of the head's weights
					const int ni = n.sizes[H], no = n_out, act = n.act[H - 1];
					const float* dup = Ds + (size_t)node_off[H + 1] * R;
#pragma unroll 1
					for (int i = t; i < ni; i += GF_THREADS)
					{
						const size_t at = (size_t)(node_off[H] + i) * R;
						float v[R], s[R];
						gf_rows<R>(v, As + at);
#pragma unroll
						for (int r = 0; r < R; ++r) s[r] = 0.0f;
#pragma unroll 1
						for (int o = 0; o < no; ++o)
						{
							const float w = wn[o * ni + i];
							float d[R];
							gf_rows<R>(d, dup + o * R);
#pragma unroll
							for (int r = 0; r < R; ++r) s[r] = fmaf(w, d[r], s[r]);
						}
						auto put = [&](auto f) {
#pragma unroll
							for (int r = 0; r < R; ++r) Ds[at + r] = r < valid ? s[r] * f(v[r]) : 0.0f;
						};
						if (act == GL_ACT_RELU) put([](float x) { return x > 0.0f ? 1.0f : 0.0f; });
						else if (act == GL_ACT_TANH || act == GL_ACT_TANHP) put([](float x) { return 1.0f - x * x; });
						else if (act == GL_ACT_SIGMOID || act == GL_ACT_SIGMOIDP) put([](float x) { return x * (1.0f - x); });
						else put([act](float x) { return act_der_b(x, act, 0.01f); });
					}
					__syncthreads();
				}
				// the group's activations to the window scratch ([row][node])
				auto store_activations = [&](int first, int step) {
#pragma unroll 1
					for (int e = first; e < tot; e += step)
					{
						float v[R];
						gf_rows<R>(v, As + (size_t)e * R);
						float* to = a.actbuf + (size_t)j0 * tot + e;
#pragma unroll
						for (int r = 0; r < R; ++r)
							if (r < valid) to[(size_t)r * tot] = v[r];
					}
				};
				if (computes)
					for (int L = wide + 1; L >= 2; --L)
					{
						const int l = L - 1;
						const int ni = n.sizes[l], no = n.sizes[L], box = gf_box(ni), nj = box / 16;
						const float* dup = Ds + (size_t)node_off[L] * R + th * RT;
						const int act = n.act[l - 1];
						for (int chunk = 0; chunk < ni; chunk += GF_TILE)
						{
							const int i0 = chunk + cw * box;
							GfSums<R> acc;
							acc.clear();
							for (int o0 = 0; o0 < no; o0 += 32)
							{
								// tile rows = 32 nodes of the layer above, columns = this warp's nodes
								const float* w = acquire() + (use_tma ? cw * box : 0) + nj * tg;
								const float* x = dup + (size_t)o0 * R;
								const int lim = no - o0 < 32 ? no - o0 : 32;
								if (i0 >= ni) ;
								else if (box == 64) gf_delta_tile<R, 4, PITCH>(acc, w, x, lim);
								else if (box == 32) gf_delta_tile<R, 2, PITCH>(acc, w, x, lim);
								else gf_delta_tile<R, 1, PITCH>(acc, w, x, lim);
								release();
							}
							if (i0 >= ni) continue;
							const size_t at = (size_t)(node_off[l] + i0 + nj * tg) * R + th * RT;
							auto put = [&](auto f) {
								// (all loads ahead of the stores, which the compiler cannot tell apart)
								float v[4][RT];
#pragma unroll
								for (int j = 0; j < 4; ++j)
									if (j < nj) gf_rows<RT>(v[j], As + at + j * R);
#pragma unroll
								for (int j = 0; j < 4; ++j)
									if (j < nj && i0 + nj * tg + j < ni)
#pragma unroll
										for (int r = 0; r < RT; ++r) Ds[at + j * R + r] = (th * RT + r < valid) ? acc.get(j, r) * f(v[j][r]) : 0.0f;
							};
							if (act == GL_ACT_RELU) put([](float v) { return v > 0.0f ? 1.0f : 0.0f; });
							else if (act == GL_ACT_TANH || act == GL_ACT_TANHP) put([](float v) { return 1.0f - v * v; });
							else if (act == GL_ACT_SIGMOID || act == GL_ACT_SIGMOIDP) put([](float v) { return v * (1.0f - v); });
							else put([act](float v) { return act_der_b(v, act, 0.01f); });
						}
						sync_computing();  // the next layer reads these deltas
					}
				else
				{
					// (beside the deltas: these warps have nothing else to do)
					if (use_tma && warp > 4) store_activations(t - 160, 96);
					if (fetches)
					{
						// the rest of the group's tiles, and the first ones of the next group's
						fetch_tiles(nsteps);
						next_group();
					}
				}
				if (!use_tma && computes) store_activations(t, GF_COMPUTE);
				__syncthreads();
				if (timed) { t_d = now(); tm[13] += t_d - t_c; t_c = t_d; }
				// ---- the group's deltas to the window scratch, times what phase 2 wants of them; partial sums
				for (int L = 1; L <= H + 1; ++L)
				{
					const int nodes = n.sizes[L];
					const float lr = n.lr[L - 1];
					const bool whole = nodes > GF_NARROW && n.wd1[L - 1] * lr == 0.0f && n.wd2[L - 1] * lr == 0.0f;
#pragma unroll 1
					for (int e = t; e < nodes; e += GF_THREADS)
					{
						float v[R], c[R];
						gf_rows<R>(v, Ds + (size_t)(node_off[L] + e) * R);
						float* to = a.delbuf + (size_t)j0 * tot + node_off[L] + e;
						if (whole)
#pragma unroll
							for (int r = 0; r < R; ++r) c[r] = scale[L - 1][r];
#pragma unroll
						for (int r = 0; r < R; ++r) v[r] = whole ? v[r] * lr * c[r] : v[r] * lr;
#pragma unroll
						for (int r = 0; r < R; ++r)
							if (r < valid) to[(size_t)r * tot] = v[r];
					}
				}
				if (warp >= 1 && warp <= H)
				{
					// scalar-bias delta of hidden layer `warp`: sum of the deltas of the layer above, this group's rows
					const int l = warp, no = n.sizes[l + 1];
					double s0 = 0.0, s1 = 0.0;
					const float* d = Ds + (size_t)node_off[l + 1] * R;
#pragma unroll 4
					for (int e = lane; e < no * R; e += 64)
					{
						s0 += (double)d[e];
						s1 += e + 32 < no * R ? (double)d[e + 32] : 0.0;
					}
					const double s = warp_sum_d(s0 + s1);
					if (lane == 0) s_part[2 + l] += s;
				}
				if (t == 0)
				{
					for (int r = 0; r < valid; ++r)
					{
						s_part[0] += (double)rowm[2 * r];
						s_part[1] += (double)rowm[2 * r + 1];
					}
				}
			}
			__syncthreads();
			if (t < GF_PART) a.part[(size_t)blockIdx.x * GF_PART + t] = s_part[t];
			{
				// the next window's inputs travel under phase 2 (this window's are in the scratch)
				const long long next = r0 + mb < a.rows ? r0 + mb : 0;
				const int next_len = (int)((a.rows - next) < mb ? (a.rows - next) : mb), j0 = (int)blockIdx.x * R;
				if ((next || !last_epoch) && j0 < next_len)
				{
					fetch_inputs(next + j0, (next_len - j0) < R ? (next_len - j0) : R);
					fetched = true;
				}
			}
			if (timed) { t_b = now(); tm[0] += t_b - t_a; if (t_c) tm[14] += t_b - t_c; }
			grid.sync();
			if (timed) { t_a = now(); tm[1] += t_a - t_b; }

			// ================= phase 2: gradient + update per weight tile; the last CTA also the scalars
			// (the copies of this phase read through the asynchronous proxy what phase 1 wrote through the generic one)
			if (lane == 0) asm volatile("fence.proxy.async;" ::: "memory");
			const float inv_len = 1.0f / (float)len;
			bool scalars_due = blockIdx.x == scalar_cta;
			// this lane's CTAs' partial sums, in order; the loads of five CTAs at a time
			auto sum_parts = [&](double& sum, int which) {
				for (int b = lane; b < (int)gridDim.x; b += 160)
				{
					double v[5];
#pragma unroll
					for (int k = 0; k < 5; ++k) v[k] = b + 32 * k < (int)gridDim.x ? __ldcg(a.part + (size_t)(b + 32 * k) * GF_PART + which) : 0.0;
#pragma unroll
					for (int k = 0; k < 5; ++k) sum += v[k];
				}
			};
			auto scalars = [&]() {
				if (!scalars_due) return;
				scalars_due = false;
				if (warp >= 1 && warp <= H)
				{
					const int l = warp;
					double s = 0.0;
					sum_parts(s, 2 + l);
					s = warp_sum_d(s) * (double)n.lr[l];
					if (lane == 0)
					{
						const float nb = sbias[l] - ((a.bias_rule == GL_BIAS_REFERENCE) ? (float)(s * (double)n.sizes[l]) : (float)(s / (double)len));
						if (!isfinite(nb)) bad = 1;
						n.bias[l] = nb;
					}
				}
				// the CTAs' cost and accuracy partials: lanes stride over the CTAs, then a fixed shuffle tree; a warp for each, since the
				// loads' latency is what this costs
				for (int which = 0; which < 2; ++which)
					if (warp == (which ? acc_warp : 0))
					{
						double c = 0.0;
						sum_parts(c, which);
						c = warp_sum_d(c);
						if (which == 0) ecost += c;
						else eacc += c;
					}
			};
			for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x)
			{
				int l = 0;
				while (tile >= tile_off[l + 1]) ++l;
				const int tiles_i = (n.sizes[l] + tile_i - 1) / tile_i;
				const int tl = tile - tile_off[l];
				// the weight-tile ring is idle in this phase (every tile of the window has been consumed, the next
				// window's are issued after the grid barrier): it holds the stages
				const int in = node_off[l], above = node_off[l + 1], i0 = tl * GF_NCOLS;
				switch (n.sizes[l + 1])
				{
				case 1: gf_grad_columns<1>(a, p2, l, i0, len, in, above, inv_len, bad, scalars); break;
				case 2: gf_grad_columns<2>(a, p2, l, i0, len, in, above, inv_len, bad, scalars); break;
				case 3: gf_grad_columns<3>(a, p2, l, i0, len, in, above, inv_len, bad, scalars); break;
				case 4: gf_grad_columns<4>(a, p2, l, i0, len, in, above, inv_len, bad, scalars); break;
				default: gf_grad_tile(a, p2, l, (tl / tiles_i) * GF_TO, (tl % tiles_i) * tile_i, len, in, above, inv_len, bad, scalars); break;
				}
			}
			scalars();
			if (timed) { t_b = now(); tm[2] += t_b - t_a; }
			grid.sync();
			if (timed) { t_a = now(); tm[3] += t_a - t_b; }
		}
		if (blockIdx.x == scalar_cta && t == 0) a.epoch_sums[2 * ep] = ecost;
		if (blockIdx.x == scalar_cta && t == acc_warp * 32) a.epoch_sums[2 * ep + 1] = eacc;
	}
	if (use_tma && fetches) tiles_asked.finish(*(volatile int*)&gf_abort != 0, drain_tiles);  // (its readers may have given up behind its last tile)
	if (timed)
		for (int k = 0; k < 16; ++k) a.timing[k] += tm[k];
	if (bad) atomicOr(a.flags, 1);
}

#ifndef GF_KERNEL_ROWS
// =================================================================================================
// Cluster variant of the whole-window kernel.
//
// grid_fused_kernel's phase 1 is bound by how fast ONE SM gets the network's weights delivered: every CTA
// streams all of them per sample group.  Here a thread-block cluster of CF_CS CTAs carries CF_R rows through the
// network together and every CTA owns 1/CF_CS of each layer's NODES: it keeps the weight rows of its nodes
// (forward) and the weight columns of its nodes (hidden deltas) in shared memory for the whole window -- read
// from L2 once per window instead of once per sample group -- computes its nodes' activations for the
// CF_R rows and stores them into the activation buffers of all CF_CS CTAs over distributed shared memory
// (st.shared::cluster: plain stores), one cluster barrier per layer.  The head runs on every CTA's own
// copy (side effects from cluster rank 0 only).  Activations and deltas go to the same window scratch as in
// grid_fused_kernel, and phase 2 sums the window's rows per weight tile -- here with a 4 x 4 register tile per
// lane and the 64 rows of a step dealt over the eight warps, whose partial sums are added in warp order.
// Everything is deterministic.  All barriers are executed unconditionally by every thread of every CTA.
constexpr int CF_CS = 8;   // CTAs per cluster (the portable maximum)
constexpr int CF_R = 32;   // rows a cluster carries through the network together

struct CfPlan
{
	int tot;                                  // nodes of the network
	int node_off[GL_MAX_WEIGHT_LAYERS + 2];   // first node of layer j
	int sl[GL_MAX_WEIGHT_LAYERS + 2];         // nodes of layer j one CTA owns (a multiple of 4)
	int d_off[GL_MAX_WEIGHT_LAYERS + 2];      // first row of layer j's deltas in the delta buffer (j >= 1)
	int d_rows;                               // rows of the delta buffer (each layer rounded up to 4 nodes)
	int wf[GL_MAX_WEIGHT_LAYERS + 1];         // float offset of the forward slice of weight layer l
	int wb[GL_MAX_WEIGHT_LAYERS + 1];         // float offset of the delta slice of node layer j (1..H)
	int rowm;                                 // float offset of the per-row metric scratch
	int soff[GL_MAX_WEIGHT_LAYERS + 2];       // the window scratch: first column of layer j
	int pitch;                                // and its pitch
	int floats;                               // dynamic shared memory, floats
};

__host__ __device__ inline void cf_plan(const NetView& n, CfPlan& p)
{
	const int H = n.H;
	int tot = 0;
	for (int j = 0; j <= H + 1; ++j)
	{
		p.node_off[j] = tot;
		tot += n.sizes[j];
		p.sl[j] = (((n.sizes[j] + CF_CS - 1) / CF_CS) + 3) & ~3;
	}
	p.tot = tot;
	int dr = 0;
	p.d_off[0] = 0;
	for (int j = 1; j <= H + 1; ++j)
	{
		p.d_off[j] = dr;
		dr += (n.sizes[j] + 3) & ~3;
	}
	p.d_rows = dr;
	int f = (tot + dr) * CF_R;
	for (int l = 0; l <= H; ++l)
	{
		p.wf[l] = f;
		f += p.sl[l + 1] * (n.sizes[l] + 4);
	}
	p.wb[0] = 0;
	for (int j = 1; j <= H; ++j)
	{
		p.wb[j] = f;
		f += p.sl[j] * (((n.sizes[j + 1] + 3) & ~3) + 4);
	}
	p.rowm = f;
	f += 2 * CF_R;
	p.pitch = gf_scratch_layout(n, p.soff);
	p.floats = f > GF_P2_MAX_FLOATS ? f : GF_P2_MAX_FLOATS;  // the phase-2 stages alias the phase-1 buffers
}

__device__ __forceinline__ uint32_t cl_rank()
{
	uint32_t r;
	asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
	return r;
}
// every thread of every CTA of the cluster; orders shared::cluster stores before it against loads after it
__device__ __forceinline__ void cl_sync()
{
	asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cl_map(uint32_t local_addr, uint32_t rank)
{
	uint32_t r;
	asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(rank));
	return r;
}
__device__ __forceinline__ void cl_store4(uint32_t cluster_addr, float x, float y, float z, float w)
{
	asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

// s[q] = sum_k InT[k][4 * sq + q] * Wsl[n][k] (q = 0..3) for the CTA's `cnt` nodes n; InT is [K][CF_R], Wsl is
// [cnt][K + 4], K a multiple of 4.  Thread = one node and four rows (eight row quads x 32 nodes per pass); where
// the CTA owns at most 8 nodes a warp takes one node and its four lane groups a quarter of k each, added in
// lane-group order.  epi(n, sq, s0, s1, s2, s3) runs once per node and row quad.
template <typename Epi>
__device__ __forceinline__ void cf_product(const float* InT, int K, const float* Wsl, int cnt, Epi epi)
{
	const int t = threadIdx.x, sq = t & 7;
	const int ws = K + 4;
	const float* in = InT + 4 * sq;
	auto dot = [&](const float* w, int k0, int k1, float& a0, float& a1, float& a2, float& a3) {
#pragma unroll 2
		for (int k = k0; k < k1; k += 4)
		{
			const float4 wv = *reinterpret_cast<const float4*>(w + k);
			const float4 x0 = *reinterpret_cast<const float4*>(in + (size_t)(k + 0) * CF_R);
			const float4 x1 = *reinterpret_cast<const float4*>(in + (size_t)(k + 1) * CF_R);
			const float4 x2 = *reinterpret_cast<const float4*>(in + (size_t)(k + 2) * CF_R);
			const float4 x3 = *reinterpret_cast<const float4*>(in + (size_t)(k + 3) * CF_R);
			a0 = fmaf(wv.x, x0.x, a0); a1 = fmaf(wv.x, x0.y, a1); a2 = fmaf(wv.x, x0.z, a2); a3 = fmaf(wv.x, x0.w, a3);
			a0 = fmaf(wv.y, x1.x, a0); a1 = fmaf(wv.y, x1.y, a1); a2 = fmaf(wv.y, x1.z, a2); a3 = fmaf(wv.y, x1.w, a3);
			a0 = fmaf(wv.z, x2.x, a0); a1 = fmaf(wv.z, x2.y, a1); a2 = fmaf(wv.z, x2.z, a2); a3 = fmaf(wv.z, x2.w, a3);
			a0 = fmaf(wv.w, x3.x, a0); a1 = fmaf(wv.w, x3.y, a1); a2 = fmaf(wv.w, x3.z, a2); a3 = fmaf(wv.w, x3.w, a3);
		}
	};
	if (cnt <= 8)
	{
		const int n = t >> 5, kc = (t >> 3) & 3;
		const int chunk = (((K + 3) / 4) + 3) & ~3;
		float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
		if (n < cnt)
		{
			const int k0 = kc * chunk, k1 = (k0 + chunk) < K ? (k0 + chunk) : K;
			dot(Wsl + (size_t)n * ws, k0, k1, a0, a1, a2, a3);
		}
		// whole warps take part in the shuffles (n is uniform in a warp)
#pragma unroll
		for (int off = 8; off <= 16; off <<= 1)
		{
			a0 += __shfl_xor_sync(0xffffffffu, a0, off);
			a1 += __shfl_xor_sync(0xffffffffu, a1, off);
			a2 += __shfl_xor_sync(0xffffffffu, a2, off);
			a3 += __shfl_xor_sync(0xffffffffu, a3, off);
		}
		if (n < cnt && kc == 0) epi(n, sq, a0, a1, a2, a3);
		return;
	}
	for (int nb = 0; nb < cnt; nb += 32)
	{
		const int n = nb + (t >> 3);
		if (n < cnt)
		{
			float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
			dot(Wsl + (size_t)n * ws, 0, K, a0, a1, a2, a3);
			epi(n, sq, a0, a1, a2, a3);
		}
	}
}

__global__ void __launch_bounds__(GF_THREADS, 1) cluster_fused_kernel(const __grid_constant__ GridFusedArgs a)
{
	extern __shared__ __align__(16) float sm[];
	cg::grid_group grid = cg::this_grid();
	const NetView& n = a.net;
	const int H = n.H;
	const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
	const int n_out = n.sizes[H + 1];
	const int mb = n.mb;
	const int crank = (int)cl_rank();
	const int cid = (int)blockIdx.x / CF_CS, nclusters = (int)gridDim.x / CF_CS;
	__shared__ CfPlan P;
	__shared__ double s_part[GF_PART];
	if (t == 0) cf_plan(n, P);
	__syncthreads();
	const int tot = P.tot;
	const int pitch = P.pitch;
	float* AT = sm;                          // [tot][CF_R] activations, node-major
	float* DT = sm + (size_t)tot * CF_R;     // [d_rows][CF_R] deltas of node layers 1..H+1
	float* rowm = sm + P.rowm;               // [CF_R][2]: cost, accuracy of the pass's rows
	// the phase-2 stages alias the phase-1 region (the phases are separated by grid barriers)
	const uint32_t at_addr = smem_u32(AT), dt_addr = smem_u32(DT);

	const bool classify = n.out_type != GL_OUT_REGRESSION;
	const bool softmax = n.act[H] == GL_ACT_SOFTMAX;
	const float data_size = a.data_size;

	// phase-2 work items: layer l has ceil(no/16) * ceil(ni/32) tiles, or ceil(ni/64) column groups where no <= 4
	int tile_off[GL_MAX_WEIGHT_LAYERS + 2];
	int tiles = 0;
	for (int l = 0; l <= H; ++l)
	{
		tile_off[l] = tiles;
		tiles += (n.sizes[l + 1] <= GF_NARROW) ? (n.sizes[l] + GF_NCOLS - 1) / GF_NCOLS
		                                       : ((n.sizes[l + 1] + GF_TO - 1) / GF_TO) * ((n.sizes[l] + GF_P2_TI - 1) / GF_P2_TI);
	}
	tile_off[H + 1] = tiles;

	const bool timed = a.timing != nullptr && blockIdx.x == 0 && t == 0;
	unsigned long long tm[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, t_a = 0, t_b = 0, t_c = 0, t_d = 0;
	auto now = []() {
		unsigned long long v;
		asm volatile("mov.u64 %0, %%clock64;" : "=l"(v));
		return v;
	};

	cl_sync();  // every CTA of the cluster is running before the first store into its shared memory
	int bad = 0;
	for (int ep = 0; ep < a.n_epochs; ++ep)
	{
		const bool last_epoch = ep == a.n_epochs - 1;
		double ecost = 0.0, eacc = 0.0;  // CTA 0, thread 0
		for (long long r0 = 0; r0 < a.rows; r0 += mb)
		{
			const int len = (int)((a.rows - r0) < mb ? (a.rows - r0) : mb);
			const int passes = (len + CF_R - 1) / CF_R;
			if (t < GF_PART) s_part[t] = 0.0;
			if (timed) t_a = now();
			// ---- this window's weights of the CTA's nodes: rows of W_l (forward), columns of W_j (hidden deltas)
			for (int l = 0; l <= H; ++l)
			{
				const int K = n.sizes[l], nb0 = crank * P.sl[l + 1];
				int cnt = n.sizes[l + 1] - nb0;
				cnt = cnt < 0 ? 0 : (cnt > P.sl[l + 1] ? P.sl[l + 1] : cnt);
				const float* src = n.W[l] + (size_t)nb0 * K;
				float* dst = sm + P.wf[l];
				const int kq = K >> 2;
				for (int e = t; e < cnt * kq; e += GF_THREADS)
				{
					const int r = e / kq, k = (e - r * kq) << 2;
					*reinterpret_cast<float4*>(dst + (size_t)r * (K + 4) + k) = __ldcg(reinterpret_cast<const float4*>(src + (size_t)r * K + k));
				}
			}
			for (int j = 1; j <= H; ++j)
			{
				const int ni = n.sizes[j], no = n.sizes[j + 1], K4 = (no + 3) & ~3, i0 = crank * P.sl[j];
				int cnt = ni - i0;
				cnt = cnt < 0 ? 0 : (cnt > P.sl[j] ? P.sl[j] : cnt);
				const float* src = n.W[j] + i0;
				float* dst = sm + P.wb[j];
				for (int e = t; e < cnt * K4; e += GF_THREADS)
				{
					const int o = e / cnt, i = e - o * cnt;
					dst[(size_t)i * (K4 + 4) + o] = (o < no) ? __ldcg(src + (size_t)o * ni + i) : 0.0f;
				}
			}
			__syncthreads();
			if (timed) { t_c = now(); tm[4] += t_c - t_a; }
			// ================= phase 1: forward, head, deltas, CF_R rows per cluster pass
			for (int pass = cid; pass < passes; pass += nclusters)
			{
				const int j0 = pass * CF_R;
				const int valid = (len - j0) < CF_R ? (len - j0) : CF_R;
				{
					// inputs of the pass, transposed to [node][row]; every CTA reads them itself
					const int n0 = n.sizes[0], kq = n0 >> 2;
					for (int e = t; e < CF_R * kq; e += GF_THREADS)
					{
						const int r = e / kq, i = (e - r * kq) << 2;
						float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
						if (r < valid) v = *reinterpret_cast<const float4*>(a.X + (size_t)(r0 + j0 + r) * n0 + i);
						AT[(i + 0) * CF_R + r] = v.x;
						AT[(i + 1) * CF_R + r] = v.y;
						AT[(i + 2) * CF_R + r] = v.z;
						AT[(i + 3) * CF_R + r] = v.w;
					}
				}
				__syncthreads();
				for (int l = 0; l <= H; ++l)
				{
					const int nb0 = crank * P.sl[l + 1];
					int cnt = n.sizes[l + 1] - nb0;
					cnt = cnt < 0 ? 0 : (cnt > P.sl[l + 1] ? P.sl[l + 1] : cnt);
					const float b = (l >= 1) ? __ldcg(n.bias + l) : 0.0f;
					const int act = n.act[l];
					const float par = n.par[l];
					const int out_node = P.node_off[l + 1] + nb0, out_col = P.soff[l + 1] + nb0;
					const bool hidden = l < H;
					cf_product(AT + (size_t)P.node_off[l] * CF_R, n.sizes[l], sm + P.wf[l], cnt,
					           [&](int nn, int sq, float s0, float s1, float s2, float s3) {
						           const float v0 = squash_b(s0 + b, act, par), v1 = squash_b(s1 + b, act, par);
						           const float v2 = squash_b(s2 + b, act, par), v3 = squash_b(s3 + b, act, par);
						           const uint32_t local = at_addr + (uint32_t)(((out_node + nn) * CF_R + 4 * sq) * 4);
#pragma unroll
						           for (int dst = 0; dst < CF_CS; ++dst) cl_store4(cl_map(local, (uint32_t)dst), v0, v1, v2, v3);
						           if (hidden)
						           {
							           float* ga = a.actbuf + (size_t)(j0 + 4 * sq) * pitch + out_col + nn;
							           if (4 * sq + 0 < valid) ga[0] = v0;
							           if (4 * sq + 1 < valid) ga[(size_t)pitch] = v1;
							           if (4 * sq + 2 < valid) ga[(size_t)2 * pitch] = v2;
							           if (4 * sq + 3 < valid) ga[(size_t)3 * pitch] = v3;
						           }
					           });
					cl_sync();  // the layer's activations have landed in every CTA of the cluster
				}
				if (timed) { t_d = now(); tm[5] += t_d - t_c; t_c = t_d; }
				// ---- head on this CTA's copy: warp = four rows of the pass; side effects from cluster rank 0 only
				for (int rr = 0; rr < CF_R / 8; ++rr)
				{
					const int r = warp * (CF_R / 8) + rr;
					float* p = AT + (size_t)P.node_off[H + 1] * CF_R + r;  // stride CF_R
					float* dout = DT + (size_t)P.d_off[H + 1] * CF_R + r;
					float c_acc = 0.0f, a_acc = 0.0f, be = 0.0f, bp = 0.0f;
					int ie = -1, ip = -1;
					if (r < valid)
					{
						const float* y = a.Y + (r0 + j0 + r) * n_out;
						float mx = -INFINITY, inv_den = 1.0f;
						if (softmax)
						{
							for (int o = lane; o < n_out; o += 32) mx = fmaxf(mx, p[(size_t)o * CF_R]);
							mx = warp_max(mx);
							float den = 0.0f;
							for (int o = lane; o < n_out; o += 32) den += expf(p[(size_t)o * CF_R] - mx);
							inv_den = 1.0f / warp_sum(den);
						}
						for (int o = lane; o < n_out; o += 32)
						{
							float pv = p[(size_t)o * CF_R];
							const float e = y[o];
							float cost, d;
							if (softmax)
							{
								pv = expf(pv - mx) * inv_den;
								p[(size_t)o * CF_R] = pv;
								cost = (e != 0.0f) ? -(e * logf(pv)) / data_size : 0.0f;
								d = pv - e;
							}
							else if (n.out_type == GL_OUT_REGRESSION)
							{
								const float tt = e - pv;
								cost = tt * tt / data_size;
								d = 2.0f * (pv - e);
							}
							else if (n.out_type == GL_OUT_CLASSIFICATION)
							{
								cost = -((e * logf(pv)) + ((1.0f - e) * logf(1.0f - pv))) / data_size;
								d = (pv - e) / ((1.0f - pv) * pv);
							}
							else
							{
								cost = logf(e / pv) / data_size;
								d = -(e / pv);
							}
							dout[(size_t)o * CF_R] = d;
							if (crank == 0)
							{
								a.actbuf[(size_t)(j0 + r) * pitch + P.soff[H + 1] + o] = pv;
								a.delbuf[(size_t)(j0 + r) * pitch + P.soff[H + 1] + o] = d;
							}
							c_acc += cost;
							a_acc += fmaxf((1.0f - fminf(fabsf(pv - e), 1.0f)) * 100.0f, 0.0f);
							if (e > be) { be = e; ie = o; }
							if (pv > bp) { bp = pv; ip = o; }
						}
						c_acc = warp_sum(c_acc);
						a_acc = warp_sum(a_acc);
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
						if (crank == 0)
						{
							if (lane == 0 && classify && last_epoch && ie >= 0 && ip >= 0) atomicAdd(a.confusion + ie * n_out + ip, 1);
							if (a.last_out && last_epoch && r0 + j0 + r == a.rows - 1)
								for (int o = lane; o < n_out; o += 32) a.last_out[o] = p[(size_t)o * CF_R];
						}
					}
					else
					{
						for (int o = lane; o < n_out; o += 32) dout[(size_t)o * CF_R] = 0.0f;
					}
					// rows of the delta buffer beyond the layer's nodes (rounded up to 4) take part in the next product as zeros
					for (int o = n_out + lane; o < ((n_out + 3) & ~3); o += 32) dout[(size_t)o * CF_R] = 0.0f;
					if (lane == 0)
					{
						rowm[2 * r] = c_acc;
						rowm[2 * r + 1] = a_acc;
					}
				}
				__syncthreads();
				if (timed) { t_d = now(); tm[6] += t_d - t_c; t_c = t_d; }
				// ---- hidden deltas of the CTA's nodes: D_j = (D_{j+1} W_j) * act'(A_j)
				for (int j = H; j >= 1; --j)
				{
					const int i0 = crank * P.sl[j];
					int cnt = n.sizes[j] - i0;
					cnt = cnt < 0 ? 0 : (cnt > P.sl[j] ? P.sl[j] : cnt);
					const int act = n.act[j - 1];
					const int node = P.node_off[j] + i0, drow = P.d_off[j] + i0, dcol = P.soff[j] + i0;
					const bool gather = j >= 2;
					cf_product(DT + (size_t)P.d_off[j + 1] * CF_R, (n.sizes[j + 1] + 3) & ~3, sm + P.wb[j], cnt,
					           [&](int nn, int sq, float s0, float s1, float s2, float s3) {
						           const float4 av = *reinterpret_cast<const float4*>(AT + (size_t)(node + nn) * CF_R + 4 * sq);
						           const float d0 = (4 * sq + 0 < valid) ? s0 * act_der_b(av.x, act, 0.01f) : 0.0f;
						           const float d1 = (4 * sq + 1 < valid) ? s1 * act_der_b(av.y, act, 0.01f) : 0.0f;
						           const float d2 = (4 * sq + 2 < valid) ? s2 * act_der_b(av.z, act, 0.01f) : 0.0f;
						           const float d3 = (4 * sq + 3 < valid) ? s3 * act_der_b(av.w, act, 0.01f) : 0.0f;
						           if (gather)
						           {
							           const uint32_t local = dt_addr + (uint32_t)(((drow + nn) * CF_R + 4 * sq) * 4);
#pragma unroll
							           for (int dst = 0; dst < CF_CS; ++dst) cl_store4(cl_map(local, (uint32_t)dst), d0, d1, d2, d3);
						           }
						           float* gd = a.delbuf + (size_t)(j0 + 4 * sq) * pitch + dcol + nn;
						           if (4 * sq + 0 < valid) gd[0] = d0;
						           if (4 * sq + 1 < valid) gd[(size_t)pitch] = d1;
						           if (4 * sq + 2 < valid) gd[(size_t)2 * pitch] = d2;
						           if (4 * sq + 3 < valid) gd[(size_t)3 * pitch] = d3;
					           });
					if (gather) cl_sync();
				}
				if (timed) { t_d = now(); tm[7] += t_d - t_c; t_c = t_d; }
				// the inputs of the pass belong to the window scratch too (phase 2 of layer 0 reads them)
				{
					const int n0 = n.sizes[0];
					for (int e = t + crank * GF_THREADS; e < valid * n0; e += GF_THREADS * CF_CS)
					{
						const int r = e / n0, i = e - r * n0;
						a.actbuf[(size_t)(j0 + r) * pitch + i] = AT[(size_t)i * CF_R + r];
					}
				}
				if (crank == 0)
				{
					if (warp >= 1 && warp <= H)
					{
						// scalar-bias delta of hidden layer `warp`: sum of the deltas of the layer above, this pass's rows
						const int l = warp, no = n.sizes[l + 1];
						double s = 0.0;
						for (int e = lane; e < no * CF_R; e += 32) s += (double)DT[(size_t)P.d_off[l + 1] * CF_R + e];
						s = warp_sum_d(s);
						if (lane == 0) s_part[2 + l] += s;
					}
					if (t == 0)
					{
						for (int r = 0; r < valid; ++r)
						{
							s_part[0] += (double)rowm[2 * r];
							s_part[1] += (double)rowm[2 * r + 1];
						}
					}
				}
				cl_sync();  // nobody of the cluster reads this pass's buffers any more: the next pass may overwrite them
				if (timed) { t_d = now(); tm[8] += t_d - t_c; t_c = t_d; }
			}
			__syncthreads();
			if (t < GF_PART) a.part[(size_t)blockIdx.x * GF_PART + t] = s_part[t];
			if (timed) { t_b = now(); tm[0] += t_b - t_a; }
			grid.sync();
			if (timed) { t_a = now(); tm[1] += t_a - t_b; }

			// ================= phase 2: gradient + update per weight tile; CTA 0 also the scalars
			const float inv_len = 1.0f / (float)len;
			for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x)
			{
				int l = 0;
				while (tile >= tile_off[l + 1]) ++l;
				const int tiles_i = (n.sizes[l] + GF_P2_TI - 1) / GF_P2_TI;
				const int tl = tile - tile_off[l];
				const float* ckl = a.ck + (size_t)l * (mb + 1);
				if (n.sizes[l + 1] <= GF_NARROW)
					gf_grad_narrow(a, l, tl * GF_NCOLS, len, pitch, P.soff[l], P.soff[l + 1], ckl, inv_len, sm, bad);
				else
					gf_grad_tile_async(a, l, (tl / tiles_i) * GF_TO, (tl % tiles_i) * GF_P2_TI, len, pitch, P.soff[l], P.soff[l + 1], sm,
					                   ckl, inv_len, bad);
			}
			if (blockIdx.x == 0)
			{
				if (warp >= 1 && warp <= H)
				{
					const int l = warp;
					double s = 0.0;
					for (int b = lane; b < (int)gridDim.x; b += 32) s += __ldcg(a.part + (size_t)b * GF_PART + 2 + l);
					s = warp_sum_d(s) * (double)n.lr[l];
					if (lane == 0)
					{
						const float nb = __ldcg(n.bias + l) -
						                 ((a.bias_rule == GL_BIAS_REFERENCE) ? (float)(s * (double)n.sizes[l]) : (float)(s / (double)len));
						if (!isfinite(nb)) bad = 1;
						n.bias[l] = nb;
					}
				}
				if (warp == 0)
				{
					double c = 0.0, q = 0.0;
					for (int b = lane; b < (int)gridDim.x; b += 32)
					{
						c += __ldcg(a.part + (size_t)b * GF_PART);
						q += __ldcg(a.part + (size_t)b * GF_PART + 1);
					}
					c = warp_sum_d(c);
					q = warp_sum_d(q);
					if (lane == 0)
					{
						ecost += c;
						eacc += q;
					}
				}
			}
			if (timed) { t_b = now(); tm[2] += t_b - t_a; }
			grid.sync();
			if (timed) { t_a = now(); tm[3] += t_a - t_b; }
		}
		if (blockIdx.x == 0 && t == 0)
		{
			a.epoch_sums[2 * ep] = ecost;
			a.epoch_sums[2 * ep + 1] = eacc;
		}
	}
	if (timed)
		for (int k = 0; k < 9; ++k) a.timing[k] += tm[k];
	if (bad) atomicOr(a.flags, 1);
}

#endif  // GF_KERNEL_ROWS

}  // namespace

// This file is compiled once per group size (GF_KERNEL_ROWS) for grid_fused_kernel's two instantiations, and once more for the cluster variant
// and the host side: a process loads the code of the group sizes that it runs, not of all ten kernels (13 against 3 ms of a first call).
#ifdef GF_KERNEL_ROWS
void* GL_CAT(grid_fused_function_, GF_KERNEL_ROWS)(bool tma)
{
	return tma ? (void*)grid_fused_kernel<true, GF_KERNEL_ROWS> : (void*)grid_fused_kernel<false, GF_KERNEL_ROWS>;
}
#else
void* grid_fused_function_2(bool tma);
void* grid_fused_function_4(bool tma);
void* grid_fused_function_8(bool tma);
void* grid_fused_function_12(bool tma);
void* grid_fused_function_16(bool tma);

static size_t gf_smem_bytes(const NetView& n, int rows)
{
	int off[GL_MAX_WEIGHT_LAYERS + 2];
	const int tot = gf_scratch_layout(n, off);
	size_t f = 2 * (size_t)tot * rows + 2 * rows + GF_SEQ_MAX;
	if (n.sizes[n.H + 1] <= GF_NARROW && n.H >= 1)  // the narrow head's weights and the partial sums of its forward product
		f += (((size_t)n.sizes[n.H + 1] * n.sizes[n.H] + 3) & ~(size_t)3) + 8 * rows * GF_NARROW;
	// + alignment slack + the ring
	return f * sizeof(float) + 1024 + (size_t)GF_NS * GF_STAGE + 64;
}

int grid_fused_box(int nodes) { return gf_box(nodes); }

// (eight rows: more are taken where they fit)
size_t grid_fused_smem_bytes(const NetView& n) { return gf_smem_bytes(n, 8); }

int grid_fused_scratch_pitch(const NetView& n)
{
	int soff[GL_MAX_WEIGHT_LAYERS + 2];
	return gf_scratch_layout(n, soff);
}

int grid_fused_total_nodes(const NetView& n)
{
	int tot = 0;
	for (int l = 0; l <= n.H + 1; ++l) tot += n.sizes[l];
	return tot;
}

static void* grid_fused_function(int rows, bool tma)
{
	switch (rows)
	{
	case 2: return grid_fused_function_2(tma);
	case 4: return grid_fused_function_4(tma);
	case 8: return grid_fused_function_8(tma);
	case 12: return grid_fused_function_12(tma);
	default: return grid_fused_function_16(tma);
	}
}

cudaError_t launch_grid_fused(const GridFusedArgs& a, cudaStream_t s)
{
	if (a.part_ctas < 1) return cudaErrorInvalidValue;
	// Rows per group: a CTA's time is its groups times (a part that goes with the weights' way from L2 and the steps' latency, about six
	// rows' worth) + (the rows' multiply-adds).
	int rows = 2;
	long long best = 0;
	for (int r : {2, 4, 8, 12, 16})
	{
		const long long groups = (a.net.mb + r - 1) / r, time = (groups + a.part_ctas - 1) / a.part_ctas * (6 + r);
		if ((best == 0 || time < best) && (r <= 8 || gf_smem_bytes(a.net, r) <= (size_t)220 * 1024))
		{
			best = time;
			rows = r;
		}
	}
	const size_t bytes = gf_smem_bytes(a.net, rows);
	void* fn = grid_fused_function(rows, a.tma != nullptr);
	// the attribute belongs to the current device: set it per launch (a cheap call) rather than cache it per process
	const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
	if (e != cudaSuccess) return e;
	GridFusedArgs copy = a;
	void* params[] = {&copy};
	// one CTA per SM (the shared-memory footprint allows no more), all co-resident as the grid barrier needs
	return cudaLaunchCooperativeKernel(fn, dim3((unsigned)a.part_ctas), dim3(GF_THREADS), params, bytes, s);
}

// ---- cluster variant: host side ------------------------------------------------------------------
size_t cluster_fused_smem_bytes(const NetView& n)
{
	CfPlan p;
	cf_plan(n, p);
	return (size_t)p.floats * sizeof(float);
}

// The variant wants every layer that is read as an input (0..H) to be a multiple of 4 nodes (16-byte rows for
// the vector loads), at least one hidden layer, and its buffers inside one SM's shared memory.
bool cluster_fused_fits(const NetView& n)
{
	if (n.H < 1) return false;
	for (int l = 0; l <= n.H; ++l)
		if (n.sizes[l] % 4 != 0) return false;
	return cluster_fused_smem_bytes(n) <= (size_t)226 * 1024;
}

static cudaError_t cluster_fused_config(const NetView& n, cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attrs, unsigned grid, cudaStream_t s)
{
	const size_t bytes = cluster_fused_smem_bytes(n);
	cudaError_t e = cudaFuncSetAttribute(cluster_fused_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
	if (e != cudaSuccess) return e;
	memset(&cfg, 0, sizeof cfg);
	cfg.gridDim = dim3(grid);
	cfg.blockDim = dim3(GF_THREADS);
	cfg.dynamicSmemBytes = bytes;
	cfg.stream = s;
	attrs[0].id = cudaLaunchAttributeClusterDimension;
	attrs[0].val.clusterDim.x = CF_CS;
	attrs[0].val.clusterDim.y = 1;
	attrs[0].val.clusterDim.z = 1;
	attrs[1].id = cudaLaunchAttributeCooperative;
	attrs[1].val.cooperative = 1;
	cfg.attrs = attrs;
	cfg.numAttrs = 2;
	return cudaSuccess;
}

// CTAs of the largest co-resident grid of whole clusters on the current device (0: the variant cannot run here)
int cluster_fused_max_ctas(const NetView& n)
{
	cudaLaunchConfig_t cfg;
	cudaLaunchAttribute attrs[2];
	if (cluster_fused_config(n, cfg, attrs, CF_CS, 0) != cudaSuccess)
	{
		cudaGetLastError();
		return 0;
	}
	cfg.numAttrs = 1;  // the occupancy query takes the cluster shape; co-residency is what it reports
	int clusters = 0;
	if (cudaOccupancyMaxActiveClusters(&clusters, cluster_fused_kernel, &cfg) != cudaSuccess)
	{
		cudaGetLastError();
		return 0;
	}
	return clusters * CF_CS;
}

cudaError_t launch_cluster_fused(const GridFusedArgs& a, cudaStream_t s)
{
	if (a.part_ctas < CF_CS || a.part_ctas % CF_CS != 0) return cudaErrorInvalidValue;
	cudaLaunchConfig_t cfg;
	cudaLaunchAttribute attrs[2];
	cudaError_t e = cluster_fused_config(a.net, cfg, attrs, (unsigned)a.part_ctas, s);
	if (e != cudaSuccess) return e;
	return cudaLaunchKernelEx(&cfg, cluster_fused_kernel, a);
}

#endif  // GF_KERNEL_ROWS

}  // namespace glb
