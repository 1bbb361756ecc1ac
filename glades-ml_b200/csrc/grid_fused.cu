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
// scheduler; two per scheduler would double the loads -- head, activations, stores and latencies at the layers' ends 16 k, phase 2 14 k, two
// grid barriers 7 k.  55 k clocks, 81 k when a step ended in a block barrier, the block copied phase 2's stages by 16-byte
// asynchronous copies and every element's activation was a copy of its own of the code.
// Arithmetic = the batched mode of batched.cu / small_fused.cu (reference loop
// Networks/network.cpp:457-668 with aligned windows, frozen weights and a plain error sum); c_j is
// the closed form of the reference's intra-window momentum history (State/node.cpp:278-292).
#include <cooperative_groups.h>
#include <type_traits>

#include "copy_ring.h"
#include "grid_fused.cuh"
#include "tc_device.cuh"

namespace cg = cooperative_groups;

namespace glb {
using namespace tc;
namespace {

constexpr int GF_NS = 3;                // stages of the weight-tile ring (bulk tensor copies, 32 KB each)
constexpr int GF_STAGE = 32768;
constexpr int GF_SEQ_MAX = 704;         // weight tiles one sample group walks through, at most: 8 layers of at most 1024 nodes and 2^19 weights
                                        // have less than 64 + 8 * 37 forward and 64 + 7 * 37 back
// nodes of a layer that one of phase 1's computing warps takes at a time
__host__ __device__ inline int gf_box(int nodes) { return nodes <= 64 ? 16 : (nodes <= 128 ? 32 : 64); }

#ifdef GF_KERNEL_ROWS
constexpr int GF_ROWS = 16;     // samples a CTA carries through the network together, at most
constexpr int GF_TILE = 256;    // weight tile: 256 output nodes x 32 inputs (forward), 32 output nodes x 256 inputs (deltas)
static_assert(GF_TILE * 32 * 4 == GF_STAGE, "a stage holds one weight tile");

// ---- phase 2 ----------------------------------------------------------------------------------------
// Rows 8w..8w+7 of every 64-row stage are warp w's chain, the warps' sums are added in warp order.  Every warp fetches the rows of its
// own chain, by bulk tensor copies of two stages (16 rows) each into a ring of its own, so that no
// barrier of the block stands between two stages; and the factors that do not depend on the weight (learning rate and, without
// decay, the momentum weight) are multiplied into the deltas when phase 1 writes them.  18 instructions per row and warp, of which two are
// loads of two clocks each (the cluster variant's functions take 27, three loads of seven clocks, three asynchronous copies per thread and
// stage with their addresses, and two barriers' worth of waits per stage).
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

// The arithmetic of phase 1.  The first four warps compute, one per scheduler: a warp takes 16, 32 or 64 neighbouring nodes of a layer
// (of 256 at a time, gf_box), lane (g, h) = (lane / 2, lane % 2) 1, 2 or 4 of them and half of the group's rows.  Neighbouring lanes read the
// same weights, so that a 16-byte load costs two clocks (32 rows of weights, one per lane, cost four), and what the next four k need is
// read ahead of the current ones' multiply-adds.  Every sum is one chain, k ascending.  The warps wait for one another at the ends of layers
// only.
constexpr int GF_COMPUTE = 128;
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
	// tm[9], tm[11..14]: inside phase 1 -- waits for weight tiles, then forward, head, deltas, tail
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
	bool dead = false;     // computing warps: a bounded wait ran out; stop waiting, finish the launch
	auto drain_tiles = [&](unsigned lo, unsigned hi) { mbar_drain<GF_NS>(smem_u32(&full_bars[0][0]), lo, hi); };
	// up to `most` more tiles of the current group; each waits for the tile three before it to be read
	auto fetch_tiles = [&](int most) {
		for (; most > 0 && group_left > 0; --most, --group_left, --p_left)
		{
			const unsigned e = seq[p_at], ps = tiles_asked.base, st = ps % GF_NS;
			if (++p_at == nsteps) p_at = 0;
			uint64_t* const full = &full_bars[use_tma ? 0 : cw][st];
			auto read = [&](unsigned stage, unsigned parity) { return mbar_wait(smem_u32(&empty_bars[use_tma ? 0 : cw][stage]), parity, &gf_abort, a.flags + 1, 32); };
			if (use_tma && !tiles_asked.may_ask(read, drain_tiles)) return;
			if (!use_tma && ps >= GF_NS && !read(st, (ps / GF_NS - 1) & 1u))
			{
				nsteps = group_left = 0;  // nothing more to copy, in this window or another
				asm volatile("cp.async.wait_all;" ::: "memory");
				return;
			}
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
#endif  // GF_KERNEL_ROWS

}  // namespace

// This file is compiled once per group size (GF_KERNEL_ROWS) for grid_fused_kernel's two instantiations, and once more for
// the host side: a process loads the code of the group sizes that it runs, not of all ten kernels (2.3 against 13 ms of a first call).
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
#endif  // GF_KERNEL_ROWS

}  // namespace glb
