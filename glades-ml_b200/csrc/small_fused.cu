// Batched mode for small networks: one persistent CTA trains n_epochs * windows in a single launch
// with ALL weights resident in shared memory.
//
// Per window (aligned, `mb` rows, weights frozen inside it):
//   phase 1  one warp per SR samples: forward (lane = output node, one fmaf chain per node and sample, k ascending), optional
//            softmax and the output delta, a group of lanes per sample, then the deltas of the hidden layers (lane = input
//            node, plain error sum);
//   phase 2  2 x 4 weights per thread, or per 2 or 4 threads that take every 2nd or 4th row where there are few:
//            G = sum_j c_j * (lr*d_jo*a_ji + decay terms) over the window's samples in a fixed order (deterministic),
//            W -= G / len; the last warps sum the hidden layers' scalar-bias deltas.
// Two block-wide barriers per window; the next window's rows travel during the current one.
// Arithmetic = the batched mode of batched.cu (reference loop Networks/network.cpp:457-668 with
// aligned windows, frozen weights and a plain error sum); c_j is the closed form of the reference's
// intra-window momentum history (State/node.cpp:278-292).
//
// What bounds a window is the 32 words per clock that shared memory delivers into registers (a broadcast quad counts as four),
// then the latency of the chains and of the activations.  So a weight that has been read serves SR samples and, in phase 2, a
// row's 7 words eight products; rows are padded to whole quads with a pitch of an odd number of them, so that 16-byte reads of
// 8 neighbouring rows hit all banks.  Measured, 10-32-32-1 with windows of 32 rows: one warp per sample and one thread per weight
// 12.5 us per window, 6.0 us now.
#include "common.cuh"
#include "internal.h"

namespace glb {

constexpr int SF_THREADS = 512;

__host__ __device__ __forceinline__ int sf_quads(int n) { return (n + 3) >> 2; }
__host__ __device__ __forceinline__ int sf_pitch(int ni) { return 4 * (sf_quads(ni) | 1); }

// What the phases ask about a weight layer, in shared memory: the kernel's parameters and arrays indexed by the layer would be
// read through the constant cache and local memory, a chain of such reads at the head of every layer of every window.
// Offsets are in floats from the start of shared memory, so that every access is known to be one to shared memory.
struct __align__(16) SfLayer
{
	int ni, no, iquads, oquads;
	int w, ld, in, ipitch;           // weights and their pitch; the layer's input (layer 0: of window buffer 0) and its pitch
	int out, act, act_below, tiles;  // out: the layer above inside a row of A and of D
	float par, lr, w1, w2;
};

template <int SR>
__global__ void __launch_bounds__(SF_THREADS, 1) small_fused_kernel(const __grid_constant__ SmallFusedArgs a)
{
	extern __shared__ __align__(16) float sm[];
	__shared__ SfLayer layer[GL_MAX_WEIGHT_LAYERS];
	__shared__ float sbias[GL_MAX_WEIGHT_LAYERS];
	__shared__ double swarp[SF_THREADS / 32][2];
	const NetView& n = a.net;
	const int H = n.H;
	const int T = blockDim.x, t = threadIdx.x;
	const int lane = t & 31, warp = t >> 5, nwarps = T >> 5;
	const int n_in = n.sizes[0], n_out = n.sizes[H + 1], out_type = n.out_type;
	const int mb = n.mb, mbp = (mb + SR - 1) / SR * SR;
	const long long rows = a.rows;

	// shared memory: padded weights | activations and deltas of layers 1..H+1, [mbp][tot] each | inputs of two windows
	// [2][mbp][ipitch] | targets of two windows | momentum weights and the same times the learning rate, [H+1][mb] each
	int tot = 0, tiles = 0, A = 0;
	for (int l = 0; l <= H; ++l)
	{
		tot += 4 * sf_quads(n.sizes[l + 1]);
		tiles += (n.sizes[l] + 1) / 2 * sf_quads(n.sizes[l + 1]);
		A += 4 * sf_quads(n.sizes[l + 1]) * sf_pitch(n.sizes[l]);
	}
	const int ipitch = 4 * sf_quads(n_in);
	const int split = tiles * 4 <= T ? 2 : (tiles * 2 <= T ? 1 : 0);  // log2 of the threads that share a tile of phase 2
	const int D = A + mbp * tot, X0 = D + mbp * tot, Y0 = X0 + 2 * mbp * ipitch;
	const int cw = Y0 + 2 * mbp * n_out, clr = cw + (H + 1) * mb, end = clr + (H + 1) * mb;
	if (t == 0)
		for (int l = 0, w = 0, out = 0; l <= H; ++l)
		{
			SfLayer& y = layer[l];
			y.ni = n.sizes[l];
			y.no = n.sizes[l + 1];
			y.iquads = sf_quads(y.ni);
			y.oquads = sf_quads(y.no);
			y.w = w;
			y.ld = sf_pitch(y.ni);
			y.in = l ? A + out - 4 * y.iquads : X0;
			y.ipitch = l ? tot : ipitch;
			y.out = out;
			y.act = n.act[l];
			y.act_below = l ? n.act[l - 1] : 0;
			y.tiles = (y.ni + 1) / 2 * y.oquads;
			y.par = n.par[l];
			y.lr = n.lr[l];
			y.w1 = n.wd1[l] * y.lr;
			y.w2 = n.wd2[l] * y.lr;
			w += 4 * y.oquads * y.ld;
			out += 4 * y.oquads;
		}
	for (int p = t; p < end; p += T) sm[p] = 0.0f;  // (paddings stay zero)
	__syncthreads();
	for (int l = 0; l <= H; ++l)
	{
		const int ni = layer[l].ni, cells = ni * layer[l].no;
		for (int e = t; e < cells; e += T) sm[layer[l].w + (e / ni) * layer[l].ld + (e % ni)] = n.W[l][e];
	}
	if (t < GL_MAX_WEIGHT_LAYERS) sbias[t] = n.bias[t];
	const bool classify = out_type != GL_OUT_REGRESSION;
	if (classify)
		for (int e = t; e < n_out * n_out; e += T) a.confusion[e] = 0;

	const uint32_t smem = (uint32_t)__cvta_generic_to_shared(sm);
	// e / n_in by a multiplication with 2^32 / n_in, rounded up: exact for e * n_in < 2^32
	const unsigned in_magic = n_in == 1 ? 0 : (unsigned)(0x100000000ull / (unsigned)n_in) + 1;
	auto fetch = [&](long long r0, int buf) {
		const int len = (int)((rows - r0) < mb ? (rows - r0) : mb);
		for (int e = t; e < len * n_in; e += T)  // (the rows lie one after the other)
		{
			const int j = n_in == 1 ? e : (int)__umulhi((unsigned)e, in_magic);
			cp_async4(smem + (uint32_t)(X0 + (buf * mbp + j) * ipitch + (e - j * n_in)) * 4, a.X + r0 * n_in + e, true);
		}
		for (int e = t; e < len * n_out; e += T) cp_async4(smem + (uint32_t)(Y0 + buf * mbp * n_out + e) * 4, a.Y + r0 * n_out + e, true);
		cp_async_commit();
	};
	fetch(0, 0);
	cp_async_wait<0>();
	__syncthreads();

	const float data_size = (float)(rows * (long long)n_out);
	const bool softmax = n.act[H] == GL_ACT_SOFTMAX;
	const int head = layer[H].out;
	int gw = 1;  // lanes per sample at the head
	while (gw < n_out && gw < 32) gw <<= 1;
	int cur_len = -1, buf = 0;

	for (int ep = 0; ep < a.n_epochs; ++ep)
	{
		const bool last_epoch = ep == a.n_epochs - 1;
		double ecost = 0.0, eacc = 0.0;  // this thread's share
		for (long long r0 = 0; r0 < rows; r0 += mb, buf ^= 1)
		{
			const int len = (int)((rows - r0) < mb ? (rows - r0) : mb);
			if (len != cur_len)
			{
				// c_j = sum_{t=0}^{len-1-j} m^t
				for (int e = t; e < (H + 1) * len; e += T)
				{
					const int l = e / len, j = e - l * len;
					const double m = (double)n.mom[l];
					double s = 0.0, pw = 1.0;
					if (m != 0.0)
						for (int q = 0; q < len - j; ++q)
						{
							s += pw;
							pw *= m;
							if (pw < 1e-30) break;
						}
					const float c = (m == 0.0) ? 1.0f : (float)s;
					sm[cw + l * mb + j] = c;
					sm[clr + l * mb + j] = layer[l].lr * c;
				}
				cur_len = len;
			}
			const long long next = r0 + mb < rows ? r0 + mb : 0;
			if (next || !last_epoch) fetch(next, buf ^ 1);
			const int X = X0 + buf * mbp * ipitch, Y = Y0 + buf * mbp * n_out;
			// ---------------- phase 1: one warp per SR samples (rows beyond `len` are computed from what lies there, and not used)
			for (int j0 = warp * SR; j0 < len; j0 += nwarps * SR)
			{
				const int aj = A + j0 * tot, dj = D + j0 * tot;
				for (int l = 0; l <= H; ++l)
				{
					const SfLayer y = layer[l];
					const int in = (l ? y.in : X) + j0 * y.ipitch;
					const float b = (l >= 1) ? sbias[l] : 0.0f;
					for (int o = lane; o < y.no; o += 32)
					{
						const float4* w = reinterpret_cast<const float4*>(sm + y.w + o * y.ld);
						float z[SR];
#pragma unroll
						for (int s = 0; s < SR; ++s) z[s] = 0.0f;
#pragma unroll 2
						for (int q = 0; q < y.iquads; ++q)
						{
							const float4 wv = w[q];
							float4 v[SR];
#pragma unroll
							for (int s = 0; s < SR; ++s) v[s] = *reinterpret_cast<const float4*>(sm + in + s * y.ipitch + 4 * q);
#pragma unroll
							for (int s = 0; s < SR; ++s) z[s] = fmaf(wv.x, v[s].x, z[s]);
#pragma unroll
							for (int s = 0; s < SR; ++s) z[s] = fmaf(wv.y, v[s].y, z[s]);
#pragma unroll
							for (int s = 0; s < SR; ++s) z[s] = fmaf(wv.z, v[s].z, z[s]);
#pragma unroll
							for (int s = 0; s < SR; ++s) z[s] = fmaf(wv.w, v[s].w, z[s]);
						}
#pragma unroll
						for (int s = 0; s < SR; ++s) z[s] = squash_b(z[s] + b, y.act, y.par);
#pragma unroll
						for (int s = 0; s < SR; ++s) sm[aj + y.out + s * tot + o] = z[s];
					}
					__syncwarp();
				}
				// head: optional softmax, output delta, figures; gw lanes per sample
				for (int s0 = 0; s0 < SR; s0 += 32 / gw)
				{
					const int s = s0 + lane / gw, og = lane & (gw - 1);
					const bool row = s < SR && j0 + s < len;
					const int j = row ? j0 + s : j0;
					float* const p = sm + A + j * tot + head;
					float* const dout = sm + D + j * tot + head;
					const float* const y = sm + Y + j * n_out;
					float mx = -INFINITY, inv_den = 1.0f;
					if (softmax)
					{
						for (int o = og; o < n_out; o += gw) mx = fmaxf(mx, p[o]);
						for (int off = gw >> 1; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
						float den = 0.0f;
						for (int o = og; o < n_out; o += gw) den += expf(p[o] - mx);
						for (int off = gw >> 1; off > 0; off >>= 1) den += __shfl_xor_sync(0xffffffffu, den, off);
						inv_den = 1.0f / den;
					}
					__syncwarp();  // (lanes without a row of their own have read the first row's sums)
					float be = 0.0f, bp = 0.0f;
					int ie = -1, ip = -1;
					if (row)
						for (int o = og; o < n_out; o += gw)
						{
							float pv = p[o];
							const float e = y[o];
							float cost, d;
							if (softmax)
							{
								pv = expf(pv - mx) * inv_den;
								p[o] = pv;
								cost = (e != 0.0f) ? -(e * logf(pv)) / data_size : 0.0f;
								d = pv - e;
							}
							else if (out_type == GL_OUT_REGRESSION)
							{
								const float tt = e - pv;
								cost = tt * tt / data_size;
								d = 2.0f * (pv - e);
							}
							else if (out_type == GL_OUT_CLASSIFICATION)
							{
								cost = -((e * logf(pv)) + ((1.0f - e) * logf(1.0f - pv))) / data_size;
								d = (pv - e) / ((1.0f - pv) * pv);
							}
							else
							{
								cost = logf(e / pv) / data_size;
								d = -(e / pv);
							}
							dout[o] = d;
							ecost += (double)cost;
							eacc += (double)fmaxf((1.0f - fminf(fabsf(pv - e), 1.0f)) * 100.0f, 0.0f);
							if (e > be) { be = e; ie = o; }
							if (pv > bp) { bp = pv; ip = o; }
							if (a.last_out && last_epoch && r0 + j == rows - 1) a.last_out[o] = pv;
						}
					if (classify && last_epoch)
					{
						for (int off = gw >> 1; off > 0; off >>= 1)
						{
							const float oe = __shfl_xor_sync(0xffffffffu, be, off);
							const int oie = __shfl_xor_sync(0xffffffffu, ie, off);
							if (oie >= 0 && (ie < 0 || oe > be || (oe == be && oie < ie))) { be = oe; ie = oie; }
							const float op = __shfl_xor_sync(0xffffffffu, bp, off);
							const int oip = __shfl_xor_sync(0xffffffffu, ip, off);
							if (oip >= 0 && (ip < 0 || op > bp || (op == bp && oip < ip))) { bp = op; ip = oip; }
						}
						if (row && og == 0 && ie >= 0 && ip >= 0) atomicAdd(a.confusion + ie * n_out + ip, 1);
					}
				}
				__syncwarp();
				// deltas of the hidden layers: D_l = (D_{l+1} W_l) * act'(A_l)
				for (int l = H; l >= 1; --l)
				{
					const SfLayer y = layer[l];
					const int below = y.in - A;  // the layer's input nodes inside a row of A and of D
					for (int i = lane; i < y.ni; i += 32)
					{
						const float* w = sm + y.w + i;
						const float* dup = sm + dj + y.out;
						float e[SR], av[SR];
#pragma unroll
						for (int s = 0; s < SR; ++s)
						{
							e[s] = 0.0f;
							av[s] = sm[aj + s * tot + below + i];
						}
#pragma unroll 2
						for (int q = 0; q < y.oquads; ++q, w += 4 * y.ld)
						{
							const float w0 = w[0], w1 = w[y.ld], w2 = w[2 * y.ld], w3 = w[3 * y.ld];
							float4 v[SR];
#pragma unroll
							for (int s = 0; s < SR; ++s) v[s] = *reinterpret_cast<const float4*>(dup + s * tot + 4 * q);
#pragma unroll
							for (int s = 0; s < SR; ++s) e[s] = fmaf(v[s].x, w0, e[s]);
#pragma unroll
							for (int s = 0; s < SR; ++s) e[s] = fmaf(v[s].y, w1, e[s]);
#pragma unroll
							for (int s = 0; s < SR; ++s) e[s] = fmaf(v[s].z, w2, e[s]);
#pragma unroll
							for (int s = 0; s < SR; ++s) e[s] = fmaf(v[s].w, w3, e[s]);
						}
#pragma unroll
						for (int s = 0; s < SR; ++s) sm[dj + s * tot + below + i] = e[s] * act_der_b(av[s], y.act_below, 0.01f);
					}
					__syncwarp();
				}
			}
			__syncthreads();
			// ---------------- phase 2: gradient + update
			const float inv_len = 1.0f / (float)len;
			for (int e0 = t; e0 < ((tiles << split) + 31) / 32 * 32; e0 += T)
			{
				const bool mine = (e0 >> split) < tiles;
				int l = 0, e = mine ? e0 >> split : 0;
				for (; e >= layer[l].tiles; ++l) e -= layer[l].tiles;
				const SfLayer y = layer[l];
				const int pairs = (y.ni + 1) >> 1, oq = e / pairs, i = 2 * (e - oq * pairs);
				const int j0 = e0 & ((1 << split) - 1);
				const float* av = sm + (l ? y.in : X) + i;
				const float* dv = sm + D + y.out + 4 * oq;
				const float* c = sm + cw + l * mb;
				const float* cl = sm + clr + l * mb;
				float g[4][2] = {};
#pragma unroll 4
				for (int j = j0; j < len; j += 1 << split)
				{
					const float2 x = *reinterpret_cast<const float2*>(av + j * y.ipitch);
					const float4 d = *reinterpret_cast<const float4*>(dv + j * tot);
					const float s = cl[j], sd[4] = {s * d.x, s * d.y, s * d.z, s * d.w};
#pragma unroll
					for (int k = 0; k < 4; ++k)
					{
						g[k][0] = fmaf(sd[k], x.x, g[k][0]);
						g[k][1] = fmaf(sd[k], x.y, g[k][1]);
					}
				}
				if (y.w1 != 0.0f || y.w2 != 0.0f)
				{
					float decay[2] = {0.0f, 0.0f};
					for (int j = j0; j < len; j += 1 << split)
					{
						const float2 x = *reinterpret_cast<const float2*>(av + j * y.ipitch);
						decay[0] = fmaf(c[j], fmaf(y.w1, fabsf(x.x), y.w2 * x.x), decay[0]);
						decay[1] = fmaf(c[j], fmaf(y.w1, fabsf(x.y), y.w2 * x.y), decay[1]);
					}
#pragma unroll
					for (int k = 0; k < 4; ++k)
					{
						g[k][0] += decay[0];
						g[k][1] += decay[1];
					}
				}
				for (int off = 1; off < 1 << split; off <<= 1)
#pragma unroll
					for (int k = 0; k < 4; ++k)
					{
						g[k][0] += __shfl_xor_sync(0xffffffffu, g[k][0], off);
						g[k][1] += __shfl_xor_sync(0xffffffffu, g[k][1], off);
					}
				float* w = sm + y.w + 4 * oq * y.ld + i;
				if (mine && j0 == 0)
#pragma unroll
					for (int k = 0; k < 4; ++k)
					{
						if (4 * oq + k < y.no) w[k * y.ld] -= g[k][0] * inv_len;
						if (4 * oq + k < y.no && i + 1 < y.ni) w[k * y.ld + 1] -= g[k][1] * inv_len;
					}
			}
			// scalar biases of the hidden layers: lr * sum of the deltas of the layer above, on the warps that have the fewest weights
			if (nwarps - 1 - warp < H)
			{
				const int l = nwarps - warp;
				const SfLayer y = layer[l];
				const float* d = sm + D + y.out;
				// lanes side by side on a row's nodes, as many rows at once as fit
				int w = 1, lw = 0;
				while (w < y.no && w < 32)
				{
					w <<= 1;
					++lw;
				}
				double s0 = 0.0, s1 = 0.0;
				const int step = 32 >> lw;
				for (int o = lane & (w - 1); o < y.no; o += w)
				{
					int j = lane >> lw;
#pragma unroll 4
					for (; j + step < len; j += 2 * step)
					{
						s0 += (double)d[j * tot + o];
						s1 += (double)d[(j + step) * tot + o];
					}
					if (j < len) s0 += (double)d[j * tot + o];
				}
				const double s = warp_sum_d(s0 + s1) * (double)y.lr;
				if (lane == 0) sbias[l] -= (a.bias_rule == GL_BIAS_REFERENCE) ? (float)(s * (double)y.ni) : (float)(s / (double)len);
			}
			cp_async_wait<0>();
			__syncthreads();
		}
		ecost = warp_sum_d(ecost);
		eacc = warp_sum_d(eacc);
		if (lane == 0)
		{
			swarp[warp][0] = ecost;
			swarp[warp][1] = eacc;
		}
		__syncthreads();
		if (t < 2)
		{
			double s = 0.0;
			for (int w = 0; w < nwarps; ++w) s += swarp[w][t];
			a.epoch_sums[2 * ep + t] = s;
		}
		// (the next epoch's sums are written behind its windows' barriers)
	}
	// write the weights back and look for non-finite values
	int bad = 0;
	for (int l = 0; l <= H; ++l)
	{
		const int ni = layer[l].ni, cells = ni * layer[l].no;
		for (int e = t; e < cells; e += T)
		{
			const float w = sm[layer[l].w + (e / ni) * layer[l].ld + (e % ni)];
			n.W[l][e] = w;
			if (!isfinite(w)) bad = 1;
		}
	}
	if (t >= 1 && t <= H)
	{
		n.bias[t] = sbias[t];
		if (!isfinite(sbias[t])) bad = 1;
	}
	if (bad) atomicOr(a.flags, 1);
}

// This file is compiled once per number of samples (SF_KERNEL_SAMPLES), and once more for the host side: a process loads the code of the
// kernel that it runs, not of all seven (10-32-32-1, a process's first call of one epoch: 1.5 ms with all of them in one object, 0.95 ms with three, 0.7 ms now).
#ifdef SF_KERNEL_SAMPLES
const void* GL_CAT(small_fused_function_, SF_KERNEL_SAMPLES)() { return reinterpret_cast<const void*>(small_fused_kernel<SF_KERNEL_SAMPLES>); }
#else
const void* small_fused_function_1();
const void* small_fused_function_2();
const void* small_fused_function_4();
const void* small_fused_function_5();
const void* small_fused_function_6();
const void* small_fused_function_7();
const void* small_fused_function_8();

static const void* small_fused_function(int samples)
{
	switch (samples)
	{
	case 1: return small_fused_function_1();
	case 2: return small_fused_function_2();
	case 4: return small_fused_function_4();
	case 5: return small_fused_function_5();
	case 6: return small_fused_function_6();
	case 7: return small_fused_function_7();
	default: return small_fused_function_8();
	}
}

// Samples per warp in phase 1: as few as the sixteen warps allow.  More samples per warp read a weight less often, but the
// activations are chains of dependent instructions with branches, which only other warps fill (10-32-32-1, windows of 32: 6.6 us
// per window with two, 7.6 us with four, 7.4 us with one on 32 warps).
static int sf_least_samples(int mb) { return mb > 32 ? 4 : (mb > 16 ? 2 : 1); }

static size_t sf_smem_bytes(const NetView& n, int samples)
{
	const size_t sr = samples, mbp = ((size_t)n.mb + sr - 1) / sr * sr;
	size_t f = 0, tot = 0;
	for (int l = 0; l <= n.H; ++l)
	{
		tot += 4 * sf_quads(n.sizes[l + 1]);
		f += (size_t)4 * sf_quads(n.sizes[l + 1]) * sf_pitch(n.sizes[l]);
	}
	f += 2 * mbp * (tot + 4 * sf_quads(n.sizes[0]) + n.sizes[n.H + 1]) + 2 * (size_t)(n.H + 1) * n.mb;
	return f * sizeof(float);
}
size_t small_fused_smem_bytes(const NetView& n) { return sf_smem_bytes(n, sf_least_samples(n.mb)); }

// Windows of more than 64 rows give some warps a second turn at four samples each; five to eight samples in one turn take less (a
// window of 74 rows of 24-50-36-9: phase 1 39 k clocks with four).  Where that shares 16 warps out evenly, and where the rows that it
// rounds up to fit the block's shared memory.
static int sf_samples(const NetView& n)
{
	const int least = sf_least_samples(n.mb), even = (n.mb + SF_THREADS / 32 - 1) / (SF_THREADS / 32);
	return n.mb > 64 && even <= 8 && sf_smem_bytes(n, even) <= (size_t)220 * 1024 ? even : least;
}

cudaError_t launch_small_fused(const SmallFusedArgs& a, cudaStream_t s)
{
	const int sr = sf_samples(a.net);
	const size_t bytes = sf_smem_bytes(a.net, sr);
	const void* const kernel = small_fused_function(sr);
	const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
	if (e != cudaSuccess) return e;
	int tiles = 0;
	for (int l = 0; l <= a.net.H; ++l) tiles += (a.net.sizes[l] + 1) / 2 * sf_quads(a.net.sizes[l + 1]);
	const int least = sf_least_samples(a.net.mb);
	int warps = (a.net.mb + least - 1) / least;  // (not by sr: how phase 2 shares its sums out goes with the threads)
	if (warps < (tiles + 31) / 32 + a.net.H) warps = (tiles + 31) / 32 + a.net.H;  // phase 2: a warp for every 32 tiles and for every bias
	if (warps < a.net.H + 1) warps = a.net.H + 1;
	if (warps < 4) warps = 4;
	if (warps > SF_THREADS / 32) warps = SF_THREADS / 32;
	SmallFusedArgs copy = a;
	void* params[] = {&copy};
	return cudaLaunchKernel(kernel, dim3(1), dim3(warps * 32), params, bytes, s);
}
#endif  // SF_KERNEL_SAMPLES

}  // namespace glb
