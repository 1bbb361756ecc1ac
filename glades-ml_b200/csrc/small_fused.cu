// Batched mode for small networks: one persistent CTA trains n_epochs * windows in a single launch
// with ALL weights resident in shared memory.
//
// Per window (aligned, `mb` rows, weights frozen inside it):
//   phase 1  one warp per SR samples: forward (lane = output node, one fmaf chain per node and sample, k ascending), optional
//            softmax and the output delta, a group of lanes per sample, then the deltas of the hidden layers (lane = input
//            node, plain error sum);
//   phase 2  one thread per four weights of a row: G = sum_j c_j * (lr*d_jo*a_ji + decay terms) over the window's
//            samples in row order (deterministic), W -= G / len; the last warps sum the hidden layers' scalar-bias deltas.
// Two block-wide barriers per window; the next window's rows travel during the current one.
// Arithmetic = the batched mode of batched.cu (reference loop Networks/network.cpp:457-668 with
// aligned windows, frozen weights and a plain error sum); c_j is the closed form of the reference's
// intra-window momentum history (State/node.cpp:278-292).
//
// What bounds a window is shared memory's one row of 128 bytes per clock, then the latency of the chains.  So a weight that has
// been read serves SR samples and, in phase 2, an activation quad serves four weights; rows are padded to whole quads with a
// pitch of an odd number of them, so that 16-byte reads of 8 neighbouring rows hit all banks.  Measured, 10-32-32-1 with
// windows of 32 rows: one warp per sample and one thread per weight 12.5 us per window, MEASURED now.
#include "common.cuh"
#include "internal.h"

namespace glb {

__host__ __device__ __forceinline__ int sf_quads(int n) { return (n + 3) >> 2; }
__host__ __device__ __forceinline__ int sf_pitch(int ni) { return 4 * (sf_quads(ni) | 1); }

template <int SR>
__global__ void __launch_bounds__(1024, 1) small_fused_kernel(const __grid_constant__ SmallFusedArgs a)
{
	extern __shared__ __align__(16) float sm[];
	const NetView& n = a.net;
	const int H = n.H;
	const int T = blockDim.x, t = threadIdx.x;
	const int lane = t & 31, warp = t >> 5, nwarps = T >> 5;
	const int n_in = n.sizes[0], n_out = n.sizes[H + 1];
	const int mb = n.mb, mbp = (mb + SR - 1) / SR * SR;

	// shared memory: padded weights | activations and deltas of layers 1..H+1, [mbp][tot] each | inputs of two windows
	// [2][mbp][ipitch] | targets of two windows | momentum weights and the same times the learning rate, [H+1][mb] each | biases
	int node_off[GL_MAX_WEIGHT_LAYERS + 2];
	int tot = 0, tiles = 0;
	float* Wp[GL_MAX_WEIGHT_LAYERS];
	float* cur = sm;
	for (int l = 0; l <= H; ++l)
	{
		node_off[l + 1] = tot;
		tot += 4 * sf_quads(n.sizes[l + 1]);
		tiles += sf_quads(n.sizes[l]) * n.sizes[l + 1];
		Wp[l] = cur;
		cur += 4 * sf_quads(n.sizes[l + 1]) * sf_pitch(n.sizes[l]);
	}
	const int ipitch = 4 * sf_quads(n_in);
	float* const A = cur;
	float* const D = A + (size_t)mbp * tot;
	float* const Xs = D + (size_t)mbp * tot;
	float* const Ys = Xs + (size_t)2 * mbp * ipitch;
	float* const cw = Ys + (size_t)2 * mbp * n_out;
	float* const clr = cw + (H + 1) * mb;
	float* const sbias = clr + (H + 1) * mb;
	float* const end = sbias + GL_MAX_WEIGHT_LAYERS;
	__shared__ double swarp[32][2];

	for (float* p = sm + t; p < end; p += T) *p = 0.0f;  // (paddings stay zero)
	__syncthreads();
	for (int l = 0; l <= H; ++l)
	{
		const int ni = n.sizes[l], no = n.sizes[l + 1], ld = sf_pitch(ni);
		for (int e = t; e < ni * no; e += T) Wp[l][(e / ni) * ld + (e % ni)] = n.W[l][e];
	}
	if (t < GL_MAX_WEIGHT_LAYERS) sbias[t] = n.bias[t];
	const bool classify = n.out_type != GL_OUT_REGRESSION;
	if (classify)
		for (int e = t; e < n_out * n_out; e += T) a.confusion[e] = 0;

	const uint32_t xaddr = (uint32_t)__cvta_generic_to_shared(Xs), yaddr = (uint32_t)__cvta_generic_to_shared(Ys);
	auto fetch = [&](long long r0, int buf) {
		const int len = (int)((a.rows - r0) < mb ? (a.rows - r0) : mb);
		for (int j = warp; j < len; j += nwarps)
		{
			for (int i = lane; i < n_in; i += 32) cp_async4(xaddr + (uint32_t)((buf * mbp + j) * ipitch + i) * 4, a.X + (r0 + j) * n_in + i, true);
			for (int o = lane; o < n_out; o += 32) cp_async4(yaddr + (uint32_t)((buf * mbp + j) * n_out + o) * 4, a.Y + (r0 + j) * n_out + o, true);
		}
		cp_async_commit();
	};
	fetch(0, 0);
	cp_async_wait<0>();
	__syncthreads();

	const float data_size = (float)(a.rows * (long long)n_out);
	const bool softmax = n.act[H] == GL_ACT_SOFTMAX;
	int gw = 1;  // lanes per sample at the head
	while (gw < n_out && gw < 32) gw <<= 1;
	int cur_len = -1, buf = 0;

	for (int ep = 0; ep < a.n_epochs; ++ep)
	{
		const bool last_epoch = ep == a.n_epochs - 1;
		double ecost = 0.0, eacc = 0.0;  // this thread's share
		for (long long r0 = 0; r0 < a.rows; r0 += mb, buf ^= 1)
		{
			const int len = (int)((a.rows - r0) < mb ? (a.rows - r0) : mb);
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
					cw[l * mb + j] = c;
					clr[l * mb + j] = n.lr[l] * c;
				}
				cur_len = len;
			}
			if (r0 + mb < a.rows) fetch(r0 + mb, buf ^ 1);
			else if (!last_epoch) fetch(0, buf ^ 1);
			const float* const X = Xs + (size_t)buf * mbp * ipitch;
			const float* const Y = Ys + (size_t)buf * mbp * n_out;
			// ---------------- phase 1: one warp per SR samples (rows beyond `len` are computed from what lies there, and not used)
			for (int j0 = warp * SR; j0 < len; j0 += nwarps * SR)
			{
				float* const aj = A + (size_t)j0 * tot;
				float* const dj = D + (size_t)j0 * tot;
				for (int l = 0; l <= H; ++l)
				{
					const int no = n.sizes[l + 1], ld = sf_pitch(n.sizes[l]), quads = sf_quads(n.sizes[l]);
					const float* in = l ? aj + node_off[l] : X + (size_t)j0 * ipitch;
					const int ipt = l ? tot : ipitch;
					float* out = aj + node_off[l + 1];
					const float b = (l >= 1) ? sbias[l] : 0.0f;
					for (int o = lane; o < no; o += 32)
					{
						const float4* w = reinterpret_cast<const float4*>(Wp[l] + o * ld);
						float z[SR];
#pragma unroll
						for (int s = 0; s < SR; ++s) z[s] = 0.0f;
#pragma unroll 2
						for (int q = 0; q < quads; ++q)
						{
							const float4 wv = w[q];
							float4 v[SR];
#pragma unroll
							for (int s = 0; s < SR; ++s) v[s] = *reinterpret_cast<const float4*>(in + s * ipt + 4 * q);
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
						for (int s = 0; s < SR; ++s) out[s * tot + o] = squash_b(z[s] + b, n.act[l], n.par[l]);
					}
					__syncwarp();
				}
				// head: optional softmax, output delta, figures; gw lanes per sample
				for (int s0 = 0; s0 < SR; s0 += 32 / gw)
				{
					const int s = s0 + lane / gw, og = lane & (gw - 1);
					const bool row = s < SR && j0 + s < len;
					const int j = row ? j0 + s : j0;
					float* p = A + (size_t)j * tot + node_off[H + 1];
					float* dout = D + (size_t)j * tot + node_off[H + 1];
					const float* y = Y + (size_t)j * n_out;
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
							dout[o] = d;
							ecost += (double)cost;
							eacc += (double)fmaxf((1.0f - fminf(fabsf(pv - e), 1.0f)) * 100.0f, 0.0f);
							if (e > be) { be = e; ie = o; }
							if (pv > bp) { bp = pv; ip = o; }
							if (a.last_out && last_epoch && r0 + j == a.rows - 1) a.last_out[o] = pv;
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
					const int ni = n.sizes[l], ld = sf_pitch(ni), quads = sf_quads(n.sizes[l + 1]);
					const float* dup = dj + node_off[l + 1];
					for (int i = lane; i < ni; i += 32)
					{
						const float* w = Wp[l] + i;
						float e[SR];
#pragma unroll
						for (int s = 0; s < SR; ++s) e[s] = 0.0f;
#pragma unroll 2
						for (int q = 0; q < quads; ++q)
						{
							const float w0 = w[(4 * q) * ld], w1 = w[(4 * q + 1) * ld], w2 = w[(4 * q + 2) * ld], w3 = w[(4 * q + 3) * ld];
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
						for (int s = 0; s < SR; ++s)
							dj[s * tot + node_off[l] + i] = e[s] * act_der_b(aj[s * tot + node_off[l] + i], n.act[l - 1], 0.01f);
					}
					__syncwarp();
				}
			}
			__syncthreads();
			// ---------------- phase 2: gradient + update, one thread per four weights of a row
			const float inv_len = 1.0f / (float)len;
			for (int e0 = t; e0 < tiles; e0 += T)
			{
				int l = 0, e = e0;
				for (; e >= sf_quads(n.sizes[l]) * n.sizes[l + 1]; ++l) e -= sf_quads(n.sizes[l]) * n.sizes[l + 1];
				const int quads = sf_quads(n.sizes[l]), o = e / quads, iq = e - o * quads;
				const float* av = l ? A + node_off[l] + 4 * iq : X + 4 * iq;
				const int apt = l ? tot : ipitch;
				const float* dv = D + node_off[l + 1] + o;
				const float* c = cw + l * mb;
				const float* cl = clr + l * mb;
				float4 g = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
				for (int j = 0; j < len; ++j)
				{
					const float4 x = *reinterpret_cast<const float4*>(av + (size_t)j * apt);
					const float s = cl[j] * dv[(size_t)j * tot];
					g.x = fmaf(s, x.x, g.x);
					g.y = fmaf(s, x.y, g.y);
					g.z = fmaf(s, x.z, g.z);
					g.w = fmaf(s, x.w, g.w);
				}
				const float w1 = n.wd1[l] * n.lr[l], w2 = n.wd2[l] * n.lr[l];
				if (w1 != 0.0f || w2 != 0.0f)
					for (int j = 0; j < len; ++j)
					{
						const float4 x = *reinterpret_cast<const float4*>(av + (size_t)j * apt);
						g.x = fmaf(c[j], fmaf(w1, fabsf(x.x), w2 * x.x), g.x);
						g.y = fmaf(c[j], fmaf(w1, fabsf(x.y), w2 * x.y), g.y);
						g.z = fmaf(c[j], fmaf(w1, fabsf(x.z), w2 * x.z), g.z);
						g.w = fmaf(c[j], fmaf(w1, fabsf(x.w), w2 * x.w), g.w);
					}
				float4* w = reinterpret_cast<float4*>(Wp[l] + o * sf_pitch(n.sizes[l]) + 4 * iq);
				float4 v = *w;
				v.x -= g.x * inv_len;
				v.y -= g.y * inv_len;
				v.z -= g.z * inv_len;
				v.w -= g.w * inv_len;
				*w = v;
			}
			// scalar biases of the hidden layers: lr * sum of the deltas of the layer above, on the warps that have the fewest weights
			if (nwarps - 1 - warp < H)
			{
				const int l = nwarps - warp, no = n.sizes[l + 1];
				const float* d = D + node_off[l + 1];
				// lanes side by side on a row's nodes, as many rows at once as fit
				int w = 1;
				while (w < no && w < 32) w <<= 1;
				double s0 = 0.0, s1 = 0.0;
				for (int o = lane & (w - 1); o < no; o += w)
				{
					int j = lane / w;
					const int step = 32 / w;
					for (; j + step < len; j += 2 * step)
					{
						s0 += (double)d[(size_t)j * tot + o];
						s1 += (double)d[(size_t)(j + step) * tot + o];
					}
					if (j < len) s0 += (double)d[(size_t)j * tot + o];
				}
				const double s = warp_sum_d(s0 + s1) * (double)n.lr[l];
				if (lane == 0) sbias[l] -= (a.bias_rule == GL_BIAS_REFERENCE) ? (float)(s * (double)n.sizes[l]) : (float)(s / (double)len);
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
		const int ni = n.sizes[l], no = n.sizes[l + 1], ld = sf_pitch(ni);
		for (int e = t; e < ni * no; e += T)
		{
			const float w = Wp[l][(e / ni) * ld + (e % ni)];
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

// Samples per warp in phase 1: four where that leaves eight warps or more, two per scheduler.
static int sf_samples(int mb) { return mb > 28 ? 4 : (mb > 8 ? 2 : 1); }

size_t small_fused_smem_bytes(const NetView& n)
{
	const size_t sr = sf_samples(n.mb), mbp = ((size_t)n.mb + sr - 1) / sr * sr;
	size_t f = 0, tot = 0;
	for (int l = 0; l <= n.H; ++l)
	{
		tot += 4 * sf_quads(n.sizes[l + 1]);
		f += (size_t)4 * sf_quads(n.sizes[l + 1]) * sf_pitch(n.sizes[l]);
	}
	f += 2 * mbp * (tot + 4 * sf_quads(n.sizes[0]) + n.sizes[n.H + 1]) + 2 * (size_t)(n.H + 1) * n.mb + GL_MAX_WEIGHT_LAYERS;
	return f * sizeof(float);
}

cudaError_t launch_small_fused(const SmallFusedArgs& a, cudaStream_t s)
{
	const size_t bytes = small_fused_smem_bytes(a.net);
	const int sr = sf_samples(a.net.mb);
	void (*kernel)(SmallFusedArgs) = sr == 4 ? small_fused_kernel<4> : (sr == 2 ? small_fused_kernel<2> : small_fused_kernel<1>);
	cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
	if (e != cudaSuccess) return e;
	int tiles = 0;
	for (int l = 0; l <= a.net.H; ++l) tiles += sf_quads(a.net.sizes[l]) * a.net.sizes[l + 1];
	int warps = (a.net.mb + sr - 1) / sr;
	if (warps < (tiles + 31) / 32 + a.net.H) warps = (tiles + 31) / 32 + a.net.H;  // phase 2: a warp for every 128 weights and for every bias
	if (warps < a.net.H + 1) warps = a.net.H + 1;
	if (warps < 4) warps = 4;
	if (warps > 32) warps = 32;
	kernel<<<1, warps * 32, bytes, s>>>(a);
	return cudaGetLastError();
}

}  // namespace glb
