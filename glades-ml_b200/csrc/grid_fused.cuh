// What the two whole-window kernels (grid_fused.cu and its cluster variant in cluster_fused.cu) share: the window scratch, how
// the gradient phase cuts the weights into work items, and the CTAs' partial sums.
#pragma once
#include "common.cuh"
#include "internal.h"

namespace glb {

constexpr int GF_THREADS = 256;
constexpr int GF_TO = 16, GF_P2_TI = 32, GF_TJ = 64;  // phase 2: weight tiles of 16 outputs x 32 inputs, 64 rows per stage
// Layers with at most GF_NARROW output nodes (the usual regression head): work items of GF_NCOLS input columns.
constexpr int GF_NARROW = 4;
constexpr int GF_NCOLS = 64;
constexpr int GF_PART = 2 + GL_MAX_WEIGHT_LAYERS;  // doubles per CTA: cost, accuracy, bias-delta sums per layer

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

}  // namespace glb
