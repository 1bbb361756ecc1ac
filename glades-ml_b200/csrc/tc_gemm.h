// Tensor-core matrix product of batched mode: TMA-fed tcgen05.mma (kind::f16) on operands split into a high and
// a low fp16 part under a per-matrix power-of-two scale ("3xFP16"), fp32 accumulation in tensor memory.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "internal.h"

namespace glb {

// Scale record of a split matrix (device memory).  Stored parts of an element x:
//   hi = fp16(x * 2^e),  lo = fp16((x * 2^e - hi) * 2^11)
// amax: bits of the largest finite |x|; e is chosen so that |x| * 2^e < 2^15 for every element.
struct TensorScale
{
	unsigned amax;
	int e;
};

// A split matrix as an operand X(r, k).  mn == 0: stored [r][k] (K-contiguous), mn == 1: stored [k][r].  ld halfs per row, a
// multiple of 8; for mn == 1 the columns from the true width up to the next multiple of 64 must exist in every row
// (ld a multiple of 64) and hold zeros.
struct SplitOperand
{
	const __half* hi;
	const __half* lo;
	long long ld;
	const TensorScale* sc;
	int mn;
};

struct TcGemmArgs
{
	SplitOperand A, B;  // C[m][n] = sum_k A(m,k) * B(n,k); any M, N, K >= 1
	int M, N, K;
	int epi;            // EPI_*
	float* C;           // fp32 output, pitch ldc, or NULL
	long long ldc;
	__half* Chi;        // split output, pitch ldch (multiple of 8), scale record csc (amax is maxed into, e is set); or NULL
	__half* Clo;
	long long ldch;
	TensorScale* csc;
	float* Clo32;           // low TF32 parts of C (pitch ldc), with W of the new weights (pitch N); or NULL
	const float* bias_ptr;  // EPI_FORWARD: device scalar or NULL
	int act;
	float par;
	const float* aux;       // EPI_ERRPROP without mask: activations, 16-byte aligned rows
	long long ld_aux;
	float alpha;            // EPI_GRAD
	const float* colterm;
	unsigned* relu_mask_out;       // [M][mask_ld] words, mask_ld a multiple of 4
	const unsigned* relu_mask_in;
	int mask_ld;
	double* dsum;           // EPI_ERRPROP: [tc_dsum_parts(M, N)] partial sums of the output, one per tile and epilogue warp; or NULL
	int* dsum_count;        // host: how many were written
	// EPI_GRAD with W != NULL: the update W -= C * inv_mb is applied in place (W [M][N] fp32, pitch N), C is not stored;
	// Chi/Clo/csc receive the new weights' split, wsc is the old weights' record
	float* W;
	const TensorScale* wsc;
	float inv_mb;
	float decay_bound;      // largest |colterm| per unit of the activations' amax
	int* bad_flag;          // bit 0 set when a new weight is not finite
	int sm_reserve;
	const void* peer_maps;
	int band_rows;
	int peer_self;
	const TcSplitK* sk;
};

bool tc_gemm_available();

// An fp32 matrix with its low TF32 parts as an operand of the 3xTF32 product (gemm_tf32.cu): X(r, k) stored [r][k] (mn == 0) or
// [k][r] (mn == 1), pitch ld floats.
struct Tf32Operand
{
	const float* x;
	const float* lo;
	long long ld;
	int mn;
};
// M % 128 == 0, N % 128 == 0, K % 16 == 0, rows on 16-byte boundaries
bool tf32_gemm_fits(const Tf32Operand& A, const Tf32Operand& B, int M, int N, int K);
// The same epilogues and outputs as launch_gemm_tc (plus Clo32); of g.A and g.B only the scale records are read, and those only
// for a split output.
cudaError_t launch_gemm_tf32(const TcGemmArgs& g, const Tf32Operand& A, const Tf32Operand& B, int* err_flag, cudaStream_t s);
cudaError_t launch_scale_split_lo(const float* src, const float* rowscale, int ld, float* dst, float* lo, long long count, cudaStream_t s);
// lo[i] = low TF32 part of src[i]; count a multiple of 4, pointers 16-byte aligned
cudaError_t launch_split_lo(const float* src, float* lo, long long count, cudaStream_t s);
// One launch of engine 0 (3xFP16) or 1 (3xTF32), for the counts below.
void tc_count_launch(int engine, bool wide, bool several_tiles, bool peer, bool split);
cudaError_t prepare_tc_launch(const void* kernel, int smem_bytes, int* sm_count);
// fp32 operand for 16-deep k-blocks: K-contiguous rows (64-byte swizzle), or MN-contiguous as [r/32][k][r%32]
bool tc_make_operand_map_f32(void* out128, const float* ptr, int mn, long long rows, long long k, long long ld, int box_rows);
// the shapes that the public matrix-product entry points take on this engine: M % 128 == 0, N % 128 == 0, K % 16 == 0, every
// operand contiguous in k or in m/n with 16-byte aligned rows
bool tc_matmul_shape_ok(const GemmArgs& g);
// C = A * B^T of such a product: the operands' parts go to a_scratch / b_scratch (tc_matmul_operand_bytes each, 256-byte aligned),
// their scale records to header (64 bytes, zeroed by the caller).  bands (optional): a data-parallel gradient's epilogue and
// stores in place of C.
size_t tc_matmul_operand_bytes(long long r, long long k);
cudaError_t tc_matmul(const GemmArgs& g, void* header, void* a_scratch, void* b_scratch, const TcSplitK* sk, int* err_flag, cudaStream_t s,
                      const TcGemmArgs* bands = nullptr);
// number of doubles launch_gemm_tc writes to dsum
long long tc_dsum_parts(int M, int N);
// err_flag: device int, set non-zero if a bounded wait inside the kernel ran out.
cudaError_t launch_gemm_tc(const TcGemmArgs& g, int* err_flag, cudaStream_t s);

// Launch counts per tile variant since the library was loaded: [0] tiles of at most 128 columns, [1] 256-wide tiles,
// [2] launches whose persistent CTAs walked more than one tile each, [3] data-parallel (peer-store) launches,
// [4] launches that split their last wave of tiles along k.
void tc_variant_counts(long long out5[5]);
// The same launches per engine: [0] 3xFP16 (gemm_tcgen05.cu), [1] 3xTF32 (gemm_tf32.cu).
void tc_engine_counts(long long out2[2]);

// Tensor map (128 bytes, 64-byte aligned storage) over a row-major [rows][cols] fp32 matrix with 32 x 32
// boxes, as the epilogue's bulk stores use it; for the per-owner bands of a data-parallel gradient.
bool tc_make_store_map(void* out128, const float* base, long long rows, long long cols, long long ld);

// General 2-D map over a row-major [rows][cols] fp32 matrix (row pitch ld floats, a multiple of 4; base
// 16-byte aligned): boxes of box_rows x box_cols, 128-byte swizzle (box_cols must then be 32) or none.
bool tc_make_map2d(void* out128, const float* base, long long rows, long long cols, long long ld, int box_cols, int box_rows,
                   int swizzle128);
// A [stages][8 groups][8 rows][ld] view of a row-major fp32 matrix of 64 * stages rows (pitch ld, a multiple of 4), in boxes of box_stages x
// box_groups x 8 rows x box_cols.
bool tc_make_rows_map(void* out128, const float* base, long long stages, long long ld, int box_cols, int box_groups, int box_stages);

// sc->amax = max(sc->amax, largest finite |src|) over a [rows][cols] matrix of pitch ld (the caller presets amax)
cudaError_t launch_amax(const float* src, long long rows, int cols, long long ld, TensorScale* sc, cudaStream_t s);
// hi / lo of src under the scale that sc->amax asks for; writes sc->e.  Columns cols..ldo-1 are written as zeros.
cudaError_t launch_split(const float* src, long long rows, int cols, long long ld, TensorScale* sc, __half* hi, __half* lo, long long ldo,
                         cudaStream_t s);
// the same from an already split matrix (src scale ssc), row r times rowscale[r] (|rowscale| <= rowscale_max): for
// momentum-weighted deltas
cudaError_t launch_rescale_split(const __half* shi, const __half* slo, const TensorScale* ssc, long long rows, int cols, long long lds,
                                 const float* rowscale, float rowscale_max, TensorScale* sc, __half* hi, __half* lo, long long ldo,
                                 cudaStream_t s);

}  // namespace glb
