// Interface of the product kernel for few rows (gemm_skinny.cu).
#pragma once
#include "gemm_tcgen05.cuh"

constexpr int UGB_SKINNY_ROWS = 8;      // most rows of A it takes
constexpr int UGB_SKINNY_SPLITS = 8;     // most partials it writes

// Whether a decode step of `rows` rows runs its products on this kernel.  Measured at 8 rows: a 2048 x 2048 projection
// takes 2.5 us in the chain of a step against 4.5 on 64-row tcgen05 tiles; beyond 8 rows the activations no longer fit
// the registers beside the weights in flight (with half of those in flight 16 rows took 1.22 ms a step against 1.16).
inline bool ugb_skinny_rows(size_t rows) { return rows >= 1 && rows <= (size_t)UGB_SKINNY_ROWS; }

// Whether every CTA has one piece (16 rows of W) of an unsplit product at most.
bool ugb_skinny_one_round(int sm_count, size_t n, size_t batch);

// k splits of a product with a f32 result that the consumer sums: 2048 inputs or fewer each, more where the columns alone do
// not fill the SMs.
int ugb_skinny_splits(int sm_count, size_t n, size_t k);

// gelu_tanh
static __device__ __forceinline__ float ugb_gelu_tanh(float x) { return 0.5f * x * (1.0f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x))); }

// Activations that the kernel forms itself: A[r, j] = bf16(gelu_tanh(sum_p part[p][r][j]) * table[tok[r]][off + j]), j < n = k; 0 for a
// token outside the table.
struct ugb_skinny_gate {
  const float *part;
  int n_part;
  size_t part_stride;
  int ld, n;
  const int *tok;
  const __nv_bfloat16 *table;
  size_t table_ld;
  int off, vocab;
};

// out = A . W^T for up to 8 rows, arguments and epilogues as ugb_tc_gemm (no rope, no n-major B, no pair_k); `splits` as
// given, rounded as ugb_skinny_effective_splits says.  Grouped rows: tiles of g.tile_m rows of which the first
// `rows_per_tile` may hold something; m is their total.  UGB_ERR_UNSUPPORTED (last_error untouched) for what it does not take.
// With `gate`, g.a is not read (f32 or bf16 result, k of 512 at most).
int32_t ugb_skinny_gemm(ugb_device *dev, const ugb_tc_gemm_args &g, int rows_per_tile = 0, const ugb_skinny_gate *gate = nullptr);
int ugb_skinny_effective_splits(size_t k, int splits);
