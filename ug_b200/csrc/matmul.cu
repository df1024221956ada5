// ug::Device::matmul for the B200 backend.
//
// The reference forwards every matmul to cublasGemmStridedBatchedEx after
// deriving transposition flags, leading dimensions and batch strides from the
// two operand layouts (ug-cuda/src/gemm.rs:8-83,292-332).  Here the same
// layout rules pick between
//   * the tcgen05 / TMEM tensor-core kernel (bf16 operands, fp32 accumulate),
//     declared in gemm_tcgen05.cuh, and
//   * for f32 (the dtype ug-llama casts every weight to, model.rs:118,140,313) two FP32-pipe kernels, a
//     warp-per-column streaming kernel for the skinny products of a decode step and a register-blocked FFMA kernel
//     for short sums, and for the rest the tensor cores on three bf16 parts of every value (gemm_f32_split.cu), and
//   * the same FFMA kernel on 16-bit operands for the shapes and layouts the tensor-core kernels do not take.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "gemm_f32_split.cuh"
#include "gemm_plan.h"
#include "gemm_skinny.cuh"
#include "gemm_tcgen05.cuh"
#include "ugb_internal.h"

namespace {

struct MatLayout {
  long long rs, cs;   // element strides of the last two dims
  long long batch;    // element stride between batch steps
  bool transposed;    // true when the minor stride is on the row index
};

// gemm.rs:18-43 (minor dims) and :59-74 (batch stride).  `rows`/`cols` are the
// logical extents of the last two dims (m,k for lhs; k,n for rhs).
int32_t parse_layout(ugb_device *dev, const char *which, int rank, const size_t *dims,
                     const size_t *strides, size_t rows, size_t cols, MatLayout *out) {
  UGB_REQUIRE(dev, rank >= 2 && rank <= 4, UGB_ERR_SHAPE, "matmul: %s rank %d not in 2..4", which, rank);
  const size_t m1 = strides[rank - 1], m2 = strides[rank - 2];
  if ((m1 == 1 || cols == 1) && (m2 == cols || rows == 1)) {
    out->rs = (long long)cols;
    out->cs = 1;
    out->transposed = false;
  } else if ((m1 == rows || cols == 1) && (m2 == 1 || rows == 1)) {
    out->rs = 1;
    out->cs = (long long)rows;
    out->transposed = true;
  } else {
    return ugb_fail(dev, UGB_ERR_SHAPE, "non contiguous matmul, %s strides (..., %zu, %zu) for %zux%zu",
                    which, m2, m1, rows, cols);
  }
  const int nb = rank - 2;
  if (nb == 0) {
    out->batch = (long long)(rows * cols);
  } else if (nb == 1) {
    out->batch = (long long)strides[0];
  } else {
    const size_t s1 = strides[0], s2 = strides[1];
    if (s1 == s2 * dims[1]) out->batch = (long long)s2;
    else if (dims[0] == 1) out->batch = (long long)s2;
    else if (dims[1] == 1) out->batch = (long long)s1;
    else
      return ugb_fail(dev, UGB_ERR_SHAPE, "non contiguous matmul, %s batch strides (%zu, %zu)", which, s1, s2);
  }
  return UGB_OK;
}

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }

// The kernels below are dependent launches: they are resident while the kernels that write their operands may still run.  So
// no operand is read through the non-coherent path (__ldg, or const __restrict__), which wants memory that nothing writes as
// long as the kernel lives; ordinary loads behind the wait see what was written before it.
// The 16-byte ones are written out: the compiler's own sink to their uses, one behind the other ([12, 8192] x [64, 8192]^T
// 122 us so, 58 with all in flight).  Single values of a guarded piece are left to it (64 times [1339, 597] x [597, 19] in bf16
// 506 us so, 931 written out).
__device__ __forceinline__ float4 ld_global(const float4 *p) {
  float4 v;
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

// ---- fp32 on the FP32 pipe (the reference's default for f32 is CUBLAS_COMPUTE_32F, gemm.rs:87-128: no reduced
// precision), two shapes -------------------------------------------------------------------------------------
// (1) Skinny products, m <= 16 rows against a [n, k] operand with k contiguous (Linear::fwd = matmul_t with a
// weight, model.rs:147-149, for the one new token of a decode step): HBM-bound on the weight.  One warp per output
// column: the lanes stream the column's k values with 128-bit loads, every value is used for all m rows, the
// partial dot products are summed by warp shuffles.
template <int MR>
__global__ void __launch_bounds__(256)
f32_skinny_kernel(float *C, const float *A, const float *B, int m, int n, int k, long long a_b, long long b_b) {
  ugb_pdl_trigger();
  ugb_pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * 8 + warp;
  if (col >= n) return;
  const int batch = blockIdx.y;
  const float4 *w = reinterpret_cast<const float4 *>(B + (long long)batch * b_b + (long long)col * k);
  const float *a = A + (long long)batch * a_b;
  float acc[MR];
#pragma unroll
  for (int r = 0; r < MR; ++r) acc[r] = 0.f;
  const int k4 = k >> 2;
#pragma unroll 4
  for (int c = lane; c < k4; c += 32) {
    const float4 wv = __ldcs(w + c);                 // streamed once
#pragma unroll
    for (int r = 0; r < MR; ++r) {
      if (r < m) {
        const float4 x = ld_global(reinterpret_cast<const float4 *>(a + (long long)r * k) + c);
        acc[r] = fmaf(x.x, wv.x, fmaf(x.y, wv.y, fmaf(x.z, wv.z, fmaf(x.w, wv.w, acc[r]))));
      }
    }
  }
#pragma unroll
  for (int r = 0; r < MR; ++r) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
    if (lane == 0 && r < m) C[(long long)batch * m * n + (long long)r * n + col] = acc[r];
  }
}

// (1b) Skinny products against a [k, n] operand with n contiguous (Attention::fwd's probabilities x values for the
// one new token, model.rs:243: [1, T] x [T, 64] per head): one CTA per (128-column chunk, batch step); its warps (32 for
// m <= 2, fewer for more rows) split k, a lane keeps 4 adjacent columns, so every k row of the chunk is one coalesced 512-byte read per warp and
// is used for all m rows; the partial sums meet in shared memory.  (32 heads x [1, 1024] x [1024, 64] took 199 us
// on 128 x 128 tiles.)
template <int MR>
__global__ void __launch_bounds__(MR <= 2 ? 1024 : (MR <= 4 ? 512 : 256))
f32_skinny_n_kernel(float *C, const float *A, const float *B, int m, int n, int k, long long a_rs, long long a_b, long long b_rs, long long b_b) {
  constexpr int WARPS = MR <= 2 ? 32 : (MR <= 4 ? 16 : 8);       // 32 KiB of partial sums at most
  __shared__ __align__(16) float red[WARPS][MR][128];
  ugb_pdl_trigger();
  ugb_pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int batch = blockIdx.y, col = blockIdx.x * 128 + lane * 4;
  const float *a = A + (long long)batch * a_b;
  const float *bp = B + (long long)batch * b_b + col;
  float acc[MR][4];
#pragma unroll
  for (int r = 0; r < MR; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
  if (col < n) {                                       // n % 4 == 0: a lane's 4 columns are all in or all out
#pragma unroll 8
    for (int kk = warp; kk < k; kk += WARPS) {
      const float4 bv = __ldcs(reinterpret_cast<const float4 *>(bp + (long long)kk * b_rs));
#pragma unroll
      for (int r = 0; r < MR; ++r) {
        if (r < m) {
          const float x = a[(long long)r * a_rs + kk];
          acc[r][0] = fmaf(x, bv.x, acc[r][0]); acc[r][1] = fmaf(x, bv.y, acc[r][1]);
          acc[r][2] = fmaf(x, bv.z, acc[r][2]); acc[r][3] = fmaf(x, bv.w, acc[r][3]);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < MR; ++r)
    *reinterpret_cast<float4 *>(&red[warp][r][lane * 4]) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
  __syncthreads();
  for (int i = threadIdx.x; i < MR * 128; i += WARPS * 32) {
    const int r = i >> 7, c = i & 127, gc = blockIdx.x * 128 + c;
    if (r < m && gc < n) {
      float sum = 0.f;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) sum += red[w][r][c];
      C[(long long)batch * m * n + (long long)r * n + gc] = sum;
    }
  }
}

// (2) Everything else in f32.  A warp owns 32 x 128 outputs, a thread 8 x 16 of them; of the four warps of a CTA, WM lie side by
// side over rows and WK take parts of every k slice.  With p.split > 1 the CTAs of a cluster take equal parts of k as well.
// All partial sums meet in shared memory, in a fixed order.
//
// Bound: the FP32 pipe (74 TFLOP/s), with the shared-memory reads close behind: a 16-byte read of a warp takes four passes
// whatever its lanes have in common, so 8 x 8 outputs per thread (4 reads per 64 FFMA) leave no room above 100 % of both, 8 x 16
// (6 reads per 128) a quarter.  Two products per instruction (fma.rn.f32x2: the same roundings) halve the issue slots that the
// products take; the column pairs come out of shared memory as they are needed, the eight row values are doubled by moves.
// k slices of 16 go through registers into one of two buffers, 16-byte global reads where the layout allows (VEC), zeros behind
// the edges; the columns of slice k are permuted by 8 (k / 4 mod 4), so that four lanes along k and eight along the rows write
// without conflicts.
//
// [2048, 2048] x [4096, 2048]^T runs at 45 TFLOP/s with k unsplit, FMA pipe 75 % busy while its CTAs run, and at 50 with k split in two, as it is
// (two CTAs of 256 threads with 8 x 8 outputs on 128 x 128 tiles: 41, 64 %).  Against those: [257, 2048] x [5632, 2048]^T 288 -> 180 us,
// [1619, 1768] x [984, 1768]^T 246 -> 136, [120, 7144] x [1352, 7144]^T 978 -> 112, [2, 6045] x [338, 6045]^T 977 -> 44.  Slices of 8 were
// slower (683 -> 770 us on the first), and CTAs whose warps lie over columns no faster than these.
// The next kernel is let in by this one's end, not by a trigger: let in earlier, the CTAs of a product of 75 to 148 tiles come to SMs that are
// still taken, two on one and none on another, and that product takes nearly twice as long (2 of [526, 216] x [1080, 216]^T one behind the other
// 43 us with a trigger at the start, 34 with one behind the last slice, 26 without; 64 of [128, 64] x [128, 64]^T 12.4, 9.0, 8.8).
// 16-bit operands (E) that no tensor-core kernel takes, odd rows above all: [500, 999] x [1001, 999]^T 168 -> 44 us, [11, 2001] x
// [200, 2001]^T 271 -> 36 on 64 x 64 tiles of one 16-deep buffer before.
template <int WM, int WK> struct F32Tile {
  static constexpr int BM = 32 * WM, BN = 128, BK = 16, THREADS = 32 * WM * WK;
  static constexpr int STAGE = BK * (BM + BN);                                     // floats
  static constexpr int SMEM = 2 * STAGE * 4, SMEM_REDUCE = WK * BM * BN * 4;       // bytes; the sums come after the slices
};
struct F32Params {
  void *c;
  const void *a, *b;
  int m, n, k;
  long long a_rs, a_cs, a_b, b_rs, b_cs, b_b, c_rs, c_b;
  int split, k_per_split;                              // CTAs of a cluster along k
};

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint64_t twice(float x) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float2 halves(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

// TURNED: the product's rows are the tile's columns, C^T = B^T A^T.
template <typename E, int WM, int WK, bool VEC, bool TURNED>
__global__ void __launch_bounds__(128, 2)
f32_tile_kernel(const F32Params p) {
  using T = F32Tile<WM, WK>;
  constexpr int BM = T::BM, BN = T::BN, BK = T::BK, QK = BK / 4, SW = 32 / QK;
  static_assert(T::THREADS == 128, "four warps");
  extern __shared__ __align__(16) float smem[];
  ugb_pdl_wait();
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int rank = p.split > 1 ? (int)(blockIdx.x % p.split) : 0, n0 = (int)(p.split > 1 ? blockIdx.x / p.split : blockIdx.x) * BN;
  const int m0 = blockIdx.y * BM;
  const E *A = (const E *)p.a + (long long)blockIdx.z * p.a_b, *B = (const E *)p.b + (long long)blockIdx.z * p.b_b;
  static_assert(!VEC || sizeof(E) == 4, "16-byte pieces are four floats");
  const int k_lo = rank * p.k_per_split, k_hi = min(p.k, k_lo + p.k_per_split);

  // One operand's slice: R rows of 16 k, in pieces of four values along the contiguous direction
  auto fetch = [&](auto &reg, const E *src, long long rs, long long ks, int r0, int rows, int R, int k0) {
    const bool kc = ks == 1;
#pragma unroll
    for (int i = 0; i < (int)(sizeof(reg) / sizeof(float4)); ++i) {
      const int q = t + i * 128;
      const int r = r0 + (kc ? q / QK : q % (R / 4) * 4), k = k0 + (kc ? q % QK * 4 : q / (R / 4));
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      const E *at = src + r * rs + k * ks;
      if constexpr (VEC) {                             // a piece is all in or all out
        if (r < rows && k < k_hi) {
          const float4 w = ld_global(reinterpret_cast<const float4 *>(at));
          v[0] = w.x; v[1] = w.y; v[2] = w.z; v[3] = w.w;
        }
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (kc ? r < rows && k + e < k_hi : r + e < rows && k < k_hi) v[e] = to_f32<E>(at[e * (kc ? ks : rs)]);
      }
      reg[i] = make_float4(v[0], v[1], v[2], v[3]);
    }
  };
  auto stage = [&](const auto &reg, float *dst, long long ks, int R) {
    const bool kc = ks == 1;
#pragma unroll
    for (int i = 0; i < (int)(sizeof(reg) / sizeof(float4)); ++i) {
      const int q = t + i * 128;
      if (kc) {
        const int r = q / QK ^ q % QK * SW, k = q % QK * 4;
        dst[k * R + r] = reg[i].x; dst[(k + 1) * R + r] = reg[i].y; dst[(k + 2) * R + r] = reg[i].z; dst[(k + 3) * R + r] = reg[i].w;
      } else {
        const int k = q / (R / 4), r = q % (R / 4) * 4 ^ (k >> 2) * SW;
        *reinterpret_cast<float4 *>(dst + k * R + r) = reg[i];
      }
    }
  };
  float4 ra[BM * BK / 512], rb[BN * BK / 512];
  auto fetch_both = [&](int k0) {
    fetch(ra, A, p.a_rs, p.a_cs, m0, p.m, BM, k0);
    fetch(rb, B, p.b_cs, p.b_rs, n0, p.n, BN, k0);
  };
  auto stage_both = [&](int buf) {
    stage(ra, smem + buf * T::STAGE, p.a_cs, BM);
    stage(rb, smem + buf * T::STAGE + BK * BM, p.b_rs, BN);
  };

  const int wk = warp % WK, wm = warp / WK;
  // Halves of this warp's part of a slice that hold anything.  The guarded reads of !VEC lose more by a bound that varies than
  // they gain ([65536, 63] x [63, 63]^T 37.4 -> 39.8 us); the others gain where k is short ([3694, 8] x [15392, 8]^T 58.8 -> 51.7,
  // 64 times [595, 8] x [8, 344] 18.5 -> 15.5).
  const bool live = m0 + wm * 32 < p.m;
  auto halves_of = [&](int k0) {
    constexpr int HALF = BK / WK / 2;
    return !VEC ? 2 : !live ? 0 : min(2, (k_hi - k0 - wk * 2 * HALF + HALF - 1) / HALF);
  };
  const int ty = lane >> 3, tx = lane & 7;
  uint64_t acc[8][8];                                  // columns in pairs
#pragma unroll
  for (int u = 0; u < 8; ++u)
#pragma unroll
    for (int v = 0; v < 8; ++v) acc[u][v] = 0ull;
  if (k_lo < k_hi) {
    fetch_both(k_lo);
    stage_both(0);
  }
  __syncthreads();
  int buf = 0;
  for (int k0 = k_lo; k0 < k_hi; k0 += BK) {
    const bool more = k0 + BK < k_hi;
    if (more) fetch_both(k0 + BK);
    const float *as = smem + buf * T::STAGE, *bs = as + BK * BM;
#pragma unroll 1
    for (int h = 0; h < halves_of(k0); ++h)               // rolled, or the compiler moves the global reads down to their use
#pragma unroll
    for (int j = 0; j < BK / WK / 2; ++j) {
      const int kk = wk * (BK / WK) + h * (BK / WK / 2) + j, x = (kk >> 2) * SW;
      const float *ar = as + kk * BM + wm * 32, *br = bs + kk * BN + (tx * 4 ^ x);
      const float4 a0 = *reinterpret_cast<const float4 *>(ar + (ty * 4 ^ x)), a1 = *reinterpret_cast<const float4 *>(ar + (16 + ty * 4 ^ x));
      const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      uint64_t b[8];
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(br + g * 32);
        b[2 * g] = w.x; b[2 * g + 1] = w.y;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const uint64_t aa = twice(a[u]);
#pragma unroll
        for (int v = 0; v < 8; ++v) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[u][v]) : "l"(aa), "l"(b[v]));
      }
    }
    if (more) {
      stage_both(buf ^ 1);
      __syncthreads();
      buf ^= 1;
    }
  }

  E *C = (E *)p.c + (long long)blockIdx.z * p.c_b;
  auto store = [&](int row, int col, float4 v) {       // row, col inside the tile
    const int gi = m0 + row, gj = n0 + col;
    if (gi >= p.m) return;
    E *at = TURNED ? C + gj * p.c_rs + gi : C + gi * p.c_rs + gj;
    if (VEC && !TURNED && gj + 3 < p.n) {
      if constexpr (VEC) *reinterpret_cast<float4 *>(at) = v;
    } else {
      const float w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (gj + e < p.n) at[TURNED ? e * p.c_rs : e] = from_f32<E>(w[e]);
    }
  };
  const bool alone = WK == 1 && p.split == 1;
  if (!alone) __syncthreads();                         // the sums take the place of the slices
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int row = wm * 32 + ty * 4 + (u & 3) + (u >> 2) * 16;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int col = g * 32 + tx * 4;
      const float2 lo = halves(acc[u][2 * g]), hi = halves(acc[u][2 * g + 1]);
      const float4 v = make_float4(lo.x, lo.y, hi.x, hi.y);
      if (alone) store(row, col, v);
      else *reinterpret_cast<float4 *>(smem + (wk * BM + row) * BN + col) = v;
    }
  }
  if (alone) return;
  if (p.split > 1) cluster_barrier(); else __syncthreads();
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem);
  for (int i = rank * 128 + t; i < BM * BN / 4; i += p.split * 128) {
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < p.split; ++s) {
      uint32_t from = base;
      if (p.split > 1) asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(from) : "r"(base), "r"(s));
#pragma unroll
      for (int w = 0; w < WK; ++w) {
        float4 v;
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(from + (uint32_t)(w * BM * BN + 4 * i) * 4u) : "memory");
        sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
      }
    }
    store(4 * i / BN, 4 * i % BN, sum);
  }
  if (p.split > 1) cluster_barrier();                  // the others have read this CTA's sums
}

// (3) k of one slice or less: hardly anything to sum, so what counts is how soon the first result leaves.  64 x 64 tiles, 4 x 4 results per
// thread, everything staged once; eight CTAs to an SM where the kernel above has two.  Its time against that kernel's, k = 1 to 16: bf16 [137, k] x
// [k, 202] 4.1 us against 7, [1920, k] x [k, 104] 6 against 9, 64 times [24, k] x [k, 4920] 0.66, [3694, k] x [k, 8001] as much; from k = 20 on,
// with a second slice, it is behind.  f32: 0.6 to 0.95 up to 8 M results, [3694, k] x [k, 8001] 1.4 (as many bytes again to store); where the
// kernel above moves 16 bytes at a time only [30, 8] x [8, 8] and the like are ahead here (0.65; 64 times [595, 8] x [8, 344] 1.6).
constexpr int SHORT_K = 16;
constexpr size_t SHORT_K_F32_RESULTS = 1u << 24, SHORT_K_F32_VEC_RESULTS = 1u << 16;

template <typename E>
__global__ void __launch_bounds__(256)
short_k_kernel(const F32Params p) {
  constexpr int BM = 64, BN = 64;
  __shared__ float as[SHORT_K][BM + 1], bs[SHORT_K][BN + 1];
  ugb_pdl_trigger();
  ugb_pdl_wait();
  const E *A = (const E *)p.a + (long long)blockIdx.z * p.a_b, *B = (const E *)p.b + (long long)blockIdx.z * p.b_b;
  E *C = (E *)p.c + (long long)blockIdx.z * p.c_b;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
#pragma unroll
  for (int e = threadIdx.x; e < BM * SHORT_K; e += 256) {               // along an operand's contiguous direction
    const int i = p.a_cs == 1 ? e / SHORT_K : e % BM, kk = p.a_cs == 1 ? e % SHORT_K : e / BM;
    as[kk][i] = m0 + i < p.m && kk < p.k ? to_f32<E>(A[(m0 + i) * p.a_rs + kk * p.a_cs]) : 0.f;
  }
#pragma unroll
  for (int e = threadIdx.x; e < BN * SHORT_K; e += 256) {
    const int j = p.b_cs == 1 ? e % BN : e / SHORT_K, kk = p.b_cs == 1 ? e / BN : e % SHORT_K;
    bs[kk][j] = n0 + j < p.n && kk < p.k ? to_f32<E>(B[kk * p.b_rs + (n0 + j) * p.b_cs]) : 0.f;
  }
  __syncthreads();
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  float acc[4][4] = {};
#pragma unroll 4
  for (int kk = 0; kk < p.k; ++kk) {
    float a[4], b[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) { a[u] = as[kk][ty * 4 + u]; b[u] = bs[kk][tx * 4 + u]; }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[u][v] = fmaf(a[u], b[v], acc[u][v]);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int i = m0 + ty * 4 + u, j = n0 + tx * 4 + v;
      if (i < p.m && j < p.n) C[i * p.c_rs + j] = from_f32<E>(acc[u][v]);
    }
}

inline bool al16(const void *p) { return ((uintptr_t)p & 15) == 0; }

template <typename E, int WM, int WK, bool VEC, bool TURNED = false>
int32_t launch_f32_shape(ugb_device *dev, const F32Params &p, size_t b, bool pdl) {
  using T = F32Tile<WM, WK>;
  const dim3 grid((unsigned)((p.n + T::BN - 1) / T::BN * p.split), (unsigned)((p.m + T::BM - 1) / T::BM), (unsigned)b);
  const size_t smem = WK * p.split > 1 ? std::max(T::SMEM, T::SMEM_REDUCE) : T::SMEM;
  constexpr unsigned bit = 1u << ((sizeof(E) == 4 ? VEC : std::is_same<E, __half>::value ? 2 : 3) * 6 + (TURNED ? 3 : 0) + (WM == 4 ? 0 : WM == 2 ? 1 : 2));
  if (smem > 48 * 1024 && !(dev->f32_smem_set & bit)) {      // once: a step that is captured has run eagerly before
    UGB_CUDA(dev, cudaFuncSetAttribute(f32_tile_kernel<E, WM, WK, VEC, TURNED>, cudaFuncAttributeMaxDynamicSharedMemorySize, std::max(T::SMEM, T::SMEM_REDUCE)));
    dev->f32_smem_set |= bit;
  }
  const cudaError_t e = ugb_launch_cluster(f32_tile_kernel<E, WM, WK, VEC, TURNED>, grid, dim3(T::THREADS), smem, dev->stream, pdl, p.split, p);
  if (e != cudaSuccess) return ugb_fail(dev, UGB_ERR_CUDA, "launch of f32_tile_kernel failed: %s", cudaGetErrorString(e));
  return ugb_after_launch(dev, "f32_tile_kernel");
}

template <typename E, bool VEC>
int32_t launch_f32_tile(ugb_device *dev, F32Params p, size_t b, bool pdl) {
  if constexpr (sizeof(E) == 4) {
    const ugb_f32_split_plan s = ugb_f32_gemm_split_plan(dev->sm_count, b, p.m, p.n, p.k, p.a_cs != 1);
    if (s.bn) {
      const ugb_f32_split_args g{(float *)p.c, (const float *)p.b, (const float *)p.a, b, (size_t)p.n, (size_t)p.m, (size_t)p.k, p.b_cs, p.b_rs, p.b_b, p.a_rs, p.a_cs, p.a_b, p.c_rs, p.c_b, pdl};
      const int32_t rc = ugb_f32_split(dev, g, s.bn, s.split);
      if (rc != UGB_ERR_UNSUPPORTED) return rc;
    }
  }
  UGB_REQUIRE(dev, b <= 65535 && ((size_t)p.m + 127) / 128 <= 65535, UGB_ERR_UNSUPPORTED, "matmul: m or batch too large for the FP32-pipe kernel");
  if (p.k <= SHORT_K && (p.m + 63) / 64 <= 65535 && (sizeof(E) == 2 || b * (size_t)p.m * (size_t)p.n <= (VEC ? SHORT_K_F32_VEC_RESULTS : SHORT_K_F32_RESULTS))) {
    const cudaError_t e = ugb_launch(short_k_kernel<E>, dim3((unsigned)((p.n + 63) / 64), (unsigned)((p.m + 63) / 64), (unsigned)b), dim3(256), 0, dev->stream, pdl, p);
    if (e != cudaSuccess) return ugb_fail(dev, UGB_ERR_CUDA, "launch of short_k_kernel failed: %s", cudaGetErrorString(e));
    return ugb_after_launch(dev, "short_k_kernel");
  }
  const ugb_f32_shape s = ugb_f32_gemm_shape(dev->sm_count, b, p.m, p.n, p.k);
  p.split = s.split;
  p.k_per_split = (int)((((size_t)p.k + s.split - 1) / s.split + 15) / 16 * 16);
  if (s.turned) {
    std::swap(p.m, p.n);
    std::swap(p.a, p.b);
    std::swap(p.a_b, p.b_b);
    std::swap(p.a_rs, p.b_cs);
    std::swap(p.a_cs, p.b_rs);
    return s.wk == 4 ? launch_f32_shape<E, 1, 4, VEC, true>(dev, p, b, pdl) : launch_f32_shape<E, 2, 2, VEC, true>(dev, p, b, pdl);
  }
  if (s.wk == 4) return launch_f32_shape<E, 1, 4, VEC>(dev, p, b, pdl);
  if (s.wk == 2) return launch_f32_shape<E, 2, 2, VEC>(dev, p, b, pdl);
  return launch_f32_shape<E, 4, 1, VEC>(dev, p, b, pdl);
}

int32_t launch_f32(ugb_device *dev, float *dst, const float *lhs, const float *rhs, size_t b, size_t m, size_t n, size_t k,
                   const MatLayout &L, const MatLayout &R, bool pdl) {
  if (k == 0) {
    UGB_CUDA(dev, cudaMemsetAsync(dst, 0, b * m * n * sizeof(float), dev->stream));
    return UGB_OK;
  }
  UGB_REQUIRE(dev, b <= 65535, UGB_ERR_UNSUPPORTED, "matmul: batch too large");
  const bool bases = al16(dst) && al16(lhs) && al16(rhs) && L.batch % 4 == 0 && R.batch % 4 == 0;
  if (m <= 16 && !L.transposed && R.transposed && k % 4 == 0 && bases) {
    const dim3 grid((unsigned)((n + 7) / 8), (unsigned)b);
#define UGB_SKINNY(MR) ugb_launch(f32_skinny_kernel<MR>, grid, dim3(256), 0, dev->stream, pdl, dst, lhs, rhs, (int)m, (int)n, (int)k, L.batch, R.batch)
    if (m <= 1) UGB_SKINNY(1); else if (m <= 2) UGB_SKINNY(2); else if (m <= 4) UGB_SKINNY(4); else if (m <= 8) UGB_SKINNY(8); else UGB_SKINNY(16);
#undef UGB_SKINNY
    return ugb_after_launch(dev, "f32_skinny_kernel");
  }
  // only the right operand is read in 128-bit pieces: the left rows may start anywhere (their length is the KV length)
  if (m <= 8 && !L.transposed && !R.transposed && (L.cs == 1 || k == 1) && (R.cs == 1 || n == 1) && n % 4 == 0 &&
      R.rs % 4 == 0 && R.batch % 4 == 0 && al16(rhs)) {
    const dim3 grid((unsigned)((n + 127) / 128), (unsigned)b);
#define UGB_SKINNY_N(MR) ugb_launch(f32_skinny_n_kernel<MR>, grid, dim3((MR) <= 2 ? 1024 : ((MR) <= 4 ? 512 : 256)), 0, dev->stream, pdl, dst, lhs, rhs, (int)m, (int)n, (int)k, L.rs, L.batch, R.rs, R.batch)
    if (m <= 1) UGB_SKINNY_N(1); else if (m <= 2) UGB_SKINNY_N(2); else if (m <= 4) UGB_SKINNY_N(4); else UGB_SKINNY_N(8);
#undef UGB_SKINNY_N
    return ugb_after_launch(dev, "f32_skinny_n_kernel");
  }
  // 128-bit pieces: the contiguous extent and the leading stride of each operand in whole float4s
  const size_t a_c = L.transposed ? m : k, a_ld = (size_t)(L.transposed ? L.cs : L.rs);
  const size_t b_c = R.transposed ? k : n, b_ld = (size_t)(R.transposed ? R.cs : R.rs);
  const bool vec = bases && a_c % 4 == 0 && a_ld % 4 == 0 && b_c % 4 == 0 && b_ld % 4 == 0 && n % 4 == 0;
  {
    const F32Params p{dst, lhs, rhs, (int)m, (int)n, (int)k, L.rs, L.cs, L.batch, R.rs, R.cs, R.batch, (long long)n, (long long)(m * n), 1, 0};
    return vec ? launch_f32_tile<float, true>(dev, p, b, pdl) : launch_f32_tile<float, false>(dev, p, b, pdl);
  }
}

}  // namespace

namespace {
// 64 x 64 tiles of grouped rows: rows [i tile_m, (i + 1) tile_m) multiply weights groups[i] (< 0: nothing to do).
__global__ void __launch_bounds__(256)
f32_grouped_kernel(float *__restrict__ c, const float *__restrict__ a, const float *__restrict__ b, const int *__restrict__ groups, int tile_m, int n, int k) {
  __shared__ float as[16][64 + 4], bs[16][64 + 4];
  const int m0 = blockIdx.y * 64, n0 = blockIdx.x * 64, g = groups[m0 / tile_m];
  if (g < 0) return;
  const float *ga = a + (size_t)m0 * k, *gb = b + (size_t)g * n * k;
  const int lr = threadIdx.x >> 2, lk = (threadIdx.x & 3) * 4, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[4][4] = {};
  for (int k0 = 0; k0 < k; k0 += 16) {
    float4 va = make_float4(0.f, 0.f, 0.f, 0.f), vb = va;
    if (k0 + lk < k) {                                       // k % 4 == 0
      va = *reinterpret_cast<const float4 *>(ga + (size_t)lr * k + k0 + lk);
      if (n0 + lr < n) vb = *reinterpret_cast<const float4 *>(gb + (size_t)(n0 + lr) * k + k0 + lk);
    }
    __syncthreads();
    as[lk][lr] = va.x; as[lk + 1][lr] = va.y; as[lk + 2][lr] = va.z; as[lk + 3][lr] = va.w;
    bs[lk][lr] = vb.x; bs[lk + 1][lr] = vb.y; bs[lk + 2][lr] = vb.z; bs[lk + 3][lr] = vb.w;
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) {
      const float4 x = *reinterpret_cast<const float4 *>(&as[kk][4 * ty]), y = *reinterpret_cast<const float4 *>(&bs[kk][4 * tx]);
      const float xv[4] = {x.x, x.y, x.z, x.w}, yv[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xv[i], yv[j], acc[i][j]);
    }
  }
  if (n0 + 4 * tx >= n) return;                              // n % 4 == 0
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<float4 *>(c + (size_t)(m0 + 4 * ty + i) * n + n0 + 4 * tx) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
}
}  // namespace

int32_t ugb_f32_grouped_gemm(ugb_device *dev, float *c, const float *a, const float *b, const int *groups, size_t m, int tile_m, int n, int k) {
  if (m == 0 || n == 0) return UGB_OK;
  UGB_REQUIRE(dev, tile_m % 64 == 0 && m % tile_m == 0 && m / 64 <= 65535 && n % 4 == 0 && k % 4 == 0, UGB_ERR_UNSUPPORTED,
              "f32 grouped product: %zu rows in tiles of %d, n %d, k %d", m, tile_m, n, k);
  f32_grouped_kernel<<<dim3((unsigned)((n + 63) / 64), (unsigned)(m / 64)), 256, 0, dev->stream>>>(c, a, b, groups, tile_m, n, k);
  return ugb_after_launch(dev, "f32_grouped_kernel");
}

int32_t ugb_f32_gemm(ugb_device *dev, float *c, const float *a, const float *b, size_t batch, size_t m, size_t n, size_t k,
                     size_t a_ld, size_t a_batch, bool b_is_nk, size_t b_batch, size_t c_ld, size_t c_batch, bool pdl) {
  if (batch == 0 || m == 0 || n == 0) return UGB_OK;
  if (batch == 1 && a_ld == k && c_ld == n && b_is_nk && k > 0) {   // a Linear: the skinny kernel takes few rows
    const MatLayout L{(long long)k, 1, (long long)a_batch, false}, R{1, (long long)k, (long long)b_batch, true};
    return launch_f32(dev, c, a, b, batch, m, n, k, L, R, pdl);
  }
  UGB_REQUIRE(dev, batch <= 65535 && (m + 127) / 128 <= 65535 && m < (1u << 31) && n < (1u << 31) && k < (1u << 31), UGB_ERR_UNSUPPORTED,
              "f32 product: extent too large");
  const bool vec = al16(c) && al16(a) && al16(b) && k % 4 == 0 && n % 4 == 0 && a_ld % 4 == 0 && c_ld % 4 == 0 &&
                   a_batch % 4 == 0 && b_batch % 4 == 0 && c_batch % 4 == 0;
  const long long b_rs = b_is_nk ? 1 : (long long)n, b_cs = b_is_nk ? (long long)k : 1;
  {
    const F32Params p{c, a, b, (int)m, (int)n, (int)k, (long long)a_ld, 1, (long long)a_batch, b_rs, b_cs, (long long)b_batch, (long long)c_ld, (long long)c_batch, 1, 0};
    return vec ? launch_f32_tile<float, true>(dev, p, batch, pdl) : launch_f32_tile<float, false>(dev, p, batch, pdl);
  }
}

extern "C" {

void ugb_gemm_state_free(ugb_device *dev) { ugb_tc_state_free(dev); }

int32_t ugb_matmul(ugb_device *dev, ugb_slice *dst, const ugb_slice *lhs, const ugb_slice *rhs,
                   size_t b, size_t m, size_t n, size_t k, int32_t rank, const size_t *lhs_dims,
                   const size_t *lhs_strides, size_t lhs_off, const size_t *rhs_dims,
                   const size_t *rhs_strides, size_t rhs_off) {
  if (!dev) return UGB_ERR_INVALID;
  UGB_REQUIRE(dev, dst && lhs && rhs, UGB_ERR_INVALID, "matmul: null slice");
  UGB_REQUIRE(dev, lhs_dims && lhs_strides && rhs_dims && rhs_strides, UGB_ERR_INVALID,
              "matmul: null layout");
  // gemm.rs:301-331: the three dtypes must agree and be one of bf16/f16/f32.
  const int32_t dt = dst->dtype;
  UGB_REQUIRE(dev, dt == lhs->dtype && dt == rhs->dtype && (dt == UGB_BF16 || dt == UGB_F16 || dt == UGB_F32),
              UGB_ERR_DTYPE, "incorrect dtypes for matmul, dst: %s, lhs: %s, rhs: %s",
              ugb_dtype_name(dst->dtype), ugb_dtype_name(lhs->dtype), ugb_dtype_name(rhs->dtype));
  UGB_REQUIRE(dev, dst->dev == dev && lhs->dev == dev && rhs->dev == dev, UGB_ERR_INVALID,
              "matmul: slice belongs to another device");
  MatLayout L, R;
  int32_t rc = parse_layout(dev, "lhs", rank, lhs_dims, lhs_strides, m, k, &L);
  if (rc) return rc;
  rc = parse_layout(dev, "rhs", rank, rhs_dims, rhs_strides, k, n, &R);
  if (rc) return rc;
  UGB_REQUIRE(dev, m < (1u << 31) && n < (1u << 31) && k < (1u << 31), UGB_ERR_SHAPE, "matmul: extent too large");
  UGB_REQUIRE(dev, dst->len >= b * m * n, UGB_ERR_SHAPE, "matmul: dst holds %zu elements, %zu needed",
              dst->len, b * m * n);
  if (b == 0 || m == 0 || n == 0) return UGB_OK;
  // extent of each operand in elements, from its strides
  auto extent = [&](const MatLayout &X, size_t rows, size_t cols) {
    return (size_t)((long long)(b - 1) * X.batch + (long long)(rows - 1) * X.rs +
                    (long long)(cols - 1) * X.cs + 1);
  };
  if (k > 0) {
    UGB_REQUIRE(dev, lhs->len >= lhs_off + extent(L, m, k), UGB_ERR_SHAPE, "matmul: lhs slice too short");
    UGB_REQUIRE(dev, rhs->len >= rhs_off + extent(R, k, n), UGB_ERR_SHAPE, "matmul: rhs slice too short");
  }
  const size_t es = ugb_dtype_size(dt);
  const char *lp = (const char *)lhs->ptr + lhs_off * es;
  const char *rp = (const char *)rhs->ptr + rhs_off * es;

  // Few rows against [n, k] rows: the kernel that streams the matrix through registers, whatever n (it reads every step of a
  // batch that shares its matrix again, so those go on as one tall product).  Its CTAs take about 1.5 us for each 16 columns
  // however short k is.  Where they have one piece each it is ahead of the tensor-core tiles for every k ([4, 64] x [2048, 64]^T 3.4
  // us against 3.7, k = 2048 4.7 against 9.6), with more of them from about k = 1024 on ([4, k] x [65536, k]^T for k = 64, 512, 1024,
  // 2048: 31, 31, 32, 47 us against 9.5, 20, 36, 70; 8 times [4, k] x [2048, k]^T 11, 11, 11, 16 against 5, 8, 11, 18).  Columns or
  // bases that those tiles do not take are still better off here than on the FFMA kernel from about k = 128 on ([65536, k]: 31
  // us against 8, 19, 31, 57 for k = 8, 64, 128, 256).
  const bool few = (dt == UGB_BF16 || dt == UGB_F16) && !L.transposed && R.transposed && ugb_skinny_rows(R.batch == 0 ? b * m : m);
  auto stream_rows = [&]() {
    ugb_tc_gemm_args g;
    g.out = dst->ptr; g.a = lp; g.b = rp;
    g.batch = b; g.m = m; g.n = n; g.k = k;
    g.a_batch = L.batch; g.b_batch = R.batch; g.b_is_nk = true; g.f16 = dt == UGB_F16;
    g.epi = UGB_EPI_BF16; g.splits = 1; g.bn = 0; g.b_static = false; g.pdl = true;
    return ugb_skinny_gemm(dev, g);
  };
  const bool stream = few && (k >= 1024 || ugb_skinny_one_round(dev->sm_count, n, R.batch == 0 ? 1 : b));
  if (stream) {
    const int32_t src = stream_rows();
    if (src != UGB_ERR_UNSUPPORTED) return src;
  }
  // Whatever has the alignment is faster on the tensor cores, also the smallest: [1, 8] x [8, 8] 3.5 us against 4.2 on the FFMA kernel, [1, 32] x
  // [32, 8] 3.5 against 5.6, [9, 192] x [64, 192]^T 4.1 against 11.1, [100, 64] x [64, 64]^T 4.2 against 8.1, 64 of [64, 128] x [64, 128]^T
  // 4.0 against 16.3.  Only long rows of results with next to nothing to sum are not ([8, 8] x [65536, 8]^T 16.6 against 9.1; with k = 32 9.7
  // against 12.1).
  if ((dt == UGB_BF16 || dt == UGB_F16) && !L.transposed && !(few && !stream && k <= 16)) {
    // tensor-core path (bf16 and f16 are the same tcgen05.mma.kind::f16 instruction with another format field, as
    // both go to cublasGemmStridedBatchedEx in the reference, gemm.rs:130-232): A [m,k] row-major, B either
    // [n,k] row-major ("TN", matmul_t with a weight) or [k,n] row-major ("NN").
    int32_t trc = ugb_tc_gemm_bf16(dev, dst->ptr, lp, rp, b, m, n, k, L.batch, R.batch, R.transposed, dt == UGB_F16);
    if (trc != UGB_ERR_UNSUPPORTED) return trc;
  }
  if (few && !stream && k >= 128) {
    const int32_t src = stream_rows();
    if (src != UGB_ERR_UNSUPPORTED) return src;
  }
  switch (dt) {
    case UGB_F32: return launch_f32(dev, (float *)dst->ptr, (const float *)lp, (const float *)rp, b, m, n, k, L, R, true);
    default: {
      if (k == 0) {
        UGB_CUDA(dev, cudaMemsetAsync(dst->ptr, 0, b * m * n * es, dev->stream));
        return UGB_OK;
      }
      const F32Params p{dst->ptr, lp, rp, (int)m, (int)n, (int)k, L.rs, L.cs, L.batch, R.rs, R.cs, R.batch, (long long)n, (long long)(m * n), 1, 0};
      return dt == UGB_BF16 ? launch_f32_tile<__nv_bfloat16, false>(dev, p, b, true) : launch_f32_tile<__half, false>(dev, p, b, true);
    }
  }
}

}  // extern "C"
