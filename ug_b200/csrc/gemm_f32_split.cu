// f32 products on the tensor cores: every value is the exact sum of three bf16 parts, and eight of the nine products of parts are
// formed by tcgen05.mma with f32 accumulators.
//
//   x = hi + mid + lo     hi = bf16(x), mid = bf16(x - hi), lo = x - hi - mid: 8 bits each, nothing is lost
//   a b = hi hi           16 products at a time, each time in an accumulator of its own, from where they are added up in f32 registers
//       + hi mid + mid hi + mid mid + hi lo + lo hi + mid lo + lo mid          (2^-8 of it and less: an accumulator for 960 k)
//       + lo lo                                              left out: 2^-33 of |a b|
//
// The tensor core cuts off what an FFMA rounds: of 16 products and the accumulator what lies 2^-25 below the largest, then their sum to
// f32 (sums formed that way on a CPU have the errors measured here).  Sums of one sign lose a little of themselves every time, so
// nothing is added to hi hi there.  The error against 64 bits, beside that of the FFMA kernel, by what is summed (2-norm, 257 x 1024
// results):
//                                     k = 1000                2048                    4096
//   normal                            7.6e-8 against 2.1e-7   8.1e-8 against 2.2e-7   9.0e-8 against 3.0e-7
//   uniform in 0 .. 1                 4.4e-8 against 7.0e-8   4.7e-8 against 7.1e-8   4.8e-8 against 8.0e-8
//   softmax (deviation 3) x uniform   9.5e-8 against 1.1e-7   9.8e-8 against 1.1e-7   9.9e-8 against 1.4e-7
// With 64 k in an accumulator and six products the last of these was 2.8e-7 to 3.0e-7.  At k = 64 it is 8e-8 here and 6e-8 with FFMA: see
// ugb_f32_gemm_split_plan for the sums that stay there.
//
// What the parts cannot hold is found as it is read and as it is stored, and that result is then formed again with FFMA: one that is not
// finite, and, where parts left the normal range or products of parts may have lost more than 2^-30 of a product of values (it loses no more as long as
// the smallest exponents add up to -96 or more), one so small that what was lost may be 2^-26 of it.
//
// Tile: 128 columns of the result (lanes of the tensor memory: a warp stores whole lines) x BN rows.  16 warps read both operands, two
// stages of 32 k ahead in registers, split them into the six swizzled shared-memory planes of a stage, and add what the tensor core
// has finished to their f32 sums: hi hi of a stage while its other products are formed.  Every six stages those sums go back into the
// tensor memory, added to those of the stages before, so that no chain of additions is long.  A warp of its own issues (issued by one of the
// 16, its conversion and its issuing were in line, and every stage waited for both).  Few tiles: CTAs of a cluster along k, sums through
// distributed shared memory in rank order.
//
// Bound: the conversion (about ten instructions a value on 28 values per thread and stage), the products' own reads of shared memory
// (an MMA of 128 x 96 x 16 takes 56 cycles for its operands, sixteen a stage) and the sums' way out of the tensor memory, 1.0 us a stage
// together (with hi hi waited for together with the rest of its stage the first product below took 85 us).  The loads wait in the L1, which
// is what the stages leave of 256 KB: 32 k a stage, not 64.  The fence between the planes and the tensor core is that of shared memory
// alone: the general one also waits for the loads ahead.  Other forms were measured with six products and 64 k in an accumulator, when the
// first product below took 56 us: the general fence 86, 8 warps with twice the work each 68, three stages ahead 61, lines asked into the
// L2 six stages ahead 59, and tiles of 128 rows for 2048 x 4096 x 2048 299 against 283.
// Against the FFMA kernel: [257, 2048] x [5632, 2048]^T 182 -> 73 us, [2048, 2048] x [4096, 2048]^T 679 -> 352, [777, 5632] x [2048, 5632]^T 482 -> 205,
// [128, 2048] x [2048, 2048]^T 56 -> 20, [500, 999] x [1001, 999]^T 35 -> 22.  The first with an infinity or a row of NaN 120 us, with a column of NaN 111;
// with some in most rows, so that most results are formed again, 595, and the second 2900: three to four and a half times the FFMA kernel's time.
#include "gemm_f32_split.cuh"
#include "tc_ptx.cuh"

namespace {

using namespace ugb_tc;

constexpr int BM = 128, BK = 32, WORKERS = 512, AHEAD = 2, WARPS = WORKERS / 32, THREADS = WORKERS + 32;
constexpr int PLANE_P = BM * BK * 2;
constexpr int RED_LD = BM;                 // floats between a tile's rows of q in shared memory
constexpr int GROUP = 6, REST = 30;        // stages whose sums stay in registers; between two transfers of the rest
constexpr int D_STRIDE = 96, TMEM_COLS = 512;         // hi hi of the two 16 k of a stage, the rest, the sums of whole groups

template <int BN> struct Shape {
  static constexpr int SLOTS = 3;
  static constexpr int PLANE_Q = BN * BK * 2, STAGE = 3 * (PLANE_P + PLANE_Q), SMEM = SLOTS * STAGE + 1024;
};

struct Params {
  float *c;
  const float *p, *q;
  long long p_rs, p_ks, p_b, q_rs, q_ks, q_b, c_q, c_b;
  int rows_p, rows_q, k, split, k_per_split;
  ugb_status_word *status;
};

// Zero where `on` is not set.  Written out: behind a branch the value is chosen, and waited for, where it is asked for, and the
// compiler's own loads sink to their uses.
static __device__ __forceinline__ float4 ld4(const float *p, bool on) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %5, 0;\n @q ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n}"
               : "+f"(v.x), "+f"(v.y), "+f"(v.z), "+f"(v.w) : "l"(p), "r"((uint32_t)on));
  return v;
}
static __device__ __forceinline__ float ld1(const float *p, bool on) {
  float v = 0.f;
  asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q ld.global.f32 %0, [%1];\n}" : "+f"(v) : "l"(p), "r"((uint32_t)on));
  return v;
}
static __device__ __forceinline__ uint32_t pack(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
static __device__ __forceinline__ uint32_t abs_max(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
static __device__ __forceinline__ void st2(uint32_t at, uint32_t a, uint32_t b) { asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(a), "r"(b) : "memory"); }
static __device__ __forceinline__ void tmem_ld8(uint32_t at, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(at) : "memory");
}
static __device__ __forceinline__ void tmem_st8(uint32_t at, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               :: "r"(at), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

// R rows x 32 k of an operand in pieces of four values along its contiguous direction (KC: k), N of them per worker:
// the first at (row, k), the others STEP rows or k steps further.
template <int R, bool KC, bool VEC> struct Operand {
  static constexpr int N = (R * BK / 4 + WORKERS - 1) / WORKERS, STEP = KC ? WORKERS * 4 / BK : WORKERS / (R / 4);
  const float *at;                         // of the first piece, of the stage that is read next
  long long step, stage;                   // elements to the next piece, to the next stage
  uint32_t to;                             // of the first piece inside a plane
  int row, k, rows;                        // rows: behind the first row of the tile
  uint32_t least = 0xffffffffu;            // the smallest 2 |x| - 1 seen, in bits; zeros are the largest value
  uint32_t most = 0;                       // the largest hi, in both halves; signs mean nothing
  __device__ __forceinline__ Operand(const float *src, long long rs, long long ks, int rows_, int t) : rows(rows_) {
    if (KC) { row = t / (BK / 4); k = t % (BK / 4) * 4; }
    else { k = t / (R / 4); row = t % (R / 4) * 4; }
    at = src + row * rs + k * ks;
    step = STEP * (KC ? rs : ks);
    stage = BK * ks;
    to = KC ? row * 64 + ((k >> 3 ^ (row >> 1 & 3)) << 4) + (k & 4) * 2            // rows of 64 bytes, 64-byte swizzle
            : (row >> 6) * (BK * 128) + k * 128 + (((row & 63) >> 3 ^ (k & 7)) << 4) + (row & 4) * 2;      // k of 128, 128-byte swizzle
  }
  // Whether this worker has piece i: the last is not everyone's where the pieces do not come out even.
  static __device__ __forceinline__ bool mine(int i, int row, int k) { return (i + 1) * WORKERS * 4 <= R * BK || (KC ? row + STEP * i < R : k + STEP * i < BK); }
  __device__ __forceinline__ void load(float4 (&v)[N], int k_left) {
    const float *from = at;
#pragma unroll
    for (int i = 0; i < N; ++i, from += step) {
      const int r = row + (KC ? STEP * i : 0), kk = k + (KC ? 0 : STEP * i);
      const bool on = mine(i, row, k) && r < rows && kk < k_left;
      if constexpr (VEC) v[i] = ld4(from, on);          // a piece is all in or all out
      else if constexpr (KC) v[i] = make_float4(ld1(from, on), ld1(from + 1, on && kk + 1 < k_left), ld1(from + 2, on && kk + 2 < k_left), ld1(from + 3, on && kk + 3 < k_left));
      else v[i] = make_float4(ld1(from, on), ld1(from + 1, on && r + 1 < rows), ld1(from + 2, on && r + 2 < rows), ld1(from + 3, on && r + 3 < rows));
    }
    at += stage;
  }
  __device__ __forceinline__ void store(const float4 (&v)[N], uint32_t base, int plane) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (!mine(i, row, k)) break;
      float x[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) least = min(least, 2u * __float_as_uint(x[e]) - 1u);
#pragma unroll
      for (int part = 0; part < 3; ++part) {
        const uint32_t a = pack(x[0], x[1]), b = pack(x[2], x[3]);
        if (part == 0) most = abs_max(abs_max(most, a), b);
        st2(base + to + (uint32_t)(part * plane + i * STEP * (KC ? 64 : 128)), a, b);
        if (part < 2) {
          x[0] -= __uint_as_float(a << 16); x[1] -= __uint_as_float(a & 0xffff0000u);
          x[2] -= __uint_as_float(b << 16); x[3] -= __uint_as_float(b & 0xffff0000u);
        }
      }
    }
  }
};

// Bit j of a worker's `odd`: its sum j is formed again, in f32.  The others keep what they have, so that no result depends on what its
// neighbours in the tile hold.  Up to LIST of them (a row or a column of the product) are dot products of a warp each; more are
// formed by all workers from slices in shared memory, eight columns of a warp without one passed over.  Not inlined: a tile comes here once at
// most, and the arrays would be the main loop's registers.  All threads of the block.
template <int BN, bool PK, bool QK>
static __device__ __noinline__ void again_with_ffma(const float *P, const float *Q, long long p_rs, long long p_ks, long long q_rs, long long q_ks, int rows_p, int rows_q,
                                                    int k_lo, int k_hi, float (&result)[BN * 4 / WARPS], uint32_t odd) {
  extern __shared__ uint8_t smem_raw[];    // not handed over: its loads would be generic ones
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int CK = 32, COLS = BN * 4 / WARPS, NP = (BM * CK + THREADS - 1) / THREADS, NQ = (BN * CK + THREADS - 1) / THREADS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = (warp & 3) * 32 + lane, col0 = (warp >> 2) * COLS;
  const uint32_t needed = __reduce_or_sync(0xffffffffu, odd);
  {
    constexpr int LIST = 512;
    int *count = reinterpret_cast<int *>(smem);
    uint16_t *list = reinterpret_cast<uint16_t *>(smem + 16);
    float *sums = reinterpret_cast<float *>(smem + 16 + 2 * LIST);
    if (threadIdx.x == 0) *count = 0;
    __syncthreads();
    const int first = odd ? atomicAdd(count, __popc(odd)) : 0;
    int at = first;
#pragma unroll
    for (int j = 0; j < COLS; ++j)
      if (odd >> j & 1) {
        if (at < LIST) list[at] = (uint16_t)((col0 + j) * BM + row);
        ++at;
      }
    __syncthreads();
    const int n = *count;
    if (n <= LIST) {
      for (int i = warp; i < n; i += WARPS + 1) {
        const float *x = P + (list[i] % BM) * p_rs, *y = Q + (list[i] / BM) * q_rs;
        float sum = 0.f;
#pragma unroll 8
        for (int k = k_lo + lane; k < k_hi; k += 32) sum = fmaf(x[k * p_ks], y[k * q_ks], sum);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) sums[i] = sum;
      }
      __syncthreads();
      at = first;
#pragma unroll
      for (int j = 0; j < COLS; ++j)
        if (odd >> j & 1) result[j] = sums[at++];
      __syncthreads();                     // the caller writes shared memory
      return;
    }
    __syncthreads();
  }
  float(*sp)[BM + 1] = reinterpret_cast<float(*)[BM + 1]>(smem);
  float(*sq)[BN + 4] = reinterpret_cast<float(*)[BN + 4]>(smem + CK * (BM + 1) * 4 + 64 - CK * (BM + 1) * 4 % 64);
  float acc[COLS] = {}, np[NP], nq[NQ];    // np, nq: the next slice
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int e = threadIdx.x + i * THREADS, r = PK ? e / CK : e % BM, k = k0 + (PK ? e % CK : e / BM);
      np[i] = ld1(P + r * p_rs + k * p_ks, e < BM * CK && r < rows_p && k < k_hi);
    }
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
      const int e = threadIdx.x + i * THREADS, r = QK ? e / CK : e % BN, k = k0 + (QK ? e % CK : e / BN);
      nq[i] = ld1(Q + r * q_rs + k * q_ks, e < BN * CK && r < rows_q && k < k_hi);
    }
  };
  fetch(k_lo);
  for (int k0 = k_lo; k0 < k_hi; k0 += CK) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int e = threadIdx.x + i * THREADS;
      if (e < BM * CK) sp[PK ? e % CK : e / BM][PK ? e / CK : e % BM] = np[i];
    }
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
      const int e = threadIdx.x + i * THREADS;
      if (e < BN * CK) sq[QK ? e % CK : e / BN][QK ? e / CK : e % BN] = nq[i];
    }
    __syncthreads();
    fetch(k0 + CK);
#pragma unroll
    for (int j = 0; j < COLS; j += 8) {
      if (!(needed >> j & 0xff)) continue;
      float sum[8] = {};                   // of this slice, so that no sum is long
#pragma unroll 8
      for (int k = 0; k < CK; ++k) {
        const float x = sp[k][row];
        const float4 y = *reinterpret_cast<const float4 *>(&sq[k][col0 + j]), z = *reinterpret_cast<const float4 *>(&sq[k][col0 + j + 4]);
        sum[0] = fmaf(x, y.x, sum[0]); sum[1] = fmaf(x, y.y, sum[1]); sum[2] = fmaf(x, y.z, sum[2]); sum[3] = fmaf(x, y.w, sum[3]);
        sum[4] = fmaf(x, z.x, sum[4]); sum[5] = fmaf(x, z.y, sum[5]); sum[6] = fmaf(x, z.z, sum[6]); sum[7] = fmaf(x, z.w, sum[7]);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[j + e] += sum[e];
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < COLS; ++j)
    if (odd >> j & 1) result[j] = acc[j];
}

template <int BN, bool PK, bool QK, bool VEC>
__global__ void __launch_bounds__(THREADS, 1)
f32_split_kernel(const Params p) {
  using S = Shape<BN>;
  constexpr int SLOTS = S::SLOTS, COLS = BN * 4 / WARPS;              // COLS: of a worker's sums
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full[SLOTS], lead[SLOTS], rest, last;               // lead: hi hi of a stage
  __shared__ uint32_t tmem_slot, least_p, least_q, most;
  __shared__ int aborted, again;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = p.split > 1 ? (int)(blockIdx.x % p.split) : 0;
  const int p0 = (int)(p.split > 1 ? blockIdx.x / p.split : blockIdx.x) * BM, q0 = blockIdx.y * BN;
  const float *P = p.p + (long long)blockIdx.z * p.p_b + p0 * p.p_rs, *Q = p.q + (long long)blockIdx.z * p.q_b + q0 * p.q_rs;
  const int k_lo = min(p.k, rank * p.k_per_split), k_hi = min(p.k, k_lo + p.k_per_split), stages = (k_hi - k_lo + BK - 1) / BK;
  if (threadIdx.x == 0) {
    for (int i = 0; i < SLOTS; ++i) {
      mbar_init(smem_u32(&full[i]), WARPS);
      mbar_init(smem_u32(&lead[i]), 1);
    }
    mbar_init(smem_u32(&rest), 1);
    mbar_init(smem_u32(&last), 1);
    aborted = again = 0;
    least_p = least_q = 0xffffffffu;
    most = 0x3f80u;                        // 1
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == WARPS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = tmem_slot;
  volatile int *abort_flag = &aborted;
  ugb_pdl_wait();

  float acc[COLS];
#pragma unroll
  for (int j = 0; j < COLS; ++j) acc[j] = 0.f;
  const uint32_t idesc = make_idesc(BM, BN, !QK) | (PK ? 0u : 1u << 15);
  // k-contiguous planes: 8-row groups 512 bytes apart, a k step of 16 moves 32 bytes inside the swizzled row.  The others: 64-row
  // chunks 4 KiB apart, 8-k groups 1024 bytes, a k step moves 16 rows of 128 bytes.
  auto desc = [&](uint32_t at, bool kc) {
    const uint64_t d = make_smem_desc(at, kc ? 0 : BK * 128, kc ? 512 : 1024);
    return kc ? (d & ~(7ull << 61)) | 4ull << 61 : d;                  // layout 4: 64-byte swizzle
  };
  const uint64_t pd = desc(smem_u32(smem), PK), qd = desc(smem_u32(smem) + 3 * PLANE_P, QK);
  constexpr uint32_t PSTEP = (PK ? 32 : 2048) >> 4, QSTEP = (QK ? 32 : 2048) >> 4, PP = PLANE_P >> 4, QP = S::PLANE_Q >> 4;
  auto multiply = [&](int s, int slot) { // one thread
    const uint32_t d0 = tmem, d1 = tmem + 2 * D_STRIDE;
    const uint64_t p0 = pd + (uint32_t)slot * (S::STAGE >> 4), q0 = qd + (uint32_t)slot * (S::STAGE >> 4);
#pragma unroll
    for (int j = 0; j < BK / UMMA_K; ++j) umma_bf16(d0 + j * D_STRIDE, p0 + j * PSTEP, q0 + j * QSTEP, idesc, 0);
    umma_commit(smem_u32(&lead[slot]));
#pragma unroll
    for (int j = 0; j < BK / UMMA_K; ++j) {
      const uint64_t a = p0 + j * PSTEP, b = q0 + j * QSTEP;
      umma_bf16(d1, a, b + QP, idesc, s % REST > 0 || j > 0);
      umma_bf16(d1, a + PP, b, idesc, 1);
      umma_bf16(d1, a + PP, b + QP, idesc, 1);
      umma_bf16(d1, a, b + 2 * QP, idesc, 1);
      umma_bf16(d1, a + 2 * PP, b, idesc, 1);
      umma_bf16(d1, a + PP, b + 2 * QP, idesc, 1);
      umma_bf16(d1, a + 2 * PP, b + QP, idesc, 1);
    }
    if (s + 1 == stages || (s + 1) % REST == 0) umma_commit(smem_u32(&rest));
  };
  const int row = (warp & 3) * 32 + lane, col0 = (warp >> 2) * COLS;            // of this worker's sums
  const bool worker = warp < WARPS;
  // the same answer in all lanes
  auto wait = [&](uint64_t &bar, uint32_t parity, unsigned site) {
    return __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar), parity, abort_flag, p.status, site)) != 0;
  };
  bool alive = true;
  if (!worker) {
    for (int s = 0; s < stages && alive; ++s) {
      alive = wait(full[s % SLOTS], s / SLOTS & 1, 0x62);
      tcgen05_fence_after();
      if (alive && elect_one()) multiply(s, s % SLOTS);
      __syncwarp();
    }
    if (!alive && elect_one()) {           // nothing may be at work on shared or tensor memory when they are given back
      int none = 0;
      umma_commit(smem_u32(&last));
      mbar_wait(smem_u32(&last), 0, &none, p.status, 0x64);
    }
  } else {
    using OP = Operand<BM, PK, VEC>;
    using OQ = Operand<BN, QK, VEC>;
    OP op(P + k_lo * p.p_ks, p.p_rs, p.p_ks, p.rows_p - p0, threadIdx.x);
    OQ oq(Q + k_lo * p.q_ks, p.q_rs, p.q_ks, p.rows_q - q0, threadIdx.x);
    float4 vp[AHEAD][OP::N], vq[AHEAD][OQ::N];
    auto load = [&](int s, float4 (&a)[OP::N], float4 (&b)[OQ::N]) {     // stages in turn
      op.load(a, k_hi - k_lo - s * BK);
      oq.load(b, k_hi - k_lo - s * BK);
    };
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    auto add = [&]() {                     // hi hi of the last stage
#pragma unroll
      for (int j = 0; j < COLS; j += 8) {
        uint32_t v[8], w[8];
        const uint32_t at = tmem + lanes + (uint32_t)(col0 + j);
        tmem_ld8(at, v);
        tmem_ld8(at + D_STRIDE, w);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[j + e] += __uint_as_float(v[e]) + __uint_as_float(w[e]);
      }
    };
    auto add_from = [&](uint32_t from) {   // 2: the rest; 3: the groups before, which no one else touches
#pragma unroll
      for (int j = 0; j < COLS; j += 8) {
        uint32_t v[8];
        tmem_ld8(tmem + lanes + from * D_STRIDE + (uint32_t)(col0 + j), v);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[j + e] += __uint_as_float(v[e]);
      }
    };
    uint32_t rests = 0;                    // transfers of the rest so far
    auto put_away = [&]() {
#pragma unroll
      for (int j = 0; j < COLS; j += 8) {
        uint32_t v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) { v[e] = __float_as_uint(acc[j + e]); acc[j + e] = 0.f; }
        tmem_st8(tmem + lanes + (uint32_t)(3 * D_STRIDE + col0 + j), v);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    };
    auto stage = [&](int s, int slot, bool new_group, float4 (&a)[OP::N], float4 (&b)[OQ::N]) {
      if (!alive) return;
      const uint32_t base = smem_u32(smem) + slot * S::STAGE;
      op.store(a, base, PLANE_P);
      oq.store(b, base + 3 * PLANE_P, S::PLANE_Q);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      if (s + AHEAD < stages) load(s + AHEAD, a, b);
      // hi hi of the stage before, which this one starts anew; its other products are still being formed, and with it all of the stage before that
      // is complete, whose planes the next stage writes over.
      if (s >= 1) {
        alive = wait(lead[(s - 1) % SLOTS], (s - 1) / SLOTS & 1, 0x61);
        if (new_group && s % REST == 0 && alive) alive = wait(rest, rests++ & 1, 0x65);
        if (!alive) return;
        tcgen05_fence_after();
        add();
        if (new_group) {
          if (s % REST == 0) add_from(2);
          if (s > GROUP) add_from(3);
          put_away();
        }
        tcgen05_fence_before();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&full[slot]));
    };
#pragma unroll
    for (int s = 0; s < AHEAD; ++s)
      if (s < stages) load(s, vp[s], vq[s]);
    static_assert(GROUP % SLOTS == 0 && GROUP % AHEAD == 0 && REST % GROUP == 0, "");
    for (int s = 0; s < stages; s += GROUP)
#pragma unroll
      for (int i = 0; i < GROUP; ++i)
        if (s + i < stages) stage(s + i, i % SLOTS, i == 0, vp[i % AHEAD], vq[i % AHEAD]);
    if (stages > 0) {
      if (alive) alive = wait(rest, rests & 1, 0x63);        // and all before it
      tcgen05_fence_after();
      if (alive) {
        add();
        add_from(2);
        if (stages > GROUP) add_from(3);
      }
    }
    const uint32_t lp = __reduce_min_sync(0xffffffffu, op.least), lq = __reduce_min_sync(0xffffffffu, oq.least);
    const uint32_t both = abs_max(op.most, oq.most), top = __reduce_max_sync(0xffffffffu, max(both >> 16 & 0x7fffu, both & 0x7fffu));
    if (lane == 0) {
      atomicMin(&least_p, lp);
      atomicMin(&least_q, lq);
      atomicMax(&most, top);
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == WARPS) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
  }
  // Biased exponents of the smallest values: products of parts stay above 2^-126, or each of the k products has lost up to 2^-123
  // times the largest value.
  const uint32_t ep = least_p == 0xffffffffu ? 255u : (least_p + 1u) >> 24, eq = least_q == 0xffffffffu ? 255u : (least_q + 1u) >> 24;
  const float floor_ = ep < 24u || eq < 24u || ep + eq < 158u ? (float)p.k * __uint_as_float(most << 16) * 0x1p-97f : 0.f;
  uint32_t odd = 0;                        // of this worker's sums
  if (worker) {
#pragma unroll
    for (int j = 0; j < COLS; ++j)
      if (p0 + row < p.rows_p && q0 + col0 + j < p.rows_q && !(fabsf(acc[j]) <= 3.402823466e38f && fabsf(acc[j]) >= floor_)) odd |= 1u << j;
    if (__any_sync(0xffffffffu, odd) && lane == 0) atomicOr(&again, 1);
  }
  __syncthreads();
  if (again) {
    float sums[COLS];
#pragma unroll
    for (int j = 0; j < COLS; ++j) sums[j] = acc[j];
    again_with_ffma<BN, PK, QK>(P, Q, p.p_rs, p.p_ks, p.q_rs, p.q_ks, p.rows_p - p0, p.rows_q - q0, k_lo, k_hi, sums, odd);
#pragma unroll
    for (int j = 0; j < COLS; ++j) acc[j] = sums[j];
  }

  float *C = p.c + (long long)blockIdx.z * p.c_b;
  if (p.split == 1) {                      // a warp's lanes are neighbours in memory
    if (worker && p0 + row < p.rows_p) {
#pragma unroll
      for (int j = 0; j < COLS; ++j)
        if (q0 + col0 + j < p.rows_q) C[(long long)(q0 + col0 + j) * p.c_q + p0 + row] = acc[j];
    }
    return;
  }
  float *red = reinterpret_cast<float *>(smem);
  if (worker)
#pragma unroll
    for (int j = 0; j < COLS; ++j) red[(col0 + j) * RED_LD + row] = acc[j];
  cluster_sync_all();
  for (int e = rank * THREADS + (int)threadIdx.x; e < BM * BN; e += p.split * THREADS) {
    const int r = e % BM, c = e / BM;
    if (p0 + r >= p.rows_p || q0 + c >= p.rows_q) continue;
    const uint32_t at = smem_u32(red + c * RED_LD + r);
    float sum = 0.f;
    for (int x = 0; x < p.split; ++x) {
      float v;
      asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(mapa_u32(at, (uint32_t)x)) : "memory");
      sum = x ? sum + v : v;
    }
    C[(long long)(q0 + c) * p.c_q + p0 + r] = sum;
  }
  cluster_sync_all();                      // the others have read this CTA's sums
}

template <int BN, bool PK, bool QK, bool VEC>
cudaError_t launch(ugb_device *dev, const Params &p, dim3 grid, bool pdl) {
  constexpr unsigned long long bit = 1ull << (((BN / 32 - 1) * 2 + PK) * 4 + QK * 2 + VEC);
  if (!(dev->f32_split_smem_set & bit)) {  // once: a step that is captured has run eagerly before
    const cudaError_t e = cudaFuncSetAttribute(f32_split_kernel<BN, PK, QK, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<BN>::SMEM);
    if (e != cudaSuccess) return e;
    dev->f32_split_smem_set |= bit;
  }
  return ugb_launch_cluster(f32_split_kernel<BN, PK, QK, VEC>, grid, dim3(THREADS), Shape<BN>::SMEM, dev->stream, pdl, p.split, p);
}

template <int BN>
cudaError_t launch_any(ugb_device *dev, const Params &p, dim3 grid, bool pk, bool qk, bool vec, bool pdl) {
#define UGB_GO(PK, QK) (vec ? launch<BN, PK, QK, true>(dev, p, grid, pdl) : launch<BN, PK, QK, false>(dev, p, grid, pdl))
  if (pk) return qk ? UGB_GO(true, true) : UGB_GO(true, false);
  return qk ? UGB_GO(false, true) : UGB_GO(false, false);
#undef UGB_GO
}

}  // namespace

int32_t ugb_f32_split(ugb_device *dev, const ugb_f32_split_args &a, int bn, int split) {
  const size_t tiles_p = (a.rows_p + BM - 1) / BM, tiles_q = (a.rows_q + bn - 1) / bn;
  if (a.batch == 0 || a.batch > 65535 || tiles_q > 65535 || a.rows_p == 0 || a.rows_q == 0 || a.k == 0) return UGB_ERR_UNSUPPORTED;
  if (a.rows_p >= 1u << 30 || a.rows_q >= 1u << 30 || a.k >= 1u << 30 || split < 1 || split > 8) return UGB_ERR_UNSUPPORTED;
  const bool pk = a.p_ks == 1, qk = a.q_ks == 1;
  if ((!pk && a.p_rs != 1) || (!qk && a.q_rs != 1)) return UGB_ERR_UNSUPPORTED;
  auto pieces = [&](const float *at, bool kc, long long rs, long long ks, long long batch, size_t rows) {
    return ((uintptr_t)at & 15) == 0 && batch % 4 == 0 && (kc ? rs % 4 == 0 && a.k % 4 == 0 : ks % 4 == 0 && rows % 4 == 0);
  };
  const bool vec = pieces(a.p, pk, a.p_rs, a.p_ks, a.p_batch, a.rows_p) && pieces(a.q, qk, a.q_rs, a.q_ks, a.q_batch, a.rows_q);
  Params p{a.c, a.p, a.q, a.p_rs, a.p_ks, a.p_batch, a.q_rs, a.q_ks, a.q_batch, a.c_q, a.c_batch, (int)a.rows_p, (int)a.rows_q, (int)a.k, split,
           (int)(((a.k + split - 1) / split + BK - 1) / BK * BK), dev->status_dev};
  const dim3 grid((unsigned)(tiles_p * split), (unsigned)tiles_q, (unsigned)a.batch);
  cudaError_t e;
  switch (bn) {
    case 32: if (!qk) return UGB_ERR_UNSUPPORTED; e = launch_any<32>(dev, p, grid, pk, qk, vec, a.pdl); break;
    case 64: e = launch_any<64>(dev, p, grid, pk, qk, vec, a.pdl); break;
    case 96: if (!qk) return UGB_ERR_UNSUPPORTED; e = launch_any<96>(dev, p, grid, pk, qk, vec, a.pdl); break;
    default: return UGB_ERR_UNSUPPORTED;
  }
  if (e != cudaSuccess) return ugb_fail(dev, UGB_ERR_CUDA, "launch of f32_split_kernel failed: %s", cudaGetErrorString(e));
  return ugb_after_launch(dev, "f32_split_kernel");
}
