// Products of few rows with a large matrix: out[r, n] = sum_k A[r, k] W[n, k], up to 8 rows, bf16 or f16, f32 sums.
// The projections of a decode step of one to eight sequences (ug-llama's own case, ug-llama/src/model.rs:171-374, is one).
//
// Bound: the weight stream, and, since a step is a chain of dependent kernels, whatever lies between two of them.  So the
// weights go from HBM straight into registers: a thread has up to 16 loads of 16 bytes in flight (64 KiB per CTA), the first
// 64 KiB of a CTA are requested before the wait for the preceding kernel, and each register is refilled with the next piece
// as soon as it has been used.  What is left behind the wait is a read of the activations from L2, a few MMAs, one
// reduction through shared memory and the store; no ring, no barriers, no TMEM, no tensor maps.
//
// Requesting the rest of a CTA's share into L2 before the wait as well made single kernels faster (46 MB: 10.9 to 10.3 us) and
// the chain slower (Llama 836 to 845 us a step, Kabidra 798 to 827): the requests delay the reads that the chain waits for.
//
// Work is cut into units of 16 rows of W x one k split x one batch step (or group), dealt to the CTAs in equal contiguous
// shares.  Inside a unit the 8 warps take 64-wide k chunks in turn.  The products are mma.sync m16n8k16 with the rows of W as
// the 16 and the rows of A as the 8; the order of k inside a chunk is permuted so that a lane's
// fragments are 16 contiguous bytes of a row of W and of A alike.  The contraction is 8 columns wide: tcgen05 would run
// it as 64 and needs its operands in shared memory first.  The activations of a warp's chunks stay in registers while its
// CTA walks the units of one split.  Partial sums are added in the order of the warps: the same bits on every run.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "gemm_skinny.cuh"

namespace {

constexpr int WARPS = 8, THREADS = WARPS * 32;
constexpr int CHUNK = 64;                  // k of one step of a warp: a 128-byte line of every row
constexpr int MAX_CHUNKS = 4;              // of a warp in flight
constexpr int TILE_N = 16;                 // rows of W
constexpr int RED_LD = 20;                 // floats between the columns of the reduction tile: 8 t + g are distinct banks

struct Params {
  const void *w, *a;
  void *out;
  long long w_batch, a_ld, a_batch, c_ld, c_batch, c_split;      // elements
  int rows, n, k, tiles, splits, chunks, chunks_per_split, spans, units;
  int epi, late_trigger, wait_first;       // wait_first: a kernel of the stream may write W
  const int *groups;                       // expert of group tile i, -1 behind the last; or null
  int n_groups_tiles, tile_m;
  ugb_skinny_gate gate;                    // GATE: where the activations come from
};

// A piece of W, read once: past L1.  FIXED: nothing writes it as long as the kernel lives, as the non-coherent load wants it.  A
// kernel that a W's writer may still run beside (Params::wait_first) takes the ordinary load.
template <bool FIXED>
static __device__ __forceinline__ uint4 ld_stream(const void *p) {
  uint4 v;
  if constexpr (FIXED)
    asm volatile("ld.global.nc.L1::no_allocate.L2::256B.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  else
    asm volatile("ld.global.L1::no_allocate.L2::256B.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
template <bool F16>
static __device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if constexpr (F16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <bool F16> static __device__ __forceinline__ void store16(void *out, long long i, float v) {
  if constexpr (F16) reinterpret_cast<__half *>(out)[i] = __float2half_rn(v);
  else reinterpret_cast<__nv_bfloat16 *>(out)[i] = __float2bfloat16_rn(v);
}

// Activations k .. k + 7 of row r, formed from the product before: gelu_tanh(sum of its partials) * the row's token in the table,
// rounded to bf16.  Every CTA does it again for all of its k (2048 values of 1024 bytes of partials and table each); what it
// saves is a kernel between two products of 1 MB (Zidevik, 8 sequences: 28 of them a step, request of 32 steps 96.4 -> 95.0 ms).
static __device__ __forceinline__ uint4 gate_entry(const ugb_skinny_gate &q, int r, int k) {
  const int id = q.tok[r];
  return id >= 0 && id < q.vocab ? __ldg(reinterpret_cast<const uint4 *>(q.table + (size_t)id * q.table_ld + q.off + k)) : make_uint4(0, 0, 0, 0);
}
// `e`: the table's values, asked for ahead of the wait: the token is the step's own, and its row comes from HBM.
static __device__ __forceinline__ uint4 gated_act(const ugb_skinny_gate &q, int r, int k, uint4 e) {
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const float *row = q.part + (size_t)r * q.ld + k;
  for (int p = 0; p < q.n_part; p += 4) {  // the partials are added in order
    float4 v[4][2];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        v[j][h] = p + j < q.n_part ? __ldcg(reinterpret_cast<const float4 *>(row + (size_t)(p + j) * q.part_stride) + h) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) { s[4 * h] += v[j][h].x; s[4 * h + 1] += v[j][h].y; s[4 * h + 2] += v[j][h].z; s[4 * h + 3] += v[j][h].w; }
  }
  const uint32_t w[4] = {e.x, e.y, e.z, e.w};
  uint32_t o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&w[j]));
    const __nv_bfloat162 y = __floats2bfloat162_rn(ugb_gelu_tanh(s[2 * j]) * t.x, ugb_gelu_tanh(s[2 * j + 1]) * t.y);
    o[j] = *reinterpret_cast<const uint32_t *>(&y);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// KC: chunks of a warp per piece; a unit whose split is longer runs in p.spans pieces.  FIXED: no kernel of the stream writes W.
// AHEAD: see ugb_tc_gemm_args::a_ahead.  Up to two chunks leave registers for a ninth warp, which waits and then lets the next kernel in;
// with more chunks the CTA does so behind its first unit.
template <int KC, bool F16, bool FIXED, bool GATE = false, bool AHEAD = false>
__global__ void __launch_bounds__(AHEAD && KC <= 2 ? THREADS + 32 : THREADS, 2)
skinny_gemm_kernel(const Params p) {
  __shared__ float red[2][WARPS][8 * RED_LD];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  int units = p.units, first_groups = -1;  // lane i: the group of tile i
  if (p.groups) {                          // the map is the preceding kernel's: only live tiles are dealt
    ugb_pdl_wait();
    if (p.late_trigger) ugb_pdl_trigger();
    int live = 0;
    for (int i = 0; i < p.n_groups_tiles; i += 32) {
      const int e = i + lane < p.n_groups_tiles ? __ldcg(p.groups + i + lane) : -1;
      if (i == 0) first_groups = e;
      live += __popc(__ballot_sync(0xffffffffu, e >= 0));
    }
    units = live * p.tiles;
  }
  if (!p.late_trigger) ugb_pdl_trigger();
  if (p.wait_first) ugb_pdl_wait();
  if (AHEAD && KC <= 2 && warp == WARPS) {
    ugb_pdl_wait();
    ugb_pdl_trigger();
    return;
  }
  const int u1 = (int)((long long)(blockIdx.x + 1) * units / gridDim.x);
  int u = (int)((long long)blockIdx.x * units / gridDim.x), s = 0;

  // piece being loaded: this lane's two rows of W, the warp's first chunk and the end of the piece
  const char *r0 = nullptr, *r1 = nullptr;
  int lc = 0, lc1 = 0;
  auto aim = [&](int unit, int span) {
    const int tile = unit % p.tiles, rest = unit / p.tiles;
    const int sp = p.groups ? 0 : rest % p.splits, b = p.groups ? 0 : rest / p.splits;
    size_t row = 0;
    if (p.groups) {                        // a read of the map here would stand between every two pieces
      const int e = rest < 32 ? __shfl_sync(0xffffffffu, first_groups, rest) : __ldcg(p.groups + rest);
      row = (size_t)max(0, e) * p.n;
    }
    const char *base = (const char *)p.w + 2 * (b * p.w_batch + (long long)(row * p.k));
    const int n0 = tile * TILE_N;
    r0 = base + 2 * (size_t)min(n0 + g, p.n - 1) * p.k;
    r1 = base + 2 * (size_t)min(n0 + g + 8, p.n - 1) * p.k;
    const int c0 = sp * p.chunks_per_split + span * (KC * WARPS);
    lc = c0 + warp;
    lc1 = min(min(p.chunks, (sp + 1) * p.chunks_per_split), c0 + KC * WARPS);
  };
  uint4 w[KC][4];
  auto load = [&](int i) {
    const int c = lc + i * WARPS, k = c * CHUNK + 8 * t;
    const bool lo = c < lc1 && k < p.k, hi = c < lc1 && k + 32 < p.k;
    const uint4 z = make_uint4(0, 0, 0, 0);
    w[i][0] = lo ? ld_stream<FIXED>(r0 + 2 * (size_t)k) : z;
    w[i][1] = lo ? ld_stream<FIXED>(r1 + 2 * (size_t)k) : z;
    w[i][2] = hi ? ld_stream<FIXED>(r0 + 2 * (size_t)k + 64) : z;
    w[i][3] = hi ? ld_stream<FIXED>(r1 + 2 * (size_t)k + 64) : z;
  };
  if (u < u1) {
    aim(u, 0);
#pragma unroll
    for (int i = 0; i < KC; ++i) load(i);
  }
  uint4 entry[2] = {};
  if constexpr (GATE) {                    // all of k is one piece
    if (u < u1 && g < p.rows)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (warp * CHUNK + 32 * h + 8 * t < p.k) entry[h] = gate_entry(p.gate, g, warp * CHUNK + 32 * h + 8 * t);
  }
  bool waits = AHEAD && KC > 2 && u < u1;
  if (!p.groups && !(AHEAD && KC <= 2) && !waits) {
    ugb_pdl_wait();
    if (p.late_trigger) ugb_pdl_trigger();
  }
  if (u >= u1) return;

  uint4 act[KC][2];
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  int have = -1, buf = 0;
  for (;;) {
    const int rest = u / p.tiles, key = rest * p.spans + s;
    if (key != have) {                     // the chunks of this piece of every row of A, as the MMA wants them
      have = key;
      const long long at = p.groups ? (long long)rest * p.tile_m * p.a_ld : (rest / p.splits) * p.a_batch;
      const char *row = (const char *)p.a + 2 * (at + g * p.a_ld);
#pragma unroll
      for (int i = 0; i < KC; ++i) {
        const int c = lc + i * WARPS, k = c * CHUNK + 8 * t;
        const bool on = g < p.rows && c < lc1;
        if constexpr (GATE) {
          act[i][0] = on && k < p.k ? gated_act(p.gate, g, k, entry[0]) : make_uint4(0, 0, 0, 0);
          act[i][1] = on && k + 32 < p.k ? gated_act(p.gate, g, k + 32, entry[1]) : make_uint4(0, 0, 0, 0);
          continue;
        }
        act[i][0] = on && k < p.k ? __ldcg(reinterpret_cast<const uint4 *>(row + 2 * (size_t)k)) : make_uint4(0, 0, 0, 0);
        act[i][1] = on && k + 32 < p.k ? __ldcg(reinterpret_cast<const uint4 *>(row + 2 * (size_t)k + 64)) : make_uint4(0, 0, 0, 0);
      }
    }
    int nu = u, ns = s + 1;
    if (ns == p.spans) { ns = 0; ++nu; }
    const bool more = nu < u1;
    if (more) aim(nu, ns);
#pragma unroll
    for (int i = 0; i < KC; ++i) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        mma<F16>(acc, w[i][2 * h].x, w[i][2 * h + 1].x, w[i][2 * h].y, w[i][2 * h + 1].y, act[i][h].x, act[i][h].y);
        mma<F16>(acc, w[i][2 * h].z, w[i][2 * h + 1].z, w[i][2 * h].w, w[i][2 * h + 1].w, act[i][h].z, act[i][h].w);
      }
      if (more) load(i);
    }
    if (ns == 0) {                         // the unit is complete
      float *c0 = red[buf][warp] + 2 * t * RED_LD + g, *c1 = c0 + RED_LD;
      c0[0] = acc[0]; c1[0] = acc[1]; c0[8] = acc[2]; c1[8] = acc[3];
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[e] = 0.f;
      asm volatile("bar.sync 1, 256;" ::: "memory");   // one per unit: the other buffer's readers have passed it before it is written again
      if (threadIdx.x < 128) {
        const int r = threadIdx.x >> 4, e = threadIdx.x & 15;
        float v = 0.f;
#pragma unroll
        for (int x = 0; x < WARPS; ++x) v += red[buf][x][r * RED_LD + e];
        const int n = (u % p.tiles) * TILE_N + e;
        const bool live = r < p.rows && n < p.n;
        const int sp = p.groups ? 0 : rest % p.splits;
        const long long row = p.groups ? ((long long)rest * p.tile_m + r) * p.c_ld : (rest / p.splits) * p.c_batch + sp * p.c_split + r * p.c_ld;
        if (p.epi == UGB_EPI_SILU_MUL_BF16) {
          const float up = __shfl_down_sync(0xffffffffu, v, 1);       // columns are (gate, up) pairs
          if (live && !(n & 1)) store16<false>(p.out, row + (n >> 1), __fdividef(v, __expf(-v) + 1.0f) * up);
        } else if (live) {
          if (p.epi == UGB_EPI_F32) reinterpret_cast<float *>(p.out)[row + n] = v;
          else if (p.epi == UGB_EPI_RELU2_BF16) { v = fmaxf(v, 0.f); store16<false>(p.out, row + n, v * v); }
          else store16<F16>(p.out, row + n, v);
        }
      }
      buf ^= 1;
      if (waits) {
        ugb_pdl_wait();
        ugb_pdl_trigger();
        waits = false;
      }
    }
    if (!more) return;
    u = nu; s = ns;
  }
}

// Two CTAs per SM at most, all with the same number of units where that comes out: what bounds the stream is how much of it is in flight
// (a step of Llama, one sequence, with up to 1.33, 1.5 and 2 CTAs per SM: 822, 822, 792 us; with one 901).
//
// Loads into registers wait for their data in the L1, which is what a launch leaves of an SM's 256 KB as shared memory.  A chain whose
// kernels want different splits pays for it twice: with much shared memory the L1 holds less than two CTAs have in flight, and an SM
// changes the split only when it is empty, so that a kernel that needs more than there is cannot start beside this one.  64 KB hold this
// kernel's sums and a CTA of attention beside them (the same step without a preference 792 us, with 32, 64 and 100 KB 726, 724 and 723, with
// next to none 943).
constexpr size_t CARVEOUT_BYTES = 64 * 1024;
// CTAs that a product may have so that it still counts as one round (ugb_skinny_one_round).
long long round_ctas(int sm_count) { return (long long)sm_count * 4 / 3; }

int chunks_of(size_t k) { return (int)((k + CHUNK - 1) / CHUNK); }

}  // namespace

int ugb_skinny_effective_splits(size_t k, int splits) {
  const int chunks = chunks_of(k);
  splits = std::max(1, std::min(splits, chunks));
  const int per = (chunks + splits - 1) / splits;
  return (chunks + per - 1) / per;
}

bool ugb_skinny_one_round(int sm_count, size_t n, size_t batch) { return (n + TILE_N - 1) / TILE_N * batch <= (size_t)round_ctas(sm_count); }

int ugb_skinny_splits(int sm_count, size_t n, size_t k) {
  const int chunks = chunks_of(k), tiles = (int)((n + TILE_N - 1) / TILE_N);
  const int need = (chunks + MAX_CHUNKS * WARPS - 1) / (MAX_CHUNKS * WARPS);
  const int fill = std::min(sm_count / std::max(1, tiles), chunks / WARPS);
  return ugb_skinny_effective_splits(k, std::min(UGB_SKINNY_SPLITS, std::max(need, fill)));
}

int32_t ugb_skinny_gemm(ugb_device *dev, const ugb_tc_gemm_args &args, int rows_per_tile, const ugb_skinny_gate *gate) {
  ugb_tc_gemm_args g = args;
  const long long dense_c = (long long)g.m * (long long)(g.epi == UGB_EPI_SILU_MUL_BF16 ? g.n / 2 : g.n);
  if (g.batch > 1 && g.b_batch == 0 && g.a_ld == 0 && g.c_ld == 0 && g.a_batch == (long long)(g.m * g.k) && (g.c_batch == 0 || g.c_batch == dense_c)) {
    g.m *= g.batch;                        // one matrix under densely stacked rows
    g.batch = 1;
  }
  const size_t rows = g.groups ? (size_t)rows_per_tile : g.m;
  if (!ugb_skinny_rows(rows) || !g.b_is_nk || g.pair_k || g.query_grid || g.query_ctas_per_sm || g.n == 0 || g.k == 0 || g.k % 8 != 0) return UGB_ERR_UNSUPPORTED;
  if (((uintptr_t)g.a | (uintptr_t)g.b) & 15) return UGB_ERR_UNSUPPORTED;                 // 16-byte loads of both operands
  if (g.a_ld < 0 || g.c_ld < 0 || g.a_ld % 8 != 0 || g.a_batch % 8 != 0 || g.b_batch % 8 != 0 || g.a_batch < 0 || g.b_batch < 0) return UGB_ERR_UNSUPPORTED;
  if (g.epi != UGB_EPI_F32 && g.epi != UGB_EPI_BF16 && g.epi != UGB_EPI_SILU_MUL_BF16 && g.epi != UGB_EPI_RELU2_BF16) return UGB_ERR_UNSUPPORTED;
  if ((g.splits > 1 && g.epi != UGB_EPI_F32) || (g.f16 && g.epi != UGB_EPI_F32 && g.epi != UGB_EPI_BF16)) return UGB_ERR_UNSUPPORTED;
  if (g.epi == UGB_EPI_SILU_MUL_BF16 && g.n % 2 != 0) return UGB_ERR_UNSUPPORTED;
  if (g.groups && (g.batch != 1 || g.splits > 1 || g.tile_m < (int)rows || g.m % g.tile_m != 0)) return UGB_ERR_UNSUPPORTED;
  if (g.n > (1u << 30) || g.k > (1u << 30) || g.batch < 1 || g.batch > 65535) return UGB_ERR_UNSUPPORTED;
  Params p{};
  p.w = g.b; p.a = g.a; p.out = g.out;
  const size_t out_cols = g.epi == UGB_EPI_SILU_MUL_BF16 ? g.n / 2 : g.n;
  p.a_ld = g.a_ld ? g.a_ld : (long long)g.k;
  p.c_ld = g.c_ld ? g.c_ld : (long long)out_cols;
  p.w_batch = g.b_batch; p.a_batch = g.a_batch;
  p.c_batch = g.c_batch ? g.c_batch : (long long)g.m * p.c_ld;
  p.c_split = (long long)g.batch * g.m * p.c_ld;
  p.rows = (int)rows; p.n = (int)g.n; p.k = (int)g.k;
  p.tiles = (int)((g.n + TILE_N - 1) / TILE_N);
  p.chunks = chunks_of(g.k);
  p.splits = ugb_skinny_effective_splits(g.k, g.splits);
  p.chunks_per_split = (p.chunks + p.splits - 1) / p.splits;
  const int kc = std::min(MAX_CHUNKS, (p.chunks_per_split + WARPS - 1) / WARPS);
  p.spans = (p.chunks_per_split + kc * WARPS - 1) / (kc * WARPS);
  if (gate) {                              // 16-byte pieces of the table's and the partials' rows, all of k in registers
    if (g.groups || g.f16 || g.batch != 1 || p.splits != 1 || kc != 1 || p.spans != 1 || gate->n_part < 1) return UGB_ERR_UNSUPPORTED;
    if (!g.b_static || ((uintptr_t)gate->part | (uintptr_t)gate->table) & 15 || gate->part_stride % 4 != 0 || gate->ld % 4 != 0 || gate->table_ld % 8 != 0 || gate->off % 8 != 0 ||
        gate->n % 8 != 0 || (size_t)gate->n != g.k)
      return UGB_ERR_UNSUPPORTED;
    p.gate = *gate;
  }
  p.epi = g.epi;
  p.late_trigger = g.late_trigger ? 1 : 0;
  p.wait_first = !g.b_static && !g.groups ? 1 : 0;
  const bool ahead = g.a_ahead && g.b_static && !g.groups && !gate && g.late_trigger && g.pdl && !g.f16;
  p.groups = g.groups; p.tile_m = g.tile_m;
  p.n_groups_tiles = g.groups ? (int)(g.m / g.tile_m) : 0;
  const long long units = (long long)p.tiles * (g.groups ? p.n_groups_tiles : (long long)p.splits * (long long)g.batch);
  if (units > (1ll << 30)) return UGB_ERR_UNSUPPORTED;
  p.units = (int)units;
  const ugb_launch_form form{g.pdl, 1, ugb_carveout(CARVEOUT_BYTES)};
  const long long most = 2ll * dev->sm_count;
  const long long rounds = (units + most - 1) / most;
  const unsigned grid = (unsigned)((units + rounds - 1) / rounds);
  cudaError_t e = cudaErrorInvalidValue;
#define UGB_SKINNY(KC) \
  e = ahead          ? ugb_launch_as(skinny_gemm_kernel<KC, false, true, false, true>, dim3(grid), dim3(KC <= 2 ? THREADS + 32 : THREADS), 0, dev->stream, form, p) \
      : g.f16        ? ugb_launch_as(skinny_gemm_kernel<KC, true, false>, dim3(grid), dim3(THREADS), 0, dev->stream, form, p) \
      : p.wait_first ? ugb_launch_as(skinny_gemm_kernel<KC, false, false>, dim3(grid), dim3(THREADS), 0, dev->stream, form, p) \
                     : ugb_launch_as(skinny_gemm_kernel<KC, false, true>, dim3(grid), dim3(THREADS), 0, dev->stream, form, p)
  if (gate) e = ugb_launch_as(skinny_gemm_kernel<1, false, true, true>, dim3(grid), dim3(THREADS), 0, dev->stream, form, p);
  else switch (kc) { case 1: UGB_SKINNY(1); break; case 2: UGB_SKINNY(2); break; case 3: UGB_SKINNY(3); break; default: UGB_SKINNY(4); }
#undef UGB_SKINNY
  if (e != cudaSuccess) return ugb_fail(dev, UGB_ERR_CUDA, "launch of skinny_gemm_kernel failed: %s", cudaGetErrorString(e));
  return ugb_after_launch(dev, "skinny_gemm_kernel");
}
