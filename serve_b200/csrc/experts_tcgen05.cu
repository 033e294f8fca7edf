// The products of routed experts in bfloat16 on the fifth-generation tensor cores (tcgen05 + TMA), for any number of tokens.
//
// An expert's matrices are far larger than what its few tokens bring, so these products are bound by reading the weights
// once. The roles are therefore swapped: 128 rows of a weight matrix are the 128 rows of the tensor core's tile, the
// expert's tokens (rounded up to 16, at most 256 of them) are its columns. No work goes into padding tokens up to a tile of
// 64 or 128, and an expert of at most 256 tokens has every weight read exactly once.
//
// A unit of work is (an expert's run of tokens, some rows of its matrix). Persistent CTAs, one an SM, take units in turn.
// Warp 0 feeds a ring of stages of 64 k-values with TMA: weight rows, and the tokens' rows from an operand in grouped
// order (moe_gather_kernel makes it for gate/up: fetching the rows from the activations with tile::gather4 instead took
// 115 cycles for every four rows, and the gate/up product of 2,048 tokens 170 us). Warp 1 issues the products (both walk their loops
// as whole warps, see elect_one: issued by one thread of a divergent warp, behind a division by the number of stages, 8 tokens' gate/up took
// 44.7 us in place of 32.7);
// sixteen warps take the finished sums out of tensor memory. The ring runs on into the next unit while sums are taken out,
// so the weights keep streaming although a wide unit has a single set of accumulators.
//
// A unit with two accumulators is 256 weight rows: many tokens an expert, where the tokens' rows are what the SMs fetch
// most. A unit with one is at most 128 rows, of a count that shares the step's rows out evenly over the SMs (pick_unit):
// few tokens an expert, where a unit is nothing but weights and a last round of a few units would leave most SMs idle.
// Every TMA instruction costs its issuer time however little it fetches, so a stage takes as few as possible: there is a map for every
// count of weight rows a unit may have, and maps of 128, 64 and 16 tokens.
//
//   gate/up:  act[row, c] = f(g, u): with two accumulators the gate rows are one and the up rows of the same outputs the
//             other, so a thread holds both sums; with one, 16 gate rows and the 16 up rows of the same outputs take turns
//             along the tile's rows and half-warps exchange what the other needs.
//   up:       act[row, c] = relu(x W^T)^2 (experts without a gate)
//   down:     out[pair, c] = act[row] W^T, times the pair's weight if that belongs to the output
//
// Every sum runs over k in ascending order whatever else is in the step. Waits are bounded; one that runs out raises *error.
#include "tcgen05_ops.cuh"

using namespace sb;
typedef __nv_bfloat16 bf16;

namespace {

constexpr int BK = 64, W_BYTES = 128 * BK * 2;   // a stage's k-values; bytes of 128 weight rows
constexpr int EPI_WARPS = 16, THREADS = 64 + 32 * EPI_WARPS;
constexpr int MAX_STAGES = 12, MAX_TOKENS = 256;
constexpr int UNITS = 5;                         // counts of outputs a unit with one accumulator may have
constexpr int SMEM_LIMIT = 224 * 1024;
constexpr uint32_t TMEM_COLS = 512;
enum { GATED = 0, RELU2 = 1, DOWN = 2 };
__host__ __device__ constexpr int unit_outputs(int mode, int i) {
  return mode == GATED ? (i < 3 ? 64 - 16 * i : 16) : (i < 2 ? 128 - 32 * i : 96 - 16 * i);        // 64 48 32 16 16, 128 96 64 48 32
}

struct Args {
  const int* order;
  const int* offsets;
  const int* tiles;        // (expert, first row in grouped order) of every run of at most ``cap`` tokens of an expert
  const int* n_tiles;
  const float* wts;
  void* out;
  int* error;
  int K;                   // the product's k
  int cols;                // outputs of a row of ``out``: ff, or N of the down product
  int w_rows;              // rows of one expert in the weight map
  int cap, stages, scale, act_kind;
  float limit, alpha;
};

struct Maps {
  CUtensorMap w[UNITS];    // two accumulators: only the first
  CUtensorMap x[3];        // 128, 64 and 16 tokens
};

__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + expf(-x)); }

__device__ __forceinline__ float gated(float g, float u, const Args& a) {
  if (a.act_kind == 1) {
    g = fminf(g, a.limit);
    u = fminf(fmaxf(u, -a.limit), a.limit);
    return g * sigmoid_f(a.alpha * g) * (u + 1.f);
  }
  return g * sigmoid_f(g) * u;
}

// rows of a stage's room for tokens: what the boxes of the longest run fill
__host__ __device__ inline int x_rows_of(int cap) { return cap <= 16 ? 16 : (cap <= 64 ? 64 : (cap + 127) / 128 * 128); }

// What a step costs with units of r outputs: the units of the CTA that has the most of them, times a unit's length. A stage
// takes about as long as reading 10 KB more than it holds (80 weight rows of 64 k-values, or the gate and up rows of 40 outputs).
__host__ __device__ constexpr int unit_cost(int mode, int runs, int cols, int r, int ctas) {
  return (runs * ((cols + r - 1) / r) + ctas - 1) / ctas * (r + (mode == GATED ? 40 : 80));
}

// Which count of outputs a unit with one accumulator has: the cheapest.
__host__ __device__ inline int pick_unit(int mode, int runs, int cols, int ctas) {
  int best = 0;
  for (int i = 1; i < UNITS; ++i)
    if (unit_cost(mode, runs, cols, unit_outputs(mode, i), ctas) < unit_cost(mode, runs, cols, unit_outputs(mode, best), ctas)) best = i;
  return best;
}

template <int MODE, int ACCS, typename O>
__global__ void __launch_bounds__(THREADS) experts_kernel(const __grid_constant__ Maps maps, const Args a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t full_bar[MAX_STAGES];
  __shared__ __align__(8) uint64_t empty_bar[MAX_STAGES];
  __shared__ __align__(8) uint64_t acc_full[2];
  __shared__ __align__(8) uint64_t acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~(uintptr_t)1023);

  constexpr bool TURNS = MODE == GATED && ACCS == 1;         // gate and up rows take turns in one accumulator
  constexpr int MOST = MODE == GATED ? 64 * ACCS : 128 * ACCS;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int stage_bytes = ACCS * W_BYTES + x_rows_of(a.cap) * BK * 2;
  const int k_blocks = (a.K + BK - 1) / BK;
  const int acc_cols = a.cap <= 128 ? 128 : 256;             // tensor-memory columns of an accumulator
  const int bufs = ACCS * acc_cols <= 256 ? 2 : 1;           // sets of accumulators

  if (threadIdx.x == 0) {
    for (int s = 0; s < MAX_STAGES; ++s) {
      tc::mbar_init(&full_bar[s], 1);
      tc::mbar_init(&empty_bar[s], 1);
    }
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&acc_full[b], 1);
      tc::mbar_init(&acc_empty[b], EPI_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(&tmem_base_s)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  // set up; the runs, the tokens and the right to overwrite the output come with the end of the kernel before
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t tmem_base = tmem_base_s;
  const int runs = a.n_tiles[0];
  const int which = ACCS == 2 || a.cap > 16 ? 0 : pick_unit(MODE, runs, a.cols, gridDim.x);
  const int unit_cols = ACCS == 2 ? MOST : unit_outputs(MODE, which);
  const int col_blocks = (a.cols + unit_cols - 1) / unit_cols;
  const int units = runs * col_blocks;
  bool failed = false;

  if (warp == 0) {
    int it = 0, s = 0;                                       // stages filled so far, the next one, its barrier's parity
    unsigned phase = 1;                                      // (fresh barriers pass a wait on parity 1)
    for (int unit = blockIdx.x; unit < units && !failed; unit += gridDim.x) {
      const int tile = unit / col_blocks, c0 = (unit - tile * col_blocks) * unit_cols;
      const int e = a.tiles[2 * tile], row0 = a.tiles[2 * tile + 1];
      const int rows = min(a.cap, a.offsets[e + 1] - row0), n = (rows + 15) & ~15;
      const int w0 = e * a.w_rows + c0;
      const int w_bytes = ACCS == 2 ? 2 * W_BYTES : (TURNS ? 2 : 1) * unit_cols * BK * 2;
      // the run's tokens: whole boxes of 128, then one of 128, 64 or 16 for the rest (its rows beyond the run are another's)
      const int rest = n & 127, full = n >> 7, rest_rows = rest > 64 ? 128 : (rest > 16 ? 64 : rest);
      const CUtensorMap* map_rest = &maps.x[rest > 64 ? 0 : (rest > 16 ? 1 : 2)];
      const unsigned bytes = w_bytes + (full * 128 + rest_rows) * BK * 2;
      for (int kb = 0; kb < k_blocks; ++kb, ++it) {
        if (!tc::warp_wait(&empty_bar[s], phase)) { failed = true; break; }
        if (tc::elect_one()) {
          unsigned char* w_dst = ring + (size_t)s * stage_bytes;
          unsigned char* x_dst = w_dst + ACCS * W_BYTES;
          tc::mbar_expect_tx(&full_bar[s], bytes);
          if (ACCS == 2) {
            tc::load_2d(w_dst, &maps.w[0], &full_bar[s], kb * BK, w0);
            tc::load_2d(w_dst + W_BYTES, &maps.w[0], &full_bar[s], kb * BK, w0 + (MODE == GATED ? a.cols : 128));
          } else if (TURNS) {
            tc::load_5d(w_dst, &maps.w[which], &full_bar[s], kb * BK, 0, 0, c0 / 16, e);
          } else {
            tc::load_2d(w_dst, &maps.w[which], &full_bar[s], kb * BK, w0);
          }
          for (int i = 0; i < full; ++i) tc::load_2d(x_dst + i * 128 * BK * 2, &maps.x[0], &full_bar[s], kb * BK, row0 + i * 128);
          if (rest) tc::load_2d(x_dst + full * 128 * BK * 2, map_rest, &full_bar[s], kb * BK, row0 + full * 128);
        }
        __syncwarp();
        if (++s == a.stages) { s = 0; phase ^= 1; }
      }
    }
    // a wait that ran out: the copies under way land before the block's shared memory is given back (every other wait fails first)
    for (int f = max(0, it - a.stages); failed && f < it; ++f) tc::mbar_wait(&full_bar[f % a.stages], (f / a.stages) & 1);
  } else if (warp == 1) {
    const uint32_t ring_lo = tc::desc_lo(tc::smem_u32(ring));
    int s = 0, local = 0;
    unsigned phase = 0;
    for (int unit = blockIdx.x; unit < units && !failed; unit += gridDim.x, ++local) {
      const int tile = unit / col_blocks;
      const int e = a.tiles[2 * tile], row0 = a.tiles[2 * tile + 1];
      const int n = (min(a.cap, a.offsets[e + 1] - row0) + 15) & ~15;
      const uint32_t idesc = tc::make_idesc(128, n);
      const int buf = bufs == 2 ? local & 1 : 0, round = bufs == 2 ? local >> 1 : local;
      if (!tc::warp_wait(&acc_empty[buf], (round & 1) ^ 1)) { failed = true; break; }
      const uint32_t acc = tmem_base + (uint32_t)(buf * 256);
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!tc::warp_wait(&full_bar[s], phase)) { failed = true; break; }
        tc::fence_after();
        const uint32_t dw = ring_lo + (uint32_t)(s * (stage_bytes >> 4)), dx = dw + (uint32_t)(ACCS * W_BYTES >> 4);
        if (tc::elect_one()) {
#pragma unroll
          for (int j = 0; j < BK / 16; ++j)
#pragma unroll
            for (int i = 0; i < ACCS; ++i)
              tc::mma_lo(acc + (uint32_t)(i * acc_cols), dw + (uint32_t)((i * W_BYTES >> 4) + j * 2), dx + (uint32_t)(j * 2), idesc, (kb | j) != 0 ? 1u : 0u);
          tc::commit(&empty_bar[s]);
          if (kb + 1 == k_blocks) tc::commit(&acc_full[buf]);
        }
        __syncwarp();
        if (++s == a.stages) { s = 0; phase ^= 1; }
      }
    }
  } else {
    // a warp may touch the 32 tensor-memory lanes of its rank modulo 4; the four warps of a quarter take the chunks of 32
    // tokens in turn. A lane is a weight row, so the 32 lanes of a store lie side by side in the output.
    const int q = warp & 3, first = ((warp - 2) >> 2) * 32;
    int local = 0;
    for (int unit = blockIdx.x; unit < units && !failed; unit += gridDim.x, ++local) {
      const int tile = unit / col_blocks, c0 = (unit - tile * col_blocks) * unit_cols;
      const int e = a.tiles[2 * tile], row0 = a.tiles[2 * tile + 1];
      const int rows = min(a.cap, a.offsets[e + 1] - row0);
      const int buf = bufs == 2 ? local & 1 : 0, round = bufs == 2 ? local >> 1 : local;
      const bool ok = tc::mbar_wait(&acc_full[buf], round & 1);
      if (!__all_sync(0xffffffffu, ok)) { failed = true; break; }
      tc::fence_after();
      const uint32_t acc = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * 256);
#pragma unroll 1
      for (int ch = first; ch < rows; ch += 128) {
        const int here = min(32, rows - ch);
        const int pair = lane < here ? a.order[row0 + ch + lane] : 0;
        const float wt = (a.scale && lane < here) ? a.wts[pair] : 1.f;
        uint32_t v[32], u[32];
        tc::load32(acc + (uint32_t)ch, v);
        if (ACCS == 2) tc::load32(acc + (uint32_t)(acc_cols + ch), u);
        tc::wait_loads();
        if (TURNS) {
          // lanes 0..15 hold gate rows, 16..31 the up rows of the same outputs: the lower half takes tokens 0..15, the upper 16..31
          const bool low = lane < 16;
          const int col = q * 16 + (lane & 15) < unit_cols ? c0 + q * 16 + (lane & 15) : a.cols;
          bf16* dst = (bf16*)a.out + (size_t)(row0 + ch + (low ? 0 : 16)) * a.cols + col;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float mine = __uint_as_float(low ? v[i] : v[i + 16]);
            const float other = __uint_as_float(__shfl_xor_sync(0xffffffffu, low ? v[i + 16] : v[i], 16));
            const float w = __shfl_sync(0xffffffffu, wt, i + (low ? 0 : 16));
            const float y = gated((low ? mine : other) * w, (low ? other : mine) * w, a);
            if (i + (low ? 0 : 16) < here && col < a.cols) dst[(size_t)i * a.cols] = __float2bfloat16_rn(y);
          }
        } else if (MODE == GATED) {
          const int col = c0 + q * 32 + lane;
          bf16* dst = (bf16*)a.out + (size_t)(row0 + ch) * a.cols + col;
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const float w = __shfl_sync(0xffffffffu, wt, i);
            const float y = gated(__uint_as_float(v[i]) * w, __uint_as_float(u[i]) * w, a);
            if (i < here && col < a.cols) dst[(size_t)i * a.cols] = __float2bfloat16_rn(y);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const float w = __shfl_sync(0xffffffffu, wt, i);
            const int p = __shfl_sync(0xffffffffu, pair, i);
            if (i >= here) continue;
#pragma unroll
            for (int h = 0; h < ACCS; ++h) {
              const int col = ACCS == 2 || q * 32 + lane < unit_cols ? c0 + h * 128 + q * 32 + lane : a.cols;
              float y = __uint_as_float(h == 0 ? v[i] : u[i]);
              if (col >= a.cols) continue;
              if (MODE == RELU2) {
                y = fmaxf(y, 0.f);
                ((bf16*)a.out)[(size_t)(row0 + ch + i) * a.cols + col] = __float2bfloat16_rn(y * y);
              } else {
                ((O*)a.out)[(size_t)p * a.cols + col] = from_float<O>(y * w);
              }
            }
          }
        }
      }
      tc::fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&acc_empty[buf]);
    }
  }
  if (failed) atomicExch(a.error, 1);
  tc::fence_before();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

template <int MODE, int ACCS, typename O>
int launch(const void* w, const void* x, int n_pairs, int E, Args a, cudaStream_t stream) {
  Maps maps;
  const uint64_t K = (uint64_t)a.K;
  // (an encoding is host time: only what the kernel may read, which chooses among the counts of outputs for up to 16 tokens alone)
  for (int i = 0; i < UNITS; ++i) {
    int rc;
    if (i && (ACCS == 2 || a.cap > 16 || unit_outputs(MODE, i) == unit_outputs(MODE, i - 1))) { maps.w[i] = maps.w[i - 1]; continue; }
    if (ACCS == 2) {
      rc = tc::make_map_2d(&maps.w[0], w, (uint64_t)E * a.w_rows, K, K, 128);
    } else if (MODE == GATED) {
      // [expert][group of 16 outputs][gate, up][16][k]: one box is the gate and up rows of some groups, taking turns
      const uint64_t ff = (uint64_t)a.cols;
      const uint64_t dims[5] = {K, 16, 2, ff / 16, (uint64_t)E}, strides[4] = {K, ff * K, 16 * K, 2 * ff * K};
      const uint32_t box[5] = {(uint32_t)BK, 16, 2, (uint32_t)unit_outputs(GATED, i) / 16, 1};
      rc = tc::make_map(&maps.w[i], w, 5, dims, strides, box);
    } else {
      rc = tc::make_map_2d(&maps.w[i], w, (uint64_t)E * a.w_rows, K, K, (uint32_t)unit_outputs(MODE, i));
    }
    if (rc) return rc;
  }
  for (int i = 2; i >= 0; --i) {                    // 128 tokens only for runs of more than 64, 64 for more than 16
    if (a.cap <= (i == 0 ? 64 : (i == 1 ? 16 : 0))) { maps.x[i] = maps.x[i + 1]; continue; }
    const int rc = tc::make_map_2d(&maps.x[i], x, (uint64_t)n_pairs, K, K, i == 0 ? 128 : (i == 1 ? 64 : 16));
    if (rc) return rc;
  }
  const int stage = ACCS * W_BYTES + x_rows_of(a.cap) * BK * 2;
  a.stages = (SMEM_LIMIT - 1024) / stage < MAX_STAGES ? (SMEM_LIMIT - 1024) / stage : MAX_STAGES;
  const size_t smem = (size_t)a.stages * stage + 1024;
  auto k = experts_kernel<MODE, ACCS, O>;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const long long units = (long long)(n_pairs / a.cap + (E < n_pairs ? E : n_pairs)) * ((a.cols + 15) / 16);      // (at most)
  const int sms = sm_count();
  SB_PDL_CHECK(launch_pdl(k, dim3((unsigned)(units < sms ? units : sms)), dim3(THREADS), smem, stream, maps, a));
  return 0;
}

// One accumulator a unit or two. Up to 16 tokens (a run is one group of 16 columns): what costs less for the number of
// experts that as many uniform choices hit. Gate/up with one | two at width 2,048, 64 experts, 4 a token: 1 token 14.2 | 17.8 us, 4 tokens 23.8 | 22.9,
// 8 tokens 32.4 | 39.7 (156 units of two for 148 SMs), 16 tokens 45.6 | 43.9. Up to 128 tokens two: the tokens' rows are then fetched half as often
// (64 tokens 69.6 | 68.4). With more there is room in tensor memory for two sets of sums only if a unit has one accumulator, and taking
// sums out overlaps the next unit's products: gate/up of 256 tokens 77.2 | 79.4, 2,048 tokens 92.4 | 105.4, 4,096 tokens 118 | 146; down of 2,048
// tokens 47.7 | 54.5. Long rows of few tokens an expert are the exception (width 4,096, 64 experts, 8 a token: gate/up of 512
// tokens 113.9 | 110.4, of 1,024 125.2 | 127.9).
int pick_accs(int mode, const Args& a, int n_pairs, int E) {
  if (a.cap > 128) return mode == GATED && a.K > 3072 && n_pairs < 100 * E ? 2 : 1;
  if (a.cap > 16) return 2;
  float miss = 1.f;
  for (int i = 0; i < n_pairs && i < 256; ++i) miss *= 1.f - 1.f / (float)E;
  const int runs = (int)((float)E * (1.f - miss) + 0.5f), sms = sm_count();
  const int one = unit_cost(mode, runs, a.cols, unit_outputs(mode, pick_unit(mode, runs, a.cols, sms)), sms);
  return unit_cost(mode, runs, a.cols, mode == GATED ? 128 : 256, sms) < one ? 2 : 1;
}

template <int MODE, typename O>
int launch_accs(const void* w, const void* x, int n_pairs, int E, const Args& a, cudaStream_t stream) {
  return pick_accs(MODE, a, n_pairs, E) == 2 ? launch<MODE, 2, O>(w, x, n_pairs, E, a, stream) : launch<MODE, 1, O>(w, x, n_pairs, E, a, stream);
}

// xg[i] = x[order[i] / top]: a warp a row, 16 bytes a lane and step. Like the kernels of routed_experts.cu it may begin before the kernel
// that writes what it reads has ended, so it reads with plain loads (no __ldg, no __restrict__: both say that nobody writes meanwhile).
__global__ void __launch_bounds__(256) moe_gather_kernel(const bf16* x, int x_stride, const int* order, const int* offsets, int E, int top, int K, bf16* xg) {
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  pdl_launch_dependents();
  pdl_wait();
  if (i >= offsets[E]) return;                      // (choices that name no expert have no place)
  const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)(order[i] / top) * x_stride);
  uint4* dst = reinterpret_cast<uint4*>(xg + (size_t)i * K);
  for (int c = lane; c < K / 8; c += 128) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c + 32 * u < K / 8) v[u] = src[c + 32 * u];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c + 32 * u < K / 8) dst[c + 32 * u] = v[u];
  }
}

}  // namespace

// Tokens a run of these products holds at most for a step of n_tokens (the grouping's tile_rows), or 0 if they do not take
// the sizes: bfloat16, k of both products a multiple of 32 (so rows are whole 16-byte pieces, as TMA needs them).
SB_EXPORT int sb_moe_tensor_rows(int dtype, int K, int ff, int x_stride, int n_tokens) {
  if (dtype != SB_DTYPE_BF16 || K < 32 || K % 32 || ff < 32 || ff % 32 || x_stride % 8 || n_tokens < 1) return 0;
  return n_tokens >= MAX_TOKENS ? MAX_TOKENS : (n_tokens + 15) / 16 * 16;
}

// act [n_pairs rows in grouped order, ff]: gated = 1: f(x W_gate^T, x W_up^T) with w [E, 2 ff, K] (gate rows, then up rows), the
// pair's weight on both sums if scale_input, act_kind 0: silu(g) u, 1: the clamped form; gated = 0: relu(x W^T)^2, w [E, ff, K].
// xg [n_pairs, K]: room for the activations in grouped order.
SB_EXPORT int sb_moe_gate_up_tensor(const void* x, int x_stride, int n_tokens, void* xg, const void* w, const int* order, const int* offsets,
                                    const int* tiles, const int* n_tiles, const float* wts, int top, int n_pairs, int E, int K, int ff, int gated,
                                    int scale_input, int act_kind, float limit, float alpha, void* act, int tile_rows, int* error,
                                    cudaStream_t stream) {
  if (n_pairs <= 0) return 0;
  if (tile_rows != sb_moe_tensor_rows(SB_DTYPE_BF16, K, ff, x_stride, n_tokens) || tile_rows == 0 || top <= 0 || E <= 0) return SB_ERR_SHAPE;
  if (!aligned16(x) || !aligned16(w) || !aligned16(xg) || !error) return SB_ERR_ALIGN;
  SB_PDL_CHECK(launch_pdl(moe_gather_kernel, dim3((n_pairs + 7) / 8), dim3(256), 0, stream, (const bf16*)x, x_stride, order, offsets, E, top, K, (bf16*)xg));
  Args a = {};
  a.order = order; a.offsets = offsets; a.tiles = tiles; a.n_tiles = n_tiles; a.wts = wts; a.out = act; a.error = error;
  a.K = K; a.cols = ff; a.w_rows = gated ? 2 * ff : ff; a.cap = tile_rows; a.scale = gated && scale_input;
  a.act_kind = act_kind; a.limit = limit; a.alpha = alpha;
  return gated ? launch_accs<GATED, bf16>(w, xg, n_pairs, E, a, stream) : launch_accs<RELU2, bf16>(w, xg, n_pairs, E, a, stream);
}

// out [n_pairs, N] at the pair's own place, of dtype out_dtype; act [n_pairs, ff] in grouped order, w_down [E, N, ff].
SB_EXPORT int sb_moe_down_tensor(const void* act, const void* w_down, const int* order, const int* offsets, const int* tiles, const int* n_tiles,
                                 const float* wts, int n_pairs, int E, int ff, int N, int scale_output, void* out, int out_dtype, int tile_rows,
                                 int* error, cudaStream_t stream) {
  if (n_pairs <= 0) return 0;
  if (tile_rows <= 0 || tile_rows % 16 || tile_rows > MAX_TOKENS || ff % 32 || ff < 32 || N <= 0 || E <= 0) return SB_ERR_SHAPE;
  if (!aligned16(act) || !aligned16(w_down) || !error) return SB_ERR_ALIGN;
  Args a = {};
  a.order = order; a.offsets = offsets; a.tiles = tiles; a.n_tiles = n_tiles; a.wts = wts; a.out = out; a.error = error;
  a.K = ff; a.cols = N; a.w_rows = N; a.cap = tile_rows; a.scale = scale_output;
  if (out_dtype == SB_DTYPE_F32) return launch_accs<DOWN, float>(w_down, act, n_pairs, E, a, stream);
  if (out_dtype == SB_DTYPE_BF16) return launch_accs<DOWN, bf16>(w_down, act, n_pairs, E, a, stream);
  return SB_ERR_DTYPE;
}
