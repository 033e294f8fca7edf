// Matrix products for many rows (prompt portions) on the fifth-generation tensor cores:
// out[M,N] = a[M,K] * w[N,K]^T, bfloat16 in, float accumulation in tensor memory, bfloat16 out.
// With gate_up, w is [2N, K] (gate rows, then up rows) and out[m,n] = silu(gate) * up (serve/model.py:85):
// the activation is applied while the accumulator leaves tensor memory, and the [M, 2N] intermediate of the
// unfused path is never written. A third epilogue is the q/k/v product's (serve/model.py:120-124, 234-244): query and
// key columns are rotated by their token's position, queries go to out, keys and values straight into the
// request's cache pages, so the rotary kernel and its pass over q, k and v are not needed.
//
// A persistent CTA per SM walks over 128 x 256 tiles of the accumulator (with gate_up: 128 gate columns and
// their 128 up columns, i.e. 128 output columns). Warp 0 feeds a ring of four shared-memory stages with TMA
// (cp.async.bulk.tensor, 128-byte swizzle: one 128 x 64 box of a and a 256 x 64 box, or two 128 x 64 boxes, of
// w per stage, completion counted on an mbarrier); one thread of warp 1 issues tcgen05.mma (128 x 256 x 16,
// operands read from shared memory through matrix descriptors, accumulator in tensor memory) and releases
// stages with tcgen05.commit; warps 2..17 read a finished accumulator back with tcgen05.ld, apply the epilogue
// and store. Tensor memory holds two accumulators (2 x 256 columns), so the epilogue of one tile runs while
// the products of the next are issued. Tiles that share a panel of w run at the same time on neighbouring
// CTAs, so w comes from HBM once. Rows beyond M and k-values beyond K are zero-filled by TMA; stores are guarded.
//
// Every wait is bounded; a wait that runs out raises *error, and the CTA still frees its tensor memory.
#include <cuda.h>

#include "common.cuh"
#include "tcgen05_ops.cuh"

using namespace sb;
typedef __nv_bfloat16 bf16;

namespace {

constexpr int BM = 128, BN = 256, BK = 64;      // accumulator tile and k-values per stage
constexpr int NSTAGE = 4;
constexpr int A_BYTES = BM * BK * 2, B_BYTES = BN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int EPI_WARPS = 16;                    // four warps per quarter of the tensor-memory lanes
constexpr int THREADS = 64 + 32 * EPI_WARPS;     // warp 0: TMA, warp 1: MMA + tensor memory, warps 2..17: epilogue
constexpr uint32_t TMEM_COLS = 512;              // two accumulators of BN columns

constexpr int EPI_STORE = 0, EPI_GATE_UP = 1, EPI_ROPE = 2;

// What the q/k/v epilogue needs: columns are [q heads | k heads | v heads] x D, D a multiple of 32 so that the 32
// columns a thread holds at a time lie in one head. Adjacent pairs (2j, 2j+1) turn by position * inv_freq[j]; the
// cosine and sine of that angle come from a table [rot/2, rows] made once per step (sb_rope_angles): an epilogue
// warp has its scheduler to itself, so every instruction of a sincosf would be paid at full latency, 16 times per
// 32 columns, and the epilogue, not the tensor core, would set the kernel's pace.
struct RopeEpilogue {
  const int* positions;
  const int* token_row;
  const float2* cos_sin;
  const int* block_table;
  bf16* kc;
  bf16* vc;
  int* errors;
  int rot, H, Hkv, D, bt_width, ps, num_pages, write_cache;
  // gate/up epilogue: limit < 0 asks for gelu(g) * u; limit > 0 for the clamped activation g <- min(g, limit), u <- clamp(u, -limit, limit),
  // g * sigmoid(alpha g) * (u + 1) in place of silu(g) * u
  float act_limit, act_alpha;
  // plain products: an activation on every output, after its rounding to bfloat16 (0: none, 1: relu squared, 2: gelu in
  // its tanh form, 3: silu, 4: tanh)
  int store_act;
};

__device__ __forceinline__ float plain_act(float z, int kind) {
  if (kind == 1) { const float r = fmaxf(z, 0.f); return r * r; }
  if (kind == 2) return 0.5f * z * (1.f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
  if (kind == 3) return z / (1.f + expf(-z));
  return kind == 4 ? tanhf(z) : z;
}

__device__ __forceinline__ float gated_act(float g, float u, float limit, float alpha) {
  if (limit > 0.f) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return g / (1.0f + expf(-alpha * g)) * (u + 1.0f);
  }
  if (limit < 0.f) return 0.5f * g * (1.f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g))) * u;      // gelu (tanh form) as the gate
  return g / (1.0f + expf(-g)) * u;
}

// Where the keys and values of this thread's row go: element offset of (page, kv head 0, slot, 0) or -1.
__device__ __forceinline__ long long rope_row_slot(const RopeEpilogue& ra, int row, int pos) {
  const int blk = pos / ra.ps;
  const int page = (blk < ra.bt_width && pos >= 0) ? ra.block_table[(size_t)ra.token_row[row] * ra.bt_width + blk] : -1;
  if (page < 0 || page >= ra.num_pages) return -1;
  return ((long long)page * ra.Hkv * ra.ps + (pos - blk * ra.ps)) * ra.D;
}

// 32 accumulator columns n .. n+31 of one row: rounded to bfloat16 as the unfused path stores them, q and k pairs
// rotated, then q to out and k, v to the row's slot in the cache.
__device__ __forceinline__ void rope_store_chunk(const RopeEpilogue& ra, const uint32_t (&v)[32], int row, int n, int M, int N,
                                                 long long slot, bf16* __restrict__ out) {
  const int head = n / ra.D, d0 = n - head * ra.D;
  uint32_t packed[16];
  const bool turns = head < ra.H + ra.Hkv;
  // the table is [pair][row]: the 32 rows of a warp read 256 consecutive bytes per pair. All loads first, so that
  // their latencies overlap (a warp alone on its scheduler has nothing else to run meanwhile). Plain loads: the angles are made in the
  // same step, by a kernel that need not have ended when this one begins.
  float2 a[16];
  const float2* angles = ra.cos_sin + (size_t)(d0 >> 1) * M + row;
#pragma unroll
  for (int i = 0; i < 16; ++i) a[i] = (turns && d0 + 2 * i < ra.rot) ? angles[(size_t)i * M] : make_float2(1.f, 0.f);
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float x = to_float(__float2bfloat16_rn(__uint_as_float(v[2 * i]))), y = to_float(__float2bfloat16_rn(__uint_as_float(v[2 * i + 1])));
    __nv_bfloat162 o;
    if (turns && d0 + 2 * i < ra.rot) o = __floats2bfloat162_rn(x * a[i].x - y * a[i].y, y * a[i].x + x * a[i].y);
    else o = __floats2bfloat162_rn(x, y);
    packed[i] = *reinterpret_cast<uint32_t*>(&o);
  }
  bf16* dst;
  if (head < ra.H) {
    dst = out + (size_t)row * N + n;
  } else {
    if (!ra.write_cache) return;
    if (slot < 0) {
      if (n == ra.H * ra.D) atomicAdd(ra.errors, 1);       // once per token
      return;
    }
    const bool is_k = turns;
    const int kvh = is_k ? head - ra.H : head - ra.H - ra.Hkv;
    dst = (is_k ? ra.kc : ra.vc) + slot + (long long)kvh * ra.ps * ra.D + d0;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<uint4*>(dst + i * 8) = make_uint4(packed[4 * i], packed[4 * i + 1], packed[4 * i + 2], packed[4 * i + 3]);
}

template <int EPI>
__global__ void __launch_bounds__(THREADS) gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a,
                                                               const __grid_constant__ CUtensorMap map_w, bf16* __restrict__ out,
                                                               int M, int N, int K, int bn, int* __restrict__ error,
                                                               const RopeEpilogue ra) {
  constexpr bool GU = EPI == EPI_GATE_UP;
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t full_bar[NSTAGE];
  __shared__ __align__(8) uint64_t empty_bar[NSTAGE];
  __shared__ __align__(8) uint64_t acc_full[2];
  __shared__ __align__(8) uint64_t acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  // the dynamic region is aligned by hand: the 128-byte swizzle wants 1024-byte aligned tiles
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~(uintptr_t)1023);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  // bn: accumulator columns of a tile (a multiple of 32, at most BN), chosen by the host so that the tiles
  // fill whole waves of CTAs
  const int OUT_COLS = GU ? bn / 2 : bn;             // output columns of one tile
  const int m_tiles = (M + BM - 1) / BM, n_tiles = (N + OUT_COLS - 1) / OUT_COLS;
  const int total_tiles = m_tiles * n_tiles;
  const int k_blocks = (K + BK - 1) / BK;

  if (threadIdx.x == 0) {
#pragma unroll
    for (int s = 0; s < NSTAGE; ++s) {
      tc::mbar_init(&full_bar[s], 1);
      tc::mbar_init(&empty_bar[s], 1);
    }
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&acc_full[b], 1);
      tc::mbar_init(&acc_empty[b], EPI_WARPS);       // one arrival per epilogue warp
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(&tmem_base_s)), "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  // barriers, tensor memory and descriptors are ready; the activations (and the right to overwrite out) come with
  // the end of the kernel before this one
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t tmem_base = tmem_base_s;
  bool failed = false;

  // tile t of this CTA: consecutive CTAs take the row tiles of one panel of w
  const uint32_t tiles_lo = tc::desc_lo(tc::smem_u32(tiles));
  if (warp == 0) {
    int s = 0;
    unsigned phase = 1;                                // a fresh barrier passes a wait on parity 1: the first round finds every stage free
    for (int tile = blockIdx.x; tile < total_tiles && !failed; tile += gridDim.x) {
      const int m0 = (tile % m_tiles) * BM, n0 = (tile / m_tiles) * OUT_COLS;
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!tc::warp_wait(&empty_bar[s], phase)) { failed = true; break; }
        if (tc::elect_one()) {
          unsigned char* a_dst = tiles + s * STAGE_BYTES;
          unsigned char* b_dst = a_dst + A_BYTES;
          tc::mbar_expect_tx(&full_bar[s], (unsigned)(A_BYTES + bn * BK * 2));
          tc::load_2d(a_dst, &map_a, &full_bar[s], kb * BK, m0);
          tc::load_2d(b_dst, &map_w, &full_bar[s], kb * BK, n0);                         // with gate_up the gate rows
          if (GU) tc::load_2d(b_dst + bn * BK, &map_w, &full_bar[s], kb * BK, N + n0);   // and their up rows
        }
        __syncwarp();
        if (++s == NSTAGE) { s = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    const uint32_t idesc = tc::make_idesc(BM, bn);
    int s = 0, local = 0;
    unsigned phase = 0;
    for (int tile = blockIdx.x; tile < total_tiles && !failed; tile += gridDim.x, ++local) {
      const int buf = local & 1;
      // the epilogue must have emptied this accumulator (first use of each: passes at once)
      if (!tc::warp_wait(&acc_empty[buf], ((local >> 1) & 1) ^ 1)) { failed = true; break; }
      const uint32_t acc = tmem_base + (uint32_t)(buf * BN);
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!tc::warp_wait(&full_bar[s], phase)) { failed = true; break; }
        tc::fence_after();
        const uint32_t da = tiles_lo + (uint32_t)(s * (STAGE_BYTES >> 4)), db = da + (A_BYTES >> 4);
        if (tc::elect_one()) {
#pragma unroll
          for (int j = 0; j < BK / 16; ++j) {
            // 16 k-values further along the swizzled row: 32 bytes, two 16-byte units of the start address
            tc::mma_lo(acc, da + (uint32_t)(j * 2), db + (uint32_t)(j * 2), idesc, (kb | j) != 0 ? 1u : 0u);
          }
          tc::commit(&empty_bar[s]);          // the stage is free once these products have read it
          if (kb + 1 == k_blocks) tc::commit(&acc_full[buf]);     // the accumulator is complete once all products are done
        }
        __syncwarp();
        if (++s == NSTAGE) { s = 0; phase ^= 1; }
      }
    }
  } else {
    // epilogue warps: a warp may touch the 32 tensor-memory lanes of its rank modulo 4; the warps of a quarter take
    // the chunks of 32 columns in turn. With a tile or two per CTA the last tile's epilogue is not hidden behind any
    // product, and a warp alone on its scheduler pays every instruction's latency in full: with four warps (one per
    // quarter) the q/k/v product with rotation took 41.7 us inside a 2,048-token step, with eight 40.7, with sixteen 35.6.
    const int q = warp & 3, c_first = ((warp - 2) >> 2) * 32;
    int local = 0;
    for (int tile = blockIdx.x; tile < total_tiles && !failed; tile += gridDim.x, ++local) {
      const int m0 = (tile % m_tiles) * BM, n0 = (tile / m_tiles) * OUT_COLS;
      const int buf = local & 1;
      if (!tc::warp_wait(&acc_full[buf], (local >> 1) & 1)) { failed = true; break; }
      tc::fence_after();
      const int row = m0 + q * 32 + lane;
      const uint32_t acc = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN);
      int pos = 0;
      long long slot = -1;
      if (EPI == EPI_ROPE && row < M) {
        pos = ra.positions[row];
        if (ra.write_cache && n0 + OUT_COLS > ra.H * ra.D) slot = rope_row_slot(ra, row, pos);
      }
#pragma unroll 1
      for (int c = c_first; c < OUT_COLS; c += 32 * (EPI_WARPS / 4)) {
        if (n0 + c >= N) break;
        uint32_t v[32];
        tc::load32(acc + (uint32_t)c, v);
        if (!GU) tc::wait_loads();
        if (EPI == EPI_ROPE) {
          if (row < M) rope_store_chunk(ra, v, row, n0 + c, M, N, slot, out);
          continue;
        }
        uint32_t packed[16];
        if (GU) {
          uint32_t u[32];
          tc::load32(acc + (uint32_t)(OUT_COLS + c), u);
          tc::wait_loads();
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            // both halves rounded to the activation type first, as the unfused path stores them
            const float g0 = to_float(__float2bfloat16_rn(__uint_as_float(v[2 * i]))), g1 = to_float(__float2bfloat16_rn(__uint_as_float(v[2 * i + 1])));
            const float u0 = to_float(__float2bfloat16_rn(__uint_as_float(u[2 * i]))), u1 = to_float(__float2bfloat16_rn(__uint_as_float(u[2 * i + 1])));
            __nv_bfloat162 o = __floats2bfloat162_rn(gated_act(g0, u0, ra.act_limit, ra.act_alpha), gated_act(g1, u1, ra.act_limit, ra.act_alpha));
            packed[i] = *reinterpret_cast<uint32_t*>(&o);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            __nv_bfloat162 o = __floats2bfloat162_rn(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
            if (ra.store_act)          // on the rounded product, as the unfused path stores it first
              o = __floats2bfloat162_rn(plain_act(__low2float(o), ra.store_act), plain_act(__high2float(o), ra.store_act));
            packed[i] = *reinterpret_cast<uint32_t*>(&o);
          }
        }
        if (row < M) {
          bf16* dst = out + (size_t)row * N + n0 + c;
          if (n0 + c + 32 <= N) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              *reinterpret_cast<uint4*>(dst + i * 8) = make_uint4(packed[4 * i], packed[4 * i + 1], packed[4 * i + 2], packed[4 * i + 3]);
          } else {
            for (int i = 0; i < 32; ++i)
              if (n0 + c + i < N) dst[i] = reinterpret_cast<const bf16*>(packed)[i];
          }
        }
      }
      // this warp has read its part of the accumulator: the next tile but one may overwrite it
      tc::fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&acc_empty[buf]);
    }
  }
  if (failed) atomicExch(error, 1);
  tc::fence_before();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// ------------------------------------------------------------------------------------------------------------
// The same product with two CTAs (a cluster of two, on neighbouring SMs) working on one 256 x bn tile:
// tcgen05.mma.cta_group::2. CTA r of the pair holds rows 128 r .. 128 r + 127 of the tile's a operand and the r-th
// half of its w operand in its own shared memory, and its 128 rows of the accumulator in its own tensor memory.
// One thread of the first CTA issues the products for both; each product reads both shared memories, so every CTA
// loads (and the tensor core reads) only half of w per tile: shared-memory traffic per flop is 2/3 of the
// one-CTA kernel's, which is what that kernel is bound by. A stage is 16 KB of a + at most 16 KB of w, six stages.
//
// Barriers: both CTAs' TMA loads count their bytes on the first CTA's full barrier (its address with the pair bit
// cleared); tcgen05.commit arrives on the empty / accumulator-full barriers of both CTAs at once (multicast);
// the epilogue warps of both CTAs arrive on the first CTA's accumulator-empty barrier (a remote arrive for the second).
constexpr int PAIR_STAGES = 6;
constexpr int PAIR_A_BYTES = 128 * BK * 2, PAIR_STAGE_BYTES = PAIR_A_BYTES + 128 * BK * 2;
constexpr uint32_t PAIR_LEADER_MASK = 0xFEFFFFFFu;   // clears the bit of a shared-memory address that tells the two CTAs apart

__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, uint32_t leader_bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(tc::smem_u32(dst)), "l"(map), "r"(leader_bar), "r"(x), "r"(y) : "memory");
}
// arrives, once the products issued so far are done, on the barrier at this address in both CTAs of the pair
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(tc::smem_u32(bar)), "h"((unsigned short)3) : "memory");
}
__device__ __forceinline__ void cluster_sync_all_threads() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS)
    gemm_tcgen05_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                             bf16* __restrict__ out, int M, int N, int K, int bn, int* __restrict__ error,
                             const RopeEpilogue ra) {
  constexpr bool GU = EPI == EPI_GATE_UP;
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t full_bar[PAIR_STAGES];
  __shared__ __align__(8) uint64_t empty_bar[PAIR_STAGES];
  __shared__ __align__(8) uint64_t acc_full[2];
  __shared__ __align__(8) uint64_t acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  unsigned char* tiles = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~(uintptr_t)1023);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const int OUT_COLS = GU ? bn / 2 : bn;
  const int half = bn / 2;                              // rows of w this CTA loads per stage
  const int m_tiles = (M + 255) / 256, n_tiles = (N + OUT_COLS - 1) / OUT_COLS;
  const int total_tiles = m_tiles * n_tiles;
  const int k_blocks = (K + BK - 1) / BK;

  if (threadIdx.x == 0) {
#pragma unroll
    for (int s = 0; s < PAIR_STAGES; ++s) {
      tc::mbar_init(&full_bar[s], 1);
      tc::mbar_init(&empty_bar[s], 1);
    }
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&acc_full[b], 1);
      tc::mbar_init(&acc_empty[b], 2 * EPI_WARPS);   // one arrival per epilogue warp of both CTAs
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
  }
  if (warp == 1) {
    // the same warp of both CTAs allocates: the accumulators get the same address in both tensor memories
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(&tmem_base_s)), "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc::fence_before();
  __syncthreads();
  cluster_sync_all_threads();            // the other CTA's barriers exist before anything arrives on them
  tc::fence_after();
  pdl_launch_dependents();
  pdl_wait();                            // as in the one-CTA kernel
  const uint32_t tmem_base = tmem_base_s;
  bool failed = false;

  const uint32_t tiles_lo = tc::desc_lo(tc::smem_u32(tiles));
  if (warp == 0) {
    int s = 0;
    unsigned phase = 1;
    for (int tile = pair; tile < total_tiles && !failed; tile += num_pairs) {
      const int m0 = (tile % m_tiles) * 256 + (int)rank * 128, n0 = (tile / m_tiles) * OUT_COLS;
      // with gate_up the first CTA loads the gate rows and the second their up rows: accumulator columns
      // 0 .. half-1 are gate, half .. bn-1 are up, for the rows of both CTAs
      const int w_row = GU ? (rank == 0 ? n0 : N + n0) : n0 + (int)rank * half;
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!tc::warp_wait(&empty_bar[s], phase)) { failed = true; break; }
        if (tc::elect_one()) {
          unsigned char* a_dst = tiles + s * PAIR_STAGE_BYTES;
          const uint32_t leader_bar = tc::smem_u32(&full_bar[s]) & PAIR_LEADER_MASK;
          if (rank == 0) tc::mbar_expect_tx(&full_bar[s], (unsigned)(2 * (PAIR_A_BYTES + half * BK * 2)));
          tma_load_2d_pair(a_dst, &map_a, leader_bar, kb * BK, m0);
          tma_load_2d_pair(a_dst + PAIR_A_BYTES, &map_w, leader_bar, kb * BK, w_row);
        }
        __syncwarp();
        if (++s == PAIR_STAGES) { s = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    const uint32_t idesc = tc::make_idesc(256, bn);
    int s = 0, local = 0;
    unsigned phase = 0;
    for (int tile = pair; rank == 0 && tile < total_tiles && !failed; tile += num_pairs, ++local) {
      const int buf = local & 1;
      if (!tc::warp_wait(&acc_empty[buf], ((local >> 1) & 1) ^ 1)) { failed = true; break; }
      const uint32_t acc = tmem_base + (uint32_t)(buf * BN);
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!tc::warp_wait(&full_bar[s], phase)) { failed = true; break; }
        tc::fence_after();
        const uint32_t da = tiles_lo + (uint32_t)(s * (PAIR_STAGE_BYTES >> 4)), db = da + (PAIR_A_BYTES >> 4);
        if (tc::elect_one()) {
#pragma unroll
          for (int j = 0; j < BK / 16; ++j)
            tc::mma_pair_lo(acc, da + (uint32_t)(j * 2), db + (uint32_t)(j * 2), idesc, (kb | j) != 0 ? 1u : 0u);
          tc_commit_pair(&empty_bar[s]);
          if (kb + 1 == k_blocks) tc_commit_pair(&acc_full[buf]);
        }
        __syncwarp();
        if (++s == PAIR_STAGES) { s = 0; phase ^= 1; }
      }
    }
  } else {
    const int q = warp & 3, c_first = ((warp - 2) >> 2) * 32;
    uint32_t leader_acc_empty[2];
#pragma unroll
    for (int b = 0; b < 2; ++b)
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(leader_acc_empty[b]) : "r"(tc::smem_u32(&acc_empty[b])), "r"(0u));
    int local = 0;
    for (int tile = pair; tile < total_tiles && !failed; tile += num_pairs, ++local) {
      const int m0 = (tile % m_tiles) * 256 + (int)rank * 128, n0 = (tile / m_tiles) * OUT_COLS;
      const int buf = local & 1;
      if (!tc::warp_wait(&acc_full[buf], (local >> 1) & 1)) { failed = true; break; }
      tc::fence_after();
      const int row = m0 + q * 32 + lane;
      const uint32_t acc = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN);
      int pos = 0;
      long long slot = -1;
      if (EPI == EPI_ROPE && row < M) {
        pos = ra.positions[row];
        if (ra.write_cache && n0 + OUT_COLS > ra.H * ra.D) slot = rope_row_slot(ra, row, pos);
      }
#pragma unroll 1
      for (int c = c_first; c < OUT_COLS; c += 32 * (EPI_WARPS / 4)) {
        if (n0 + c >= N) break;
        uint32_t v[32];
        tc::load32(acc + (uint32_t)c, v);
        if (!GU) tc::wait_loads();
        if (EPI == EPI_ROPE) {
          if (row < M) rope_store_chunk(ra, v, row, n0 + c, M, N, slot, out);
          continue;
        }
        uint32_t packed[16];
        if (GU) {
          uint32_t u[32];
          tc::load32(acc + (uint32_t)(OUT_COLS + c), u);
          tc::wait_loads();
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float g0 = to_float(__float2bfloat16_rn(__uint_as_float(v[2 * i]))), g1 = to_float(__float2bfloat16_rn(__uint_as_float(v[2 * i + 1])));
            const float u0 = to_float(__float2bfloat16_rn(__uint_as_float(u[2 * i]))), u1 = to_float(__float2bfloat16_rn(__uint_as_float(u[2 * i + 1])));
            __nv_bfloat162 o = __floats2bfloat162_rn(gated_act(g0, u0, ra.act_limit, ra.act_alpha), gated_act(g1, u1, ra.act_limit, ra.act_alpha));
            packed[i] = *reinterpret_cast<uint32_t*>(&o);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            __nv_bfloat162 o = __floats2bfloat162_rn(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
            if (ra.store_act)          // on the rounded product, as the unfused path stores it first
              o = __floats2bfloat162_rn(plain_act(__low2float(o), ra.store_act), plain_act(__high2float(o), ra.store_act));
            packed[i] = *reinterpret_cast<uint32_t*>(&o);
          }
        }
        if (row < M) {
          bf16* dst = out + (size_t)row * N + n0 + c;
          if (n0 + c + 32 <= N) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              *reinterpret_cast<uint4*>(dst + i * 8) = make_uint4(packed[4 * i], packed[4 * i + 1], packed[4 * i + 2], packed[4 * i + 3]);
          } else {
            for (int i = 0; i < 32; ++i)
              if (n0 + c + i < N) dst[i] = reinterpret_cast<const bf16*>(packed)[i];
          }
        }
      }
      tc::fence_before();
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(leader_acc_empty[buf]) : "memory");
    }
  }
  if (failed) atomicExch(error, 1);
  tc::fence_before();
  __syncthreads();
  cluster_sync_all_threads();            // neither CTA leaves, or frees tensor memory, while the other may still use it
  if (warp == 1) {
    tc::fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// rows x cols bfloat16, row-major; box of box_rows x 64 columns, 128-byte swizzle, zero fill outside
int make_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows) {
  const tc::EncodeTiledFn encode = tc::encode_fn();
  if (!encode) return -300;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols * 2};
  const cuuint32_t box[2] = {(cuuint32_t)BK, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -301 - (int)r;
}

int g_pair_enabled = 1;
int g_forced_width = 0;      // tests: accumulator columns per tile instead of the tile plan's choice
int g_pair_capacity[3] = {0, 0, 0};

bool pair_mode(int M) { return g_pair_enabled && M > 128; }

template <int EPI>
int pair_capacity_of(int sms) {
  const size_t smem = (size_t)PAIR_STAGES * PAIR_STAGE_BYTES + 1024;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sms / 2 * 2, 1, 1);
  cfg.blockDim = dim3(THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  int clusters = 0;
  cudaFuncSetAttribute(gemm_tcgen05_pair_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const cudaError_t e = cudaOccupancyMaxActiveClusters(&clusters, gemm_tcgen05_pair_kernel<EPI>, &cfg);
  if (e != cudaSuccess || clusters < 1) { cudaGetLastError(); clusters = sms / 2; }
  return clusters > sms / 2 ? sms / 2 : clusters;
}

// CTA pairs of the two-CTA kernel that the device holds at a time (the persistent grid's size)
int pair_capacity(int epi, int sms) {
  int& cached = g_pair_capacity[epi];
  if (cached > 0) return cached;
  cached = epi == EPI_GATE_UP ? pair_capacity_of<EPI_GATE_UP>(sms) : epi == EPI_ROPE ? pair_capacity_of<EPI_ROPE>(sms)
                                                                                      : pair_capacity_of<EPI_STORE>(sms);
  return cached;
}

template <int EPI>
cudaError_t launch_single(dim3 grid, size_t smem, cudaStream_t stream, const CUtensorMap& map_a, const CUtensorMap& map_w, bf16* out,
                          int M, int N, int K, int bn, int* error, const RopeEpilogue& ra) {
  auto k = gemm_tcgen05_kernel<EPI>;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  return launch_pdl(k, grid, dim3(THREADS), smem, stream, map_a, map_w, out, M, N, K, bn, error, ra);
}

template <int EPI>
cudaError_t launch_pair(dim3 grid, size_t smem, cudaStream_t stream, const CUtensorMap& map_a, const CUtensorMap& map_w, bf16* out,
                        int M, int N, int K, int bn, int* error, const RopeEpilogue& ra) {
  return launch_pdl(gemm_tcgen05_pair_kernel<EPI>, grid, dim3(THREADS), smem, stream, map_a, map_w, out, M, N, K, bn, error, ra);
}

int supports(int M, int N, int K, int epi) {
  if (M < 1 || N < 8 || K < 8 || (K % 8) || (N % 8)) return 0;     // 16-byte row pitch for TMA, vector stores
  if (epi == EPI_GATE_UP && (N % 128)) return 0;                    // a tile's 128 gate rows must not reach into the up rows
  return 1;
}

// a [M,K], w [N,K] (or [2N,K] with gate/up), out [M,N]; all bfloat16, row-major, 16-byte aligned.
int run_product(const void* a, const void* w, void* out, int M, int N, int K, int epi, const RopeEpilogue& ra, int* error,
                cudaStream_t stream) {
  if (!supports(M, N, K, epi)) return SB_ERR_SHAPE;
  if (!aligned16(a) || !aligned16(w) || !aligned16(out) || !error) return SB_ERR_ALIGN;
  const bool gate_up = epi == EPI_GATE_UP;
  CUtensorMap map_a, map_w;
  int rc = make_map(&map_a, a, (uint64_t)M, (uint64_t)K, BM);
  if (rc) return rc;
  const int sms = sm_count();
  // Tile plan. A wave of tiles takes about (tile width + a fixed part worth 32 columns) whether its tiles are 128 rows
  // on one CTA or 256 rows on a CTA pair (each SM works on 128 rows either way), so the two kernels' costs compare
  // directly: whole waves needed x that time, for the best width of each. Ragged row counts decide it: 330 rows are
  // three 128-row tiles but two 256-row ones (512 rows of work).
  const bool forced = g_forced_width >= 32 && g_forced_width <= BN && (g_forced_width % 32) == 0 && !gate_up;
  const int widest = forced ? g_forced_width : BN, narrowest = forced ? g_forced_width : (gate_up ? BN : 128);
  long long cost_single = -1, cost_pair = -1, waves_pair = 0;
  int bn_single = BN, bn_pair = BN;
  const int pairs = pair_mode(M) ? pair_capacity(epi, sms) : 0;
  for (int cand = widest; cand >= narrowest; cand -= 32) {
    const int out_cols = gate_up ? cand / 2 : cand;
    const long long n_tiles = (N + out_cols - 1) / out_cols;
    const long long w1 = (((M + 127) / 128) * n_tiles + sms - 1) / sms;
    if (cost_single < 0 || w1 * (cand + 32) < cost_single) { cost_single = w1 * (cand + 32); bn_single = cand; }
    if (pairs > 0) {
      const long long w2 = (((M + 255) / 256) * n_tiles + pairs - 1) / pairs;
      if (cost_pair < 0 || w2 * (cand + 32) < cost_pair) { cost_pair = w2 * (cand + 32); bn_pair = cand; waves_pair = w2; }
    }
  }
  cudaError_t e;
  // At equal cost the pair kernel wins where a CTA has more than a tile of 32 blocks of k-values or more to do: starting and ending a
  // cluster costs it about 1 us more than the one-CTA kernel, and with shorter rows its tiles' ends come too often (one CTA | pair: q/k/v, 2,048
  // k-values, 600 rows 12.1 | 12.2 us, 1,700 rows 25.9 | 21.6, 2,048 rows 26.7 | 23.9; gate/up to 768, 2,048 rows 20.7 | 21.3; gate/up to 8,192 of 3,072, 1,700 rows
  // 135.6 | 126.4; of 1,024 k-values, gate/up to 4,096, 2,048 rows 33.1 | 35.2, to 8,192, 4,096 rows 109.9 | 116.4, of 1,536 to 2,048, 4,096 rows 42.3 | 43.3; one tile of
  // 4,096, gate/up to 768, 1,000 rows 44.4 | 45.7).
  const long long k_blocks = (K + BK - 1) / BK;
  const bool pair_wins = cost_pair < cost_single || (cost_pair == cost_single && k_blocks >= 32 && waves_pair * k_blocks >= (waves_pair > 1 ? 64 : 96));
  if (pairs > 0 && (pair_wins || g_pair_enabled == 2)) {
    const long long m_tiles = (M + 255) / 256;
    const int bn = bn_pair;
    rc = make_map(&map_w, w, (uint64_t)(gate_up ? 2 * N : N), (uint64_t)K, bn / 2);
    if (rc) return rc;
    const size_t smem = (size_t)PAIR_STAGES * PAIR_STAGE_BYTES + 1024;
    const int out_cols = gate_up ? bn / 2 : bn;
    const long long tiles = (long long)((N + out_cols - 1) / out_cols) * m_tiles;
    dim3 grid((unsigned)(2 * (tiles < pairs ? tiles : pairs)));
    e = epi == EPI_GATE_UP ? launch_pair<EPI_GATE_UP>(grid, smem, stream, map_a, map_w, (bf16*)out, M, N, K, bn, error, ra)
        : epi == EPI_ROPE  ? launch_pair<EPI_ROPE>(grid, smem, stream, map_a, map_w, (bf16*)out, M, N, K, bn, error, ra)
                           : launch_pair<EPI_STORE>(grid, smem, stream, map_a, map_w, (bf16*)out, M, N, K, bn, error, ra);
    SB_PDL_CHECK(e);
    return 0;
  }
  const long long m_tiles = (M + BM - 1) / BM;
  const int bn = bn_single;
  rc = make_map(&map_w, w, (uint64_t)(gate_up ? 2 * N : N), (uint64_t)K, gate_up ? bn / 2 : bn);
  if (rc) return rc;
  const size_t smem = (size_t)NSTAGE * STAGE_BYTES + 1024;
  const int out_cols = gate_up ? bn / 2 : bn;
  const long long tiles = (long long)((N + out_cols - 1) / out_cols) * m_tiles;
  dim3 grid((unsigned)(tiles < sms ? tiles : sms));
  e = epi == EPI_GATE_UP ? launch_single<EPI_GATE_UP>(grid, smem, stream, map_a, map_w, (bf16*)out, M, N, K, bn, error, ra)
      : epi == EPI_ROPE  ? launch_single<EPI_ROPE>(grid, smem, stream, map_a, map_w, (bf16*)out, M, N, K, bn, error, ra)
                         : launch_single<EPI_STORE>(grid, smem, stream, map_a, map_w, (bf16*)out, M, N, K, bn, error, ra);
  SB_PDL_CHECK(e);
  return 0;
}

}  // namespace

// 0 keeps every product on the one-CTA kernel, 1 (the default) lets products of more than 128 rows go to CTA pairs
// where the tile plan says they are no slower, 2 sends all of those to CTA pairs (tests).
SB_EXPORT void sb_gemm_tcgen05_use_pairs(int on) { g_pair_enabled = on; }
// 0: the tile plan chooses; a multiple of 32 up to 256: every product without gate/up uses tiles of that many columns
SB_EXPORT void sb_gemm_tcgen05_force_width(int bn) { g_forced_width = bn; }
SB_EXPORT int sb_gemm_tcgen05_pair_capacity(int gate_up) { return pair_capacity(gate_up ? EPI_GATE_UP : EPI_STORE, sm_count()); }

// 1 if sb_gemm_tcgen05 takes these sizes (else the caller uses the library product).
SB_EXPORT int sb_gemm_tcgen05_supports(int M, int N, int K, int gate_up) { return supports(M, N, K, gate_up ? EPI_GATE_UP : EPI_STORE); }

// The gate/up product with the clamped activation in its epilogue (see RopeEpilogue): w [2N, K], out [M, N].
SB_EXPORT int sb_gemm_tcgen05_gate_up_clamped(const void* a, const void* w, void* out, int M, int N, int K, float limit, float alpha,
                                              int* error, cudaStream_t stream) {
  if (!(limit > 0.f)) return SB_ERR_SHAPE;
  RopeEpilogue ra{};
  ra.act_limit = limit; ra.act_alpha = alpha;
  return run_product(a, w, out, M, N, K, EPI_GATE_UP, ra, error, stream);
}

// The gate/up product with gelu(g) * u (the tanh form of gelu) in its epilogue: w [2N, K], out [M, N].
SB_EXPORT int sb_gemm_tcgen05_gate_up_gelu(const void* a, const void* w, void* out, int M, int N, int K, int* error, cudaStream_t stream) {
  RopeEpilogue ra{};
  ra.act_limit = -1.f; ra.act_alpha = 1.f;
  return run_product(a, w, out, M, N, K, EPI_GATE_UP, ra, error, stream);
}

// error: device int set to 1 if a bounded wait inside the kernel ran out.
// out [M, N] = act(a w^T), the activation (see RopeEpilogue::store_act) on the product rounded to bfloat16.
SB_EXPORT int sb_gemm_tcgen05_act(const void* a, const void* w, void* out, int M, int N, int K, int act, int* error, cudaStream_t stream) {
  if (act < 1 || act > 4) return SB_ERR_SHAPE;
  RopeEpilogue ra = {};
  ra.store_act = act;
  return run_product(a, w, out, M, N, K, EPI_STORE, ra, error, stream);
}

SB_EXPORT int sb_gemm_tcgen05(const void* a, const void* w, void* out, int M, int N, int K, int gate_up, int* error,
                              cudaStream_t stream) {
  return run_product(a, w, out, M, N, K, gate_up ? EPI_GATE_UP : EPI_STORE, RopeEpilogue{}, error, stream);
}

// 1 if sb_gemm_tcgen05_qkv_rope takes these sizes: whole heads of a multiple of 32 elements, an even rotary width.
SB_EXPORT int sb_gemm_tcgen05_qkv_rope_supports(int M, int K, int rot, int H, int Hkv, int D) {
  if (H < 1 || Hkv < 1 || D < 32 || (D % 32) || rot < 0 || rot > D || (rot & 1)) return 0;
  return supports(M, (H + 2 * Hkv) * D, K, EPI_ROPE);
}

// The q/k/v product of an attention layer: out[M, (H + 2 Hkv) D] gets the rotated queries (its key and value columns
// are left untouched); rotated keys and the values go to kc / vc [pages, Hkv, ps, D] at each token's position, through
// its request's row of the block table. cos_sin [rot/2, M] pairs of floats from sb_rope_angles for the same positions. errors counts tokens without a page; wait_error as in sb_gemm_tcgen05.
SB_EXPORT int sb_gemm_tcgen05_qkv_rope(const void* a, const void* w, void* out, int M, int K, const int* positions,
                                       const int* token_row, const float* cos_sin, int rot, int H, int Hkv, int D, void* kc,
                                       void* vc, const int* block_table, int bt_width, int ps, int num_pages, int write_cache,
                                       int* errors, int* wait_error, cudaStream_t stream) {
  if (!sb_gemm_tcgen05_qkv_rope_supports(M, K, rot, H, Hkv, D) || ps <= 0) return SB_ERR_SHAPE;
  if (!positions || !errors || (rot > 0 && (!cos_sin || ((uintptr_t)cos_sin & 7)))) return SB_ERR_ALIGN;
  if (write_cache && (!kc || !vc || !block_table || !token_row || !aligned16(kc) || !aligned16(vc))) return SB_ERR_ALIGN;
  RopeEpilogue ra = {};
  ra.positions = positions;
  ra.token_row = token_row;
  ra.cos_sin = (const float2*)cos_sin;
  ra.block_table = block_table;
  ra.kc = (bf16*)kc;
  ra.vc = (bf16*)vc;
  ra.errors = errors;
  ra.rot = rot; ra.H = H; ra.Hkv = Hkv; ra.D = D;
  ra.bt_width = bt_width; ra.ps = ps; ra.num_pages = num_pages; ra.write_cache = write_cache;
  return run_product(a, w, out, M, (H + 2 * Hkv) * D, K, EPI_ROPE, ra, wait_error, stream);
}
