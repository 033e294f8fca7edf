// Paged causal attention for prompt portions on the fifth-generation tensor cores (head_dim 64 or 128, and rows of 256 that are
// keys and values at once, bfloat16), over all keys or behind a window that may keep the sequence's first keys.
//
// Work is cut as in attention_mma.cu: per (request, kv head), with the G = H / Hkv query heads that share the kv
// head folded into the row dimension: row m stands for (token m / G, head hk*G + m % G). A CTA owns 128 such
// rows (128 / G tokens) and walks over the request's keys in tiles of 64:
//   warp 0     feeds shared memory with TMA: the query tile once (a 4-d box over the q/k/v buffer), then per tile the key and value
//              pages named by the block table (4-d boxes over the caches, 128-byte swizzle) through a ring of stages;
//   warp 1     issues tcgen05.mma: S = Q K^T (128 x 64) into a score buffer in tensor memory, and, once the probabilities of a tile are
//              in tensor memory too, O += P V (V read MN-major) into the output accumulator, which stays there for the whole walk;
//              tcgen05.commit signals the readers and frees stages and buffers;
//   warps 2..9 two threads a row, 32 keys of a tile each: they read their part of S (tcgen05.ld), scale, causal mask on the diagonal
//              tiles, exp2 against a reference maximum, and leave the probabilities as bfloat16 in tensor memory, the first operand
//              of the second product. The reference maximum only follows the running maximum when that has moved by more than 8 (a
//              factor 256, harmless in bfloat16 and float): one barrier with a vote a tile tells the two threads of a row whether it
//              does; then, and only then, they exchange their maxima and rescale the accumulator in tensor memory after the products
//              issued so far have finished. So in the steady state nobody waits for the second product. At the end each thread
//              divides its half of the output row by the row's sum and stores it.
// What bounds it: a step's latencies, not its work (head_dim 64, 2,048 tokens: of 1,860 cycles a tile takes, 390 wait for the scores, 300 load them
// and take the maximum, 80 are the pair's vote, 120 moved references, 780 the exponentials and their stores, of which the exp2 unit itself
// needs 512 for the rows of a CTA, 180 the wait for the stores and the arrival; tensor pipe active 19 % of the time). What
// that led to, 2,048 tokens, 32/8 heads of 64 | 16/4 of 128 behind a window of 1,024 | 16 heads over a row of 256: a thread a row and one thread of a divergent warp to issue 53.9 | 45.8 | 60.5 us;
// two threads a row and the probabilities in tensor memory 52.4 | 41.7 | 52.8; products issued from a warp that has come together, with
// 32-bit additions in place of descriptors made anew, 50.7 | 38.3 | 49.6; waits that cost one instruction when there is nothing to wait for,
// 48.4 | 36.0 | 49.8; copies issued like the products, a tile's page looked up a tile ahead, 47.2 | 35.2 | 48.8 (a loop of a few
// more branches there: 52.3 | 39.0 | 49.2); two CTAs an SM at head_dim 128 (TIGHT) 28.9. Packed
// arithmetic (fma2, add2, max3): a whole layer 77.3 -> 76.35 | 84.8 -> 84.3 | 106.45 -> 106.2. No difference: two sets of softmax warps for even and odd tiles, longer hardware waits, a single polling lane. Slower: tiles of 128
// keys (one buffer each of scores and probabilities: eight prompts of 256 26 us against 24; 55.7 over rows of 256).
// Two CTAs share an SM at head_dim 64 (96 KB of shared memory, 256 columns of tensor memory each).
// At head_dim 128 an operand row is two 128-byte swizzle atoms: queries, keys and values arrive as two TMA boxes of 64
// elements each, the first product walks over both atoms of Q and K, the second product covers the 128 output
// columns in one instruction (the descriptor's leading byte offset names the distance between the atoms of V).
// At head_dim 256 keys and values are the same rows (latent attention), so a tile is loaded once for both products; with its
// 256 output columns and two score buffers the kernel holds all of tensor memory.
// Behind a window only the tiles that a row of the CTA can see are walked.
// The recurrences are those of serve/kernels/attn_prefill.py:58-72 with exp2 and a folded log2(e)
// (attn_prefill.py:330-331); probabilities are rounded to bfloat16 before the second product (attn_prefill.py:71),
// or split into two (FINE, below).
// Every wait is bounded; a wait that runs out raises *error and the CTA still frees its tensor memory.
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "tcgen05_ops.cuh"

#if SB_HEAD_DIM == 64 || SB_HEAD_DIM == 128 || SB_HEAD_DIM == 256

using namespace sb;
typedef __nv_bfloat16 bf16;

namespace {

constexpr int D = SB_HEAD_DIM;
constexpr int KA = D / 64;            // 128-byte swizzle atoms (64 elements) per operand row
constexpr bool SHARED = D == 256;     // keys are the values (latent attention): one load a tile serves both products
constexpr int BM = 128;              // rows per CTA
constexpr int BN = 64;               // keys per tile
constexpr int BT_CACHE = D == 256 ? 512 : 1024;       // block-table entries kept in shared memory
constexpr int SOFTMAX_WARPS = 8;
constexpr int THREADS = 64 + 32 * SOFTMAX_WARPS;
constexpr float LOG2E = 1.4426950408889634f;
constexpr int Q_BYTES = BM * D * 2, KV_BYTES = BN * D * 2, P_COLS = BN / 2;      // (two probabilities a column)

// FINE: a probability is two bfloat16 numbers, its leading bits and what they leave, and the second product runs over both. With
// exponentials taken against a reference that lags behind the maximum, the heaviest key of a row is not 1 but any number up to 256, so
// its rounding (2^-9) is the result's; a kernel that follows the maximum, as attention_mma.cu does, has no error there. From 64 bits
// (2-norms; 700 tokens, window 200, head size 128; the output's own rounding is 1.61e-3 to 1.64e-3 of it), one part | mma.sync | two
// parts: scores of a deviation of 1 2.08e-3 | 2.00e-3 | 1.61e-3, of 2 2.10e-3 | 1.83e-3 | 1.64e-3, of 6 1.96e-3 | 1.68e-3 | 1.63e-3.
// Following the maximum instead would rescale the accumulator in nearly every tile.
// TIGHT: the form at head_dim 128 that lets two CTAs share an SM (96 KB, 256 columns): one score buffer, two stages, and keys and values
// with stages of their own, so that the next keys are on their way while the values are still read.
template <bool FINE, bool TIGHT>
struct Layout {
  static_assert(!TIGHT || D == 128, "a form of head_dim 128");
  static constexpr int CTAS_PER_SM = D == 64 || TIGHT ? 2 : 1;
  static constexpr bool SPLIT = TIGHT;                  // keys and values have stages of their own
  static constexpr int NK = TIGHT ? 2 : D == 256 ? 4 : 5;     // stages of keys, and as many of values (none where the keys are the values)
  static constexpr int NSB = TIGHT ? 1 : 2;             // score buffers
  static constexpr uint32_t TMEM_COLS = CTAS_PER_SM == 2 ? 256 : 512;
  static constexpr int P_BUF = (FINE ? 2 : 1) * P_COLS; // columns of tensor memory a buffer of probabilities takes
  static constexpr int NP = NSB * BN + D + 2 * P_BUF <= (int)TMEM_COLS ? 2 : 1;     // buffers of probabilities
  static_assert(NSB * BN + D + NP * P_BUF <= (int)TMEM_COLS, "tensor memory");
  // 96 KB at head_dim 64 and in the tight form at 128, else 192
  static constexpr int TILE_BYTES = Q_BYTES + (SHARED ? 1 : 2) * NK * KV_BYTES;
  // + barriers, what the threads of a row tell one another, table entries
  static constexpr int XCH_OFF = TILE_BYTES + 256, BT_OFF = XCH_OFF + 2 * BM * 4, SMEM_BYTES = BT_OFF + BT_CACHE * 4;
  static_assert(SMEM_BYTES <= 227 * 1024 / CTAS_PER_SM - 1024, "shared memory of an SM");
};

// A wait that runs out is noted in *gave_up; from then on no wait of the CTA lasts, every loop and barrier runs to its end, and what is
// computed is not valid (*error is raised).
__device__ __noinline__ void mbar_wait_long(uint32_t bar, unsigned parity, int* gave_up) {
  for (unsigned i = 0; i < tc::WAIT_LIMIT; ++i) {
    if (tc::mbar_try(bar, parity)) return;
    if ((i & 1023u) == 1023u && *reinterpret_cast<volatile int*>(gave_up)) return;
  }
  *reinterpret_cast<volatile int*>(gave_up) = 1;
}
__device__ __forceinline__ void mbar_wait(uint64_t* bar, unsigned parity, int* gave_up) {
  const uint32_t addr = tc::smem_u32(bar);
  if (!tc::mbar_try(addr, parity)) mbar_wait_long(addr, parity, gave_up);
}
// A product whose first operand lies in tensor memory: row i of it is lane i, two bfloat16 numbers to a column.
__device__ __forceinline__ void tc_mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 b;\n mov.b64 b, {%2, %5};\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %3, p;\n}\n"
      ::"r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(tc::DESC_HI) : "memory");
}
// Stores and the wait for them, as loads, are the warp's instructions: lanes that a branch before them has parted meet first, or (_met) have
// just met and taken no branch of their own since (meeting again for each of them cost a windowed prompt 1.2 %).
__device__ __forceinline__ void tc_store32(uint32_t taddr, const float* r) {
  __syncwarp();
  const uint32_t* u = reinterpret_cast<const uint32_t*>(r);
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(u[8]), "r"(u[9]),
        "r"(u[10]), "r"(u[11]), "r"(u[12]), "r"(u[13]), "r"(u[14]), "r"(u[15]), "r"(u[16]), "r"(u[17]), "r"(u[18]), "r"(u[19]),
        "r"(u[20]), "r"(u[21]), "r"(u[22]), "r"(u[23]), "r"(u[24]), "r"(u[25]), "r"(u[26]), "r"(u[27]), "r"(u[28]), "r"(u[29]),
        "r"(u[30]), "r"(u[31])
      : "memory");
}
__device__ __forceinline__ void tc_store16_met(uint32_t taddr, const uint32_t (&u)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(u[8]), "r"(u[9]),
        "r"(u[10]), "r"(u[11]), "r"(u[12]), "r"(u[13]), "r"(u[14]), "r"(u[15])
      : "memory");
}
__device__ __forceinline__ void tc_wait_st_met() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ bool any_lane(int yes) { return __any_sync(0xffffffffu, yes) != 0; }
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// Two floats at a time: one instruction each, rounded as the single ones are.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n .reg .b64 x, y, z, w;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n mov.b64 z, {%6, %7};\n fma.rn.f32x2 w, x, y, z;\n mov.b64 {%0, %1}, w;\n}\n"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n .reg .b64 x, y, w;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n add.rn.f32x2 w, x, y;\n mov.b64 {%0, %1}, w;\n}\n"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// Barriers of the 64 threads that share 32 rows (two warps, each of which comes as a whole); the second tells all of them whether any of
// them says yes.
__device__ __forceinline__ void pair_sync(int id) {
  __syncwarp();
  asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory");
}
__device__ __forceinline__ bool pair_any(int id, bool yes) {
  uint32_t any;
  __syncwarp();
  asm volatile("{\n .reg .pred p, q;\n setp.ne.b32 q, %2, 0;\n bar.red.or.pred p, %1, 64, q;\n selp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(any) : "r"(id), "r"(yes ? 1u : 0u) : "memory");
  return any != 0;
}

struct TcParams {
  const int* block_table; int bt_width;
  const int* cu_q; const int* kv_len;
  int H, Hkv, G, ps;
  float scale_log2;
  bf16* out;
  int* error;
  const int* rows;      // requests this launch covers (blockIdx.z indexes it); nullptr: all, in order
  int heads_in_x;       // grid (kv heads, row tiles, requests) rather than (row tiles, kv heads, requests)
  // A cap c on the scaled scores (s -> c tanh(s / c)): softcap_in = scale / c is what a raw product is multiplied by inside
  // the tanh, cap_over_scale = c / scale what the tanh is multiplied by, so that the capped value is again a raw product
  // that the code below scales; both 0 without a cap. sinks: one float per query head, or null: exp(sink) joins the
  // softmax's denominator once per row (no key, no value).
  float softcap_in, cap_over_scale;
  const float* sinks;
  int window, keep;     // window > 0: a query sees the last ``window`` keys up to its own and the sequence's first ``keep``
  int deep_group;       // requests of at most 16 rows with this many query heads a kv head are the deep shape's
};

// tanh on the special-function unit, as the exponentials (relative error about 2^-11)
__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <bool FINE, bool TIGHT>
__global__ void __launch_bounds__(THREADS, Layout<FINE, TIGHT>::CTAS_PER_SM) attention_tc_kernel(const __grid_constant__ CUtensorMap map_q,
                                                               const __grid_constant__ CUtensorMap map_k,
                                                               const __grid_constant__ CUtensorMap map_v, const TcParams p) {
  typedef Layout<FINE, TIGHT> W;
  constexpr int NP = W::NP, P_BUF = W::P_BUF, NK = W::NK, NSB = W::NSB, TILE_BYTES = W::TILE_BYTES, XCH_OFF = W::XCH_OFF, BT_OFF = W::BT_OFF;
  constexpr uint32_t TMEM_COLS = W::TMEM_COLS;
  constexpr bool SPLIT = W::SPLIT;
  constexpr uint32_t O_COL = NSB * BN, P_COL = NSB * BN + D;  // the scores, O, the probabilities
  // Blocks start in the order of blockIdx.x, then y: with the heads in x, the tiles that see the most keys start first
  // for all heads. The other way round the last heads' longest tiles would start when a third of the time is over
  // and end last: 2,048 tokens, 32/8 heads took 53 us so, against 32 key tiles x ~1.1 us for the longest tile itself.
  const int r = p.rows ? p.rows[blockIdx.z] : (int)blockIdx.z;
  const int hk = p.heads_in_x ? blockIdx.x : blockIdx.y, bx = p.heads_in_x ? blockIdx.y : blockIdx.x;
  const int q0 = p.cu_q[r], qn = p.cu_q[r + 1] - q0;
  const int G = p.G;
  const int M = qn * G;
  // (a block with nothing to do still waits for the kernel before this one: see attention_deep_kernel)
  if (qn * p.deep_group <= 16) { pdl_wait(); return; }                  // the deep shape takes this request
  const int tok_per_tile = BM / G;
  const int n_mtiles = (qn + tok_per_tile - 1) / tok_per_tile;
  if (bx >= n_mtiles) { pdl_wait(); return; }
  const int tile = n_mtiles - 1 - bx;                   // later rows see more keys: they go first
  const int tok0 = tile * tok_per_tile;
  const int L = p.kv_len[r];
  const int p0 = L - qn;                                // position of the request's first query
  const int tok_last = min(tok0 + tok_per_tile, qn) - 1;
  const int hi = p0 + tok_last + 1;                     // keys [0, hi) are seen by some row of the tile
  // The tiles of keys to walk: all of them, or, behind a window, the n_kept tiles of the kept first keys and then those from
  // the window of the first row on. Step j reads the keys from key_of(j) on.
  const int behind = p.window > 0 ? max(0, p0 + tok0 - p.window + 1) / BN : 0;
  const int n_kept = p.window > 0 ? min((p.keep + BN - 1) / BN, behind) : 0;
  const int skipped = behind - n_kept;
  const int n_tiles = (hi + BN - 1) / BN - skipped;
  auto key_of = [&](int j) { return (j < n_kept ? j : j + skipped) * BN; };

  // all shared memory is dynamic, so that the tiles start at the CTA's (1024-byte aligned) window base: the
  // 128-byte swizzle needs that alignment, and a padded request would not let two CTAs share an SM
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* base = smem;
  unsigned char* Qs = base;
  unsigned char* Ks = Qs + Q_BYTES;                     // NK stages
  unsigned char* Vs = SHARED ? Ks : Ks + NK * KV_BYTES; // NK stages
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + TILE_BYTES);
  uint64_t& q_full = bars[0];
  uint64_t* k_full = bars + 1;                          // NK: a stage's keys have landed
  uint64_t* k_empty = bars + 1 + NK;                    // NK: the products that read the stage have finished
  uint64_t* v_full = SPLIT ? bars + 1 + 2 * NK : k_full;      // the same for values
  uint64_t* v_empty = SPLIT ? bars + 1 + 3 * NK : k_empty;
  uint64_t* s_full = bars + 1 + 4 * NK;                 // NSB: a score buffer is complete
  uint64_t* s_empty = bars + 3 + 4 * NK;                // NSB: the softmax threads hold it in registers
  uint64_t* p_full = bars + 5 + 4 * NK;                 // NP: a buffer of probabilities is written
  uint64_t* p_empty = bars + 7 + 4 * NK;                // NP: the second product that read it has finished
  uint32_t& tmem_base_s = *reinterpret_cast<uint32_t*>(bars + 9 + 4 * NK);
  int* gave_up = reinterpret_cast<int*>(bars + 10 + 4 * NK);      // a wait of this CTA ran out
  float* xch = reinterpret_cast<float*>(base + XCH_OFF);      // [2][BM]
  int* bt_s = reinterpret_cast<int*>(base + BT_OFF);
  if ((tc::smem_u32(base) & 1023u) != 0) {                  // never seen; refuse rather than compute with a wrong swizzle
    if (threadIdx.x == 0) atomicExch(p.error, 1);
    pdl_wait();
    return;
  }

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    tc::mbar_init(&q_full, 1);
#pragma unroll
    for (int s = 0; s < (SPLIT ? 4 : 2) * NK; ++s) tc::mbar_init(&k_full[s], 1);
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&s_full[b], 1); tc::mbar_init(&s_empty[b], SOFTMAX_WARPS); tc::mbar_init(&p_full[b], SOFTMAX_WARPS); tc::mbar_init(&p_empty[b], 1);
    }
    *gave_up = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(&tmem_base_s)), "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  // set up; queries, this step's keys and values, and the right to overwrite out come with the end of the kernel before
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t tmem_base = tmem_base_s;

  if (warp == 0) {
    // the table entries of the tile's keys, fetched once by the whole warp instead of one dependent load per page
    const int* bt = p.block_table + (size_t)r * p.bt_width;
    const int n_blocks = min((hi + p.ps - 1) / p.ps, p.bt_width);
    if (n_blocks <= BT_CACHE) {
      for (int i = lane; i < n_blocks; i += 32) bt_s[i] = bt[i];
      __syncwarp();
      bt = bt_s;
    }
    // queries: box {64 elements, G heads, 1 kv head, tokens of the tile} -> rows (token, head)
    if (tc::elect_one()) {
      tc::mbar_expect_tx(&q_full, (unsigned)(tok_per_tile * G * D * 2));
#pragma unroll
      for (int a = 0; a < KA; ++a) tc::load_4d(Qs + (size_t)a * BM * 128, &map_q, &q_full, a * 64, 0, hk, q0 + tok0);
    }
    // The loop is on the critical path: the whole warp walks it (what it computes is equal in all lanes then), no divisions, a tile's
    // page is looked up while the tile before waits for its stage. Pages of a tile or more: a tile lies in one page, from its row ``at`` on.
    const bool one = p.ps >= BN;
    const int pages_per_tile = one ? 1 : BN / p.ps;
    int blk = one ? key_of(0) / p.ps : key_of(0) / BN * pages_per_tile, at = one ? key_of(0) - blk * p.ps : 0;
    int page = blk < p.bt_width ? bt[blk] : -1;          // the tile's first page
    int s = 0, j = 0;
    unsigned phase = 1;
    for (; j < n_tiles; ++j) {
      int n_pages = blk < p.bt_width ? 1 : 0;
      if (!one) {
        const int kt = key_of(j);
        for (int i = 1; i < pages_per_tile; ++i)
          if (kt + i * p.ps < hi && blk + i < p.bt_width) ++n_pages;
      }
      const unsigned bytes = (unsigned)(n_pages * (one ? BN : p.ps) * D * 2);
      // a tile of keys (or values) from its pages: atom a of a stage is 64 keys x 128 bytes, a page's keys at their rows of it
      auto load = [&](unsigned char* stage, const CUtensorMap* map, uint64_t* full) {
        if (n_pages > 0) {                               // (-1, a page the window has passed: outside the map, zeros)
#pragma unroll
          for (int a = 0; a < KA; ++a) tc::load_4d(stage + (size_t)a * BN * 128, map, full, a * 64, at, hk, page);
        }
        if (!one) {
          for (int i = 1; i < n_pages; ++i) {
            const int pg = bt[blk + i];
#pragma unroll
            for (int a = 0; a < KA; ++a) tc::load_4d(stage + (size_t)a * BN * 128 + (size_t)i * p.ps * 128, map, full, a * 64, 0, hk, pg);
          }
        }
      };
      mbar_wait(&k_empty[s], phase, gave_up);
      if (any_lane(*reinterpret_cast<volatile int*>(gave_up))) break;        // (no copy into a stage that may still be read)
      if (tc::elect_one()) {
        tc::mbar_expect_tx(&k_full[s], SPLIT || SHARED ? bytes : 2 * bytes);
        load(Ks + (size_t)s * KV_BYTES, &map_k, &k_full[s]);
        if (!SPLIT && !SHARED) load(Vs + (size_t)s * KV_BYTES, &map_v, &k_full[s]);
      }
      __syncwarp();
      if (SPLIT) {
        mbar_wait(&v_empty[s], phase, gave_up);
        if (any_lane(*reinterpret_cast<volatile int*>(gave_up))) { ++j; break; }
        if (tc::elect_one()) {
          tc::mbar_expect_tx(&v_full[s], bytes);
          load(Vs + (size_t)s * KV_BYTES, &map_v, &v_full[s]);
        }
        __syncwarp();
      }
      // the next tile's place
      at += BN;
      if (at >= p.ps || !one) { at = 0; blk += pages_per_tile; }
      if (j + 1 == n_kept && skipped > 0) {
        const int kt = key_of(j + 1);
        blk = one ? kt / p.ps : kt / BN * pages_per_tile;
        at = one ? kt - blk * p.ps : 0;
      }
      if (j + 1 < n_tiles && blk < p.bt_width) page = bt[blk];
      if (++s == NK) { s = 0; phase ^= 1; }
    }
    if (*reinterpret_cast<volatile int*>(gave_up)) {       // the copies under way land before the CTA leaves (with a limit again)
      for (int i = max(0, j - NK); i < j; ++i) {
        for (unsigned n = 0; n < tc::WAIT_LIMIT && !tc::mbar_try(&k_full[i % NK], (i / NK) & 1); ++n) {}
        for (unsigned n = 0; n < tc::WAIT_LIMIT && !tc::mbar_try(&v_full[i % NK], (i / NK) & 1); ++n) {}
      }
      for (unsigned n = 0; n < tc::WAIT_LIMIT && !tc::mbar_try(&q_full, 0); ++n) {}
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc_s = tc::make_idesc(BM, BN, false);
    constexpr uint32_t idesc_o = tc::make_idesc(BM, D, true);
    const uint32_t dq = tc::desc_lo(tc::smem_u32(Qs)), dk0 = tc::desc_lo(tc::smem_u32(Ks)), dv0 = tc::desc_lo(tc::smem_u32(Vs), BN * 128);
    int ks = 0, vs = 0;                                  // stages of the next scores and of the next values
    unsigned kphase = 0, vphase = 0;
    // the scores of tile t, as soon as its keys are there and its score buffer has been read
    auto scores = [&](int t) {
      mbar_wait(&k_full[ks], kphase, gave_up);
      mbar_wait(&s_empty[t % NSB], ((t / NSB) & 1) ^ 1, gave_up);
      __syncwarp();
      tc::fence_after();
      const uint32_t dk = dk0 + (uint32_t)(ks * (KV_BYTES >> 4)), acc = tmem_base + (uint32_t)((t % NSB) * BN);
      if (tc::elect_one()) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          // 16 k-values further: 32 bytes within an atom (4 steps), then the next atom of Q (128 rows) and K (64 rows)
          tc::mma_lo(acc, dq + (uint32_t)((kk >> 2) * (BM * 128 >> 4) + (kk & 3) * 2), dk + (uint32_t)((kk >> 2) * (BN * 128 >> 4) + (kk & 3) * 2), idesc_s,
                 kk != 0 ? 1u : 0u);
        }
        tc::commit(&s_full[t % NSB]);
        if (SPLIT) tc::commit(&k_empty[ks]);
      }
      __syncwarp();
      if (++ks == NK) { ks = 0; kphase ^= 1; }
    };
    mbar_wait(&q_full, 0, gave_up);
    scores(0);
    for (int j = 0; j < n_tiles; ++j) {
      if (j + 1 < n_tiles) scores(j + 1);
      mbar_wait(&p_full[j % NP], (j / NP) & 1, gave_up);
      if (SPLIT) mbar_wait(&v_full[vs], vphase, gave_up);
      __syncwarp();
      tc::fence_after();
      // O += P V: P from tensor memory (16 keys are 8 columns), FINE: both parts of it; V is MN-major, 16 keys = 2048 bytes further per step
      const uint32_t pa = tmem_base + P_COL + (uint32_t)((j % NP) * P_BUF), dv = dv0 + (uint32_t)(vs * (KV_BYTES >> 4));
      if (tc::elect_one()) {
#pragma unroll
        for (int kk = 0; kk < BN / 16; ++kk) {
          tc_mma_ts(tmem_base + O_COL, pa + (uint32_t)(kk * 8), dv + (uint32_t)(kk * (2048 >> 4)), idesc_o, (j | kk) != 0 ? 1u : 0u);
          if (FINE) tc_mma_ts(tmem_base + O_COL, pa + (uint32_t)(P_COLS + kk * 8), dv + (uint32_t)(kk * (2048 >> 4)), idesc_o, 1u);
        }
        tc::commit(&p_empty[j % NP]);                     // also: "the products up to tile j have finished"
        tc::commit(&v_empty[vs]);
      }
      __syncwarp();
      if (++vs == NK) { vs = 0; vphase ^= 1; }
    }
  } else {
    // Two warps share 32 rows: warps 2 .. 5 take the first 32 keys of every tile, warps 6 .. 9 the others, a thread a row. Both threads of a
    // row hold the same reference; a barrier of the pair tells them whether either has seen a score that moves it.
    const int q = warp & 3;                              // the 32 tensor-memory lanes this warp may touch
    const int half = (warp - 2) >> 2, pair = 1 + q;      // its half of a tile's keys; the pair's barrier
    const int row = q * 32 + lane;
    const int m = tok0 * G + row;
    const bool row_ok = row < tok_per_tile * G && m < M;
    const int tok = row_ok ? m / G : 0, head = row_ok ? hk * G + (m - tok * G) : 0;
    const int pos = row_ok ? p0 + tok : -1;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
    float *mine = xch + half * BM + row, *other = xch + (half ^ 1) * BM + row;
    float m_ref = -INFINITY;                             // what the exponentials are taken against (log2 domain)
    float l_run = 0.f;                                   // (of this thread's keys)
    const int first_pos = p0 + tok0;                     // smallest position of the tile's rows
    const int window_lo = p.window > 0 ? first_pos - p.window + 1 : 0;      // no row sees a key below it that is not kept
    for (int j = 0; j < n_tiles; ++j) {
      const int b = j % NSB, kt = key_of(j), k0 = kt + half * 32;
      mbar_wait(&s_full[b], (j / NSB) & 1, gave_up);
      // The buffer of probabilities must have been read by the product of NP tiles ago. With two buffers it has by now (these scores were
      // issued behind that product), and the wait only keeps count of the barrier's uses.
      if (NP == 2 && j >= NP) mbar_wait(&p_empty[j % NP], ((j - NP) / NP) & 1, gave_up);
      __syncwarp();
      float sv[32];
      float m_half;
      {
        tc::fence_after();
        // the tile reaches beyond what the first row may see, or behind the last row's window
        const bool masked = kt + BN - 1 > first_pos || (p.window > 0 && kt <= p0 + tok_last - p.window);
        tc::load32_met(lane_addr + (uint32_t)(b * BN + half * 32), sv);
        tc::wait_loads();
        tc::fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&s_empty[b]);         // the scores are in registers: the buffer may be reused
        if (p.cap_over_scale > 0.f) {                    // the cap comes before the mask: tanh(-inf) would be finite
#pragma unroll
          for (int i = 0; i < 32; ++i) sv[i] = p.cap_over_scale * tanh_fast(sv[i] * p.softcap_in);
        }
        if (masked) {
#pragma unroll
          for (int i = 0; i < 32; ++i) sv[i] = (k0 + i <= pos) ? sv[i] : -INFINITY;
          if (p.window > 0) {
            const int from = pos - p.window + 1;          // the row's first key, the kept ones aside
#pragma unroll
            for (int i = 0; i < 32; ++i) sv[i] = (k0 + i >= from || k0 + i < p.keep) ? sv[i] : -INFINITY;
          }
        }
        float mx[4] = {sv[0], sv[1], sv[2], sv[3]};
#pragma unroll
        for (int i = 4; i < 28; i += 8)
#pragma unroll
          for (int u = 0; u < 4; ++u) mx[u] = max3(mx[u], sv[i + u], sv[i + 4 + u]);
        m_half = max3(max3(mx[0], mx[1], sv[28]), max3(mx[2], mx[3], sv[29]), fmaxf(sv[30], sv[31])) * p.scale_log2;
      }
      // the reference follows the maximum only when that has run ahead by more than 8 (or there was none yet): false for
      // m_half = -inf, true for m_ref = -inf and m_half finite
      if (pair_any(pair, m_half > m_ref + 8.0f)) {
        // rare: some row's reference moves. Both threads of a row take the larger of their maxima.
        *mine = m_half;
        pair_sync(pair);
        const float m_tile = fmaxf(m_half, *other);
        const bool moves = m_tile > m_ref + 8.0f;
        if (__any_sync(0xffffffffu, moves && m_ref != -INFINITY)) {
          // rescale the accumulator in tensor memory, once the products issued so far (up to tile j-1) are done
          mbar_wait(&p_empty[(j - 1) % NP], ((j - 1) / NP) & 1, gave_up);
          __syncwarp();
          tc::fence_after();
          const float f = (moves && m_ref != -INFINITY) ? ex2(m_ref - m_tile) : 1.f;
#pragma unroll 1
          for (int c = 0; c < D / 64; ++c) {
            const uint32_t o_addr = lane_addr + O_COL + (uint32_t)(half * (D / 2) + c * 32);
            float ov[32];
            tc::load32(o_addr, ov);
            tc::wait_loads();
#pragma unroll
            for (int i = 0; i < 32; ++i) ov[i] *= f;
            tc_store32(o_addr, ov);
          }
          tc_wait_st_met();
          l_run *= f;
        }
        if (moves) m_ref = m_tile;                       // (with no reference yet, accumulator and sum are still zero)
      }
      const float use = (m_ref == -INFINITY) ? 0.f : m_ref;
      if (NP == 1 && j > 0) {
        mbar_wait(&p_empty[0], (j - 1) & 1, gave_up);
        __syncwarp();
        tc::fence_after();
      }
      // probabilities -> tensor memory (bfloat16, two neighbouring keys a column); ex2(-inf) = 0 takes care of masked entries
      float2 sum = make_float2(0.f, 0.f);
      const float2 scale2 = make_float2(p.scale_log2, p.scale_log2), use2 = make_float2(-use, -use);
      const uint32_t p_addr = lane_addr + P_COL + (uint32_t)((j % NP) * P_BUF + half * 16);
      uint32_t pk[16], rest[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float2 z = fma2(make_float2(sv[2 * i], sv[2 * i + 1]), scale2, use2);
        const float e0 = ex2(z.x), e1 = ex2(z.y);
        sum = add2(sum, make_float2(e0, e1));
        if (FINE) {                                      // both parts cut off, not rounded: 2^-16 of the number is left out
          const uint32_t u0 = __float_as_uint(e0), u1 = __float_as_uint(e1);
          pk[i] = __byte_perm(u0, u1, 0x7632);
          rest[i] = __byte_perm(__float_as_uint(e0 - __uint_as_float(u0 & 0xffff0000u)), __float_as_uint(e1 - __uint_as_float(u1 & 0xffff0000u)), 0x7632);
        } else {
          pk[i] = pack_bf16(e0, e1);
        }
      }
      tc_store16_met(p_addr, pk);
      if (FINE) tc_store16_met(p_addr + P_COLS, rest);
      l_run += sum.x + sum.y;
      // values that no row of the tile sees must not meet a zero probability as NaN (0 times infinity): the rows of this stage beyond
      // hi (never written, or another tile's leftovers) are cleared, and so are those behind every row's window
      if (kt + BN > hi || (kt < window_lo && kt + BN > p.keep)) {
        mbar_wait(&v_full[j % NK], (j / NK) & 1, gave_up);
        unsigned char* vt = Vs + (size_t)(j % NK) * KV_BYTES;
        auto clear = [&](int first, int last) {          // rows [first, last) of the stage
          const int n = last - first;
          for (int idx = (warp - 2) * 32 + lane; idx < n * 8 * KA; idx += 32 * SOFTMAX_WARPS) {
            const int a = idx / (n * 8), rest_ = idx - a * n * 8;
            *reinterpret_cast<uint4*>(vt + (size_t)a * BN * 128 + (size_t)(first + (rest_ >> 3)) * 128 + ((rest_ & 7) << 4)) =
                make_uint4(0u, 0u, 0u, 0u);
          }
        };
        clear(max(0, p.keep - kt), min(BN, window_lo - kt));
        clear(hi - kt, BN);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // these writes are read by the tensor core
        __syncwarp();
      }
      tc_wait_st_met();
      tc::fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&p_full[j % NP]);
    }
    // all products have finished when the last one has
    mbar_wait(&p_empty[(n_tiles - 1) % NP], ((n_tiles - 1) / NP) & 1, gave_up);
    __syncwarp();
    tc::fence_after();
    *mine = l_run;
    pair_sync(pair);
    l_run = half ? *other + l_run : l_run + *other;    // (the same sum in both threads of a row)
    {
      if (p.sinks != nullptr && row_ok) {
        // the sums were taken against m_ref; so is the sink (a sink far above every score makes the sum infinite and
        // the row zero, which is its limit)
        const float sk = p.sinks[head] * LOG2E;
        l_run += (m_ref == -INFINITY) ? 1.f : exp2f(sk - m_ref);
      }
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      constexpr int COLS = D / 2;                        // output columns a thread stores
      const int c0 = half * COLS;
      bf16* dst = p.out + (size_t)(q0 + tok) * p.H * D + (size_t)head * D + c0;
#pragma unroll 1
      for (int c = 0; c < COLS; c += 32) {
        float ov[32];
        tc::load32(lane_addr + O_COL + (uint32_t)(c0 + c), ov);
        tc::wait_loads();
        if (row_ok) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            *reinterpret_cast<uint4*>(dst + c + i * 8) =
                make_uint4(pack_bf16(ov[8 * i] * inv, ov[8 * i + 1] * inv), pack_bf16(ov[8 * i + 2] * inv, ov[8 * i + 3] * inv),
                           pack_bf16(ov[8 * i + 4] * inv, ov[8 * i + 5] * inv), pack_bf16(ov[8 * i + 6] * inv, ov[8 * i + 7] * inv));
        }
      }
    }
  }
  tc::fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *gave_up) atomicExch(p.error, 1);
  if (warp == 1) {
    tc::fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

int encode4(CUtensorMap* map, const void* basep, const cuuint64_t dims[4], const cuuint64_t strides[3], const cuuint32_t box[4]) {
  const tc::EncodeTiledFn encode = tc::encode_fn();
  if (!encode) return -300;
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUresult rc = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(basep), dims, strides, box, estr,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return rc == CUDA_SUCCESS ? 0 : -301 - (int)rc;
}

}  // namespace

// 1 if sb_attention_tc_opts takes this geometry (else the caller uses the mma.sync kernel). shared: keys and values are one tensor.
SB_EXPORT int sb_attention_tc_supports(int H, int Hkv, int ps, int shared, int q_stride) {
  if (H <= 0 || Hkv <= 0 || H % Hkv) return 0;
  const int G = H / Hkv;
  if (G > 128) return 0;                                // a tile holds whole tokens: 128 / G of them (rows beyond stay unused)
  if (ps < 8) return 0;
  if (ps <= BN ? (BN % ps) != 0 : ((ps % BN) != 0 || ps > 256)) return 0;   // pages tile a stage of keys (in whole swizzle atoms), or stages tile a page
  if (SHARED && !shared) return 0;
  if (q_stride % 8) return 0;
  return 1;
}

// The wide shape of sb_attention_mma (requests with more than 16 rows) on tcgen05; arguments as there.
// n_tokens: rows of qkv; num_pages: pages of kc / vc. rows (may be null): the n_rows requests to cover, so that a
// step of hundreds of decoding requests and a few prompt portions launches blocks for the portions only.
// softcap (0: none), sinks (float [H] or null), window (0: none), keep and deep_group: see TcParams.
SB_EXPORT int sb_attention_tc_opts(const void* qkv, int q_stride, int n_tokens, const void* kc, const void* vc, const int* block_table,
                                   int bt_width, const int* cu_q, const int* kv_len, int H, int Hkv, int ps, int num_pages, float scale,
                                   void* out, int n_rows, int max_q, const int* rows, int* error, float softcap, const float* sinks,
                                   int window, int keep, int deep_group, cudaStream_t stream) {
  if (n_rows <= 0 || max_q <= 0) return 0;
  if (!sb_attention_tc_supports(H, Hkv, ps, kc == vc, q_stride) || window < 0 || keep < 0 || deep_group <= 0) return SB_ERR_SHAPE;
  if (Hkv > 65535 || n_rows > 65535) return SB_ERR_LIMIT;
  if (!aligned16(qkv) || !aligned16(kc) || !aligned16(vc) || !aligned16(out) || !error) return SB_ERR_ALIGN;
  const int G = H / Hkv;
  CUtensorMap map_q, map_k, map_v;
  {
    const cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)G, (cuuint64_t)Hkv, (cuuint64_t)n_tokens};
    const cuuint64_t strides[3] = {(cuuint64_t)D * 2, (cuuint64_t)G * D * 2, (cuuint64_t)q_stride * 2};
    const cuuint32_t box[4] = {64, (cuuint32_t)G, 1, (cuuint32_t)(BM / G)};   // one swizzle atom of the head
    int rc = encode4(&map_q, qkv, dims, strides, box);
    if (rc) return rc;
  }
  {
    const cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)ps, (cuuint64_t)Hkv, (cuuint64_t)num_pages};
    const cuuint64_t strides[3] = {(cuuint64_t)D * 2, (cuuint64_t)ps * D * 2, (cuuint64_t)Hkv * ps * D * 2};
    const cuuint32_t box[4] = {64, (cuuint32_t)(ps < BN ? ps : BN), 1, 1};
    int rc = encode4(&map_k, kc, dims, strides, box);
    if (rc) return rc;
    rc = encode4(&map_v, vc, dims, strides, box);
    if (rc) return rc;
  }
  TcParams p;
  p.block_table = block_table; p.bt_width = bt_width; p.cu_q = cu_q; p.kv_len = kv_len;
  p.H = H; p.Hkv = Hkv; p.G = G; p.ps = ps; p.scale_log2 = scale * LOG2E; p.out = (bf16*)out; p.error = error; p.rows = rows;
  p.softcap_in = softcap > 0.f ? scale / softcap : 0.f; p.cap_over_scale = softcap > 0.f ? softcap / scale : 0.f; p.sinks = sinks;
  p.window = window; p.keep = window > 0 ? keep : 0; p.deep_group = deep_group;
  const int tok_per_tile = BM / G;
  const int m_tiles = (max_q + tok_per_tile - 1) / tok_per_tile;
  p.heads_in_x = m_tiles <= 65535 ? 1 : 0;
  const dim3 grid = p.heads_in_x ? dim3(Hkv, m_tiles, n_rows) : dim3(m_tiles, Hkv, n_rows);
  auto launch = [&](auto fine, auto tight) -> int {
    constexpr bool F = SHARED || decltype(fine)::value, T = D == 128 && decltype(tight)::value;
    auto kernel = attention_tc_kernel<F, T>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Layout<F, T>::SMEM_BYTES);
    SB_PDL_CHECK(launch_pdl(kernel, grid, dim3(THREADS), (size_t)Layout<F, T>::SMEM_BYTES, stream, map_q, map_k, map_v, p));
    return 0;
  };
  // in two parts where the mma.sync kernel would be the other choice (see the dispatch in kernels/cuda.py)
  const bool fine = SHARED || window > 0 || kc == vc;
  if (D == 128) {
    // Two CTAs an SM fill one another's gaps, but each has fewer buffers and takes longer by itself: they pay once an SM would walk a
    // second CTA after its first. 24/8 heads, whole causal prompts, one | two an SM: 600 tokens (120 CTAs) 22.1 | 25.3 us, 1,024 (200) 30.6 | 32.5,
    // 1,300 (248) 39.3 | 41.3, 1,500 (288) 42.5 | 41.9, 2,048 (392) 62.2 | 49.9, 4,096 (784) 168 | 125; 16/4 heads, window 1,024: 1,024 tokens (128)
    // 19.2 | 20.9, 1,600 (200) 24.6 | 26.6, 1,800 (228) 30.4 | 27.7, 2,048 (256) 35.5 | 28.9.
    if ((long long)Hkv * m_tiles * n_rows * 2 > 3LL * sm_count())
      return fine ? launch(std::true_type{}, std::true_type{}) : launch(std::false_type{}, std::true_type{});
  }
  return fine ? launch(std::true_type{}, std::false_type{}) : launch(std::false_type{}, std::false_type{});
}

#else

SB_EXPORT int sb_attention_tc_supports(int, int, int, int, int) { return 0; }

#endif
