// A feed-forward of routed experts: every token goes through `top` of E small gated feed-forwards.
//
//   1. sb_moe_route: from float router logits [T, E], the `top` largest scores of every token (sigmoid or softmax
//      scores; lowest index on ties) and their weights, as float.
//   2. sb_moe_sort: the (token, choice) pairs grouped by expert: offsets[E + 1] and the pairs in that order, plus
//      the list of row tiles (expert, first row) the products run over. Which place a pair gets inside its
//      expert's group depends on timing, but nothing computed from it does: a pair's result is a function of its
//      own row alone.
//   3. sb_moe_gate_up: act[row] = f( w * (x W_gate^T), w * (x W_up^T) ) for the rows of every tile, x the pair's
//      token. The weight multiplies the expert's input; a product is linear, so it is applied to the float sums.
//   4. sb_moe_down: out[pair] = act[row] W_down^T, written at the pair's own place; with top == 1 that is the result,
//      otherwise sb_moe_combine adds a token's `top` rows in order.
// Experts without a gate (sb_moe_up: act[row] = f(x W_up^T), f = relu squared) and a choice that is read from a table
// over token ids instead of router logits (sb_moe_route_table) go through the same grouping and the same down product.
// Products accumulate in float over k in ascending order, whatever else is in the step. Here they are in plain arithmetic:
// float32, and bfloat16 sizes that are no multiple of 32; experts_tcgen05.cu has the others.
#include "common.cuh"

using namespace sb;

namespace {

__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + expf(-x)); }

constexpr int ROUTE_MAX_TOP = 16;

// The kernels of a layer may begin before the ones before them have ended (common.cuh), so what those write is read with plain loads behind
// pdl_wait(): no __ldg and no __restrict__, which say that nobody writes the data while the kernel runs.
//
// A warp per token: lane l holds the logits of experts l, l + 32, ... (at most ROUTE_PER_LANE of them); the best of
// what is left is found `top` times by a shuffle tree over (logit, index), lower index first on equal logits.
constexpr int ROUTE_PER_LANE = 32;      // so at most 1024 experts

__global__ void __launch_bounds__(128) moe_route_kernel(const float* logits, int E, int top, int score_kind, int renorm,
                                                        int n_tokens, int* idx, float* wts) {
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.x * 4 + (threadIdx.x >> 5);
  pdl_launch_dependents();
  pdl_wait();
  if (t >= n_tokens) return;
  const float* z = logits + (size_t)t * E;
  float mine[ROUTE_PER_LANE];
  float zmax = -INFINITY;
#pragma unroll
  for (int u = 0; u < ROUTE_PER_LANE; ++u) {
    const int e = lane + 32 * u;
    mine[u] = e < E ? z[e] : -INFINITY;
    zmax = fmaxf(zmax, mine[u]);
  }
  float denom = 1.f;
  if (score_kind == 1) {                        // softmax over all experts
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) zmax = fmaxf(zmax, __shfl_xor_sync(0xffffffffu, zmax, o));
    float part = 0.f;
#pragma unroll
    for (int u = 0; u < ROUTE_PER_LANE; ++u)
      if (lane + 32 * u < E) part += expf(mine[u] - zmax);
    denom = warp_sum(part);
  }
  float val = 0.f, total = 0.f;                 // lane s keeps the s-th choice
  int chosen = -1;
  for (int s = 0; s < top; ++s) {
    float m = -INFINITY;
    int arg = 0x7fffffff;
#pragma unroll
    for (int u = 0; u < ROUTE_PER_LANE; ++u) {
      const int e = lane + 32 * u;
      if (e < E && (mine[u] > m || (mine[u] == m && e < arg)) && mine[u] != -INFINITY) { m = mine[u]; arg = e; }
    }
    if (arg == 0x7fffffff) {                     // nothing left in this lane (or only minus infinity): offer its first free slot last
      m = -INFINITY;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float om = __shfl_xor_sync(0xffffffffu, m, o);
      const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
      if (om > m || (om == m && oa < arg)) { m = om; arg = oa; }
    }
    if (arg != 0x7fffffff && (arg & 31) == lane) {
#pragma unroll
      for (int u = 0; u < ROUTE_PER_LANE; ++u)
        if (u == (arg >> 5)) mine[u] = -INFINITY;    // taken
    }
    const float v = score_kind == 1 ? expf(m - zmax) / denom : sigmoid_f(m);
    total += v;
    if (lane == s) { val = v; chosen = arg == 0x7fffffff ? 0 : arg; }
  }
  if (lane < top) {
    idx[(size_t)t * top + lane] = chosen;
    wts[(size_t)t * top + lane] = renorm ? val / total : val;
  }
}

// As moe_route_kernel, for a router with a bias on the choice: the scores (softmax over the first E of a row's ``stride``
// logits, or sigmoid) choose through score + bias[e], lowest index first on ties, while the weights are the scores
// themselves, divided by (their sum + sum_eps) if asked. A lane holds PER_LANE outputs (E <= 32 * PER_LANE): few for the
// usual counts, so the loops over them are short. With n_groups > 1 the E outputs form as many equal groups of neighbours;
// a group is as good as its best output, and only outputs of the keep_groups best groups can be chosen. E counts every output the router scores; an index at or beyond
// the number of real experts means "the token itself" to the kernels after this one.
template <int PER_LANE>
__global__ void __launch_bounds__(128) moe_route_bias_kernel(const float* logits, int stride, int E, int top, int score_kind,
                                                             int renorm, float sum_eps, const float* bias, int n_tokens,
                                                             int* idx, float* wts, float weight_scale,
                                                             int n_groups, int keep_groups) {
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.x * 4 + (threadIdx.x >> 5);
  pdl_launch_dependents();
  pdl_wait();
  if (t >= n_tokens) return;
  const float* z = logits + (size_t)t * stride;
  float score[PER_LANE], pick[PER_LANE];
  float zmax = -INFINITY;
#pragma unroll
  for (int u = 0; u < PER_LANE; ++u) {
    const int e = lane + 32 * u;
    score[u] = e < E ? z[e] : -INFINITY;
    zmax = fmaxf(zmax, score[u]);
  }
  if (score_kind == 1) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) zmax = fmaxf(zmax, __shfl_xor_sync(0xffffffffu, zmax, o));
    float part = 0.f;
#pragma unroll
    for (int u = 0; u < PER_LANE; ++u)
      if (lane + 32 * u < E) { score[u] = expf(score[u] - zmax); part += score[u]; }
    const float denom = warp_sum(part);
#pragma unroll
    for (int u = 0; u < PER_LANE; ++u)
      if (lane + 32 * u < E) score[u] /= denom;
  } else {
#pragma unroll
    for (int u = 0; u < PER_LANE; ++u)
      if (lane + 32 * u < E) score[u] = sigmoid_f(score[u]);
  }
#pragma unroll
  for (int u = 0; u < PER_LANE; ++u) {
    const int e = lane + 32 * u;
    pick[u] = e < E ? score[u] + (bias ? bias[e] : 0.f) : -INFINITY;
  }
  if (keep_groups < n_groups) {
    // the best output of those in no kept group yet names the next group to keep
    const int gs = E / n_groups;
    unsigned kept = 0;                          // bit u: this lane's output lane + 32 u is in a kept group
    for (int s = 0; s < keep_groups; ++s) {
      float m = -INFINITY;
      int arg = 0x7fffffff;
#pragma unroll
      for (int u = 0; u < PER_LANE; ++u) {
        const int e = lane + 32 * u;
        if (e < E && !((kept >> u) & 1u) && (pick[u] > m || (pick[u] == m && e < arg))) { m = pick[u]; arg = e; }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float om = __shfl_xor_sync(0xffffffffu, m, o);
        const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
        if (om > m || (om == m && oa < arg)) { m = om; arg = oa; }
      }
#pragma unroll
      for (int u = 0; u < PER_LANE; ++u)
        if ((lane + 32 * u) / gs == arg / gs) kept |= 1u << u;
    }
#pragma unroll
    for (int u = 0; u < PER_LANE; ++u)
      if (!((kept >> u) & 1u)) pick[u] = -INFINITY;
  }
  float val = 0.f, total = 0.f;                 // lane s keeps the s-th choice
  int chosen = 0;
  for (int s = 0; s < top; ++s) {
    float m = -INFINITY, sc = 0.f;
    int arg = 0x7fffffff;
#pragma unroll
    for (int u = 0; u < PER_LANE; ++u) {
      const int e = lane + 32 * u;
      if (e < E && pick[u] != -INFINITY && (pick[u] > m || (pick[u] == m && e < arg))) { m = pick[u]; arg = e; sc = score[u]; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float om = __shfl_xor_sync(0xffffffffu, m, o);
      const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
      const float os = __shfl_xor_sync(0xffffffffu, sc, o);
      if (om > m || (om == m && oa < arg)) { m = om; arg = oa; sc = os; }
    }
    if (arg != 0x7fffffff && (arg & 31) == lane) {
#pragma unroll
      for (int u = 0; u < PER_LANE; ++u)
        if (u == (arg >> 5)) pick[u] = -INFINITY;    // taken
    }
    total += sc;
    if (lane == s) { val = sc; chosen = arg == 0x7fffffff ? 0 : arg; }
  }
  if (lane < top) {
    idx[(size_t)t * top + lane] = chosen;
    wts[(size_t)t * top + lane] = (renorm ? val / (total + sum_eps) : val) * weight_scale;
  }
}

constexpr int TM = 32;            // rows of a tile of the plain-arithmetic products (experts_tcgen05.cu has the others)

// One block. order[offsets[e] .. offsets[e+1]) = the pairs of expert e; tiles: (expert, first row) for every tile_rows rows
// of an expert's group, n_tiles[0] of them. A pair's place among its expert's comes from the atomic that counts it, kept in registers
// for up to SORT_KEEP pairs a thread (more: counted a second time); the experts' first places and tiles from one scan over the block.
// Bound by latency: 8,192 pairs of 64 experts 13.7 -> 8.9 us, 32 pairs 6.4 -> 2.7 (one thread had walked the experts).
constexpr int SORT_KEEP = 8;
__global__ void __launch_bounds__(1024) moe_sort_kernel(const int* idx, int n_pairs, int E, int tile_rows,
                                                        int* offsets, int* order, int* tiles,
                                                        int* n_tiles) {
  extern __shared__ int sh[];
  int* count = sh;            // [E]
  int* start = sh + E;        // [E]
  __shared__ int2 warp_sums[32];
  const int tid = threadIdx.x, n_threads = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const bool keeps = n_pairs <= SORT_KEEP * n_threads;
  pdl_launch_dependents();
  pdl_wait();
  int mine[SORT_KEEP], rank[SORT_KEEP];
#pragma unroll
  for (int u = 0; u < SORT_KEEP; ++u) mine[u] = tid + u * n_threads < n_pairs && keeps ? idx[tid + u * n_threads] : -1;
  for (int e = tid; e < E; e += n_threads) count[e] = 0;
  __syncthreads();
  if (keeps) {
#pragma unroll
    for (int u = 0; u < SORT_KEEP; ++u)
      if (mine[u] >= 0 && mine[u] < E) rank[u] = atomicAdd(&count[mine[u]], 1);
  } else {
    for (int p = tid; p < n_pairs; p += n_threads) {
      const int e = idx[p];
      if (e >= 0 && e < E) atomicAdd(&count[e], 1);
    }
  }
  __syncthreads();
  // a thread takes ``per`` neighbouring experts: (pairs, tiles) before them
  const int per = (E + n_threads - 1) / n_threads, e0 = min(E, tid * per), e1 = min(E, e0 + per);
  int pairs = 0, n = 0;
  for (int e = e0; e < e1; ++e) { pairs += count[e]; n += (count[e] + tile_rows - 1) / tile_rows; }
  int sp = pairs, sn = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int ap = __shfl_up_sync(0xffffffffu, sp, o), an = __shfl_up_sync(0xffffffffu, sn, o);
    if (lane >= o) { sp += ap; sn += an; }
  }
  if (lane == 31) warp_sums[warp] = make_int2(sp, sn);
  __syncthreads();
  int at = sp - pairs, nt = sn - n, all_pairs = 0, all_tiles = 0;
  for (int w = 0; w < n_threads / 32; ++w) {
    const int2 v = warp_sums[w];
    if (w < warp) { at += v.x; nt += v.y; }
    all_pairs += v.x;
    all_tiles += v.y;
  }
  for (int e = e0; e < e1; ++e) {
    const int c = count[e];
    start[e] = at;
    offsets[e] = at;
    for (int r0 = 0; r0 < c; r0 += tile_rows, ++nt) {
      tiles[2 * nt] = e;
      tiles[2 * nt + 1] = at + r0;
    }
    at += c;
    if (!keeps) count[e] = 0;
  }
  if (tid == 0) {
    offsets[E] = all_pairs;
    n_tiles[0] = all_tiles;
  }
  __syncthreads();
  if (keeps) {
#pragma unroll
    for (int u = 0; u < SORT_KEEP; ++u)
      if (mine[u] >= 0 && mine[u] < E) order[start[mine[u]] + rank[u]] = tid + u * n_threads;
  } else {
    for (int p = tid; p < n_pairs; p += n_threads) {
      const int e = idx[p];
      if (e >= 0 && e < E) order[start[e] + atomicAdd(&count[e], 1)] = p;
    }
  }
}

// The experts of a token from a table over token ids: idx[t, j] = table[token[t], j], every weight 1 / top. A token id
// below zero, -(s + 1), stands for the token last sampled for state slot s (as in the embedding kernel).
__global__ void __launch_bounds__(256) moe_route_table_kernel(const int* __restrict__ tokens, const int* __restrict__ last_token,
                                                              int n_slots, const int* __restrict__ table, int vocab, int E, int top,
                                                              int n_tokens, int* __restrict__ idx, float* __restrict__ wts,
                                                              int* __restrict__ errors) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= n_tokens * top) return;
  const int t = w / top, j = w - t * top;
  int tok = tokens[t];
  if (tok < 0 && last_token != nullptr && -tok - 1 < n_slots) tok = last_token[-tok - 1];
  int e = (tok >= 0 && tok < vocab) ? table[(size_t)tok * top + j] : -1;
  if (e < 0 || e >= E) {
    atomicAdd(errors, 1);        // a token outside the table or an entry outside the experts: counted, expert 0 stands in
    e = 0;
  }
  idx[w] = e;
  wts[w] = 1.0f / (float)top;
}

constexpr int TK = 32;
constexpr int GU_COLS = 32;       // gate columns of a tile (and as many up columns)
constexpr int DN_COLS = 64;
constexpr int MOE_THREADS = 256;

// grid (column tiles of ff, row tiles). x [T, K] with row stride; w_gu [E, 2 ff, K] (gate rows, then up rows).
// act kinds: 0 = silu(g) * u; 1 = the clamped form: g <- min(g, limit), u <- clamp(u, -limit, limit), g * sigmoid(alpha g) * (u + 1);
// 2 = no gate: w_gu is [E, ff, K] and the output is relu(x W^T)^2.
template <typename T>
__global__ void __launch_bounds__(MOE_THREADS) moe_gate_up_kernel(const T* __restrict__ x, int x_stride, const T* __restrict__ w_gu,
                                                                  const int* __restrict__ order, const int* __restrict__ offsets,
                                                                  const int* __restrict__ tiles, const int* __restrict__ n_tiles,
                                                                  const float* __restrict__ wts, int top, int K, int ff, int scale_input,
                                                                  int act_kind, float limit, float alpha, T* __restrict__ act) {
  if ((int)blockIdx.y >= n_tiles[0]) return;
  __shared__ float As[TK][TM + 1];
  __shared__ float Bg[TK][GU_COLS + 1];
  __shared__ float Bu[TK][GU_COLS + 1];
  __shared__ int tok[TM];
  __shared__ float rw[TM];
  const int e = tiles[2 * blockIdx.y], row0 = tiles[2 * blockIdx.y + 1];
  const int rows = min(TM, offsets[e + 1] - row0);
  const int n0 = blockIdx.x * GU_COLS;
  const int tid = threadIdx.x;
  if (tid < TM) {
    const int pair = tid < rows ? order[row0 + tid] : -1;
    tok[tid] = pair >= 0 ? pair / top : -1;
    rw[tid] = pair >= 0 ? wts[pair] : 0.f;
  }
  __syncthreads();
  const bool gated = act_kind != 2;
  const T* wg = w_gu + (size_t)e * (gated ? 2 : 1) * ff * K;
  const T* wu = wg + (size_t)ff * K;
  const int ty = tid >> 4, tx = tid & 15;               // rows 2 ty, 2 ty + 1; columns 2 tx, 2 tx + 1
  float ag[2][2] = {{0.f, 0.f}, {0.f, 0.f}}, au[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
  for (int k0 = 0; k0 < K; k0 += TK) {
    for (int w = tid; w < TM * TK; w += MOE_THREADS) {
      const int m = w / TK, kk = w - m * TK;
      const int tk = tok[m];
      As[kk][m] = (tk >= 0 && k0 + kk < K) ? to_float(x[(size_t)tk * x_stride + k0 + kk]) : 0.f;
    }
    for (int w = tid; w < GU_COLS * TK; w += MOE_THREADS) {
      const int nn = w / TK, kk = w - nn * TK;
      const bool ok = n0 + nn < ff && k0 + kk < K;
      Bg[kk][nn] = ok ? to_float(wg[(size_t)(n0 + nn) * K + k0 + kk]) : 0.f;
      Bu[kk][nn] = (ok && gated) ? to_float(wu[(size_t)(n0 + nn) * K + k0 + kk]) : 0.f;
    }
    __syncthreads();
#pragma unroll 8
    for (int kk = 0; kk < TK; ++kk) {
      const float a0 = As[kk][2 * ty], a1 = As[kk][2 * ty + 1];
      const float g0 = Bg[kk][2 * tx], g1 = Bg[kk][2 * tx + 1], u0 = Bu[kk][2 * tx], u1 = Bu[kk][2 * tx + 1];
      ag[0][0] += a0 * g0; ag[0][1] += a0 * g1; ag[1][0] += a1 * g0; ag[1][1] += a1 * g1;
      au[0][0] += a0 * u0; au[0][1] += a0 * u1; au[1][0] += a1 * u0; au[1][1] += a1 * u1;
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int m = 2 * ty + i;
    if (m >= rows) continue;
    const float sc = scale_input ? rw[m] : 1.f;
#pragma unroll
    for (int jx = 0; jx < 2; ++jx) {
      const int nn = n0 + 2 * tx + jx;
      if (nn >= ff) continue;
      float g = ag[i][jx] * sc, u = au[i][jx] * sc, yv;
      if (act_kind == 2) {
        g = fmaxf(g, 0.f);
        yv = g * g;
      } else if (act_kind == 1) {
        g = fminf(g, limit);
        u = fminf(fmaxf(u, -limit), limit);
        yv = g * sigmoid_f(alpha * g) * (u + 1.f);
      } else {
        yv = g * sigmoid_f(g) * u;
      }
      act[(size_t)(row0 + m) * ff + nn] = from_float<T>(yv);
    }
  }
}

// grid (column tiles of N, row tiles). act [rows, ff]; w_down [E, N, ff]; out [pairs, N] at the pair's own place, each
// row times its weight unless the weight already went into the input.
template <typename T, typename O>
__global__ void __launch_bounds__(MOE_THREADS) moe_down_kernel(const T* __restrict__ act, const T* __restrict__ w_down,
                                                               const int* __restrict__ order, const int* __restrict__ offsets,
                                                               const int* __restrict__ tiles, const int* __restrict__ n_tiles,
                                                               const float* __restrict__ wts, int ff, int N, int scale_output,
                                                               O* __restrict__ out) {
  if ((int)blockIdx.y >= n_tiles[0]) return;
  __shared__ float As[TK][TM + 1];
  __shared__ float Bs[TK][DN_COLS + 1];
  __shared__ int pair_of[TM];
  const int e = tiles[2 * blockIdx.y], row0 = tiles[2 * blockIdx.y + 1];
  const int rows = min(TM, offsets[e + 1] - row0);
  const int n0 = blockIdx.x * DN_COLS;
  const int tid = threadIdx.x;
  if (tid < TM) pair_of[tid] = tid < rows ? order[row0 + tid] : -1;
  __syncthreads();
  const T* w = w_down + (size_t)e * N * ff;
  const int ty = tid >> 4, tx = tid & 15;               // rows 2 ty, 2 ty + 1; columns tx, tx + 16, tx + 32, tx + 48
  float acc[2][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int jx = 0; jx < 4; ++jx) acc[i][jx] = 0.f;
  for (int k0 = 0; k0 < ff; k0 += TK) {
    for (int v = tid; v < TM * TK; v += MOE_THREADS) {
      const int m = v / TK, kk = v - m * TK;
      As[kk][m] = (m < rows && k0 + kk < ff) ? to_float(act[(size_t)(row0 + m) * ff + k0 + kk]) : 0.f;
    }
    for (int v = tid; v < DN_COLS * TK; v += MOE_THREADS) {
      const int nn = v / TK, kk = v - nn * TK;
      Bs[kk][nn] = (n0 + nn < N && k0 + kk < ff) ? to_float(w[(size_t)(n0 + nn) * ff + k0 + kk]) : 0.f;
    }
    __syncthreads();
#pragma unroll 8
    for (int kk = 0; kk < TK; ++kk) {
      const float a0 = As[kk][2 * ty], a1 = As[kk][2 * ty + 1];
#pragma unroll
      for (int jx = 0; jx < 4; ++jx) {
        const float b = Bs[kk][tx + 16 * jx];
        acc[0][jx] += a0 * b;
        acc[1][jx] += a1 * b;
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int m = 2 * ty + i;
    if (m >= rows) continue;
    const int pair = pair_of[m];
    const float sc = scale_output ? wts[pair] : 1.f;
#pragma unroll
    for (int jx = 0; jx < 4; ++jx) {
      const int nn = n0 + tx + 16 * jx;
      if (nn < N) out[(size_t)pair * N + nn] = from_float<O>(acc[i][jx] * sc);
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256) moe_combine_kernel(const float* __restrict__ parts, int top, int N, long long total,
                                                          T* __restrict__ out) {
  for (long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += (long long)gridDim.x * blockDim.x) {
    const long long t = w / N;
    const int c = (int)(w - t * N);
    float s = 0.f;
    for (int k = 0; k < top; ++k) s += parts[((size_t)t * top + k) * N + c];
    out[w] = from_float<T>(s);
  }
}


// The sum over a token's choices when some of them are not experts, plus what every token gets:
//   out[t] = sum_k ( idx[t, k] < E_real ? parts[t * top + k] : wts[t * top + k] * x[t] )  +  g_t * shared[t]
// with g_t = sigmoid(gate[t * gate_stride]) if a gate is given, else 1; shared may be null.
template <typename T> __device__ __forceinline__ float4 moe_load4(const T* p);
template <> __device__ __forceinline__ float4 moe_load4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 moe_load4<__nv_bfloat16>(const __nv_bfloat16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&u.x), b = *reinterpret_cast<const __nv_bfloat162*>(&u.y);
  return make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
}
template <typename T> __device__ __forceinline__ void moe_store4(T* p, float4 v);
template <> __device__ __forceinline__ void moe_store4<float>(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
template <> __device__ __forceinline__ void moe_store4<__nv_bfloat16>(__nv_bfloat16* p, float4 v) {
  __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  uint2 u;
  u.x = *reinterpret_cast<uint32_t*>(&a);
  u.y = *reinterpret_cast<uint32_t*>(&b);
  *reinterpret_cast<uint2*>(p) = u;
}

// The same four elements a thread, a block a part of one token's row: the rows of four choices are under way at a time, and which choices
// are experts is known before the loads. idx null: all are. 2,048 tokens, 4 choices, width 2,048 (84 MB): 19.5 -> 18.8 us;
// 8 tokens 3.7 -> 3.3.
template <typename T>
__global__ void __launch_bounds__(256) moe_combine_rows_kernel(const float* parts, const int* idx, const float* wts,
                                                               int E_real, const T* x, int x_stride, const T* shared,
                                                               const float* gate, int gate_stride, int top, int N, int blocks_a_row,
                                                               T* out) {
  const int t = blockIdx.x / blocks_a_row, c = ((blockIdx.x - t * blocks_a_row) * 256 + threadIdx.x) * 4;
  pdl_launch_dependents();
  pdl_wait();
  if (c >= N) return;
  float4 sv = make_float4(0.f, 0.f, 0.f, 0.f);
  float g = 1.f;
  if (shared) {
    sv = moe_load4<T>(shared + (size_t)t * N + c);
    if (gate) g = gate[(size_t)t * gate_stride];
  }
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int k0 = 0; k0 < top; k0 += 4) {
    float4 v[4];
    float f[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const size_t pair = (size_t)t * top + k0 + u;
      f[u] = 0.f;
      if (k0 + u < top) f[u] = !idx || idx[pair] < E_real ? 1.f : wts[pair];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const size_t pair = (size_t)t * top + k0 + u;
      if (k0 + u < top) v[u] = !idx || idx[pair] < E_real ? *reinterpret_cast<const float4*>(parts + pair * N + c) : moe_load4<T>(x + (size_t)t * x_stride + c);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (k0 + u < top) {
        s.x = fmaf(f[u], v[u].x, s.x); s.y = fmaf(f[u], v[u].y, s.y); s.z = fmaf(f[u], v[u].z, s.z); s.w = fmaf(f[u], v[u].w, s.w);
      }
  }
  if (shared) {
    if (gate) g = sigmoid_f(g);
    s.x = fmaf(g, sv.x, s.x); s.y = fmaf(g, sv.y, s.y); s.z = fmaf(g, sv.z, s.z); s.w = fmaf(g, sv.w, s.w);
  }
  moe_store4<T>(out + (size_t)t * N + c, s);
}

// VEC elements a thread (4: N and x_stride multiples of 4, every pointer 16-byte aligned; else 1).
template <typename T, int VEC>
__global__ void __launch_bounds__(256) moe_combine_more_kernel(const float* __restrict__ parts, const int* __restrict__ idx,
                                                               const float* __restrict__ wts, int E_real, const T* __restrict__ x,
                                                               int x_stride, const T* __restrict__ shared, const float* __restrict__ gate,
                                                               int gate_stride, int top, int N, long long total, T* __restrict__ out) {
  const int nv = N / VEC;
  for (long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(w / nv);
    const int c = (int)(w - (long long)t * nv) * VEC;
    float s[VEC];
#pragma unroll
    for (int v = 0; v < VEC; ++v) s[v] = 0.f;
    for (int k = 0; k < top; ++k) {
      const size_t pair = (size_t)t * top + k;
      if (idx[pair] < E_real) {
        if (VEC == 4) {
          const float4 p4 = *reinterpret_cast<const float4*>(parts + pair * N + c);
          s[0] += p4.x; s[1 % VEC] += p4.y; s[2 % VEC] += p4.z; s[3 % VEC] += p4.w;
        } else {
          s[0] += parts[pair * N + c];
        }
      } else {
        const float wt = wts[pair];
        if (VEC == 4) {
          const float4 x4 = moe_load4<T>(x + (size_t)t * x_stride + c);
          s[0] += wt * x4.x; s[1 % VEC] += wt * x4.y; s[2 % VEC] += wt * x4.z; s[3 % VEC] += wt * x4.w;
        } else {
          s[0] += wt * to_float(x[(size_t)t * x_stride + c]);
        }
      }
    }
    if (shared) {
      const float g = gate ? sigmoid_f(gate[(size_t)t * gate_stride]) : 1.f;
      if (VEC == 4) {
        const float4 h4 = moe_load4<T>(shared + (size_t)t * N + c);
        s[0] += g * h4.x; s[1 % VEC] += g * h4.y; s[2 % VEC] += g * h4.z; s[3 % VEC] += g * h4.w;
      } else {
        s[0] += g * to_float(shared[(size_t)t * N + c]);
      }
    }
    if (VEC == 4) moe_store4<T>(out + (size_t)t * N + c, make_float4(s[0], s[1 % VEC], s[2 % VEC], s[3 % VEC]));
    else out[(size_t)t * N + c] = from_float<T>(s[0]);
  }
}

// false: the rows are not made of whole, aligned pieces of four, or would leave more than a tenth of their blocks idle (a row of 1,100 numbers takes two
// blocks of 1,024: 4,096 tokens of 2 choices 14.7 us, 10.8 with threads dealt to the pieces of all rows; of 512 numbers 7.5 | 6.3, of 64 5.9 | 2.7; of
// 1,024 10.3 | 10.1, of 2,048 26.1 | 27.5, of 3,072 40.8 | 44.6)
template <typename T>
bool combine_rows(const float* parts, const int* idx, const float* wts, int E_real, const void* x, int x_stride, const void* shared, const float* gate,
                  int gate_stride, int top, int n_tokens, int N, void* out, cudaStream_t stream, cudaError_t& e) {
  const int per_row = (N / 4 + 255) / 256;
  e = cudaSuccess;
  if (N / 4 * 10 < per_row * 256 * 9) return false;
  if (N % 4 || x_stride % 4 || !aligned16(parts) || !aligned16(x) || !aligned16(out) || (shared && !aligned16(shared)) ||
      (long long)n_tokens * per_row > 2147483647LL)
    return false;
  e = launch_pdl(moe_combine_rows_kernel<T>, dim3(n_tokens * per_row), dim3(256), 0, stream, parts, idx, wts, E_real, (const T*)x, x_stride, (const T*)shared,
                 gate, gate_stride, top, N, per_row, (T*)out);
  return true;
}

}  // namespace

// Rows of a tile of the plain-arithmetic products (the grouping's tile_rows for them).
SB_EXPORT int sb_moe_tile_rows() { return TM; }

// logits float [T, E] -> idx int32 [T, top], wts float [T, top]. score_kind 0: sigmoid of the logit, 1: softmax over the
// experts; renorm: the chosen weights divided by their sum.
SB_EXPORT int sb_moe_route(const float* logits, int E, int top, int score_kind, int renorm, int n_tokens, int* idx, float* wts,
                           cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (E <= 0 || top <= 0 || top > E || top > ROUTE_MAX_TOP || E > 32 * ROUTE_PER_LANE) return SB_ERR_LIMIT;
  SB_PDL_CHECK(launch_pdl(moe_route_kernel, dim3((n_tokens + 3) / 4), dim3(128), 0, stream, logits, E, top, score_kind, renorm, n_tokens, idx, wts));
  return 0;
}

// idx int32 [n_pairs] -> offsets [E + 1], order [n_pairs], tiles [2 * (n_pairs / tile_rows + E)], n_tiles [1].
SB_EXPORT int sb_moe_sort(const int* idx, int n_pairs, int E, int tile_rows, int* offsets, int* order, int* tiles, int* n_tiles,
                          cudaStream_t stream) {
  if (n_pairs <= 0) return 0;
  if (E <= 0 || E > 4096 || tile_rows <= 0) return SB_ERR_LIMIT;
  // few pairs: few warps, whose barriers are short
  const int want = n_pairs / 4 > E ? n_pairs / 4 : E, threads = want >= 1024 ? 1024 : want <= 128 ? 128 : (want + 31) / 32 * 32;
  SB_PDL_CHECK(launch_pdl(moe_sort_kernel, dim3(1), dim3(threads), (size_t)(2 * E) * sizeof(int), stream, idx, n_pairs, E, tile_rows, offsets, order, tiles,
                          n_tiles));
  return 0;
}

SB_EXPORT int sb_moe_gate_up(const void* x, int x_stride, const void* w_gu, const int* order, const int* offsets, const int* tiles,
                             const int* n_tiles, const float* wts, int top, int n_pairs, int E, int K, int ff, int scale_input,
                             int act_kind, float limit, float alpha, void* act, int dtype, cudaStream_t stream) {
  if (n_pairs <= 0) return 0;
  const int max_tiles = n_pairs / TM + (E < n_pairs ? E : n_pairs);
  if (max_tiles > 65535) return SB_ERR_LIMIT;
  dim3 grid((ff + GU_COLS - 1) / GU_COLS, max_tiles);
  if (dtype == SB_DTYPE_F32)
    moe_gate_up_kernel<float><<<grid, MOE_THREADS, 0, stream>>>((const float*)x, x_stride, (const float*)w_gu, order, offsets, tiles,
                                                                 n_tiles, wts, top, K, ff, scale_input, act_kind, limit, alpha, (float*)act);
  else if (dtype == SB_DTYPE_BF16)
    moe_gate_up_kernel<__nv_bfloat16><<<grid, MOE_THREADS, 0, stream>>>((const __nv_bfloat16*)x, x_stride, (const __nv_bfloat16*)w_gu,
                                                                         order, offsets, tiles, n_tiles, wts, top, K, ff, scale_input,
                                                                         act_kind, limit, alpha, (__nv_bfloat16*)act);
  else
    return SB_ERR_DTYPE;
  SB_LAUNCH_CHECK();
  return 0;
}

// tokens int32 [T] -> idx int32 [T, top], wts float [T, top] from table int32 [vocab, top]; ``errors``: a counter that
// receives tokens outside the table and entries outside 0 .. E-1.
SB_EXPORT int sb_moe_route_table(const int* tokens, const int* last_token, int n_slots, const int* table, int vocab, int E, int top,
                                 int n_tokens, int* idx, float* wts, int* errors, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (E <= 0 || top <= 0 || top > E || vocab <= 0 || !errors) return SB_ERR_SHAPE;
  const int total = n_tokens * top;
  moe_route_table_kernel<<<(total + 255) / 256, 256, 0, stream>>>(tokens, last_token, n_slots, table, vocab, E, top, n_tokens, idx, wts,
                                                                  errors);
  SB_LAUNCH_CHECK();
  return 0;
}

// The experts' first product without a gate: act [n_pairs rows in grouped order, ff] = relu(x W_up^T)^2, w_up [E, ff, K].
SB_EXPORT int sb_moe_up(const void* x, int x_stride, const void* w_up, const int* order, const int* offsets, const int* tiles,
                        const int* n_tiles, const float* wts, int top, int n_pairs, int E, int K, int ff, void* act, int dtype,
                        cudaStream_t stream) {
  if (n_pairs <= 0) return 0;
  const int max_tiles = n_pairs / TM + (E < n_pairs ? E : n_pairs);
  if (max_tiles > 65535) return SB_ERR_LIMIT;
  dim3 grid((ff + GU_COLS - 1) / GU_COLS, max_tiles);
  if (dtype == SB_DTYPE_F32)
    moe_gate_up_kernel<float><<<grid, MOE_THREADS, 0, stream>>>((const float*)x, x_stride, (const float*)w_up, order, offsets, tiles,
                                                                 n_tiles, wts, top, K, ff, 0, 2, 0.f, 0.f, (float*)act);
  else if (dtype == SB_DTYPE_BF16)
    moe_gate_up_kernel<__nv_bfloat16><<<grid, MOE_THREADS, 0, stream>>>((const __nv_bfloat16*)x, x_stride, (const __nv_bfloat16*)w_up,
                                                                         order, offsets, tiles, n_tiles, wts, top, K, ff, 0, 2, 0.f, 0.f,
                                                                         (__nv_bfloat16*)act);
  else
    return SB_ERR_DTYPE;
  SB_LAUNCH_CHECK();
  return 0;
}

// out: [n_pairs, N] of dtype out_dtype (float for rows that are still to be added up).
SB_EXPORT int sb_moe_down(const void* act, const void* w_down, const int* order, const int* offsets, const int* tiles, const int* n_tiles,
                          const float* wts, int n_pairs, int E, int ff, int N, int scale_output, void* out, int dtype, int out_dtype,
                          cudaStream_t stream) {
  if (n_pairs <= 0) return 0;
  const int max_tiles = n_pairs / TM + (E < n_pairs ? E : n_pairs);
  if (max_tiles > 65535) return SB_ERR_LIMIT;
  dim3 grid((N + DN_COLS - 1) / DN_COLS, max_tiles);
  if (dtype == SB_DTYPE_F32 && out_dtype == SB_DTYPE_F32)
    moe_down_kernel<float, float><<<grid, MOE_THREADS, 0, stream>>>((const float*)act, (const float*)w_down, order, offsets, tiles, n_tiles,
                                                                     wts, ff, N, scale_output, (float*)out);
  else if (dtype == SB_DTYPE_BF16 && out_dtype == SB_DTYPE_BF16)
    moe_down_kernel<__nv_bfloat16, __nv_bfloat16><<<grid, MOE_THREADS, 0, stream>>>(
        (const __nv_bfloat16*)act, (const __nv_bfloat16*)w_down, order, offsets, tiles, n_tiles, wts, ff, N, scale_output,
        (__nv_bfloat16*)out);
  else if (dtype == SB_DTYPE_BF16 && out_dtype == SB_DTYPE_F32)
    moe_down_kernel<__nv_bfloat16, float><<<grid, MOE_THREADS, 0, stream>>>((const __nv_bfloat16*)act, (const __nv_bfloat16*)w_down, order,
                                                                             offsets, tiles, n_tiles, wts, ff, N, scale_output, (float*)out);
  else
    return SB_ERR_DTYPE;
  SB_LAUNCH_CHECK();
  return 0;
}

// parts float [T * top, N] -> out [T, N]: a token's rows added in the order of its choices.
SB_EXPORT int sb_moe_combine(const float* parts, int top, int n_tokens, int N, void* out, int dtype, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (dtype != SB_DTYPE_F32 && dtype != SB_DTYPE_BF16) return SB_ERR_DTYPE;
  const bool f32 = dtype == SB_DTYPE_F32;
  cudaError_t e;
  if (!(f32 ? combine_rows<float>(parts, nullptr, nullptr, 0, out, 4, nullptr, nullptr, 0, top, n_tokens, N, out, stream, e)
            : combine_rows<__nv_bfloat16>(parts, nullptr, nullptr, 0, out, 4, nullptr, nullptr, 0, top, n_tokens, N, out, stream, e))) {
    const long long total = (long long)n_tokens * N, want = (total + 255) / 256;
    const int blocks = (int)(want < sm_count() * 8 ? want : sm_count() * 8);
    if (f32) moe_combine_kernel<float><<<blocks, 256, 0, stream>>>(parts, top, N, total, (float*)out);
    else moe_combine_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>(parts, top, N, total, (__nv_bfloat16*)out);
  }
  if (e != cudaSuccess) return (int)e;
  SB_LAUNCH_CHECK();
  return 0;
}

// As sb_moe_route with more: the row stride of the logits (columns beyond E are not the router's), a float bias [E] or
// null that joins the scores for the choice only, sum_eps, added to the sum the chosen scores are divided by,
// weight_scale, a constant every weight is multiplied by, and n_groups equal groups of outputs of which only the keep_groups
// best are open to the choice (1, 1: all are).
SB_EXPORT int sb_moe_route_bias(const float* logits, int stride, int E, int top, int score_kind, int renorm, float sum_eps,
                                const float* bias, int n_tokens, int* idx, float* wts, float weight_scale, int n_groups, int keep_groups,
                                cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (E <= 0 || top <= 0 || top > E || top > ROUTE_MAX_TOP || E > 32 * ROUTE_PER_LANE) return SB_ERR_LIMIT;
  if (stride < E) return SB_ERR_SHAPE;
  if (n_groups <= 0 || E % n_groups || keep_groups <= 0 || keep_groups > n_groups || (long long)top > (long long)keep_groups * (E / n_groups)) return SB_ERR_SHAPE;
  auto k = E <= 64 ? moe_route_bias_kernel<2> : E <= 128 ? moe_route_bias_kernel<4> : E <= 256 ? moe_route_bias_kernel<8>
                                                                                               : moe_route_bias_kernel<ROUTE_PER_LANE>;
  SB_PDL_CHECK(launch_pdl(k, dim3((n_tokens + 3) / 4), dim3(128), 0, stream, logits, stride, E, top, score_kind, renorm, sum_eps, bias, n_tokens, idx, wts,
                          weight_scale, n_groups, keep_groups));
  return 0;
}

// out [T, N] = the sum of a token's rows of parts (float [T * top, N]) where idx names one of the E_real experts, and
// wts * x[t] where it names none (N must then be x's width); plus shared [T, N] (or null), times sigmoid(gate[t]) if a
// gate (float, rows gate_stride apart) is given.
SB_EXPORT int sb_moe_combine_more(const float* parts, const int* idx, const float* wts, int E_real, const void* x, int x_stride,
                                  const void* shared, const float* gate, int gate_stride, int top, int n_tokens, int N, void* out,
                                  int dtype, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (!parts || !idx || !wts || !x || top <= 0 || x_stride < N) return SB_ERR_SHAPE;
  if (dtype != SB_DTYPE_F32 && dtype != SB_DTYPE_BF16) return SB_ERR_DTYPE;
  const bool f32 = dtype == SB_DTYPE_F32;
  cudaError_t e;
  if (!(f32 ? combine_rows<float>(parts, idx, wts, E_real, x, x_stride, shared, gate, gate_stride, top, n_tokens, N, out, stream, e)
            : combine_rows<__nv_bfloat16>(parts, idx, wts, E_real, x, x_stride, shared, gate, gate_stride, top, n_tokens, N, out, stream, e))) {
    const bool vec = N % 4 == 0 && x_stride % 4 == 0 && aligned16(parts) && aligned16(x) && aligned16(out) && (!shared || aligned16(shared));
    const long long total = (long long)n_tokens * (vec ? N / 4 : N), want = (total + 255) / 256;
    const int blocks = (int)(want < sm_count() * 16 ? want : sm_count() * 16);
    if (f32) {
      auto k = vec ? moe_combine_more_kernel<float, 4> : moe_combine_more_kernel<float, 1>;
      k<<<blocks, 256, 0, stream>>>(parts, idx, wts, E_real, (const float*)x, x_stride, (const float*)shared, gate, gate_stride, top, N, total, (float*)out);
    } else {
      auto k = vec ? moe_combine_more_kernel<__nv_bfloat16, 4> : moe_combine_more_kernel<__nv_bfloat16, 1>;
      k<<<blocks, 256, 0, stream>>>(parts, idx, wts, E_real, (const __nv_bfloat16*)x, x_stride, (const __nv_bfloat16*)shared, gate, gate_stride, top, N, total,
                                    (__nv_bfloat16*)out);
    }
  }
  if (e != cudaSuccess) return (int)e;
  SB_LAUNCH_CHECK();
  return 0;
}

// ---- a whole layer in one call from the host -----------------------------------------------------------------------------------------
extern "C" int sb_moe_tensor_rows(int dtype, int K, int ff, int x_stride, int n_tokens);
extern "C" int sb_moe_gate_up_tensor(const void* x, int x_stride, int n_tokens, void* xg, const void* w, const int* order, const int* offsets,
                                     const int* tiles, const int* n_tiles, const float* wts, int top, int n_pairs, int E, int K, int ff, int gated,
                                     int scale_input, int act_kind, float limit, float alpha, void* act, int tile_rows, int* error, cudaStream_t stream);
extern "C" int sb_moe_down_tensor(const void* act, const void* w_down, const int* order, const int* offsets, const int* tiles, const int* n_tiles,
                                  const float* wts, int n_pairs, int E, int ff, int N, int scale_output, void* out, int out_dtype, int tile_rows,
                                  int* error, cudaStream_t stream);

namespace {

// Where the work space of a layer holds what, in bytes from its start (every piece 256-byte aligned).
struct LayerRoom {
  long long idx, order, offsets, tiles, n_tiles, wts, act, parts, grouped, bytes;
  int tile_rows;
  bool tensor, own_parts;
};

LayerRoom layer_room(int n_tokens, int top, int E, int K, int ff, int N, int x_stride, int dtype, int more) {
  LayerRoom r = {};
  const long long pairs = (long long)n_tokens * top, elem = dtype == SB_DTYPE_F32 ? 4 : 2;
  const int rows = sb_moe_tensor_rows(dtype, K, ff, x_stride, n_tokens);
  r.tensor = rows > 0;
  r.tile_rows = r.tensor ? rows : TM;
  r.own_parts = top > 1 || more;                    // (a single expert's output is the layer's)
  long long at = 0;
  auto take = [&](long long bytes) { const long long here = at; at += (bytes + 255) / 256 * 256; return here; };
  r.idx = take(pairs * 4);
  r.order = take(pairs * 4);
  r.offsets = take((long long)(E + 1) * 4);
  r.tiles = take(2 * (pairs / r.tile_rows + (E < pairs ? E : pairs)) * 4);
  r.n_tiles = take(4);
  r.wts = take(pairs * 4);
  r.act = take(pairs * ff * elem);
  // The pairs' tokens in grouped order are read by the first product and by nothing after it, so they lie where the second one leaves its
  // float sums, if those take as much room (2,048 tokens, 4 experts a token, width 2,048: 34 MB that a call does not take beside them).
  const long long sums = r.own_parts ? pairs * N * 4 : 0, grouped = r.tensor ? pairs * K * elem : 0;
  r.parts = r.own_parts ? take(sums) : -1;
  r.grouped = r.tensor ? (sums >= grouped ? r.parts : take(grouped)) : -1;
  r.bytes = at;
  return r;
}

}  // namespace

// Bytes of work space that sb_moe_layer needs.
SB_EXPORT long long sb_moe_layer_bytes(int n_tokens, int top, int E, int K, int ff, int N, int x_stride, int dtype, int more) {
  if (n_tokens <= 0 || top <= 0 || E <= 0 || K <= 0 || ff <= 0 || N <= 0) return 0;
  return layer_room(n_tokens, top, E, K, ff, N, x_stride, dtype, more).bytes;
}

// Choice, grouping, the experts' products and the sum over a token's choices: the entries above one after the other on ``stream``, with one call
// from the host in place of five (8 tokens, 64 experts: 24 us of host time less, the buffers included). ``more``: sb_moe_route_bias
// and sb_moe_combine_more (outputs, sum_eps, choice_bias, weight_scale, n_groups, keep_groups, shared and gate apply), else sb_moe_route and
// sb_moe_combine. Returns the number of kernels launched, or an error: a refusal (negative) or -1000 - a CUDA error.
SB_EXPORT int sb_moe_layer(const float* logits, int logit_stride, int outputs, int top, int score_kind, int renorm, float sum_eps,
                           const float* choice_bias, float weight_scale, int n_groups, int keep_groups, int more, const void* x, int x_stride,
                           int n_tokens, const void* w_gate_up, const void* w_down, int E, int K, int ff, int N, int scale_input, int act_kind,
                           float limit, float alpha, const void* shared, const float* gate, int gate_stride, void* work, void* out, int dtype,
                           int out_dtype, int* error, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (dtype != SB_DTYPE_F32 && dtype != SB_DTYPE_BF16) return SB_ERR_DTYPE;
  const LayerRoom r = layer_room(n_tokens, top, E, K, ff, N, x_stride, dtype, more);
  if (!work || ((uintptr_t)work & 255)) return SB_ERR_ALIGN;
  char* w = (char*)work;
  int *idx = (int*)(w + r.idx), *order = (int*)(w + r.order), *offsets = (int*)(w + r.offsets), *tiles = (int*)(w + r.tiles), *n_tiles = (int*)(w + r.n_tiles);
  float* wts = (float*)(w + r.wts);
  void *act = w + r.act, *parts = r.own_parts ? (void*)(w + r.parts) : out;
  const int pairs = n_tokens * top, parts_dtype = r.own_parts ? SB_DTYPE_F32 : out_dtype;
  int launched = 0;
  auto failed = [](int rc) { return rc > 0 ? -1000 - rc : rc; };
  int rc = more ? sb_moe_route_bias(logits, logit_stride, outputs, top, score_kind, renorm, sum_eps, choice_bias, n_tokens, idx, wts, weight_scale,
                                    n_groups, keep_groups, stream)
                : sb_moe_route(logits, E, top, score_kind, renorm, n_tokens, idx, wts, stream);
  if (rc) return failed(rc);
  if ((rc = sb_moe_sort(idx, pairs, E, r.tile_rows, offsets, order, tiles, n_tiles, stream))) return failed(rc);
  launched += 2;
  if (r.tensor) {
    rc = sb_moe_gate_up_tensor(x, x_stride, n_tokens, w + r.grouped, w_gate_up, order, offsets, tiles, n_tiles, wts, top, pairs, E, K, ff, 1, scale_input,
                               act_kind, limit, alpha, act, r.tile_rows, error, stream);
    if (rc) return failed(rc);
    rc = sb_moe_down_tensor(act, w_down, order, offsets, tiles, n_tiles, wts, pairs, E, ff, N, scale_input ? 0 : 1, parts, parts_dtype, r.tile_rows, error,
                            stream);
    launched += 3;
  } else {
    rc = sb_moe_gate_up(x, x_stride, w_gate_up, order, offsets, tiles, n_tiles, wts, top, pairs, E, K, ff, scale_input, act_kind, limit, alpha, act, dtype,
                        stream);
    if (rc) return failed(rc);
    rc = sb_moe_down(act, w_down, order, offsets, tiles, n_tiles, wts, pairs, E, ff, N, scale_input ? 0 : 1, parts, dtype, parts_dtype, stream);
    launched += 2;
  }
  if (rc) return failed(rc);
  if (more) {
    rc = sb_moe_combine_more((const float*)parts, idx, wts, E, x, x_stride, shared, gate, gate_stride, top, n_tokens, N, out, out_dtype, stream);
    ++launched;
  } else if (top > 1) {
    rc = sb_moe_combine((const float*)parts, top, n_tokens, N, out, out_dtype, stream);
    ++launched;
  }
  return rc ? failed(rc) : launched;
}
