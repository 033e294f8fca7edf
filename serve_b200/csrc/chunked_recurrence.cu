// The linear recurrences of sequence_ops.cu for prompt portions, 32 tokens at a time, in plain 32-bit arithmetic.
//
// The walk's time is a chain: a token's read-out and update wait for the token before (0.09 us for a fixed decay to 0.34 us for
// the delta rule a token, with one warp a scheduler). A chunk of tokens 0 .. 31 with the state S before it obeys
//   U = V                                                     (the delta rule: (I + A) U = diag(b) V - diag(b) K' S)
//   O = Q' S + P U,        S' = diag(c) S + K''^T U
// with the decays folded in: K'_t = G_t k_t and Q'_t = G_t q_t (G_t the product of the decays up to t; WKV reads out before the
// update, so its Q' uses G_(t-1)), K''_s = (c / G_s) k_s, c the product of all, P_ts = q_t . (G_t / G_s) k_s for s <= t and A_ts = b_t k_t .
// (G_t / G_s) k_s for s < t. Ratios of products are never formed by division: G_t / G_s is the product of the decays s + 1 .. t, so a
// decay that underflows is simply zero.
//   chunk_prep_kernel: a block a (chunk, head), all chunks at once: P, Q', K'', c; for the delta rule W = (I + A)^-1 diag(b) K' and
//     V' = (I + A)^-1 diag(b) V by forward substitution, a thread a column, so that U = V' - W S.
//   chunk_walk_kernel: a block a (request, head, 16 columns of S), a chain of tokens / 32 steps: [W; Q'] S, then U, then O and the
//     next S. The tiles come through a two-stage cp.async ring; S lives in registers and, for the first product, in shared memory.
// Multiply-adds per token and head are 1.25 times the walk's, but 32 tokens wide, so the FMA units and not a latency are the bound.
// 2,048 tokens, 16 heads of 128 x 128 (B200): see the launcher. All sums are float in a fixed order.
#include "chunked_recurrence.h"

#include "common.cuh"

using namespace sb;

namespace {

constexpr int CH = 32;                 // tokens of a chunk
constexpr int VC = 16;                 // columns of S a block of the walk takes
constexpr int THREADS = 256;
constexpr int TP = CH + 4;             // pitch of a [row][token] tile
enum { MODE_DECAY = 0, MODE_SSM = 1, MODE_DELTA = 2, MODE_WKV = 3, MODE_GLA = 4, MODE_RET = 5 };

// floats of one (chunk, head) in the work space: Q' and K'' (and W) [32][DKT], P [32][32], c [2][DKT]: the float nearest to the product
// of the decays and what that leaves (a fixed decay's c is off the same way in every chunk, which would add up)
__host__ __device__ constexpr int part_floats(int dkt, bool delta) { return (delta ? 3 : 2) * CH * dkt + CH * CH + 2 * dkt; }

struct Place { int row, t0, n, n_chunks; long long slot; };

// Where entry i's chunk c lies: false if there is none (the whole block). The chunks of the entries before it are counted by the block.
__device__ __forceinline__ bool find_chunk(const SbChunkedWalk& a, int i, int c, Place& p, int* red) {
  const int r = a.rows ? a.rows[i] : i;
  const int q0 = a.cu_q[r], n = a.cu_q[r + 1] - q0;
  if (n <= a.min_tokens || c * CH >= n) return false;
  int before = 0;
  for (int u = threadIdx.x; u < i; u += THREADS) {
    const int ru = a.rows ? a.rows[u] : u;
    const int nu = a.cu_q[ru + 1] - a.cu_q[ru];
    if (nu > a.min_tokens) before += (nu + CH - 1) / CH;
  }
  if (i > 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = before;
    __syncthreads();
    before = 0;
    for (int u = 0; u < THREADS / 32; ++u) before += red[u];
  }
  p.row = r;
  p.t0 = q0 + c * CH;
  p.n = min(CH, n - c * CH);
  p.n_chunks = (n + CH - 1) / CH;
  p.slot = before;
  return true;
}

template <int DKT>
constexpr int prep_floats(bool vec) { return (vec ? 3 : 2) * DKT * TP + 8 * CH * (CH + 1) + CH * TP + CH * (CH + 1) + 3 * CH; }

// grid (chunk, head, list entry). VEC: a decay per row of S; else one for all of it.
template <int DKT, bool VEC, int MODE>
__global__ void __launch_bounds__(THREADS) chunk_prep_kernel(const SbChunkedWalk a, float* __restrict__ u_rows) {
  constexpr bool DELTA = MODE == MODE_DELTA, WKV = MODE == MODE_WKV;
  extern __shared__ __align__(16) float sm[];
  __shared__ int red_i[8];
  float* kT = sm;                                  // [DKT][TP]
  float* qT = kT + DKT * TP;
  float* gT = qT + DKT * TP;                       // VEC only
  float* part = gT + (VEC ? DKT * TP : 0);         // [8 warps][CH][CH + 1]
  float* At = part + 8 * CH * (CH + 1);            // [CH][TP]
  float* Dm = At + CH * TP;                        // [CH][CH + 1]: product of the decays s + 1 .. t (scalar decays)
  float* g1 = Dm + CH * (CH + 1);                  // [CH] decays, factors, products up to t (scalar decays)
  float* fac = g1 + CH;
  float* gam = fac + CH;
  Place p;
  if (!find_chunk(a, blockIdx.z, blockIdx.x, p, red_i)) return;
  const int h = blockIdx.y, hq = h / (a.H / a.Hqk);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool live = lane < p.n;
  const size_t tok = (size_t)(p.t0 + lane);
  const float f = live ? a.sc[tok * a.H + h] : 0.f;              // beta, dt or the bonus sum of token ``lane``
  if (warp == 0) {
    float g = 1.f;
    if (!VEC && live) g = a.head_rate ? a.af[(tok * a.H + h) * a.dkp] : a.dec[tok * a.H + h];
    g1[lane] = g;
    fac[lane] = f;
  }
  // lane = token: the rows are read 16 bytes at a time and turned, [row of S][token]
#pragma unroll 4
  for (int c = warp * 4; c < DKT; c += 32) {
    float4 k = make_float4(0.f, 0.f, 0.f, 0.f), q = k, g = make_float4(1.f, 1.f, 1.f, 1.f);
    if (live && c < a.dkp) {
      k = *reinterpret_cast<const float4*>(a.kf + (tok * a.Hqk + hq) * a.dkp + c);
      q = *reinterpret_cast<const float4*>(a.qf + (tok * a.Hqk + hq) * a.dkp + c);
      if (VEC) g = *reinterpret_cast<const float4*>(a.af + (tok * a.H + h) * a.dkp + c);
    }
    if (MODE == MODE_SSM) { k.x *= f; k.y *= f; k.z *= f; k.w *= f; }          // S += (dt k) v^T
    kT[c * TP + lane] = k.x; kT[(c + 1) * TP + lane] = k.y; kT[(c + 2) * TP + lane] = k.z; kT[(c + 3) * TP + lane] = k.w;
    qT[c * TP + lane] = q.x; qT[(c + 1) * TP + lane] = q.y; qT[(c + 2) * TP + lane] = q.z; qT[(c + 3) * TP + lane] = q.w;
    if (VEC) { gT[c * TP + lane] = g.x; gT[(c + 1) * TP + lane] = g.y; gT[(c + 2) * TP + lane] = g.z; gT[(c + 3) * TP + lane] = g.w; }
  }
  __syncthreads();
  if (!VEC && warp == 0) {
    double d = 1.0, up = 1.0;                     // (products of equal factors in float would all lean the same way)
    for (int t = 0; t < CH; ++t) {                // lane = s
      const double g = (double)g1[t];
      up *= g;
      if (t > lane) d *= g;
      Dm[t * (CH + 1) + lane] = (float)d;
      if (lane == 0) gam[t] = (float)up;
    }
  }
  // lane = t, a warp takes DKT / 8 rows of S: q_t . k_s and k_t . k_s with the decays between s and t
  {
    float aq[CH], ak[DELTA ? CH : 1];
#pragma unroll
    for (int s = 0; s < CH; ++s) aq[s] = 0.f;
#pragma unroll
    for (int s = 0; s < (DELTA ? CH : 1); ++s) ak[s] = 0.f;
#pragma unroll 1
    for (int c = warp * (DKT / 8); c < (warp + 1) * (DKT / 8); ++c) {
      const float kt = kT[c * TP + lane], qt = qT[c * TP + lane];
      float d = 1.f;
#pragma unroll
      for (int s4 = CH - 4; s4 >= 0; s4 -= 4) {
        const float4 k4 = *reinterpret_cast<const float4*>(kT + c * TP + s4);
        const float kk[4] = {k4.x, k4.y, k4.z, k4.w};
        float gg[4] = {1.f, 1.f, 1.f, 1.f};
        if (VEC) { const float4 g4 = *reinterpret_cast<const float4*>(gT + c * TP + s4); gg[0] = g4.x; gg[1] = g4.y; gg[2] = g4.z; gg[3] = g4.w; }
#pragma unroll
        for (int u = 3; u >= 0; --u) {
          const int s = s4 + u;                     // (sums of s beyond t are left out below)
          const float x = VEC ? kk[u] * d : kk[u];
          aq[s] = fmaf(qt, x, aq[s]);
          if (DELTA) ak[s] = fmaf(kt, x, ak[s]);
          if (VEC && (WKV ? s < lane : s <= lane)) d *= gg[u];
        }
      }
    }
    float* mine = part + (warp * CH + lane) * (CH + 1);
    if (DELTA) {
#pragma unroll
      for (int s = 0; s < CH; ++s) mine[s] = ak[s];
      __syncthreads();
#pragma unroll
      for (int e = tid; e < CH * CH; e += THREADS) {
        const int t = e >> 5, s = e & 31;
        float x = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) x += part[(w * CH + t) * (CH + 1) + s];
        if (!VEC) x *= Dm[t * (CH + 1) + s];
        At[s * TP + t] = s < t ? fac[t] * x : 0.f;
      }
      __syncthreads();
    }
#pragma unroll
    for (int s = 0; s < CH; ++s) mine[s] = aq[s];
  }
  __syncthreads();
  float* dst = a.work + ((p.slot + blockIdx.x) * a.H + h) * (long long)part_floats(DKT, DELTA);
  float* dst_p = dst + (DELTA ? 3 : 2) * CH * DKT;
  {
    const float skip = MODE != MODE_SSM ? 0.f : a.skip_dtype == SB_DTYPE_F32 ? ((const float*)a.skip)[h] : to_float(((const __nv_bfloat16*)a.skip)[h]);
#pragma unroll
    for (int e = tid; e < CH * CH; e += THREADS) {
      const int t = e >> 5, s = e & 31;
      float x = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) x += part[(w * CH + t) * (CH + 1) + s];
      if (!VEC) x *= Dm[t * (CH + 1) + s];
      if (s == t) x = WKV ? fac[t] : x + skip;
      dst_p[e] = s <= t ? x : 0.f;
    }
  }
  // a thread a row of S: Q' forwards with the running product of the decays, K'' backwards
  if (tid < DKT) {
    const float *q = qT + tid * TP, *g = VEC ? gT + tid * TP : g1;
    double up = 1.0;
#pragma unroll
    for (int t4 = 0; t4 < CH; t4 += 4) {
      const float4 q4 = *reinterpret_cast<const float4*>(q + t4), g4 = *reinterpret_cast<const float4*>(g + t4);
      const float qq[4] = {q4.x, q4.y, q4.z, q4.w}, gg[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (!WKV) up *= (double)gg[u];
        dst[(t4 + u) * DKT + tid] = qq[u] * (float)up;
        if (WKV) up *= (double)gg[u];
      }
    }
    dst_p[CH * CH + tid] = (float)up;
    dst_p[CH * CH + DKT + tid] = (float)(up - (double)(float)up);
  } else if (tid < 2 * DKT) {
    const int i = tid - DKT;
    const float *k = kT + i * TP, *g = VEC ? gT + i * TP : g1;
    double down = 1.0;
#pragma unroll
    for (int t4 = CH - 4; t4 >= 0; t4 -= 4) {
      const float4 k4 = *reinterpret_cast<const float4*>(k + t4), g4 = *reinterpret_cast<const float4*>(g + t4);
      const float kk[4] = {k4.x, k4.y, k4.z, k4.w}, gg[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
      for (int u = 3; u >= 0; --u) {
        dst[CH * DKT + (t4 + u) * DKT + i] = kk[u] * (float)down;
        down *= (double)gg[u];
      }
    }
  }
  // forward substitution, a thread a column of [diag(b) K' | diag(b) V]
  if constexpr (DELTA) for (int c = tid; c < DKT + a.dvp; c += THREADS) {
    const bool is_k = c < DKT;                      // (a whole warp)
    const int j = c - DKT;
    float x[CH];
    double up = 1.0;
#pragma unroll
    for (int t = 0; t < CH; ++t) {
      if (is_k) {
        if (VEC) up *= (double)gT[c * TP + t];
        x[t] = fac[t] * ((VEC ? (float)up : gam[t]) * kT[c * TP + t]);
      } else {
        x[t] = t < p.n ? fac[t] * a.vf[((size_t)(p.t0 + t) * a.H + h) * a.dvp + j] : 0.f;
      }
    }
#pragma unroll
    for (int s = 0; s < CH - 1; ++s) {              // x[s] is final: taken out of every later one (independent of one another)
#pragma unroll
      for (int t4 = (s + 1) & ~3; t4 < CH; t4 += 4) {
        const float4 a4 = *reinterpret_cast<const float4*>(At + s * TP + t4);
        if (t4 > s) x[t4] = fmaf(-a4.x, x[s], x[t4]);
        if (t4 + 1 > s) x[t4 + 1] = fmaf(-a4.y, x[s], x[t4 + 1]);
        if (t4 + 2 > s) x[t4 + 2] = fmaf(-a4.z, x[s], x[t4 + 2]);
        x[t4 + 3] = fmaf(-a4.w, x[s], x[t4 + 3]);
      }
    }
#pragma unroll
    for (int t = 0; t < CH; ++t) {
      if (is_k) dst[2 * CH * DKT + t * DKT + c] = x[t];
      else if (t < p.n) u_rows[((size_t)(p.t0 + t) * a.H + h) * a.dvp + j] = x[t];
    }
  }
}

__device__ __forceinline__ void cp16(float* smem, const float* g, bool valid) {
  const int n = valid ? 16 : 0;                    // 0: nothing is read, the 16 bytes are zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(g), "r"(n));
}

// The state in shared memory: rows 20 floats apart, the four 16-byte pieces of a row turned by the row, so that what a warp
// stores (rows 0, 4, 8 .. of two columns) and what it loads (a whole row at a time) both fall into different banks.
constexpr int SP = VC + 4;
__device__ __forceinline__ int s_at(int row, int col) { return row * SP + ((col >> 2) ^ ((row >> 3) & 3)) * 4 + (col & 3); }
template <int DKT, bool DELTA>
struct Walk {
  static constexpr int ROWS = DELTA ? 2 * CH : CH;        // rows of [W; Q']
  static constexpr int AP = DKT + 4;                      // their pitch: eight rows' 16-byte pieces fall into different banks
  static constexpr int SPLITS = 8 * 32 / ROWS;            // a group of ROWS threads takes DKT / SPLITS rows of S
  static constexpr int K_OFF = ROWS * AP, P_OFF = K_OFF + CH * DKT, U_OFF = P_OFF + CH * TP, C_OFF = U_OFF + CH * VC, STAGE = C_OFF + 2 * DKT;
  static constexpr int FLOATS = 2 * STAGE + DKT * SP + SPLITS * ROWS * VC + 2 * CH * VC;
};

// grid (ceil(dv / 16), head, list entry)
template <int DKT, bool DELTA>
__global__ void __launch_bounds__(THREADS) chunk_walk_kernel(const SbChunkedWalk a, const float* __restrict__ u_rows) {
  typedef Walk<DKT, DELTA> W;
  extern __shared__ __align__(16) float sm[];
  __shared__ int red_i[8];
  float* Ss = sm + 2 * W::STAGE;                          // [DKT][SP]
  float* part = Ss + DKT * SP;                            // [SPLITS][ROWS][VC]
  float* Us = part + W::SPLITS * W::ROWS * VC;            // [CH][VC]
  float* Rs = Us + CH * VC;                               // [CH][VC]: Q' S
  Place p;
  if (!find_chunk(a, blockIdx.z, 0, p, red_i)) return;
  const int h = blockIdx.y, j0 = blockIdx.x * VC;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n_all = a.cu_q[p.row + 1] - p.t0;
  const float* tiles = a.work + (p.slot * a.H + h) * (long long)part_floats(DKT, DELTA);
  const long long step = (long long)a.H * part_floats(DKT, DELTA);

  auto fetch = [&](int c) {
    float* st = sm + (c & 1) * W::STAGE;
    const float* src = tiles + c * step;
    for (int w = tid; w < W::ROWS * (DKT / 4); w += THREADS) {
      const int r = w / (DKT / 4), i = (w - r * (DKT / 4)) * 4;
      cp16(st + r * W::AP + i, src + (DELTA ? (r < CH ? 2 * CH * DKT + r * DKT : (r - CH) * DKT) : r * DKT) + i, true);
    }
    for (int w = tid; w < CH * DKT / 4; w += THREADS) cp16(st + W::K_OFF + w * 4, src + CH * DKT + w * 4, true);
    const float* sp = src + (DELTA ? 3 : 2) * CH * DKT;
    for (int w = tid; w < CH * CH / 4; w += THREADS) cp16(st + W::P_OFF + (w >> 3) * TP + (w & 7) * 4, sp + w * 4, true);
    if (tid < DKT / 2) cp16(st + W::C_OFF + tid * 4, sp + CH * CH + tid * 4, true);
    if (tid >= 128) {                                      // 32 rows of 64 bytes
      const int t = (tid - 128) >> 2, i = (tid & 3) * 4;
      const bool there = c * CH + t < n_all;
      cp16(st + W::U_OFF + t * VC + i, u_rows + ((size_t)(p.t0 + (there ? c * CH + t : 0)) * a.H + h) * a.dvp + j0 + i, there);
    }
    asm volatile("cp.async.commit_group;");
  };

  // this thread's part of S: four neighbouring rows i0 .. of one or two columns
  constexpr int COLS = DKT == 128 ? 2 : 1;
  const int i0 = ((lane & 7) + 8 * (warp & (DKT / 32 - 1))) * 4;
  const int c0 = ((lane >> 3) + 4 * (warp / (DKT / 32))) * COLS;
  float* S = a.state + (size_t)a.slots[p.row] * a.state_stride + (size_t)h * a.dk * a.dv;
  float s[4][COLS];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int c = 0; c < COLS; ++c) {
      s[u][c] = (i0 + u < a.dk && j0 + c0 + c < a.dv) ? S[(size_t)(i0 + u) * a.dv + j0 + c0 + c] : 0.f;
      Ss[s_at(i0 + u, c0 + c)] = s[u][c];
    }
  const int group = tid / W::ROWS, rg = lane & 7, cg = (lane >> 3) * 4, half = DELTA ? (warp & 1) * CH : 0;
  fetch(0);
  for (int c = 0; c < p.n_chunks; ++c) {
    asm volatile("cp.async.wait_group 0;");
    __syncthreads();                                       // the chunk's tiles and S are there; the other stage is free
    if (c + 1 < p.n_chunks) fetch(c + 1);
    const float* st = sm + (c & 1) * W::STAGE;
    const int n = min(CH, n_all - c * CH);
    {
      float acc[4][4] = {};
#pragma unroll 4
      for (int k = group * (DKT / W::SPLITS); k < (group + 1) * (DKT / W::SPLITS); k += 4) {
        float4 b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) b[u] = *reinterpret_cast<const float4*>(Ss + s_at(k + u, cg));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 x = *reinterpret_cast<const float4*>(st + (half + rg + 8 * j) * W::AP + k);
          acc[j][0] = fmaf(x.x, b[0].x, acc[j][0]); acc[j][1] = fmaf(x.x, b[0].y, acc[j][1]); acc[j][2] = fmaf(x.x, b[0].z, acc[j][2]); acc[j][3] = fmaf(x.x, b[0].w, acc[j][3]);
          acc[j][0] = fmaf(x.y, b[1].x, acc[j][0]); acc[j][1] = fmaf(x.y, b[1].y, acc[j][1]); acc[j][2] = fmaf(x.y, b[1].z, acc[j][2]); acc[j][3] = fmaf(x.y, b[1].w, acc[j][3]);
          acc[j][0] = fmaf(x.z, b[2].x, acc[j][0]); acc[j][1] = fmaf(x.z, b[2].y, acc[j][1]); acc[j][2] = fmaf(x.z, b[2].z, acc[j][2]); acc[j][3] = fmaf(x.z, b[2].w, acc[j][3]);
          acc[j][0] = fmaf(x.w, b[3].x, acc[j][0]); acc[j][1] = fmaf(x.w, b[3].y, acc[j][1]); acc[j][2] = fmaf(x.w, b[3].z, acc[j][2]); acc[j][3] = fmaf(x.w, b[3].w, acc[j][3]);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *reinterpret_cast<float4*>(part + ((size_t)group * W::ROWS + half + rg + 8 * j) * VC + cg) = make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]);
    }
    __syncthreads();
    if (tid < W::ROWS * 4) {
      const int r = tid >> 2, i = (tid & 3) * 4;
      float4 x = *reinterpret_cast<const float4*>(part + r * VC + i);
#pragma unroll
      for (int g = 1; g < W::SPLITS; ++g) {
        const float4 y = *reinterpret_cast<const float4*>(part + ((size_t)g * W::ROWS + r) * VC + i);
        x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w;
      }
      if (DELTA && r < CH) {
        const float4 v = *reinterpret_cast<const float4*>(st + W::U_OFF + r * VC + i);
        x = r < n ? make_float4(v.x - x.x, v.y - x.y, v.z - x.z, v.w - x.w) : make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<float4*>(Us + r * VC + i) = x;
      } else {
        *reinterpret_cast<float4*>(Rs + (DELTA ? r - CH : r) * VC + i) = x;
      }
    }
    __syncthreads();
    const float* U = DELTA ? Us : st + W::U_OFF;
    {
      // the outputs: two columns of one token a thread; only tokens up to its own enter, whatever the later ones hold
      const int t = tid >> 3, i = (tid & 7) * 2;
      float2 o = *reinterpret_cast<const float2*>(Rs + t * VC + i);
      const float* P = st + W::P_OFF + t * TP;
#pragma unroll
      for (int s4 = 0; s4 < CH; s4 += 4) {
        const float4 w = *reinterpret_cast<const float4*>(P + s4);
        const float ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float2 v = *reinterpret_cast<const float2*>(U + (s4 + u) * VC + i);
          if (s4 + u <= t) { o.x = fmaf(ww[u], v.x, o.x); o.y = fmaf(ww[u], v.y, o.y); }
        }
      }
      if (t < n) {
        float* dst = a.out + (size_t)(p.t0 + c * CH + t) * a.out_stride + (size_t)h * a.dv + j0 + i;
        if (j0 + i < a.dv) dst[0] = o.x;
        if (j0 + i + 1 < a.dv) dst[1] = o.y;
      }
    }
    {
      const float4 dc = *reinterpret_cast<const float4*>(st + W::C_OFF + i0), lo = *reinterpret_cast<const float4*>(st + W::C_OFF + DKT + i0);
#pragma unroll
      for (int v = 0; v < COLS; ++v) {
        s[0][v] = fmaf(dc.x, s[0][v], lo.x * s[0][v]); s[1][v] = fmaf(dc.y, s[1][v], lo.y * s[1][v]);
        s[2][v] = fmaf(dc.z, s[2][v], lo.z * s[2][v]); s[3][v] = fmaf(dc.w, s[3][v], lo.w * s[3][v]);
      }
#pragma unroll 8
      for (int t = 0; t < CH; ++t) {
        const float4 k = *reinterpret_cast<const float4*>(st + W::K_OFF + t * DKT + i0);
#pragma unroll
        for (int v = 0; v < COLS; ++v) {
          const float x = U[t * VC + c0 + v];
          s[0][v] = fmaf(k.x, x, s[0][v]); s[1][v] = fmaf(k.y, x, s[1][v]); s[2][v] = fmaf(k.z, x, s[2][v]); s[3][v] = fmaf(k.w, x, s[3][v]);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < COLS; ++v) Ss[s_at(i0 + u, c0 + v)] = s[u][v];
    }
  }
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < COLS; ++v)
      if (i0 + u < a.dk && j0 + c0 + v < a.dv) S[(size_t)(i0 + u) * a.dv + j0 + c0 + v] = s[u][v];
}

template <int DKT, bool VEC, int MODE>
int launch(const SbChunkedWalk& a, int chunks, cudaStream_t stream) {
  constexpr bool DELTA = MODE == MODE_DELTA;
  float* u_rows = DELTA ? a.work + (long long)chunks * a.H * part_floats(DKT, DELTA) : nullptr;
  const int most = (a.max_q + CH - 1) / CH;
  {
    auto k = chunk_prep_kernel<DKT, VEC, MODE>;
    const int smem = prep_floats<DKT>(VEC) * (int)sizeof(float);
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    k<<<dim3(most, a.H, a.n_list), THREADS, smem, stream>>>(a, u_rows);
    SB_LAUNCH_CHECK();
  }
  auto k = chunk_walk_kernel<DKT, DELTA>;
  const int smem = Walk<DKT, DELTA>::FLOATS * (int)sizeof(float);
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  k<<<dim3((a.dv + VC - 1) / VC, a.H, a.n_list), THREADS, smem, stream>>>(a, DELTA ? u_rows : a.vf);
  SB_LAUNCH_CHECK();
  return 0;
}

template <int DKT>
int launch_mode(const SbChunkedWalk& a, int chunks, cudaStream_t stream) {
  switch (a.mode) {
    case MODE_DECAY: case MODE_RET: return launch<DKT, false, MODE_DECAY>(a, chunks, stream);
    case MODE_SSM: return launch<DKT, false, MODE_SSM>(a, chunks, stream);
    case MODE_DELTA: return a.head_rate ? launch<DKT, false, MODE_DELTA>(a, chunks, stream) : launch<DKT, true, MODE_DELTA>(a, chunks, stream);
    case MODE_WKV: return launch<DKT, true, MODE_WKV>(a, chunks, stream);
    case MODE_GLA: return launch<DKT, true, MODE_GLA>(a, chunks, stream);
  }
  return SB_ERR_SHAPE;
}

}  // namespace

long long sb_chunked_walk_floats(int mode, int n_tokens, int chunks, int H, int dk, int dvp) {
  if (dk < 1 || dk > 128 || chunks < 1 || H < 1 || H > 65535) return -1;
  const bool delta = mode == MODE_DELTA;
  return (long long)chunks * H * part_floats(dk <= 64 ? 64 : 128, delta) + (delta ? (long long)n_tokens * H * dvp : 0);
}

int sb_chunked_walk(const SbChunkedWalk& a, int chunks, cudaStream_t stream) {
  if (a.n_list <= 0 || a.max_q <= a.min_tokens) return 0;
  if (sb_chunked_walk_floats(a.mode, a.n_tokens, chunks, a.H, a.dk, a.dvp) < 0 || a.dvp % VC || a.dkp > (a.dk <= 64 ? 64 : 128)) return SB_ERR_SHAPE;
  if (a.n_list > 65535) return SB_ERR_LIMIT;
  if (!aligned16(a.work)) return SB_ERR_ALIGN;
  return a.dk <= 64 ? launch_mode<64>(a, chunks, stream) : launch_mode<128>(a, chunks, stream);
}
