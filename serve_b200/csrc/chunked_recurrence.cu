// The linear recurrences of sequence_ops.cu for prompt portions, 32 tokens at a time.
//
// The walk's time is a chain: a token's read-out and update wait for the token before (0.09 us for a fixed decay to 0.34 us for
// the delta rule a token, with one warp a scheduler). A chunk of tokens 0 .. 31 with the state S before it obeys
//   U = V                                                     (the delta rule: (I + A) U = diag(b) V - diag(b) K' S)
//   O = Q' S + P U,        S' = diag(c) S + K''^T U
// with the decays folded in: K'_t = G_t k_t and Q'_t = G_t q_t (G_t the product of the decays up to t; WKV reads out before the
// update, so its Q' uses G_(t-1)), K''_s = (c / G_s) k_s, c the product of all, P_ts = q_t . (G_t / G_s) k_s for s <= t and A_ts = b_t k_t .
// (G_t / G_s) k_s for s < t. Ratios of products are never formed by division: G_t / G_s is the product of the decays s + 1 .. t, so a
// decay that underflows is simply zero.
//   chunk_prep_*_kernel: a block a (chunk, head), all chunks at once: P, Q', K'', c; for the delta rule W = (I + A)^-1 diag(b) K' and
//     V' = (I + A)^-1 diag(b) V by forward substitution, a thread a column, so that U = V' - W S.
//   chunk_walk_kernel, chunk_wide_kernel: a block a (request, head, 16 columns of S, or 32 or 64), a chain of tokens / 32 steps: [W; Q'] S,
//     then U, then O and the next S. The matrices come through a ring of two stages; S lives in the accumulator layout in registers.
//
// All of this counts as 32-bit. The products run on the tensor cores (mma.sync m16n8k16) with every float x split into three bfloat16
// numbers h + m + l = x (8 bits each, nothing left), six of the nine products of the parts (the others are below 2^-24), smallest
// first, in an accumulator that starts from zero for every 16 terms and is then added in float, so that no sum is longer than 16
// terms before a rounded addition. Measured against 64 bits, read-outs and states are about 1e-7 off (2-norms), as the walk's are.
// What bounds them now: the walk's step of 1.9 us is 1,250 cycles of the tensor pipe a scheduler and as many of shared memory (each 16
// rows of [W; Q'] cross it once a block), one after the other, and two barriers; the preparation issues 29,000 instructions a block with two blocks
// an SM (three, in 80 registers, spill: 76 us). 2,048 tokens, 16 heads of 128 x 128, gated delta rule: 120 us for the walk, 67 for the
// preparation (as plain multiply-adds, bound by shared-memory reads, 209 and 105; token by token 704). A chunk's matrices come as one
// bulk copy: 22 cp.async a thread held the products' own reads up (208 us), 32 small bulk copies for the rows of V' cost their warp
// 1,700 cycles a step (163 us), so those rows come through registers, a chunk ahead.
// A number that is not finite has no parts to multiply (0 times infinity would reach back to earlier tokens): a chunk that meets one
// in its matrices, in S or in U takes plain multiply-adds instead, over the same operands.
#include "chunked_recurrence.h"

#include "bounded_wait.h"
#include "common.cuh"
#include "tcgen05_ops.cuh"
#include "walk_rule.h"

using namespace sb;
typedef __nv_bfloat16 bf16;

namespace {

constexpr int CH = 32;                 // tokens of a chunk
constexpr int VC = 16;                 // columns of S a block of the walk takes
constexpr int THREADS = 256;
constexpr int TP = CH + 4;             // pitch of a [row][token] tile of floats
constexpr int PP = CH + 8;             // pitch of the parts of P
enum { MODE_DECAY = 0, MODE_SSM = 1, MODE_DELTA = 2, MODE_WKV = 3, MODE_GLA = 4, MODE_RET = 5 };

// What the preparation leaves of a (chunk, head), as the walk's shared memory holds it: the three parts of [W; Q'] (or Q'), of K'' and
// of P, each row 16 bytes longer than it is; c as the float nearest to the product of the decays and what that leaves (a fixed
// decay's c is off the same way in every chunk, which would add up); four ints, the first not zero if something is not finite.
template <int DKT, bool DELTA>
struct Part {
  static constexpr int ROWS = DELTA ? 2 * CH : CH, AP = DKT + 8;
  static constexpr int K_OFF = 3 * ROWS * AP, P_OFF = K_OFF + 3 * CH * AP, C_OFF = P_OFF + 3 * CH * PP;      // bf16 numbers
  static constexpr int BYTES = C_OFF * 2 + 2 * DKT * 4 + 16;
};
__host__ __device__ constexpr long long part_bytes(int dkt, bool delta) {
  return dkt == 64 ? (delta ? Part<64, true>::BYTES : Part<64, false>::BYTES) : (delta ? Part<128, true>::BYTES : Part<128, false>::BYTES);
}

struct Place { int row, t0, n, n_chunks; long long slot; };

// Two numbers in three parts each (the first in the low halves), h + m + l = x exactly. A float beyond the largest bfloat16 leaves more to
// m; of one that is not finite m is not finite.
__device__ __forceinline__ float2 unpack(uint32_t u) { return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u)); }
__device__ __forceinline__ uint32_t packed(float x, float y) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ void split3(float x, float y, uint32_t (&p)[3]) {
  constexpr float MOST = 3.3895313892515355e38f;
  p[0] = packed(fminf(fmaxf(x, -MOST), MOST), fminf(fmaxf(y, -MOST), MOST));
  const float2 h = unpack(p[0]);
  x -= h.x;
  y -= h.y;
  p[1] = packed(x, y);
  const float2 m = unpack(p[1]);
  p[2] = packed(x - m.x, y - m.y);
}
__device__ __forceinline__ float whole(float h, float m, float l) { return fabsf(m) < INFINITY ? h + (m + l) : m; }
// the two numbers whose parts lie ``plane`` apart from p on
__device__ __forceinline__ float2 joined2(const bf16* p, int plane) {
  const float2 h = unpack(*reinterpret_cast<const uint32_t*>(p)), m = unpack(*reinterpret_cast<const uint32_t*>(p + plane)),
               l = unpack(*reinterpret_cast<const uint32_t*>(p + 2 * plane));
  return make_float2(whole(h.x, m.x, l.x), whole(h.y, m.y, l.y));
}
__device__ __forceinline__ float joined(const bf16* p, int plane) {
  return whole(__bfloat162float(p[0]), __bfloat162float(p[plane]), __bfloat162float(p[2 * plane]));
}
__device__ __forceinline__ bool finite(float x) { return fabsf(x) < INFINITY; }

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((unsigned)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((unsigned)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// acc[n] += the product of 32 terms, in two slices of 16 with sums of their own: 2 NT chains of six products side by side.
// b[..][..][2 n, 2 n + 1]: columns n.
template <int NT>
__device__ __forceinline__ void product32(float (&acc)[NT][4], const uint32_t (&a)[2][3][4], const uint32_t (&b)[2][3][2 * NT]) {
  float t[2][NT][4] = {};
  constexpr int LEFT[6] = {2, 0, 1, 1, 0, 0}, RIGHT[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
  for (int i = 0; i < 6; ++i)
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int n = 0; n < NT; ++n) mma(t[k][n], a[k][LEFT[i]], b[k][RIGHT[i]][2 * n], b[k][RIGHT[i]][2 * n + 1]);
#pragma unroll
  for (int k = 0; k < 2; ++k)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[n][e] += t[k][n][e];
}

// Where entry i's chunk c lies: false if there is none (the whole block). The chunks of the entries before it are counted by the block.
__device__ __forceinline__ bool find_chunk(const SbChunkedWalk& a, int i, int c, Place& p, int* red) {
  const int r = a.rows ? a.rows[i] : i;
  const int q0 = a.cu_q[r], n = a.cu_q[r + 1] - q0;
  if (n <= a.min_tokens || c * CH >= n) return false;
  int before = 0;
  for (int u = threadIdx.x; u < i; u += blockDim.x) {
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
    for (int u = 0; u < (int)blockDim.x / 32; ++u) before += red[u];
  }
  p.row = r;
  p.t0 = q0 + c * CH;
  p.n = min(CH, n - c * CH);
  p.n_chunks = (n + CH - 1) / CH;
  p.slot = before;
  return true;
}

template <int DKT>
constexpr int rows_smem() { return (3 * DKT * TP + 8 * CH * (CH + 1) + CH * TP + CH) * 4; }

// A decay per row of S: it sits inside the products of P and A, so those are multiply-adds here. grid (chunk, head, list entry).
template <int DKT, int MODE>
__global__ void __launch_bounds__(THREADS) chunk_prep_rows_kernel(const SbChunkedWalk a, float* __restrict__ u_rows) {
  constexpr bool DELTA = MODE == MODE_DELTA, WKV = MODE == MODE_WKV;
  typedef Part<DKT, DELTA> L;
  extern __shared__ __align__(16) float sm[];
  __shared__ int red_i[8];
  float* kT = sm;                                  // [DKT][TP]
  float* qT = kT + DKT * TP;
  float* gT = qT + DKT * TP;
  float* part = gT + DKT * TP;                     // [8 warps][CH][CH + 1]
  float* At = part + 8 * CH * (CH + 1);            // [s][TP]: A_ts
  float* fac = At + CH * TP;                       // [CH] beta or the bonus sum
  Place p;
  if (!find_chunk(a, blockIdx.z, blockIdx.x, p, red_i)) return;
  const int h = blockIdx.y, hq = h / (a.H / a.Hqk);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool live = lane < p.n;
  const size_t tok = (size_t)(p.t0 + lane);
  if (warp == 0) fac[lane] = live ? a.sc[tok * a.H + h] : 0.f;
  // lane = token: the rows are read 16 bytes at a time and turned, [row of S][token]
#pragma unroll 4
  for (int c = warp * 4; c < DKT; c += 32) {
    float4 k = make_float4(0.f, 0.f, 0.f, 0.f), q = k, g = make_float4(1.f, 1.f, 1.f, 1.f);
    if (live && c < a.dkp) {
      k = *reinterpret_cast<const float4*>(a.kf + (tok * a.Hqk + hq) * a.dkp + c);
      q = *reinterpret_cast<const float4*>(a.qf + (tok * a.Hqk + hq) * a.dkp + c);
      g = *reinterpret_cast<const float4*>(a.af + (tok * a.H + h) * a.dkp + c);
    }
    kT[c * TP + lane] = k.x; kT[(c + 1) * TP + lane] = k.y; kT[(c + 2) * TP + lane] = k.z; kT[(c + 3) * TP + lane] = k.w;
    qT[c * TP + lane] = q.x; qT[(c + 1) * TP + lane] = q.y; qT[(c + 2) * TP + lane] = q.z; qT[(c + 3) * TP + lane] = q.w;
    gT[c * TP + lane] = g.x; gT[(c + 1) * TP + lane] = g.y; gT[(c + 2) * TP + lane] = g.z; gT[(c + 3) * TP + lane] = g.w;
  }
  __syncthreads();
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
        const float4 g4 = *reinterpret_cast<const float4*>(gT + c * TP + s4);
        const float gg[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
        for (int u = 3; u >= 0; --u) {
          const int s = s4 + u;                     // (sums of s beyond t are left out below)
          const float x = kk[u] * d;
          aq[s] = fmaf(qt, x, aq[s]);
          if (DELTA) ak[s] = fmaf(kt, x, ak[s]);
          if (WKV ? s < lane : s <= lane) d *= gg[u];
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
        At[s * TP + t] = s < t ? fac[t] * x : 0.f;
      }
      __syncthreads();
    }
#pragma unroll
    for (int s = 0; s < CH; ++s) mine[s] = aq[s];
  }
  __syncthreads();
  unsigned char* image = reinterpret_cast<unsigned char*>(a.work) + ((p.slot + blockIdx.x) * a.H + h) * (long long)L::BYTES;
  bf16* img = reinterpret_cast<bf16*>(image);
  float* img_c = reinterpret_cast<float*>(img + L::C_OFF);
  bool bad = false;                                // something this thread leaves is not finite
  auto leave = [&](int off, int plane, float x) {
    uint32_t parts[3];
    split3(x, 0.f, parts);
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<unsigned short*>(img + off + i * plane) = (unsigned short)parts[i];
    bad |= !finite(x);
  };
#pragma unroll
  for (int e = tid; e < CH * CH; e += THREADS) {
    const int t = e >> 5, s = e & 31;
    float x = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) x += part[(w * CH + t) * (CH + 1) + s];
    if (WKV && s == t) x = fac[t];
    leave(L::P_OFF + t * PP + s, CH * PP, s <= t ? x : 0.f);
  }
  // a thread a row of S: Q' forwards with the running product of the decays, K'' backwards
  if (tid < DKT) {
    const float *q = qT + tid * TP, *g = gT + tid * TP;
    double up = 1.0;
#pragma unroll
    for (int t4 = 0; t4 < CH; t4 += 4) {
      const float4 q4 = *reinterpret_cast<const float4*>(q + t4), g4 = *reinterpret_cast<const float4*>(g + t4);
      const float qq[4] = {q4.x, q4.y, q4.z, q4.w}, gg[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (!WKV) up *= (double)gg[u];
        leave(((DELTA ? CH : 0) + t4 + u) * L::AP + tid, L::ROWS * L::AP, qq[u] * (float)up);
        if (WKV) up *= (double)gg[u];
      }
    }
    img_c[tid] = (float)up;
    img_c[DKT + tid] = finite((float)up) ? (float)(up - (double)(float)up) : 0.f;
    bad |= !finite((float)up);
  } else if (tid < 2 * DKT) {
    const int i = tid - DKT;
    const float *k = kT + i * TP, *g = gT + i * TP;
    double down = 1.0;
#pragma unroll
    for (int t4 = CH - 4; t4 >= 0; t4 -= 4) {
      const float4 k4 = *reinterpret_cast<const float4*>(k + t4), g4 = *reinterpret_cast<const float4*>(g + t4);
      const float kk[4] = {k4.x, k4.y, k4.z, k4.w}, gg[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
      for (int u = 3; u >= 0; --u) {
        leave(L::K_OFF + (t4 + u) * L::AP + i, CH * L::AP, kk[u] * (float)down);
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
        up *= (double)gT[c * TP + t];
        x[t] = fac[t] * ((float)up * kT[c * TP + t]);
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
      if (is_k) leave(t * L::AP + c, L::ROWS * L::AP, x[t]);
      else if (t < p.n) u_rows[((size_t)(p.t0 + t) * a.H + h) * a.dvp + j] = x[t];
    }
  }
  const int any = __syncthreads_or(bad);
  if (tid == 0) reinterpret_cast<int*>(image)[L::BYTES / 4 - 4] = any;
}

template <int DKT>
constexpr int head_smem() { return 6 * CH * (DKT + 8) * 2 + (CH * TP + CH * (CH + 1) + 4 * CH + 2) * 4; }

// One decay for all of S. grid (chunk, head, list entry). P and A are products of q and k as they are, the decays between the
// two tokens a factor of each element.
template <int DKT, int MODE>
__global__ void __launch_bounds__(THREADS, 2) chunk_prep_head_kernel(const SbChunkedWalk a, float* __restrict__ u_rows) {
  constexpr bool DELTA = MODE == MODE_DELTA;
  typedef Part<DKT, DELTA> L;
  constexpr int AP = L::AP, PL = CH * AP;          // pitch and distance of the parts of q and k
  extern __shared__ __align__(16) unsigned char raw[];
  __shared__ int red_i[8];
  bf16 *qp = reinterpret_cast<bf16*>(raw), *kp = qp + 3 * PL;      // [3][CH][AP]
  float* At = reinterpret_cast<float*>(kp + 3 * PL);               // [s][TP]: A_ts
  float* Dm = At + CH * TP;                        // [CH][CH + 1]: product of the decays s + 1 .. t
  float* g1 = Dm + CH * (CH + 1);                  // [CH] decays, factors, products up to t and from t + 1 on
  float *fac = g1 + CH, *gup = fac + CH, *gdn = gup + CH;
  float* c_all = gdn + CH;                         // [2] c and what the float leaves of it (not over g1: other lanes may still read it)
  Place p;
  if (!find_chunk(a, blockIdx.z, blockIdx.x, p, red_i)) return;
  const int h = blockIdx.y, hq = h / (a.H / a.Hqk);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long c_row = (long long)p.t0 * a.H + h;               // (token, head) rows are a.H apart
  // the values this thread's column of the substitution needs: under way while everything else is made
  float x[CH];
  if (DELTA) {
    const int j = tid - DKT;
#pragma unroll
    for (int t = 0; t < CH; ++t) x[t] = (j >= 0 && j < a.dvp && t < p.n) ? a.vf[(c_row + (long long)t * a.H) * a.dvp + j] : 0.f;
  }
  if (warp == 0) {
    const bool live = lane < p.n;
    const long long r = c_row + (long long)lane * a.H;
    g1[lane] = !live ? 1.f : (a.head_rate ? a.af[r * a.dkp] : a.dec[r]);
    fac[lane] = live ? a.sc[r] : 0.f;
  }
  // rows of q and k in parts: DKT / 4 lanes a token
  constexpr int LPT = DKT / 4;
#pragma unroll
  for (int u = 0; u < CH * LPT / THREADS; ++u) {
    const int e = tid + u * THREADS, t = e / LPT, c = (e - t * LPT) * 4;
    float4 k = make_float4(0.f, 0.f, 0.f, 0.f), q = k;
    if (t < p.n && c < a.dkp) {
      const long long at = ((long long)(p.t0 + t) * a.Hqk + hq) * a.dkp + c;
      k = *reinterpret_cast<const float4*>(a.kf + at);
      q = *reinterpret_cast<const float4*>(a.qf + at);
      if (MODE == MODE_SSM) {                      // S += (dt k) v^T
        const float f = a.sc[c_row + (long long)t * a.H];
        k.x *= f; k.y *= f; k.z *= f; k.w *= f;
      }
    }
    uint32_t lo[3], hi[3];
    split3(q.x, q.y, lo);
    split3(q.z, q.w, hi);
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(qp + i * PL + t * AP + c) = make_uint2(lo[i], hi[i]);
    split3(k.x, k.y, lo);
    split3(k.z, k.w, hi);
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(kp + i * PL + t * AP + c) = make_uint2(lo[i], hi[i]);
  }
  __syncthreads();
  // warps 0 .. 3: q k^T, 4 .. 7: k k^T (the delta rule); 16 tokens t by 16 tokens s each. Above the diagonal there is nothing to do:
  // that warp multiplies the decays out meanwhile (in double: products of equal factors in float would all lean the same way).
  const int m0 = (warp & 1) * 16, n0 = ((warp >> 1) & 1) * 16;
  const bool works = n0 <= m0 && (warp < 4 || DELTA);
  float acc[2][4] = {};
  if (works) {
    const bf16* left = (warp < 4 ? qp : kp) + (m0 + (lane & 15)) * AP + (lane >> 4) * 8;
    const bf16* right = kp + (n0 + (lane >> 4) * 8 + (lane & 7)) * AP + ((lane >> 3) & 1) * 8;
#pragma unroll 1
    for (int kk = 0; kk < DKT; kk += 32) {
      uint32_t av[2][3][4], bv[2][3][4];
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int i = 0; i < 3; ++i) { ldsm4(av[k][i], left + i * PL + kk + k * 16); ldsm4(bv[k][i], right + i * PL + kk + k * 16); }
      product32(acc, av, bv);
    }
  } else if (warp == 2) {
    double d = 1.0, up = 1.0, dn = 1.0;
    for (int t = 0; t < CH; ++t) {                 // lane = s
      const double g = (double)g1[t];
      up *= g;
      if (t > lane) d *= g;
      Dm[t * (CH + 1) + lane] = (float)d;
      if (lane == t) gup[t] = (float)up;
      if (t > lane) dn *= g;
    }
    gdn[lane] = (float)dn;
    if (lane == 0) {
      c_all[0] = (float)up;
      c_all[1] = finite((float)up) ? (float)(up - (double)(float)up) : 0.f;
    }
  }
  __syncthreads();
  unsigned char* image = reinterpret_cast<unsigned char*>(a.work) + ((p.slot + blockIdx.x) * a.H + h) * (long long)L::BYTES;
  bf16* img = reinterpret_cast<bf16*>(image);
  bool bad = false;                                // something this thread leaves is not finite
  auto leave2 = [&](int off, int plane, float u, float v) {
    uint32_t parts[3];
    split3(u, v, parts);
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(img + off + i * plane) = parts[i];
    bad |= !finite(u) || !finite(v);
  };
  {
    const float skip = MODE != MODE_SSM ? 0.f : a.skip_dtype == SB_DTYPE_F32 ? ((const float*)a.skip)[h] : to_float(((const bf16*)a.skip)[h]);
    const int g = lane >> 2, c2 = (lane & 3) * 2;
    if (warp < 4 || DELTA) {
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int t = m0 + g + 8 * r, s = n0 + n * 8 + c2;
          const float u = acc[n][2 * r] * Dm[t * (CH + 1) + s], v = acc[n][2 * r + 1] * Dm[t * (CH + 1) + s + 1];
          if (warp < 4) {
            leave2(L::P_OFF + t * PP + s, CH * PP, s <= t ? (s == t ? u + skip : u) : 0.f, s + 1 <= t ? (s + 1 == t ? v + skip : v) : 0.f);
          } else {
            At[s * TP + t] = s < t ? fac[t] * u : 0.f;
            At[(s + 1) * TP + t] = s + 1 < t ? fac[t] * v : 0.f;
          }
        }
    }
  }
  // Q' and K'': two neighbouring rows of S a thread, the tokens shared out
  constexpr int GROUPS = THREADS / (DKT / 2);
  {
    const int c = (tid % (DKT / 2)) * 2, first = tid / (DKT / 2) * (CH / GROUPS);
#pragma unroll 4
    for (int t = first; t < first + CH / GROUPS; ++t) {
      const float2 q = joined2(qp + t * AP + c, PL), k = joined2(kp + t * AP + c, PL);
      leave2(((DELTA ? CH : 0) + t) * AP + c, L::ROWS * AP, q.x * gup[t], q.y * gup[t]);
      leave2(L::K_OFF + t * AP + c, CH * AP, k.x * gdn[t], k.y * gdn[t]);
    }
  }
  if (tid < DKT) {
    float* img_c = reinterpret_cast<float*>(img + L::C_OFF);
    img_c[tid] = c_all[0];
    img_c[DKT + tid] = c_all[1];
    bad |= !finite(c_all[0]);
  }
  if constexpr (DELTA) {
    __syncthreads();
    // forward substitution, a thread a column of [diag(b) K' | diag(b) V]
    for (int c = tid; c < DKT + a.dvp; c += THREADS) {
      const bool is_k = c < DKT;                   // (a whole warp)
      const int j = c - DKT;
      if (c >= THREADS) {
#pragma unroll
        for (int t = 0; t < CH; ++t) x[t] = t < p.n ? a.vf[(c_row + (long long)t * a.H) * a.dvp + j] : 0.f;
      }
#pragma unroll
      for (int t = 0; t < CH; ++t) x[t] = fac[t] * (is_k ? gup[t] * joined(kp + t * AP + c, PL) : x[t]);
#pragma unroll
      for (int s = 0; s < CH - 1; ++s) {           // x[s] is final: taken out of every later one (independent of one another)
#pragma unroll
        for (int t4 = (s + 1) & ~3; t4 < CH; t4 += 4) {
          const float4 a4 = *reinterpret_cast<const float4*>(At + s * TP + t4);
          if (t4 > s) x[t4] = fmaf(-a4.x, x[s], x[t4]);
          if (t4 + 1 > s) x[t4 + 1] = fmaf(-a4.y, x[s], x[t4 + 1]);
          if (t4 + 2 > s) x[t4 + 2] = fmaf(-a4.z, x[s], x[t4 + 2]);
          x[t4 + 3] = fmaf(-a4.w, x[s], x[t4 + 3]);
        }
      }
      if (is_k) {
        // neighbouring columns swap every other token, so that each stores pairs
        const bool odd = c & 1;
#pragma unroll
        for (int t = 0; t < CH; t += 2) {
          const float other = __shfl_xor_sync(0xffffffffu, odd ? x[t] : x[t + 1], 1);
          leave2((t + (odd ? 1 : 0)) * AP + (c & ~1), L::ROWS * AP, odd ? other : x[t], odd ? x[t + 1] : other);
        }
      } else {
#pragma unroll
        for (int t = 0; t < CH; ++t)
          if (t < p.n) u_rows[(c_row + (long long)t * a.H) * a.dvp + j] = x[t];
      }
    }
  }
  const int any = __syncthreads_or(bad);
  if (tid == 0) reinterpret_cast<int*>(image)[L::BYTES / 4 - 4] = any;
}

__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(tc::smem_u32(dst)), "l"(src), "r"(bytes), "r"(tc::smem_u32(bar)) : "memory");
}

constexpr int FETCHER = 128;           // a thread of the walk that fetches (its warp waits for no loads of its own)
constexpr int SP = VC + 8;             // pitch of the parts of S and U: eight rows' 16-byte pieces fall into different banks
template <int DKT, bool DELTA>
struct Walk {
  typedef Part<DKT, DELTA> L;
  static constexpr int STAGE = L::BYTES, S_OFF = 2 * STAGE, UP_OFF = S_OFF + 3 * DKT * SP * 2,
                       PART_OFF = UP_OFF + 3 * CH * SP * 2;
  static constexpr int US_OFF = PART_OFF + THREADS * 16, BYTES = US_OFF + CH * VC * 4;
};

// grid (ceil(dv / 16), head, list entry). Warps 0 .. 3 make U, 4 .. 7 read out; all of them the next S.
template <int DKT, bool DELTA>
__global__ void __launch_bounds__(THREADS) chunk_walk_kernel(const SbChunkedWalk a, const float* __restrict__ u_rows) {
  typedef Walk<DKT, DELTA> W;
  typedef Part<DKT, DELTA> L;
  constexpr int AP = L::AP, ROWS = L::ROWS, SPL = DKT * SP, UPL = CH * SP;
  extern __shared__ __align__(16) unsigned char raw[];
  __shared__ int red_i[8];
  __shared__ __align__(8) uint64_t full[2];
  __shared__ int gave_up;
  bf16* Sp = reinterpret_cast<bf16*>(raw + W::S_OFF);              // [3][DKT][SP]
  bf16* Up = reinterpret_cast<bf16*>(raw + W::UP_OFF);             // [3][CH][SP]
  float4* part = reinterpret_cast<float4*>(raw + W::PART_OFF);     // [warp][lane]: what the warp's neighbour adds to its sums
  float* Us = reinterpret_cast<float*>(raw + W::US_OFF);           // [CH][VC]: U
  Place p;
  if (!find_chunk(a, blockIdx.z, 0, p, red_i)) return;
  const int h = blockIdx.y, j0 = blockIdx.x * VC;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c2 = (lane & 3) * 2;
  const int n_all = a.cu_q[p.row + 1] - p.t0;
  const unsigned char* images = reinterpret_cast<const unsigned char*>(a.work) + (p.slot * a.H + h) * (long long)L::BYTES;
  if (tid == 0) {
    gave_up = 0;
    tc::mbar_init(&full[0], 1);
    tc::mbar_init(&full[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  auto fetch = [&](int c) {                                // (one thread) a chunk's image is one piece: one instruction
    uint64_t* bar = &full[c & 1];
    tc::mbar_expect_tx(bar, L::BYTES);
    bulk_load(raw + (c & 1) * W::STAGE, images + (long long)c * a.H * L::BYTES, L::BYTES, bar);
  };

  // this warp's part of S, as accumulators: 16 rows i0 .. of 16 columns (128 rows) or of 8 (64 rows)
  constexpr int NT = DKT == 128 ? 2 : 1;
  const int i0 = (DKT == 128 ? warp : warp & 3) * 16, s0 = DKT == 128 ? 0 : (warp >> 2) * 8;
  float* S = a.state + (size_t)a.slots[p.row] * a.state_stride + (size_t)h * a.dk * a.dv;
  float s[NT][4];
  bool bad = false;                                        // something of S or U that this thread holds is not finite
  auto keep = [&]() {                                      // S in parts, for the next product
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        uint32_t parts[3];
        split3(s[n][2 * r], s[n][2 * r + 1], parts);
        bad |= !finite(s[n][2 * r]) || !finite(s[n][2 * r + 1]);
#pragma unroll
        for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(Sp + i * SPL + (i0 + g + 8 * r) * SP + s0 + n * 8 + c2) = parts[i];
      }
  };
  if (tid == FETCHER) fetch(0);
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = i0 + g + 8 * (e >> 1), j = j0 + s0 + n * 8 + c2 + (e & 1);
      s[n][e] = (i < a.dk && j < a.dv) ? S[(size_t)i * a.dv + j] : 0.f;
    }
  keep();
  // two neighbouring warps share 16 rows of [W; Q'], each takes half of the rows of S; then each has the sums of 8 of the columns
  const int mt = warp >> 1, half = warp & 1, n0 = half * 8;
  const bool reads_out = mt >= 2;
  const int t0 = (mt & 1) * 16, row0 = (DELTA ? mt : mt & 1) * 16;         // its tokens, their rows of [W; Q']
  // rows of V' (or v) of the warps that make U, a chunk ahead in registers
  float2 u_next[2];
  auto fetch_u = [&](int c) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int t = c * CH + t0 + g + 8 * r;
      u_next[r] = make_float2(0.f, 0.f);
      if (t < n_all) u_next[r] = *reinterpret_cast<const float2*>(u_rows + ((size_t)(p.t0 + t) * a.H + h) * a.dvp + j0 + n0 + c2);
    }
  };
  if (!reads_out) fetch_u(0);
  for (int c = 0; c < p.n_chunks; ++c) {
    if (!tc::mbar_wait(&full[c & 1], (c >> 1) & 1)) gave_up = 1;
    const bool slow_s = __syncthreads_or(bad) != 0;        // the chunk's matrices and S are there; the other stage is free
    if (gave_up) {                                         // (all of the block; nothing else is in flight)
      if (tid == 0) {
        tc::mbar_wait(&full[c & 1], (c >> 1) & 1);
        if (a.timeouts) atomicAdd(a.timeouts, 1);
      }
      return;
    }
    if (tid == FETCHER && c + 1 < p.n_chunks) fetch(c + 1);
    const unsigned char* st = raw + (c & 1) * W::STAGE;
    const bf16* A1 = reinterpret_cast<const bf16*>(st);
    const bf16 *Kp = A1 + L::K_OFF, *Pp = A1 + L::P_OFF;
    const float* cc = reinterpret_cast<const float*>(A1 + L::C_OFF);
    const bool slow1 = slow_s || reinterpret_cast<const int*>(cc + 2 * DKT)[0] != 0;
    const int n = min(CH, n_all - c * CH);
    bad = false;
    float x[4] = {0.f, 0.f, 0.f, 0.f};
    if (DELTA || reads_out) {
      float acc[2][4] = {};
      const int k0 = half * (DKT / 2);
      if (!slow1) {
        const bf16* left = A1 + (row0 + (lane & 15)) * AP + k0 + (lane >> 4) * 8;
        const bf16* right = Sp + (k0 + ((lane >> 3) & 1) * 8 + (lane & 7)) * SP + (lane >> 4) * 8;
        uint32_t av[DKT / 64][2][3][4], bv[DKT / 64][2][3][4];
#pragma unroll
        for (int k = 0; k < DKT / 32; ++k)
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            ldsm4(av[k >> 1][k & 1][i], left + i * ROWS * AP + k * 16);
            ldsm4_t(bv[k >> 1][k & 1][i], right + i * SPL + k * 16 * SP);
          }
#pragma unroll
        for (int k = 0; k < DKT / 64; ++k) product32(acc, av[k], bv[k]);
      } else {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int r = row0 + g + 8 * (e >> 1), col = m * 8 + c2 + (e & 1);
            for (int k = k0; k < k0 + DKT / 2; ++k) acc[m][e] = fmaf(joined(A1 + r * AP + k, ROWS * AP), joined(Sp + k * SP + col, SPL), acc[m][e]);
          }
      }
      part[tid] = half ? make_float4(acc[0][0], acc[0][1], acc[0][2], acc[0][3]) : make_float4(acc[1][0], acc[1][1], acc[1][2], acc[1][3]);
      asm volatile("bar.sync %0, 64;" ::"r"(mt + 1) : "memory");
      const float4 y = part[tid ^ 32];
      x[0] = (half ? acc[1][0] : acc[0][0]) + y.x;
      x[1] = (half ? acc[1][1] : acc[0][1]) + y.y;
      x[2] = (half ? acc[1][2] : acc[0][2]) + y.z;
      x[3] = (half ? acc[1][3] : acc[0][3]) + y.w;
    }
    if (!reads_out) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int t = t0 + g + 8 * r;
        float2 u = u_next[r];
        if (DELTA) u = t < n ? make_float2(u.x - x[2 * r], u.y - x[2 * r + 1]) : make_float2(0.f, 0.f);
        *reinterpret_cast<float2*>(Us + t * VC + n0 + c2) = u;
        uint32_t parts[3];
        split3(u.x, u.y, parts);
#pragma unroll
        for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(Up + i * UPL + t * SP + n0 + c2) = parts[i];
        bad |= !finite(u.x) || !finite(u.y);
      }
      fetch_u(c + 1);
    }
    const bool slow2 = __syncthreads_or(bad) != 0 || slow1;
    bad = false;
    uint32_t uv[2][3][4];                                  // the parts of U, 32 tokens by 16 columns
    float add[NT][4] = {};
    if (!slow2) {
      const bf16* right = Up + (((lane >> 3) & 1) * 8 + (lane & 7)) * SP + (lane >> 4) * 8;
      const bf16* left = Kp + ((lane >> 4) * 8 + (lane & 7)) * AP + i0 + ((lane >> 3) & 1) * 8;
      uint32_t av[2][3][4];
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          ldsm4_t(uv[k][i], right + i * UPL + k * 16 * SP);
          ldsm4_t(av[k][i], left + i * CH * AP + k * 16 * AP);
        }
      if constexpr (NT == 2) {
        product32(add, av, uv);
      } else {
        uint32_t bv[2][3][2];
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int i = 0; i < 3; ++i) { bv[k][i][0] = s0 ? uv[k][i][2] : uv[k][i][0]; bv[k][i][1] = s0 ? uv[k][i][3] : uv[k][i][1]; }
        product32(add, av, bv);
      }
    } else {
#pragma unroll
      for (int m = 0; m < NT; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = i0 + g + 8 * (e >> 1), col = s0 + m * 8 + c2 + (e & 1);
          for (int t = 0; t < CH; ++t) add[m][e] = fmaf(joined(Kp + t * AP + i, CH * AP), Us[t * VC + col], add[m][e]);
        }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const float dc = cc[i0 + g + 8 * r], lo = cc[DKT + i0 + g + 8 * r];
#pragma unroll
      for (int m = 0; m < NT; ++m)
#pragma unroll
        for (int e = 2 * r; e < 2 * r + 2; ++e) s[m][e] = fmaf(dc, s[m][e], fmaf(lo, s[m][e], add[m][e]));
    }
    keep();
    if (reads_out) {
      if (!slow2) {
        uint32_t av[2][3][4], bv[2][3][2];
        float o[1][4] = {{x[0], x[1], x[2], x[3]}};
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            ldsm4(av[k][i], Pp + i * CH * PP + (t0 + (lane & 15)) * PP + k * 16 + (lane >> 4) * 8);      // (zeros after the diagonal)
            bv[k][i][0] = half ? uv[k][i][2] : uv[k][i][0];
            bv[k][i][1] = half ? uv[k][i][3] : uv[k][i][1];
          }
        product32(o, av, bv);
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = o[0][e];
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int t = t0 + g + 8 * (e >> 1);
          for (int k = 0; k <= t; ++k) x[e] = fmaf(joined(Pp + t * PP + k, CH * PP), Us[k * VC + n0 + c2 + (e & 1)], x[e]);
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = t0 + g + 8 * (e >> 1), j = j0 + n0 + c2 + (e & 1);
        if (t < n && j < a.dv) a.out[(size_t)(p.t0 + c * CH + t) * a.out_stride + (size_t)h * a.dv + j] = x[e];
      }
    }
  }
#pragma unroll
  for (int m = 0; m < NT; ++m)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = i0 + g + 8 * (e >> 1), j = j0 + s0 + m * 8 + c2 + (e & 1);
      if (i < a.dk && j < a.dv) S[(size_t)i * a.dv + j] = s[m][e];
    }
}

// The walk for many (request, head) pairs: G groups of 16 columns in a block, KS = 2 warps a group with half of the rows of S each, and a warp that
// fetches. A chunk's matrices then cross to an SM once for 16 G columns instead of once for 16, and since S lies turned over in
// the accumulators (columns of S are the tile's rows), they are the first operand of the next product as they stand: S and U never
// pass through shared memory, and the warps of a group meet once a step, to add their sums of W S (and Q' S) up. What bounds it: mma.sync, 16
// cycles each on a scheduler by timing (1,728 of them a step with 64 columns and no delta rule: 6,900 of the step's 7,800 cycles; the tensor pipe's
// counter calls it active in half of those). With few pairs there
// are not enough blocks, and chunk_walk_kernel, whose eight warps share 16 columns, has the shorter step. Eight requests of 256 tokens, 16
// heads of 128 x 128: fixed decay 101 -> 67 us, gated delta rule 121 -> 95. (One warp for all rows of 16 columns: 91 us, registers spill;
// the sums of Q' S a step behind those of W S, so that they hide: 107, more of them spill.)
template <int DKT, bool DELTA, int G>
struct Wide {
  typedef Part<DKT, DELTA> L;
  static constexpr int KS = 2;
  static constexpr int WARPS = KS * G, THREADS = 32 * (WARPS + 1);
  static constexpr int TILES = DELTA ? 8 : 4;             // eights of rows of [W; Q'] (or Q')
  static constexpr int XCH_OFF = 2 * L::BYTES, BYTES = XCH_OFF + 2 * WARPS * TILES * 32 * 16;
  static_assert(BYTES <= 226 * 1024, "shared memory of an SM");
};

__device__ __forceinline__ void group_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ bool group_any(int id, int threads, bool yes) {
  uint32_t any;
  asm volatile("{\n .reg .pred p, q;\n setp.ne.b32 q, %3, 0;\n bar.red.or.pred p, %1, %2, q;\n selp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(any) : "r"(id), "r"(threads), "r"(yes ? 1u : 0u) : "memory");
  return any != 0;
}
// the parts of 16 columns (j) by 16 terms as a first operand, from two neighbouring accumulators' registers
__device__ __forceinline__ void parts_of(uint32_t (&p)[3][4], const float (&x)[4], const float (&y)[4]) {
  uint32_t q[4][3];
  split3(x[0], x[1], q[0]);
  split3(x[2], x[3], q[1]);
  split3(y[0], y[1], q[2]);
  split3(y[2], y[3], q[3]);
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int r = 0; r < 4; ++r) p[i][r] = q[r][i];
}

// what its waits leave (bounded_wait.h)
struct Notes {
  int *gave_up, *timeouts;
  __device__ __forceinline__ bool raise() { return atomicExch(gave_up, 1) == 0; }
  __device__ __forceinline__ bool raised() const { return *(volatile int*)gave_up != 0; }
  __device__ __forceinline__ void count() { if (timeouts) atomicAdd(timeouts, 1); }
};

// grid (ceil(dv / (16 G)), head, list entry).
template <int DKT, bool DELTA, int G>
__global__ void __launch_bounds__(Wide<DKT, DELTA, G>::THREADS) chunk_wide_kernel(const SbChunkedWalk a, const float* __restrict__ u_rows) {
  typedef Wide<DKT, DELTA, G> W;
  typedef Part<DKT, DELTA> L;
  constexpr int AP = L::AP, ROWS = L::ROWS, TILES = W::TILES, KS = W::KS, NTS = DKT / KS / 8, OT = 4 / KS;
  constexpr int LEFT[6] = {2, 0, 1, 1, 0, 0}, RIGHT[6] = {0, 2, 1, 0, 1, 0};      // six of the nine products of the parts, smallest first
  extern __shared__ __align__(16) unsigned char raw[];
  __shared__ int red_i[16];
  __shared__ __align__(8) uint64_t full[2], empty[2];
  __shared__ int gave_up;
  Place p;
  if (!find_chunk(a, blockIdx.z, 0, p, red_i)) return;
  const int h = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int groups = min(G, (a.dv - (int)blockIdx.x * 16 * G + 15) / 16);          // (at the last columns not all have any)
  const unsigned char* images = reinterpret_cast<const unsigned char*>(a.work) + (p.slot * a.H + h) * (long long)L::BYTES;
  if (tid == 0) {
    gave_up = 0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&full[i], 1);
      tc::mbar_init(&empty[i], groups * KS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  Notes notes{&gave_up, a.timeouts};
  auto wait = [&](uint64_t* bar, unsigned parity) {
    if (!tc::mbar_try(bar, parity)) wait_in_step([&] { return tc::mbar_try(bar, parity); }, notes, tc::WAIT_LIMIT);
  };

  if (warp == W::WARPS) {                                  // a chunk's matrices are one piece: one bulk copy
    int c = 0;
    for (; c < p.n_chunks; ++c) {
      wait(&empty[c & 1], ((c >> 1) & 1) ^ 1);
      if (__any_sync(0xffffffffu, notes.raised())) break;
      if (tc::elect_one()) {
        tc::mbar_expect_tx(&full[c & 1], L::BYTES);
        bulk_load(raw + (c & 1) * L::BYTES, images + (long long)c * a.H * L::BYTES, L::BYTES, &full[c & 1]);
      }
      __syncwarp();
    }
    for (int i = max(0, c - 2); i < c; ++i)                // copies under way land before the block may leave
      wait_landed([&] { return tc::mbar_try(&full[i & 1], (i >> 1) & 1); }, notes, tc::WAIT_LIMIT);
    return;
  }
  const int group = warp / KS, ks = warp - group * KS;
  if (group >= groups) return;
  const int g = lane >> 2, c2 = (lane & 3) * 2;
  const int j0 = ((int)blockIdx.x * G + group) * 16, i0 = ks * (DKT / KS);
  const int n_all = a.cu_q[p.row + 1] - p.t0;
  float* S = a.state + (size_t)a.slots[p.row] * a.state_stride + (size_t)h * a.dk * a.dv;
  // S turned over: the tile's rows are columns j0 .. of S, its columns rows i0 .. of S. An accumulator's registers are then the first
  // operand's of the next product, and S and U never leave the registers.
  float s[NTS][4];
  bool bad = false;                                        // something of S that this thread holds is not finite
#pragma unroll
  for (int m = 0; m < NTS; ++m)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = i0 + m * 8 + c2 + (e & 1), j = j0 + g + 8 * (e >> 1);
      s[m][e] = (i < a.dk && j < a.dv) ? S[(size_t)i * a.dv + j] : 0.f;
      bad |= !finite(s[m][e]);
    }
  // rows of V' (or v), a chunk ahead
  float u_next[4][4];
  auto fetch_u = [&](int c) {
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = c * CH + n * 8 + c2 + (e & 1);
        u_next[n][e] = t < n_all ? u_rows[((size_t)(p.t0 + t) * a.H + h) * a.dvp + j0 + g + 8 * (e >> 1)] : 0.f;
      }
  };
  fetch_u(0);
  for (int c = 0; c < p.n_chunks; ++c) {
    wait(&full[c & 1], (c >> 1) & 1);
    __syncwarp();
    const bf16* A1 = reinterpret_cast<const bf16*>(raw + (c & 1) * L::BYTES);
    const bf16 *Kp = A1 + L::K_OFF, *Pp = A1 + L::P_OFF;
    const float* cc = reinterpret_cast<const float*>(A1 + L::C_OFF);
    const int n_tok = min(CH, n_all - c * CH);
    bool slow = reinterpret_cast<const int*>(cc + 2 * DKT)[0] != 0;
    // [W; Q'] S of this warp's rows of S
    float x[TILES][4];
    auto first_slow = [&]() {
      float ls[NTS * 4];
#pragma unroll
      for (int m = 0; m < NTS * 4; ++m) ls[m] = s[m >> 2][m & 3];
#pragma unroll
      for (int n = 0; n < TILES; ++n) x[n][0] = x[n][1] = x[n][2] = x[n][3] = 0.f;
#pragma unroll 1
      for (int i = 0; i < NTS * 8; ++i) {
        const int r = (i >> 3) * 4 + (i & 1), src = (lane & ~3) | ((i & 7) >> 1);
        const float lo = __shfl_sync(0xffffffffu, ls[r], src), hi = __shfl_sync(0xffffffffu, ls[r + 2], src);
#pragma unroll
        for (int n = 0; n < TILES; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float w = joined(A1 + (n * 8 + c2 + e) * AP + i0 + i, ROWS * AP);
            x[n][e] = fmaf(w, lo, x[n][e]);
            x[n][2 + e] = fmaf(w, hi, x[n][2 + e]);
          }
      }
    };
    if (!slow) {
#pragma unroll
      for (int n = 0; n < TILES; ++n) x[n][0] = x[n][1] = x[n][2] = x[n][3] = 0.f;
      const bf16* right = A1 + ((lane >> 4) * 8 + (lane & 7)) * AP + i0 + ((lane >> 3) & 1) * 8;
#pragma unroll
      for (int k = 0; k < NTS / 2; ++k) {
        uint32_t sa[3][4];
        parts_of(sa, s[2 * k], s[2 * k + 1]);
#pragma unroll
        for (int n4 = 0; n4 < TILES; n4 += 4) {
          uint32_t b[2][3][4];
          float t[4][4] = {};
#pragma unroll
          for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int i = 0; i < 3; ++i) ldsm4(b[u][i], right + i * ROWS * AP + (n4 * 8 + u * 16) * AP + k * 16);
#pragma unroll
          for (int i = 0; i < 6; ++i)
#pragma unroll
            for (int n = 0; n < 4; ++n) mma(t[n], sa[LEFT[i]], b[n >> 1][RIGHT[i]][(n & 1) * 2], b[n >> 1][RIGHT[i]][(n & 1) * 2 + 1]);
#pragma unroll
          for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) x[n4 + n][e] += t[n][e];
        }
      }
    } else {
      first_slow();
    }
    float o[OT][4];
    // the group's warps add their sums up, all of them W S, each its own tokens of Q' S
    float4* xch = reinterpret_cast<float4*>(raw + W::XCH_OFF) + (size_t)((c & 1) * W::WARPS + group * KS) * TILES * 32 + lane;
    auto leave = [&]() {
#pragma unroll
      for (int n = 0; n < TILES; ++n) xch[(ks * TILES + n) * 32] = make_float4(x[n][0], x[n][1], x[n][2], x[n][3]);
    };
    leave();
    if (group_any(1 + group, 32 * KS, bad)) {            // (all of the group) S is not finite: once more, without parts
      if (!slow) first_slow();
      slow = true;
      leave();
      group_sync(1 + group, 32 * KS);
    }
    auto sum = [&](float (&y)[4], int n) {
      float4 v[KS];
#pragma unroll
      for (int w = 0; w < KS; ++w) v[w] = xch[(w * TILES + n) * 32];
      y[0] = v[0].x; y[1] = v[0].y; y[2] = v[0].z; y[3] = v[0].w;
#pragma unroll
      for (int w = 1; w < KS; ++w) { y[0] += v[w].x; y[1] += v[w].y; y[2] += v[w].z; y[3] += v[w].w; }
    };
    if (DELTA) {
#pragma unroll
      for (int n = 0; n < 4; ++n) sum(x[n], n);
    }
#pragma unroll
    for (int n = 0; n < OT; ++n) sum(o[n], TILES - 4 + ks * OT + n);
    float u[4][4];
    bool bad_u = false;
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        u[n][e] = u_next[n][e];
        if (DELTA) u[n][e] = n * 8 + c2 + (e & 1) < n_tok ? u[n][e] - x[n][e] : 0.f;
        bad_u |= !finite(u[n][e]);
      }
    fetch_u(c + 1);
    slow |= __any_sync(0xffffffffu, bad_u) != 0;           // (the warps of a group hold the same U)
    uint32_t ua[2][3][4];
    float lu[16];
    if (!slow) {
#pragma unroll
      for (int k = 0; k < 2; ++k) parts_of(ua[k], u[2 * k], u[2 * k + 1]);
    } else {
#pragma unroll
      for (int n = 0; n < 16; ++n) lu[n] = u[n >> 2][n & 3];
    }
    bad = false;
    auto step = [&](int m, const float (&add)[4]) {        // the next S
      const float2 dc = *reinterpret_cast<const float2*>(cc + i0 + m * 8 + c2), lo = *reinterpret_cast<const float2*>(cc + DKT + i0 + m * 8 + c2);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        s[m][e] = fmaf((e & 1) ? dc.y : dc.x, s[m][e], fmaf((e & 1) ? lo.y : lo.x, s[m][e], add[e]));
        bad |= !finite(s[m][e]);
      }
    };
    if (!slow) {
      const bf16* right = Kp + (((lane >> 3) & 1) * 8 + (lane & 7)) * AP + i0 + (lane >> 4) * 8;
#pragma unroll
      for (int m = 0; m < NTS; m += 2) {
        uint32_t b[2][3][4];
        float t[2][2][4] = {};
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int i = 0; i < 3; ++i) ldsm4_t(b[k][i], right + i * CH * AP + k * 16 * AP + m * 8);
#pragma unroll
        for (int i = 0; i < 6; ++i)
#pragma unroll
          for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int n = 0; n < 2; ++n) mma(t[k][n], ua[k][LEFT[i]], b[k][RIGHT[i]][n * 2], b[k][RIGHT[i]][n * 2 + 1]);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          float add[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) add[e] = t[0][n][e] + t[1][n][e];
          step(m + n, add);
        }
      }
      // O += P U: token n's eight rows of P, zeros after the diagonal
#pragma unroll
      for (int n = 0; n < OT; ++n) {
        const int tile = ks * OT + n;
        uint32_t b[3][4];                                  // the 32 terms of eight tokens
#pragma unroll
        for (int i = 0; i < 3; ++i) ldsm4(b[i], Pp + i * CH * PP + (tile * 8 + (lane & 7)) * PP + (lane >> 3) * 8);
        float t[2][4] = {};
#pragma unroll
        for (int i = 0; i < 6; ++i)
#pragma unroll
          for (int k = 0; k < 2; ++k) mma(t[k], ua[k][LEFT[i]], b[RIGHT[i]][k * 2], b[RIGHT[i]][k * 2 + 1]);
#pragma unroll
        for (int e = 0; e < 4; ++e) o[n][e] += t[0][e] + t[1][e];
      }
    } else {
      float add[NTS][4] = {};
#pragma unroll 1
      for (int t = 0; t < CH; ++t) {
        const int r = (t >> 3) * 4 + (t & 1), src = (lane & ~3) | ((t & 7) >> 1);
        const float lo = __shfl_sync(0xffffffffu, lu[r], src), hi = __shfl_sync(0xffffffffu, lu[r + 2], src);
#pragma unroll
        for (int m = 0; m < NTS; ++m)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float k = joined(Kp + t * AP + i0 + m * 8 + c2 + e, CH * AP);
            add[m][e] = fmaf(k, lo, add[m][e]);
            add[m][2 + e] = fmaf(k, hi, add[m][2 + e]);
          }
#pragma unroll
        for (int n = 0; n < OT; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int to = (ks * OT + n) * 8 + c2 + e;
            if (t > to) continue;                          // (a later token's infinity must not reach back)
            const float q = joined(Pp + to * PP + t, CH * PP);
            o[n][e] = fmaf(q, lo, o[n][e]);
            o[n][2 + e] = fmaf(q, hi, o[n][2 + e]);
          }
      }
#pragma unroll
      for (int m = 0; m < NTS; ++m) step(m, add[m]);
    }
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(&empty[c & 1]);         // the chunk's matrices have been read
#pragma unroll
    for (int n = 0; n < OT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = (ks * OT + n) * 8 + c2 + (e & 1), j = j0 + g + 8 * (e >> 1);
        if (t < n_tok && j < a.dv) a.out[(size_t)(p.t0 + c * CH + t) * a.out_stride + (size_t)h * a.dv + j] = o[n][e];
      }
  }
  if (notes.raised()) return;                              // (the state stays the one before this step)
#pragma unroll
  for (int m = 0; m < NTS; ++m)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = i0 + m * 8 + c2 + (e & 1), j = j0 + g + 8 * (e >> 1);
      if (i < a.dk && j < a.dv) S[(size_t)i * a.dv + j] = s[m][e];
    }
}

template <int DKT, bool DELTA, int G>
int launch_wide(const SbChunkedWalk& a, const float* u_rows, cudaStream_t stream) {
  typedef Wide<DKT, DELTA, G> W;
  auto k = chunk_wide_kernel<DKT, DELTA, G>;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, W::BYTES);
  k<<<dim3((a.dv + 16 * G - 1) / (16 * G), a.H, a.n_list), W::THREADS, W::BYTES, stream>>>(a, u_rows);
  SB_LAUNCH_CHECK();
  return 0;
}

template <int DKT, bool VEC, int MODE>
int launch(const SbChunkedWalk& a, int chunks, cudaStream_t stream) {
  constexpr bool DELTA = MODE == MODE_DELTA;
  float* u_rows = DELTA ? a.work + (long long)chunks * a.H * (part_bytes(DKT, DELTA) / 4) : nullptr;
  const dim3 grid((a.max_q + CH - 1) / CH, a.H, a.n_list);
  if constexpr (VEC) {
    auto k = chunk_prep_rows_kernel<DKT, MODE>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, rows_smem<DKT>());
    k<<<grid, THREADS, rows_smem<DKT>(), stream>>>(a, u_rows);
  } else {
    auto k = chunk_prep_head_kernel<DKT, MODE>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, head_smem<DKT>());
    k<<<grid, THREADS, head_smem<DKT>(), stream>>>(a, u_rows);
  }
  SB_LAUNCH_CHECK();
  const float* u = DELTA ? u_rows : a.vf;
  const int groups = walk_groups(DELTA, DKT == 128, a.H, (a.dv + 15) / 16, chunks, (a.max_q + CH - 1) / CH, sm_count());
  if constexpr (DKT == 128 && !DELTA) {
    if (groups == 4) return launch_wide<DKT, DELTA, 4>(a, u, stream);
  }
  if (groups == 2) return launch_wide<DKT, DELTA, 2>(a, u, stream);
  auto k = chunk_walk_kernel<DKT, DELTA>;
  constexpr int smem = Walk<DKT, DELTA>::BYTES;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  k<<<dim3((a.dv + VC - 1) / VC, a.H, a.n_list), THREADS, smem, stream>>>(a, u);
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
  return (long long)chunks * H * (part_bytes(dk <= 64 ? 64 : 128, delta) / 4) + (delta ? (long long)n_tokens * H * dvp : 0);
}

int sb_chunked_walk(const SbChunkedWalk& a, int chunks, cudaStream_t stream) {
  if (a.n_list <= 0 || a.max_q <= a.min_tokens) return 0;
  if (sb_chunked_walk_floats(a.mode, a.n_tokens, chunks, a.H, a.dk, a.dvp) < 0 || a.dvp % VC || a.dkp > (a.dk <= 64 ? 64 : 128)) return SB_ERR_SHAPE;
  if (a.n_list > 65535) return SB_ERR_LIMIT;
  if (!aligned16(a.work)) return SB_ERR_ALIGN;
  return a.dk <= 64 ? launch_mode<64>(a, chunks, stream) : launch_mode<128>(a, chunks, stream);
}
