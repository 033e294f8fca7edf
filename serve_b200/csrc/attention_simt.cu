// Paged causal attention in plain float arithmetic (no tensor cores): the true
// 32-bit path, and the reference the faster kernels are checked against.
//
// One kernel serves prompt portions and decoded tokens alike. Row r of the
// step brings n = cu_q[r+1] - cu_q[r] query tokens at positions
// kv_len[r] - n .. kv_len[r] - 1; a query at position p attends the cached
// keys max(0, p - window + 1) .. p of its request (window 0: all of them).
// Two options for attentions without rotation: ``slopes`` (one float per query
// head, or null) takes slope_h * (p - key) off every score, and ``chunk`` > 0
// hides the keys before floor(p / chunk) * chunk (positions count from the start
// of the sequence, so the blocks do not move with how a prompt was cut).
// Two more: ``softcap`` c > 0 turns a scaled score s into c * tanh(s / c) (before any distance bias), and ``sinks``
// (one float per query head, or null) adds exp(sink_h) to the softmax's denominator: a score without key or value,
// neither scaled nor capped, counted once per row however the keys are split.
// Scores, running maximum, sum and the output accumulator are float; the
// online-softmax recurrences are those of serve/kernels/attn_prefill.py:58-72,
// in base e. Compile with -DSB_HEAD_DIM=<multiple of 16>.
#include "common.cuh"

#ifndef SB_HEAD_DIM
#error "define SB_HEAD_DIM"
#endif

using namespace sb;

namespace {

constexpr int D = SB_HEAD_DIM;
constexpr int BM = 16;        // query rows per block
constexpr int BN = 32;        // keys per tile
constexpr int THREADS = 128;  // 16 rows x 8 threads
constexpr int KSTRIDE = D + 1;

static_assert(D % 16 == 0 && D >= 16 && D <= 256, "head_dim must be a multiple of 16 in 16..256");

template <typename T>
__global__ void __launch_bounds__(THREADS) attention_simt_kernel(
    const T* __restrict__ qkv, int q_stride, const T* __restrict__ kc, const T* __restrict__ vc,  // caches [P, Hkv, ps, D]
    const int* __restrict__ block_table, int bt_width, const int* __restrict__ cu_q, const int* __restrict__ kv_len, int H,
    int Hkv, int ps, int num_pages, float scale, int window, T* __restrict__ out, int decode_apart,
    const float* __restrict__ slopes, int chunk, float softcap, const float* __restrict__ sinks, int keep) {
  extern __shared__ float smem[];
  float* Qs = smem;                 // [BM][D]
  float* Ks = Qs + BM * D;          // [BN][KSTRIDE]
  float* Vs = Ks + BN * KSTRIDE;    // [BN][D]
  float* Ps = Vs + BN * D;          // [BM][BN]

  const int r = blockIdx.z, h = blockIdx.y, tile = blockIdx.x;
  const int q0 = cu_q[r], qn = cu_q[r + 1] - q0;
  const int m0 = tile * BM;
  if (m0 >= qn) return;
  if (decode_apart && H / Hkv <= 16 && qn * (H / Hkv) <= 16) return;     // the decoding shape below takes this request
  const int L = kv_len[r];
  const int p0 = L - qn;            // position of the row's first query
  const int hk = h / (H / Hkv);
  const int tid = threadIdx.x;
  const int i = tid >> 3, jj = tid & 7;

  for (int w = tid; w < BM * D; w += THREADS) {
    const int mi = w / D, d = w - mi * D;
    Qs[w] = (m0 + mi < qn) ? to_float(qkv[(size_t)(q0 + m0 + mi) * q_stride + (size_t)h * D + d]) : 0.f;
  }

  const int pi = p0 + m0 + i;                       // this thread's query position
  const bool row_ok = (m0 + i) < qn;
  const int first_pos = p0 + m0, last_pos = p0 + min(m0 + BM, qn) - 1;
  int lo = window > 0 ? max(0, first_pos - window + 1) : 0;
  if (chunk > 0) lo = max(lo, (first_pos / chunk) * chunk);
  const int hi = last_pos + 1;                      // exclusive; <= L
  const float slope = slopes ? slopes[h] : 0.f;
  const int chunk_lo = chunk > 0 ? (pi / chunk) * chunk : 0;

  float m_run = -INFINITY, l_run = 0.f;
  float acc[D / 8];
#pragma unroll
  for (int c = 0; c < D / 8; ++c) acc[c] = 0.f;

  const int* bt = block_table + (size_t)r * bt_width;
  // keys below ``keep`` stay visible behind the window: the tiles that hold those before the window's first tile come first
  const int keep_end = min(keep, lo), lo_tile = (lo / BN) * BN;
  for (int kt = keep_end > 0 ? 0 : lo_tile; kt < hi; kt += BN) {
    if (kt >= keep_end && kt < lo_tile) kt = lo_tile;      // nothing to read between the kept keys and the window
    __syncthreads();  // previous tile fully consumed (and Qs written, first time round)
    for (int w = tid; w < BN * D; w += THREADS) {
      const int kj = w / D, d = w - kj * D;
      const int key = kt + kj;
      float kvv = 0.f, vvv = 0.f;
      if ((key >= lo || key < keep_end) && key < hi) {
        const int blk = key / ps;
        const int page = blk < bt_width ? bt[blk] : -1;
        if (page >= 0 && page < num_pages) {
          const size_t off = (((size_t)page * Hkv + hk) * ps + (key - blk * ps)) * D + d;
          kvv = to_float(kc[off]);
          vvv = to_float(vc[off]);
        }
      }
      Ks[kj * KSTRIDE + d] = kvv;
      Vs[kj * D + d] = vvv;
    }
    __syncthreads();

    float s[BN / 8];
#pragma unroll
    for (int c = 0; c < BN / 8; ++c) s[c] = 0.f;
    for (int d = 0; d < D; ++d) {
      const float qv = Qs[i * D + d];
#pragma unroll
      for (int c = 0; c < BN / 8; ++c) s[c] += qv * Ks[(jj + 8 * c) * KSTRIDE + d];
    }
    float tmax = -INFINITY;
#pragma unroll
    for (int c = 0; c < BN / 8; ++c) {
      const int key = kt + jj + 8 * c;
      const bool ok = row_ok && key <= pi && key >= chunk_lo && (window <= 0 || key > pi - window || key < keep);
      float sv = s[c] * scale;
      if (softcap > 0.f) sv = softcap * tanhf(sv / softcap);
      s[c] = ok ? sv - slope * (float)(pi - key) : -INFINITY;
      tmax = fmaxf(tmax, s[c]);
    }
    tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, 1));
    tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, 2));
    tmax = fmaxf(tmax, __shfl_xor_sync(0xffffffffu, tmax, 4));
    const float m_new = fmaxf(m_run, tmax);
    const float alpha = (m_new == -INFINITY) ? 1.f : expf(m_run - m_new);
    float psum = 0.f;
#pragma unroll
    for (int c = 0; c < BN / 8; ++c) {
      const float p = (s[c] == -INFINITY) ? 0.f : expf(s[c] - m_new);
      Ps[i * BN + jj + 8 * c] = p;
      psum += p;
    }
    psum += __shfl_xor_sync(0xffffffffu, psum, 1);
    psum += __shfl_xor_sync(0xffffffffu, psum, 2);
    psum += __shfl_xor_sync(0xffffffffu, psum, 4);
    l_run = l_run * alpha + psum;
    m_run = m_new;
    __syncwarp();  // the 8 threads of a row are in one warp; Ps row i is read only by them
#pragma unroll
    for (int c = 0; c < D / 8; ++c) acc[c] *= alpha;
    for (int kj = 0; kj < BN; ++kj) {
      const float p = Ps[i * BN + kj];
#pragma unroll
      for (int c = 0; c < D / 8; ++c) acc[c] += p * Vs[kj * D + jj + 8 * c];
    }
  }
  if (row_ok) {
    if (sinks != nullptr) {
      const float sk = sinks[h];
      const float m_fin = fmaxf(m_run, sk);
      const float a = (m_run == -INFINITY) ? 0.f : expf(m_run - m_fin);
      l_run = l_run * a + expf(sk - m_fin);
#pragma unroll
      for (int c = 0; c < D / 8; ++c) acc[c] *= a;
    }
    const float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
    T* orow = out + (size_t)(q0 + m0 + i) * H * D + (size_t)h * D;
#pragma unroll
    for (int c = 0; c < D / 8; ++c) orow[jj + 8 * c] = from_float<T>(acc[c] * inv);
  }
}

// The decoding shape: requests that bring at most 16 / G tokens (G = H / Hkv query heads per kv head). A block per
// (request, kv head, share of the keys); the G heads of every token are rows of one tile, so a key or value is fetched once for
// the whole group. LPK lanes share a key (each holds EPL <= 8 elements of the head vector), so a warp works on
// KPW = 32 / LPK keys at a time and a score costs log2(LPK) shuffles; the 8 warps x KPW lane groups are 8 KPW
// independent streams over the keys (stream s takes keys lo + s, lo + s + 8 KPW, ...), each with its own running
// maximum, sum and output for up to DEC_ROWS rows at a time (more rows: more passes over the keys). The streams meet
// in shared memory and are merged in stream order; the shares of the keys, if there are several, go to scratch memory and are
// merged in their order by a second kernel. Same recurrences as above, base e, full-precision expf.
// A stream waits for its own chain of loads, shuffles and exponentials, so what counts is how many streams an SM has and how far
// ahead their loads are: 8 elements a lane (instead of 16) let two blocks share an SM, the number of shares fills both, and a
// lane's keys come through a ring of cp.async stages. 8 requests of 2,048 keys, 8 kv heads of 64, 32 heads, float32 (67 MB):
// 50.9 us with one block a (request, kv head), 16 elements a lane and loads one key ahead; 44.7 with 4 shares and 8 elements; 30.3
// with the ring; 23.4 (and 3.7 for the merge) with a loop of its own for scores without options.
constexpr int DEC_WARPS = 8;
constexpr int DEC_ROWS = 4;
constexpr int LPK = D <= 16 ? 2 : (D <= 32 ? 4 : (D <= 64 ? 8 : (D <= 128 ? 16 : 32)));
constexpr int NCH = D / 4;                         // a head vector in chunks of four elements
constexpr int CPL = (NCH + LPK - 1) / LPK;         // chunks per lane: lane `sub` of a key's lanes takes chunks sub, sub + LPK, ...
constexpr int EPL = CPL * 4;                       // so neighbouring lanes read neighbouring 16 bytes of a key
constexpr int KPW = 32 / LPK;
constexpr int DEC_STREAMS = DEC_WARPS * KPW;
static_assert(D % 4 == 0 && EPL <= 8, "at most 8 elements of a head vector per lane");

__device__ __forceinline__ void load4(const float* p, float* x) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
}
__device__ __forceinline__ void load4(const __nv_bfloat16* p, float* x) {
  const uint2 v = *reinterpret_cast<const uint2*>(p);
  const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&v.x), b = *reinterpret_cast<const __nv_bfloat162*>(&v.y);
  x[0] = __low2float(a); x[1] = __high2float(a); x[2] = __low2float(b); x[3] = __high2float(b);
}

// element e of lane `sub` is element dec_index(sub, e) of the head vector
__device__ __forceinline__ int dec_index(int sub, int e) { return ((e >> 2) * LPK + sub) * 4 + (e & 3); }

// A lane's part of a key (or value) comes through a ring of DEC_STAGES stages in shared memory that only this lane reads and
// writes, so nothing but its own cp.async groups has to be waited for.
constexpr int DEC_STAGES = 4;
template <typename T>
__device__ __forceinline__ void dec_fetch(const T* __restrict__ base, size_t off, int sub, bool there, T* ring) {
#pragma unroll
  for (int c = 0; c < CPL; ++c) {
    const bool valid = there && c * LPK + sub < NCH;
    const int n = valid ? 4 * (int)sizeof(T) : 0;         // 0: nothing is read, zeros are written
    const T* src = base + (valid ? off + (size_t)(c * LPK + sub) * 4 : 0);
    const unsigned dst = (unsigned)__cvta_generic_to_shared(ring + (size_t)c * DEC_WARPS * 32 * 4);
    if (sizeof(T) == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
  }
}
template <typename T>
__device__ __forceinline__ void dec_take(const T* ring, float (&x)[EPL]) {
#pragma unroll
  for (int c = 0; c < CPL; ++c) load4(ring + (size_t)c * DEC_WARPS * 32 * 4, &x[c * 4]);
}
constexpr size_t DEC_RING = (size_t)DEC_STAGES * 2 * CPL * DEC_WARPS * 32 * 4;      // elements

// Share z of n_splits of n keys: [begin, end) of their numbers.
__device__ __forceinline__ void share_of(int n, int n_splits, int z, int& begin, int& end) {
  const int per = (n + n_splits - 1) / n_splits;
  begin = min(n, z * per);
  end = min(n, begin + per);
}

// OPTS: any of window, slopes, chunk, softcap and keep; without them the loop has only the causal mask.
template <typename T, bool OPTS>
__global__ void __launch_bounds__(DEC_WARPS * 32, 2) attention_simt_decode_kernel(
    const T* __restrict__ qkv, int q_stride, const T* __restrict__ kc, const T* __restrict__ vc,
    const int* __restrict__ block_table, int bt_width, const int* __restrict__ cu_q, const int* __restrict__ kv_len, int H,
    int Hkv, int ps, int num_pages, float scale, int window, T* __restrict__ out, const float* __restrict__ slopes, int chunk,
    float softcap, const float* __restrict__ sinks, int keep, float* __restrict__ part_o, float* __restrict__ part_ml) {
  extern __shared__ float smem[];
  float* Qs = smem;                                        // [16][D]
  float* Om = Qs + 16 * D;                                 // [DEC_STREAMS][DEC_ROWS][LPK * EPL]
  float* MLm = Om + DEC_STREAMS * DEC_ROWS * LPK * EPL;    // [DEC_STREAMS][DEC_ROWS][2]
  T* ring = reinterpret_cast<T*>(MLm + DEC_STREAMS * DEC_ROWS * 2) + threadIdx.x * 4;      // [stage][key, value][CPL][thread][4]
  constexpr int HALF = CPL * DEC_WARPS * 32 * 4, STAGE = 2 * HALF;
  const int r = blockIdx.y, hk = blockIdx.x;
  const int q0 = cu_q[r], qn = cu_q[r + 1] - q0;
  const int G = H / Hkv;
  const int M = qn * G;
  if (M > 16 || M <= 0) return;                     // the tile kernel takes this request
  const int L = kv_len[r];
  const int p0 = L - qn;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gk = lane / LPK, sub = lane - gk * LPK;
  const int stream = warp * KPW + gk;
  for (int w = tid; w < M * D; w += DEC_WARPS * 32) {
    const int row = w / D, d = w - row * D;
    const int tok = row / G, hd = hk * G + (row - tok * G);
    Qs[w] = to_float(qkv[(size_t)(q0 + tok) * q_stride + (size_t)hd * D + d]) * scale;
  }
  __syncthreads();
  const int* bt = block_table + (size_t)r * bt_width;
  const int ps_shift = (ps & (ps - 1)) == 0 ? __ffs(ps) - 1 : -1;
  for (int m0 = 0; m0 < M; m0 += DEC_ROWS) {
    float q[DEC_ROWS][EPL], acc[DEC_ROWS][EPL], m_run[DEC_ROWS], l_run[DEC_ROWS];
    int pos[DEC_ROWS], first_key[DEC_ROWS];
    float slope[DEC_ROWS];
#pragma unroll
    for (int i = 0; i < DEC_ROWS; ++i) {
      const bool valid = m0 + i < M;
      pos[i] = valid ? p0 + (m0 + i) / G : -1;
      first_key[i] = (OPTS && valid && chunk > 0) ? (pos[i] / chunk) * chunk : 0;
      slope[i] = (OPTS && valid && slopes) ? slopes[hk * G + (m0 + i) % G] : 0.f;
      m_run[i] = -INFINITY;
      l_run[i] = 0.f;
#pragma unroll
      for (int e = 0; e < EPL; ++e) {
        q[i][e] = (valid && dec_index(sub, e) < D) ? Qs[(m0 + i) * D + dec_index(sub, e)] : 0.f;
        acc[i][e] = 0.f;
      }
    }
    const int last_row = min(m0 + DEC_ROWS, M) - 1;
    int lo = OPTS && window > 0 ? max(0, p0 + m0 / G - window + 1) : 0;
    if (OPTS && chunk > 0) lo = max(lo, ((p0 + m0 / G) / chunk) * chunk);
    const int hi = p0 + last_row / G + 1;             // exclusive; <= L
    // where a key lies
    auto locate = [&](int key, size_t& off) -> bool {
      if (key >= hi) return false;
      const int blk = ps_shift >= 0 ? key >> ps_shift : key / ps;
      const int page = blk < bt_width ? bt[blk] : -1;
      if (page < 0 || page >= num_pages) return false;          // (a missing page: nothing to read)
      off = (((size_t)page * Hkv + hk) * ps + (key - blk * ps)) * D;
      return true;
    };
    // The keys a stream walks are numbered without the gap between the kept first keys and the window: number n is key
    // n below keep_end and key n - keep_end + lo from there on.
    const int keep_end = OPTS ? min(keep, lo) : 0;
    auto key_of = [&](int n) { return !OPTS || n < keep_end ? n : n - keep_end + lo; };
    // this block's share of the numbers (gridDim.z shares; a stream's first number may lie beyond it)
    int begin, end;
    share_of(keep_end + max(0, hi - lo), gridDim.z, blockIdx.z, begin, end);
    unsigned found = 0;                               // bit u: the key u stages ahead of this one has a page
    int ahead = begin + stream;
    auto fetch = [&](int stage) {
      size_t off = 0;
      const bool there = ahead < end && locate(key_of(ahead), off);
      dec_fetch(kc, off, sub, there, ring + (size_t)stage * STAGE);
      dec_fetch(vc, off, sub, there, ring + (size_t)stage * STAGE + HALF);
      asm volatile("cp.async.commit_group;" ::: "memory");
      ahead += DEC_STREAMS;
      return there ? 1u : 0u;
    };
#pragma unroll
    for (int u = 0; u < DEC_STAGES - 1; ++u) found |= fetch(u) << u;
    int stage = 0, number = begin + stream;
    for (int base = begin; base < end; base += DEC_STREAMS, number += DEC_STREAMS, found >>= 1) {
      asm volatile("cp.async.wait_group %0;" ::"n"(DEC_STAGES - 2) : "memory");
      float kv[EPL], vv[EPL];
      dec_take(ring + (size_t)stage * STAGE, kv);
      dec_take(ring + (size_t)stage * STAGE + HALF, vv);
      const bool this_there = found & 1u;
      const int this_key = key_of(number);
      // (the stage that the next fetch fills was read a step ago)
      found |= fetch((stage + DEC_STAGES - 1) % DEC_STAGES) << (DEC_STAGES - 1);
      stage = (stage + 1) % DEC_STAGES;
#pragma unroll
      for (int i = 0; i < DEC_ROWS; ++i) {
        float sc = 0.f;
#pragma unroll
        for (int e = 0; e < EPL; ++e) sc += q[i][e] * kv[e];
#pragma unroll
        for (int o = LPK / 2; o > 0; o >>= 1) sc += __shfl_xor_sync(0xffffffffu, sc, o);
        const bool ok = this_there && this_key <= pos[i] &&
                        (!OPTS || (this_key >= first_key[i] && (window <= 0 || this_key > pos[i] - window || this_key < keep)));
        if (ok) {
          if (OPTS) {
            if (softcap > 0.f) sc = softcap * tanhf(sc / softcap);
            sc -= slope[i] * (float)(pos[i] - this_key);
          }
          if (!(sc <= m_run[i])) {                         // a new maximum (or NaN): what there is so far is scaled down to it
            const float m_new = fmaxf(m_run[i], sc);
            const float alpha = (m_run[i] == -INFINITY) ? 0.f : expf(m_run[i] - m_new);
            l_run[i] *= alpha;
#pragma unroll
            for (int e = 0; e < EPL; ++e) acc[i][e] *= alpha;
            m_run[i] = m_new;
          }
          const float pr = expf(sc - m_run[i]);
          l_run[i] += pr;
#pragma unroll
          for (int e = 0; e < EPL; ++e) acc[i][e] += pr * vv[e];
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int i = 0; i < DEC_ROWS; ++i) {
#pragma unroll
      for (int e = 0; e < EPL; ++e) Om[((size_t)stream * DEC_ROWS + i) * (LPK * EPL) + dec_index(sub, e)] = acc[i][e];
      if (sub == 0) { MLm[(stream * DEC_ROWS + i) * 2] = m_run[i]; MLm[(stream * DEC_ROWS + i) * 2 + 1] = l_run[i]; }
    }
    __syncthreads();
    for (int w = tid; w < DEC_ROWS * D; w += DEC_WARPS * 32) {
      const int i = w / D, d = w - i * D;
      if (m0 + i >= M) continue;
      float mm = -INFINITY;
      for (int st = 0; st < DEC_STREAMS; ++st) mm = fmaxf(mm, MLm[(st * DEC_ROWS + i) * 2]);
      float ll = 0.f, o = 0.f;
      if (sinks != nullptr && part_o == nullptr) {
        const float sk = sinks[hk * G + (m0 + i) % G];
        mm = fmaxf(mm, sk);
        ll = expf(sk - mm);
      }
      for (int st = 0; st < DEC_STREAMS; ++st) {
        const float mw = MLm[(st * DEC_ROWS + i) * 2];
        const float f = (mw == -INFINITY) ? 0.f : expf(mw - mm);
        ll += MLm[(st * DEC_ROWS + i) * 2 + 1] * f;
        o += Om[((size_t)st * DEC_ROWS + i) * (LPK * EPL) + d] * f;
      }
      const int row = m0 + i, tok = row / G, hd = hk * G + (row - tok * G);
      if (part_o != nullptr) {
        const size_t at = (((size_t)r * Hkv + hk) * gridDim.z + blockIdx.z) * 16 + row;
        part_o[at * D + d] = o;
        if (d == 0) { part_ml[2 * at] = mm; part_ml[2 * at + 1] = ll; }
        continue;
      }
      out[(size_t)(q0 + tok) * H * D + (size_t)hd * D + d] = from_float<T>(ll > 0.f ? o / ll : 0.f);
    }
    __syncthreads();
  }
}

// The shares' outputs, sums and maxima put together: grid (kv head, request).
template <typename T>
__global__ void __launch_bounds__(128) attention_simt_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml, int n_splits,
                                                                   const int* __restrict__ cu_q, int H, int Hkv, const float* __restrict__ sinks,
                                                                   T* __restrict__ out) {
  const int r = blockIdx.y, hk = blockIdx.x, G = H / Hkv;
  const int q0 = cu_q[r], M = (cu_q[r + 1] - q0) * G;
  if (M > 16 || M <= 0) return;
  const size_t first = ((size_t)r * Hkv + hk) * n_splits * 16;
  for (int w = threadIdx.x; w < M * D; w += 128) {
    const int row = w / D, d = w - row * D, tok = row / G, hd = hk * G + (row - tok * G);
    float mm = -INFINITY, ll = 0.f, o = 0.f;
    for (int z = 0; z < n_splits; ++z) mm = fmaxf(mm, part_ml[2 * (first + z * 16 + row)]);
    if (sinks != nullptr) {
      mm = fmaxf(mm, sinks[hd]);
      ll = expf(sinks[hd] - mm);
    }
    for (int z = 0; z < n_splits; ++z) {
      const size_t at = first + z * 16 + row;
      const float mz = part_ml[2 * at], f = (mz == -INFINITY) ? 0.f : expf(mz - mm);
      ll += part_ml[2 * at + 1] * f;
      o += part_o[at * D + d] * f;
    }
    out[(size_t)(q0 + tok) * H * D + (size_t)hd * D + d] = from_float<T>(ll > 0.f ? o / ll : 0.f);
  }
}

}  // namespace

SB_EXPORT int sb_attention_simt_head_dim() { return D; }

// Options of the scores: ``slopes`` (float [H] or null), ``chunk`` (0: none), ``softcap`` (0: none), ``sinks`` (float [H] or null)
// and ``keep`` (0: none; with a window: the keys below it stay visible to every later query). ``n_splits`` > 1: the keys of a
// decoding request are shared out over that many blocks; ``scratch`` then holds n_rows * Hkv * n_splits * 16 * (D + 2) floats.
SB_EXPORT int sb_attention_simt_keep(const void* qkv, int q_stride, const void* kc, const void* vc, const int* block_table,
                                     int bt_width, const int* cu_q, const int* kv_len, int H, int Hkv, int ps, int num_pages,
                                     float scale, int window, void* out, int n_rows, int max_q, int dtype, const float* slopes,
                                     int chunk, float softcap, const float* sinks, int keep, int n_splits, float* scratch, cudaStream_t stream) {
  if (n_rows <= 0 || max_q <= 0) return 0;
  if (n_splits < 1 || n_splits > 65535 || (n_splits > 1 && !scratch)) return SB_ERR_SHAPE;
  if (keep < 0 || (keep > 0 && (window <= 0 || chunk > 0))) return SB_ERR_SHAPE;
  if (H <= 0 || Hkv <= 0 || H % Hkv || ps <= 0 || bt_width <= 0) return SB_ERR_SHAPE;
  if (H > 65535 || n_rows > 65535) return SB_ERR_LIMIT;
  const size_t smem = (size_t)(BM * D + BN * KSTRIDE + BN * D + BM * BN) * sizeof(float);
  // Requests with at most 16 rows (tokens x query heads per kv head) go to the decoding shape, the others to the
  // tile kernel; each kernel's blocks leave the other's requests alone. A step of decoded tokens only launches no tiles.
  const int G = H / Hkv;
  const bool decode_shape = G <= 16 && Hkv <= 65535;
  const bool tiles_needed = !decode_shape || (long long)max_q * G > 16;
  dim3 grid((max_q + BM - 1) / BM, H, n_rows);
  dim3 dgrid(Hkv, n_rows, n_splits);
  float* part_o = n_splits > 1 ? scratch : nullptr;
  float* part_ml = n_splits > 1 ? scratch + (size_t)n_rows * Hkv * n_splits * 16 * D : nullptr;
  const bool opts = window > 0 || slopes || chunk > 0 || softcap > 0.f;
  const size_t dsmem = (size_t)(16 * D + DEC_STREAMS * DEC_ROWS * LPK * EPL + DEC_STREAMS * DEC_ROWS * 2) * sizeof(float) +
                       DEC_RING * (dtype == SB_DTYPE_F32 ? 4 : 2);
  if (dtype == SB_DTYPE_F32) {
    if (tiles_needed) {
      auto k = attention_simt_kernel<float>;
      if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      k<<<grid, THREADS, smem, stream>>>((const float*)qkv, q_stride, (const float*)kc, (const float*)vc, block_table, bt_width, cu_q,
                                         kv_len, H, Hkv, ps, num_pages, scale, window, (float*)out, decode_shape ? 1 : 0, slopes, chunk, softcap, sinks, keep);
      SB_LAUNCH_CHECK();
    }
    if (decode_shape) {
      auto kd = opts ? attention_simt_decode_kernel<float, true> : attention_simt_decode_kernel<float, false>;
      if (dsmem > 48 * 1024) cudaFuncSetAttribute(kd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dsmem);
      kd<<<dgrid, DEC_WARPS * 32, dsmem, stream>>>(
          (const float*)qkv, q_stride, (const float*)kc, (const float*)vc, block_table, bt_width, cu_q, kv_len, H, Hkv, ps, num_pages,
          scale, window, (float*)out, slopes, chunk, softcap, sinks, keep, part_o, part_ml);
      if (part_o) {
        SB_LAUNCH_CHECK();
        attention_simt_merge_kernel<float><<<dim3(Hkv, n_rows), 128, 0, stream>>>(part_o, part_ml, n_splits, cu_q, H, Hkv, sinks, (float*)out);
      }
    }
  } else if (dtype == SB_DTYPE_BF16) {
    if (tiles_needed) {
      auto k = attention_simt_kernel<__nv_bfloat16>;
      if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      k<<<grid, THREADS, smem, stream>>>((const __nv_bfloat16*)qkv, q_stride, (const __nv_bfloat16*)kc, (const __nv_bfloat16*)vc,
                                         block_table, bt_width, cu_q, kv_len, H, Hkv, ps, num_pages, scale, window,
                                         (__nv_bfloat16*)out, decode_shape ? 1 : 0, slopes, chunk, softcap, sinks, keep);
      SB_LAUNCH_CHECK();
    }
    if (decode_shape) {
      auto kd = opts ? attention_simt_decode_kernel<__nv_bfloat16, true> : attention_simt_decode_kernel<__nv_bfloat16, false>;
      if (dsmem > 48 * 1024) cudaFuncSetAttribute(kd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dsmem);
      kd<<<dgrid, DEC_WARPS * 32, dsmem, stream>>>(
          (const __nv_bfloat16*)qkv, q_stride, (const __nv_bfloat16*)kc, (const __nv_bfloat16*)vc, block_table, bt_width, cu_q, kv_len, H,
          Hkv, ps, num_pages, scale, window, (__nv_bfloat16*)out, slopes, chunk, softcap, sinks, keep, part_o, part_ml);
      if (part_o) {
        SB_LAUNCH_CHECK();
        attention_simt_merge_kernel<__nv_bfloat16><<<dim3(Hkv, n_rows), 128, 0, stream>>>(part_o, part_ml, n_splits, cu_q, H, Hkv, sinks, (__nv_bfloat16*)out);
      }
    }
  } else {
    return SB_ERR_DTYPE;
  }
  SB_LAUNCH_CHECK();
  return 0;
}
