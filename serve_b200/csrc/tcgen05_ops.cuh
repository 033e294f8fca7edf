// The fifth-generation tensor core's instructions as small inline functions: mbarriers with bounded waits, TMA loads,
// tcgen05 products, commits and accumulator loads, matrix descriptors and the making of tensor maps.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace sb {
namespace tc {

constexpr unsigned WAIT_LIMIT = 1u << 26;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar_addr, unsigned parity) {
  uint32_t done;
  asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(done) : "r"(bar_addr), "r"(parity) : "memory");
  return done != 0;
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, unsigned parity) { return mbar_try(smem_u32(bar), parity); }
// false: the wait ran out (the caller gives up and says so)
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity) {
  const uint32_t addr = smem_u32(bar);
  for (unsigned i = 0; i < WAIT_LIMIT; ++i)
    if (mbar_try(addr, parity)) return true;
  return false;
}
// the same for a whole warp: all lanes get the same answer
__device__ __forceinline__ bool warp_wait(uint64_t* bar, unsigned parity) {
  if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
  return __all_sync(0xffffffffu, mbar_wait(bar, parity)) != 0;
}
__device__ __forceinline__ void load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z, int u) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(u) : "memory");
}
__device__ __forceinline__ void load_5d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z, int u, int v) {
  asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(u), "r"(v) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// 32 lanes x 32 columns of 32-bit accumulator: thread i of the warp gets lane (base lane + i), 32 consecutive columns
// (wait_loads() before the registers are used). The instruction is the warp's: lanes that a branch before it has parted meet first, or
// (_met) have just met and taken no branch of their own since.
__device__ __forceinline__ void load32_met(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void load32_met(uint32_t taddr, float* r) { load32_met(taddr, reinterpret_cast<uint32_t*>(r)); }
template <typename T>
__device__ __forceinline__ void load32(uint32_t taddr, T* r) {
  __syncwarp();
  load32_met(taddr, r);
}
__device__ __forceinline__ void wait_loads() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor, 128-byte swizzle: rows of 128 bytes, 8 rows to a 1024-byte atom, atoms one after the
// other (stride 1024 bytes); version 1, layout type 2; a K-major operand. Its upper half is the same for all tiles, its lower half the
// address in units of 16 bytes: the thread that issues the products only ever adds to a 32-bit number instead of making a descriptor
// anew for each.
constexpr uint32_t DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t desc_lo(uint32_t smem_addr) { return (smem_addr & 0x3FFFF) >> 4; }
// ... of an MN-major operand: ``lbo``, the distance between 64-element swizzle atoms along the non-k dimension
__device__ __forceinline__ uint32_t desc_lo(uint32_t smem_addr, uint32_t lbo_bytes) { return desc_lo(smem_addr) | (lbo_bytes >> 4) << 16; }
__device__ __forceinline__ void mma_lo(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 a, b;\n mov.b64 a, {%1, %5};\n mov.b64 b, {%2, %5};\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n}\n"
      ::"r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(DESC_HI) : "memory");
}
__device__ __forceinline__ void mma_pair_lo(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 a, b;\n mov.b64 a, {%1, %5};\n mov.b64 b, {%2, %5};\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, p;\n}\n"
      ::"r"(tmem_d), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(DESC_HI) : "memory");
}
// One thread of a warp that has come together, always the same one. Loops that issue copies and products are walked by a whole warp and
// their instructions issued behind this: the compiler then knows that addresses and counters are equal in all lanes. From one
// thread of a divergent warp every such instruction cost its issuer more than a hundred cycles.
__device__ __forceinline__ bool elect_one() {
  uint32_t yes;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(yes));
  return yes != 0;
}

// kind::f16 instruction descriptor: float accumulator, bfloat16 a and b, N x M of the tile; a K-major, and b too unless its non-k dimension
// is the contiguous one in shared memory (values: rows are keys, head elements contiguous)
__host__ __device__ constexpr uint32_t make_idesc(int m, int n, bool b_mn_major = false) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static inline EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    return cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess ? (EncodeTiledFn)p : (EncodeTiledFn) nullptr;
  }();
  return fn;
}

// bfloat16, ``rank`` dimensions, the innermost first (strides in elements, of the outer ones); 128-byte swizzle, zeros outside
static inline int make_map(CUtensorMap* map, const void* base, int rank, const uint64_t* dims, const uint64_t* strides, const uint32_t* box) {
  EncodeTiledFn encode = encode_fn();
  if (!encode) return -300;
  cuuint64_t d[5], st[4];
  cuuint32_t b[5], one[5] = {1, 1, 1, 1, 1};
  for (int i = 0; i < rank; ++i) { d[i] = dims[i]; b[i] = box[i]; }
  for (int i = 0; i + 1 < rank; ++i) st[i] = strides[i] * 2;
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base), d, st, b, one,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -301 - (int)r;
}

// rows x cols, rows ``stride`` elements apart; box of box_rows x 64 columns
static inline int make_map_2d(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t stride, uint32_t box_rows) {
  const uint64_t dims[2] = {cols, rows}, strides[1] = {stride};
  const uint32_t box[2] = {64, box_rows};
  return make_map(map, base, 2, dims, strides, box);
}

}  // namespace tc
}  // namespace sb
