// Pieces of the recurrences' tcgen05 kernels (a CTA walks tiles of 128 tokens): bounded barriers, TMA copies, operands and products, tensor memory, and
// numbers in three bfloat16 terms.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "mma_split.cuh"

namespace dli {
namespace umma {

constexpr int SLAB = 128 * 128;  // bytes of 128 rows of 64 bfloat16 numbers, 128-byte swizzle
constexpr unsigned WAIT_LIMIT = 1u << 24;

__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void bar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_done(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done;
}
// Waits for a barrier's phase, `left` polls at most.  When they run out *failed says so, the caller polls once only from then on and goes on to the end;
// nothing is stored behind it.  (A tight loop: the kernel's instructions should stay in the SM's cache.)
__device__ __forceinline__ void bar_wait(uint32_t bar, uint32_t parity, unsigned& left, volatile int* failed, int* error_flag, int code) {
  uint32_t polls;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tmov.u32 %0, %3;\n"
      "AGAIN_%=:\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t@p bra DONE_%=;\n\t"
      "sub.u32 %0, %0, 1;\n\tsetp.ne.u32 q, %0, 0;\n\t@q bra AGAIN_%=;\n"
      "DONE_%=:\n\t}"
      : "=&r"(polls) : "r"(bar), "r"(parity), "r"(left) : "memory");
  if (polls == 0) {
    left = 1;
    if (!*failed) { *failed = code; atomicCAS(error_flag, 0, code); }
  }
  __syncwarp();
}
__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}
// Operand of 128-byte rows in 128-byte swizzle: 1,024 bytes between groups of eight rows; `slab`: bytes between runs of 64 of an operand whose rows are k
__device__ __forceinline__ uint64_t operand(uint32_t addr, int slab = 0) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)(slab >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
// kind::f16: float32 accumulator, bfloat16 operands, M = 128; a_rows_k / b_rows_k: the operand's rows in shared memory are k
__device__ __forceinline__ uint32_t instruction(int n, bool a_rows_k, bool b_rows_k) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_rows_k << 15) | ((uint32_t)b_rows_k << 16) | ((uint32_t)(n >> 3) << 17) | (8u << 24);
}
// Products are issued by one lane of a warp that runs together, so that descriptors stay in uniform registers: by a thread in a branch of its own an
// instruction took 100 to 180 clocks, more than the tensor cores need for it.
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t one;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
  return one;
}
__device__ __forceinline__ void product(uint32_t one, uint32_t sum, uint64_t a, uint64_t b, uint32_t idesc, bool add) {
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 q, %5, 0;\n\tsetp.ne.b32 p, %4, 0;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(sum), "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)add), "r"(one) : "memory");
}
__device__ __forceinline__ void product_tmem(uint32_t one, uint32_t sum, uint32_t a, uint64_t b, uint32_t idesc, bool add) {  // A in tensor memory
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 q, %5, 0;\n\tsetp.ne.b32 p, %4, 0;\n\t@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
               ::"r"(sum), "r"(a), "l"(b), "r"(idesc), "r"((uint32_t)add), "r"(one) : "memory");
}
__device__ __forceinline__ void commit(uint32_t one, uint32_t bar) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar), "r"(one) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&v)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
                 "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
               : "r"(addr));
}
__device__ __forceinline__ void tmem_ld8(uint32_t addr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(addr));
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&v)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
                 "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]));
}
__device__ __forceinline__ void tmem_st4(uint32_t addr, const uint32_t (&v)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void st_shared16(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void ld_shared16(uint32_t addr, uint32_t (&v)[4]) {
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ float lds(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float4 lds4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
// COUNT (1, 4 or 8) sums over the lanes: a lane keeps the half of its numbers that its bit names.  Left in sum[0]: number lane / (32 / COUNT).
template <int COUNT> __device__ __forceinline__ void sum_over_lanes(float (&sum)[COUNT], int lane) {
#pragma unroll
  for (int half = COUNT / 2, bit = 16; half >= 1; half >>= 1, bit >>= 1) {
    const bool upper = (lane & bit) != 0;
#pragma unroll
    for (int c = 0; c < half; ++c) {
      const float give = upper ? sum[c] : sum[c + half], own = upper ? sum[c + half] : sum[c];
      sum[c] = own + __shfl_xor_sync(0xffffffffu, give, bit);
    }
  }
#pragma unroll
  for (int bit = 16 / COUNT; bit >= 1; bit >>= 1) sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], bit);
}
// sixteen numbers in three terms to columns 16 part .. of row r of three slabs
__device__ __forceinline__ void store_terms(uint32_t dst, int term_bytes, int r, int part, const float (&v)[16]) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint32_t t[3][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) split3(v[8 * h + 2 * e], v[8 * h + 2 * e + 1], t[0][e], t[1][e], t[2][e]);
    const uint32_t at = dst + r * 128 + (((2 * part + h) ^ (r & 7)) << 4);
#pragma unroll
    for (int s = 0; s < 3; ++s) st_shared16(at + s * term_bytes, t[s][0], t[s][1], t[s][2], t[s][3]);
  }
}

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline EncodeTiled encode_fn() {
  static EncodeTiled fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess) fn = (EncodeTiled)ptr;
  }
  return fn;
}
// rows x columns numbers of 2 (bfloat16) or 4 (float32) bytes, rows `row` numbers apart, in boxes of box_rows x 128 bytes; zeros outside
inline bool make_map(CUtensorMap* map, const void* base, bool f32, long long rows, long long columns, long long row, int box_rows) {
  EncodeTiled fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)columns, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)row * (f32 ? 4 : 2)};
  cuuint32_t box[2] = {f32 ? 32u : 64u, (cuuint32_t)box_rows}, elem[2] = {1, 1};
  return fn(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, f32 ? CU_TENSOR_MAP_L2_PROMOTION_NONE : CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace umma
}  // namespace dli
