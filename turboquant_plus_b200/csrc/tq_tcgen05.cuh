// Fifth-generation tensor cores (tcgen05): descriptors, tensor-memory loads and stores, bounded mbarrier waits.
#pragma once
#include <cuda.h>
#include "tq_internal.cuh"

namespace {

// cuTensorMapEncodeTiled for a matrix of `rows` rows of `columns` elements, `pitch` bytes apart, in boxes of box_columns (128 bytes) x box_rows,
// 128-byte swizzle; false where no such map can be made
inline bool tc_map(CUtensorMap* map, CUtensorMapDataType type, const void* x, int64_t columns, int64_t rows, int64_t pitch, int box_columns, int box_rows) {
  using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                              const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static const Encode encode = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess) {
      (void)cudaGetLastError();
      p = nullptr;
    }
    return reinterpret_cast<Encode>(p);
  }();
  if (!encode || rows > 0x7fffff00LL) return false;   // (box coordinates are 32-bit)
  const cuuint64_t dims[2] = {(cuuint64_t)columns, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)pitch};
  const cuuint32_t box[2] = {(cuuint32_t)box_columns, (cuuint32_t)box_rows}, ones[2] = {1, 1};
  return encode(map, type, 2, const_cast<void*>(x), dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

constexpr long long TC_WAIT_CYCLES = 1LL << 30;

__device__ __forceinline__ uint32_t sptr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool tc_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  // the hint lets the hardware keep the thread suspended for up to that many nanoseconds before the instruction returns
  // false: a waiting role then spends few issue slots on polling
  asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
               : "=r"(ok) : "r"(sptr(bar)), "r"(parity), "r"(20000u) : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool tc_wait(uint64_t* bar, uint32_t parity) {
  if (tc_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (clock64() - t0 < TC_WAIT_CYCLES)
    if (tc_try_wait(bar, parity)) return true;
  return false;
}

// The wait of a role of a kernel whose roles wait for one another: `failed`, in shared memory, is set by the first one that gives up
// and ends the waits of all.  The limit is an argument for the self-tests' sake, which make a wait run out.
constexpr long long TC_SELFTEST_CYCLES = 1LL << 20;
__device__ __noinline__ bool tc_wait_on(uint64_t* bar, uint32_t parity, volatile int* failed, long long limit) {
  const long long t0 = clock64();
  while (!*failed) {
    if (tc_try_wait(bar, parity)) return true;
    if (clock64() - t0 > limit) *failed = 1;
  }
  return false;
}
// (the polls are a function of their own: inlined at every wait, they made the dense quantizer with a sketch 0.5 % slower, appends 1 %)
__device__ __forceinline__ bool tc_wait(uint64_t* bar, uint32_t parity, volatile int* failed, long long limit) {
  return tc_try_wait(bar, parity) || tc_wait_on(bar, parity, failed, limit);
}

// shared-memory matrix descriptor, no swizzle: start address, leading-dimension and stride byte offsets (16-byte
// units), descriptor version 1.  K-major operand: LBO = distance between 8-element K chunks, SBO = distance
// between 8-row groups.  MN-major operand: LBO = distance between 8-row K groups, SBO = between 8-element N chunks.
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)((lbo >> 4) & 0x3fff) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3fff) << 32) | ((uint64_t)1 << 46);
}
// instruction descriptor, kind::f16: fp32 accumulator, fp16 A and B, A K-major, B major as given, N, M
__device__ __forceinline__ uint32_t umma_idesc(int m, int n, bool b_mn_major) {
  return (1u << 4) | ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(addr) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// sixteen columns into v[OFF .. OFF + 15], no wait: the caller waits once for all of its loads
template <int OFF, int N>
__device__ __forceinline__ void tmem_ld16_nowait(uint32_t addr, uint32_t (&v)[N]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[OFF]), "=r"(v[OFF + 1]), "=r"(v[OFF + 2]), "=r"(v[OFF + 3]), "=r"(v[OFF + 4]), "=r"(v[OFF + 5]),
        "=r"(v[OFF + 6]), "=r"(v[OFF + 7]), "=r"(v[OFF + 8]), "=r"(v[OFF + 9]), "=r"(v[OFF + 10]), "=r"(v[OFF + 11]),
        "=r"(v[OFF + 12]), "=r"(v[OFF + 13]), "=r"(v[OFF + 14]), "=r"(v[OFF + 15])
      : "r"(addr) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t addr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]),
        "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
        "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]) : "memory");
}

}  // namespace
