// Dense-rotation quantize and dequantize of d = 128 (fp32 and fp16 rows) in exact integer products on the fifth-generation
// tensor cores.
//
// The dense mode's products are fp64 (turboquant/polar_quant.py:56-119, turboquant/turboquant.py:79-124), and the fp64 units do 64
// multiply-adds per SM and clock where tcgen05.mma.kind::i8 does 8,192.  Both operands are therefore written as fixed-point
// numbers in seven balanced base-256 digits (Ozaki's splitting), value = sum_p a_p 2^(-6 - 8 p), and the products of digits p and q
// with p + q = s are summed exactly, in int32, for s = 0..7: 34 products.  The eight sums are joined in fp64.  Rounding to 2^-55 of
// the largest value and the products left out (s >= 8) together are off by 1.0e-16 of the result's norm (random rotation, rows
// with outlier channels), fp64 sums of 128 terms by 4.9e-16.
//
// What only decides something -- an index, a sign of the sketch -- needs fewer: the leading ten (indices) to 21 products (the sketch) leave a known
// bound out, and what lies within it of a boundary is decided in fp64 (di_index, di_decider, di_rows_plain).  A residual is taken from 21
// products.  Reconstructions are results themselves and take all 34.
//
// One persistent CTA per SM, 128 vectors a tile:
//   warps 0-15 rows: warps w, w + 4, w + 8 and w + 12 share the 32 vectors that are lanes 32 (w & 3) .. of tensor memory, a thread
//              32 columns of a vector (64 in eight warps: their loads of sums waited behind the MMAs' own traffic).  They norm
//              the rows (in NumPy's order), write the digits of the first operand into tensor memory (32 columns a digit, four
//              elements a word) and add up the sums of its product with R: indices, whose centroids' digits are the next
//              operand; then, with the sketch, the residual's digits, and the signs.
//   warp 16    bulk copies of the matrices' digits, 16 KB each (laid out by k_dense_digits).  The sums run from the last to 0, so that
//              digit s of a matrix has been read for the last time after sum s, and the next matrix follows it.  A single matrix stays; the
//              warp then looks after the outputs that are too close to a boundary.
//   warp 17    every MMA: one s of all 128 outputs is an accumulator of 128 columns, of which two take turns.
// Shapes by measurement: an MMA of 128 x N x 32 takes 44 clocks (its issue) for N = 32 and 64, 65 for N = 128.
//
// What bounds quantize: its rows' arithmetic, 12,000 clocks a tile without the sketch (norms 1,300, digits 2,100, sums 4,000, indices 2,600, the rest
// barriers and stores) and 40,000 with it (sums 20,000, of which the MMAs take 13,000; residuals 7,000).  65,536 fp32 vectors, fp64
// tensor cores / all 34 products each / here: 134 / 78 / 33 us, with the sketch 302 / 163 / 90 (105 where a row on a CTA's way is for
// di_rows_plain; about every second call).  di_rows_plain takes 9 us for up to sixteen rows of a tile, with the sketch 16: where every row
// is one for it (copies of a vector with an output that close to a boundary, 65,536 of 3 bits) 83 us with all 34 products / 816 with
// its rows one after the other / 281 now, with the sketch (reconstructions that are quantized again) 168 / 3,600 / 540.
// What bounds dequantize: its rows, 20,000 clocks a tile where the MMAs (88 clocks each under the rows' loads of sums) take 12,000: sums 900 clocks
// each, half of it fp64 additions, the next operand 500 a digit, results 3,700, norms and factors 3,000.  65,536 vectors, fp64 tensor
// cores / all of it behind the last sum / here: 90 / 62 / 56 us, with the sketch 164 / 93 / 85.
//
// A wait that gives up ends the waits of all roles; the results of its tile and of those behind it are then not numbers, and a
// status word is set (tq_quantize_status_sync).
//
// A row that this arithmetic does not carry -- values that are not finite or too small for a norm, residuals far beyond the
// vector's length, which an arbitrary matrix can produce -- is computed by all row threads in plain fp64.
#include <mutex>
#include <type_traits>
#include "tq_tcgen05.cuh"

namespace {

constexpr int DI_DIGITS = 7, DI_SUMS = 8;
constexpr int DI_ROWS = 128, DI_ROW_THREADS = 512, DI_COPIER = 16, DI_MMA = 17, DI_THREADS = 576;
constexpr int DI_COLS = 32;                         // columns of a row thread: four threads a row
constexpr int DI_TILE = TQ_D * TQ_D;                // bytes of one digit of a matrix
constexpr float DI_LARGEST = 1.9f;                  // the leading digit holds 127/64
// tensor memory: the operand (7 x 32 columns), the signs of a sketch (32), two accumulators
constexpr uint32_t DI_SIGNS = 32 * DI_DIGITS, DI_ACC = 256;

template <typename T> __device__ __forceinline__ float di_f(T v) { return (float)v; }
template <> __device__ __forceinline__ float di_f<__half>(__half v) { return __half2float(v); }
template <typename T> __device__ __forceinline__ double di_d(T v) { return (double)v; }
template <> __device__ __forceinline__ double di_d<__half>(__half v) { return (double)__half2float(v); }

__device__ __forceinline__ void di_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sptr(bar)) : "memory");
}
__device__ __forceinline__ void di_arrive_warp(uint64_t* bar, int lane) {
  if (lane == 0) di_arrive(bar);
}
// MMAs and commits are executed by a converged warp, one elected thread of which issues them: addresses and descriptors then live
// in uniform registers (from a branch of one thread an MMA took 115 clocks to issue, not the 65 that it takes to execute)
__device__ __forceinline__ void di_commit(uint64_t* bar) {
  asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n"
               ::"r"(sptr(bar)) : "memory");
}
// D (128 x 128, int32) += A (tensor memory, 128 x 32 int8) B^T (128 x 32 int8)
__device__ __forceinline__ void di_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n .reg .pred p, q;\n elect.sync _|q, 0xffffffff;\n setp.ne.b32 p, %4, 0;\n @q tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n}\n"
               ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
// int32 accumulator, signed int8 operands, both K-major
__device__ __forceinline__ uint32_t di_idesc() { return (2u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24); }

// eight columns, no wait
__device__ __forceinline__ void di_ld8(uint32_t addr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void di_ld8_wait(uint32_t (&v)[8]) {   // (every use of v behind the wait)
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]) :: "memory");
}
__device__ __forceinline__ void di_st2(uint32_t addr, uint32_t a, uint32_t b) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1,%2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}

// value x 2^54 as balanced base-256 digits: byte 6 the leading one (signed), bytes 5..0 the others
__device__ __forceinline__ uint64_t di_digits(long long w) { return (uint64_t)(w + 0x808080808080ll) ^ 0x808080808080ull; }
__device__ __forceinline__ uint2 di_split(uint64_t u) { return make_uint2((uint32_t)u, (uint32_t)(u >> 32)); }
// of an fp64 value below 2 in magnitude: to a whole number of 2^-54 in two steps of a large constant's rounding
__device__ __forceinline__ uint2 di_digits_f64(double v) {
  constexpr double BIG = 6755399441055744.0;                            // 1.5 x 2^52: a sum's low bits are the whole number
  const double hi = fma(v, 4194304.0, BIG);                             // v x 2^22
  const double rest = fma(hi - BIG, -2.384185791015625e-07, v);         // exact
  const double lo = fma(rest, 18014398509481984.0, BIG);                // the rest x 2^54, at most 2^31
  const long long w = (__double_as_longlong(lo) - __double_as_longlong(BIG)) + ((long long)__double2loint(hi) << 32);
  return di_split(di_digits(w));
}
// byte permute by a selector as it is: where the fourth bit of a nibble is set the byte's sign bit is repeated eight times (the intrinsic masks it)
__device__ __forceinline__ uint32_t di_prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}
// byte k of four words -> operand word k of the four elements
__device__ __forceinline__ void di_transpose(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t (&w)[4]) {
  const uint32_t ab = __byte_perm(a, b, 0x5140), cd = __byte_perm(c, d, 0x5140);
  const uint32_t ab2 = __byte_perm(a, b, 0x7362), cd2 = __byte_perm(c, d, 0x7362);
  w[0] = __byte_perm(ab, cd, 0x5410);
  w[1] = __byte_perm(ab, cd, 0x7632);
  w[2] = __byte_perm(ab2, cd2, 0x5410);
  w[3] = __byte_perm(ab2, cd2, 0x7632);
}
// digits of eight consecutive elements -> the operand words of each four of them, the leading COUNT digits, stored at column `col`
// of every digit.  LOW: the byte of the last digit (its low bytes are those of x, the next of y)
template <int COUNT, int LOW> __device__ __forceinline__ void di_store8(uint32_t area, int col, const uint2 (&u)[8]) {
  uint32_t w[COUNT][2];
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    const uint2 a = u[4 * g], b = u[4 * g + 1], c = u[4 * g + 2], d = u[4 * g + 3];
    uint32_t lo[4], hi[4];
    di_transpose(a.x, b.x, c.x, d.x, lo);
    di_transpose(a.y, b.y, c.y, d.y, hi);
#pragma unroll
    for (int p = 0; p < COUNT; ++p) {
      const int byte = LOW + COUNT - 1 - p;
      w[p][g] = byte < 4 ? lo[byte & 3] : hi[byte & 3];
    }
  }
#pragma unroll
  for (int p = 0; p < COUNT; ++p) di_st2(area + 32 * p + col, w[p][0], w[p][1]);
}

// int32 -> double: 2^52 + 2^31 + v has v ^ 0x80000000 in its low word
__device__ __forceinline__ double di_double(uint32_t v) { return __hiloint2double(0x43300000, (int)(v ^ 0x80000000u)) - 4503601774854144.0; }

// Barriers and the way of the roles through them; the row warps and the MMA warp count alike.
struct DiShared {
  uint64_t b_full[DI_DIGITS], b_free[DI_DIGITS], d_full[2], d_free[2], a_ready[2], drained;
  uint32_t tmem;
  volatile int failed;   // a wait gave up: nobody waits any more
};
// SELFTEST: 0, or the product sum of the first CTA that is never reported (di_issue), or DI_LATE, an MMA warp that comes late to every
// operand, or DI_HASTY, a decider whose wait runs out at once; waits are short then
constexpr int DI_LATE = -1, DI_HASTY = -2;
template <int SELFTEST> __device__ __forceinline__ void di_wait(DiShared& s, uint64_t* bar, uint32_t parity) {
  tc_wait(bar, parity, &s.failed, SELFTEST ? TC_SELFTEST_CYCLES : TC_WAIT_CYCLES);
}
__device__ __forceinline__ void di_init(DiShared& s) {
  auto init = [](uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sptr(bar)), "r"(count) : "memory");
  };
  for (int i = 0; i < DI_DIGITS; ++i) init(&s.b_full[i], 1), init(&s.b_free[i], 1);
  for (int i = 0; i < 2; ++i) init(&s.d_full[i], 1), init(&s.d_free[i], DI_ROW_THREADS / 32), init(&s.a_ready[i], DI_ROW_THREADS / 32);
  init(&s.drained, 1);
  s.failed = 0;
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// The row warps.  None of them leaves a tile early (a wait that gave up lets all others pass), so that all come here; whether
// any has seen a failure is agreed on by all.
__device__ __forceinline__ void di_rows_sync() { asm volatile("bar.sync 1, 512;" ::: "memory"); }
__device__ __forceinline__ bool di_rows_any(bool p) {
  uint32_t any;
  asm volatile("{\n .reg .pred a, b;\n setp.ne.b32 a, %1, 0;\n barrier.red.or.pred b, 1, 512, a;\n selp.u32 %0, 1, 0, b;\n}\n"
               : "=r"(any) : "r"((uint32_t)p) : "memory");
  return any != 0;
}

// The copier's way: the digits of the matrices that `matrix(i)` gives, the leading count(i) of each, from the last to the first, each
// into the place of the matrix before.  uses(i, p): how many of the matrices before i had a digit p
template <int SELFTEST, typename M, typename C, typename U>
__device__ __forceinline__ void di_copier(DiShared& s, uint8_t* tiles, int matrices, M&& matrix, C&& count, U&& uses) {
  int i = 0, p = 0;
  for (; i < matrices && !s.failed; ++i) {
    const uint8_t* src = matrix(i);
    for (p = count(i) - 1; p >= 0; --p) {
      const int before = uses(i, p);
      if (before > 0) di_wait<SELFTEST>(s, &s.b_free[p], (uint32_t)((before - 1) & 1));
      if (s.failed) break;
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sptr(&s.b_full[p])), "r"(DI_TILE) : "memory");
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sptr(tiles + p * DI_TILE)),
                   "l"(src + p * DI_TILE), "r"(DI_TILE), "r"(sptr(&s.b_full[p])) : "memory");
    }
    if (p >= 0) break;   // (a wait gave up in front of digit p)
  }
  for (int q = 0; q < DI_DIGITS; ++q) {   // none in flight at the end, also after a wait that gave up
    const int mine = uses(i, q) + (i < matrices && p >= 0 && q > p && q < count(i) ? 1 : 0);
    if (mine > 0) tc_wait(&s.b_full[q], (uint32_t)((mine - 1) & 1));
  }
}

// The MMA warp: the operand at `area`, of PA digits, against the leading QB digits of a matrix, sums s = LAST to 0 of the products of
// digits p + q = s.  uses(q): the matrices before that had a digit q;
// operand(s): waits for the operand's digits that the sum is the first to take
template <int PA, int QB, int LAST, int SELFTEST, typename U, typename W>
__device__ __forceinline__ void di_issue(DiShared& s, int& item, const uint8_t* tiles, U&& uses, W&& operand, uint32_t area, uint32_t acc_base) {
  const uint32_t b = sptr(tiles), idesc = di_idesc();
#pragma unroll 1
  for (int sum = LAST; sum >= 0; --sum, ++item) {
    const int sl = item & 1;
    for (int q = sum - PA + 1 > 0 ? sum - PA + 1 : 0; q < QB && (sum == LAST || q + PA - 1 == sum); ++q)   // digits used for the first time
      di_wait<SELFTEST>(s, &s.b_full[q], (uint32_t)(uses(q) & 1));
    operand(sum);
    if (item >= 2) di_wait<SELFTEST>(s, &s.d_free[sl], (uint32_t)((item / 2 - 1) & 1));
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int from = sum < QB ? 0 : sum - QB + 1, to = sum < PA ? sum : PA - 1;
#pragma unroll 1
    for (int p = from; p <= to; ++p) {
      const uint64_t desc = umma_desc(b + (sum - p) * DI_TILE, 128, 1024);
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) di_mma(acc_base + 128 * sl, area + 32 * p + 8 * ks, desc + 16 * ks, idesc, p > from || ks > 0 ? 1u : 0u);
    }
    if (!(SELFTEST && blockIdx.x == 0 && item == SELFTEST)) di_commit(&s.d_full[sl]);
    if (sum < QB) di_commit(&s.b_free[sum]);
  }
}

// ... and nothing of its in flight at the end, also after a wait that gave up (else the rows have waited for every product)
__device__ __forceinline__ void di_drain(DiShared& s) {
  if (!__any_sync(0xffffffffu, s.failed)) return;
  __syncwarp();
  di_commit(&s.drained);
  tc_wait(&s.drained, 0);
}

// A row warp waits for a sum, use(column, value) for its 32 columns; frees the accumulator once all are loaded
template <int SELFTEST, typename U>
__device__ __forceinline__ void di_columns(DiShared& s, int item, uint32_t acc_base, int lane, U&& use) {
  const int sl = item & 1;
  di_wait<SELFTEST>(s, &s.d_full[sl], (uint32_t)((item / 2) & 1));
  __syncwarp();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  uint32_t v[2][8];
  di_ld8(acc_base + 128 * sl, v[0]);
#pragma unroll
  for (int c = 0; c < DI_COLS / 8; ++c) {
    di_ld8_wait(v[c & 1]);
    if (c + 1 < DI_COLS / 8) {
      di_ld8(acc_base + 128 * sl + 8 * (c + 1), v[(c + 1) & 1]);
    } else {   // all read
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) di_arrive(&s.d_free[sl]);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) use(8 * c + k, v[c & 1][k]);
  }
}
// The same with all columns at once
template <int SELFTEST>
__device__ __forceinline__ void di_sum(DiShared& s, int& item, uint32_t acc_base, int lane, uint32_t (&v)[32]) {
  const int sl = item & 1;
  di_wait<SELFTEST>(s, &s.d_full[sl], (uint32_t)((item / 2) & 1));
  __syncwarp();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  tmem_ld32(acc_base + 128 * sl, v);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncwarp();
  if (lane == 0) di_arrive(&s.d_free[sl]);
  ++item;
}
// The product's sums s = LAST to 0 (s counts 2^(-12 - 8 s)) as a number of 2^(shift - 44), shift = 15 or 17; what is below is cut off each
// time.  Sums wrap, the result is in range
template <int LAST, int SELFTEST>
__device__ __forceinline__ void di_take32(DiShared& s, int& item, uint32_t acc_base, int lane, int shift, int32_t (&y)[DI_COLS]) {
#pragma unroll
  for (int sum = LAST; sum >= 0; --sum) {
    uint32_t v[32];
    di_sum<SELFTEST>(s, item, acc_base, lane, v);
    const int right = sum == 2 ? shift - 14 : shift - 32 + 8 * sum;
    const uint32_t left = 1u << (32 - 8 * sum - shift & 31);
#pragma unroll
    for (int k = 0; k < DI_COLS; ++k) {
      if (sum >= 2) y[k] = (sum == LAST ? 0 : y[k]) + ((sum == 2 ? (int32_t)(v[k] << 2) : (int32_t)v[k]) >> right);
      else y[k] = (int32_t)((uint32_t)y[k] + v[k] * left);
    }
  }
}
// The product's sums s = 5 to 0 as a number of 2^-44; of s = 5 what is nearest.  (A loop: unrolled, registers spill)
template <int SELFTEST>
__device__ __forceinline__ void di_take64(DiShared& s, int& item, uint32_t acc_base, int lane, long long (&y)[DI_COLS]) {
  di_columns<SELFTEST>(s, item++, acc_base, lane, [&](int k, uint32_t v) { y[k] = ((int32_t)v + 128) >> 8; });
  int32_t weight = 1;
#pragma unroll 1
  for (int sum = 4; sum > 0; --sum, weight <<= 8)
    di_columns<SELFTEST>(s, item++, acc_base, lane, [&](int k, uint32_t v) { y[k] += (long long)(int32_t)v * weight; });
  di_columns<SELFTEST>(s, item++, acc_base, lane, [&](int k, uint32_t v) { y[k] += (long long)((unsigned long long)v << 32); });
}
// A whole number below 2^51 in magnitude as fp64
__device__ __forceinline__ double di_double(long long v) {
  return __longlong_as_double(v + 0x4338000000000000ll) - 6755399441055744.0;
}

// ... for two sums, s and s - 1: of both accumulators 256 times the second plus the first
template <int SELFTEST, typename U>
__device__ __forceinline__ void di_columns2(DiShared& s, int item, uint32_t acc_base, int lane, U&& use) {
  di_wait<SELFTEST>(s, &s.d_full[item & 1], (uint32_t)((item / 2) & 1));
  di_wait<SELFTEST>(s, &s.d_full[(item + 1) & 1], (uint32_t)(((item + 1) / 2) & 1));
  __syncwarp();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t lo = acc_base + 128 * (item & 1), hi = acc_base + 128 * ((item + 1) & 1);
#pragma unroll
  for (int c = 0; c < DI_COLS / 8; ++c) {
    uint32_t v[8], w[8];
    di_ld8(lo + 8 * c, v);
    di_ld8(hi + 8 * c, w);
    di_ld8_wait(v);
    di_ld8_wait(w);
    if (c + 1 == DI_COLS / 8) {   // all read
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) di_arrive(&s.d_free[item & 1]), di_arrive(&s.d_free[(item + 1) & 1]);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) use(8 * c + k, w[k] * 256u + v[k]);
  }
}

// eight consecutive elements of a staged row (16-byte aligned) as fp32
template <typename T> __device__ __forceinline__ void di_load8(const uint8_t* p, float (&f)[8]) {
  if constexpr (sizeof(T) == 4) {
    const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  } else {
    const uint4 a = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&w[k]));
      f[2 * k] = v.x; f[2 * k + 1] = v.y;
    }
  }
}

struct DiQuant {
  const uint8_t *r, *rt, *s;          // digits of R, R^T and S (k_dense_digits)
  double r_scale;                     // sums x this: R w
  double cent_scale;                  // power of two above every centroid's magnitude
  uint2 words[DI_DIGITS];             // digits of the first eight centroids (di_store_codes)
  int32_t thr[15];                    // boundaries over r_scale, as numbers of 2^-27 or 2^-29
  uint32_t near;                      // an output that is closer to one is decided in fp64
  float step, offset[15];             // the same without the sketch (di_index_float)
  int32_t zero_idx;                   // index of the value 0
  int32_t shift;                      // sums of 2^-44 to numbers of the boundaries
  double slack;                       // of a projection, per unit of the reconstruction's factor (di_quant_args)
  float least;                        // elements of a residual that is too short are not above this many 2^-14 of its scale, likewise
  int32_t* status;                    // raised when a wait gives up
  TqDenseQuant q;
};
struct DiDequant {
  const uint8_t *rt, *st;
  uint4 words[DI_DIGITS];             // digits of the sixteen centroids, a byte each
  double r_scale, s_scale, cent_scale;
  int32_t tiled;                      // fp64 results go out by tiled copies
  int32_t* status;
  TqDenseDequant q;
};

// Centroids and boundaries in shared memory
struct DiCodes {
  double cent[16], bnd[16], square[64];   // square: of the centroids of two indices, the sum (3 bits at most), else of one
};
__device__ __forceinline__ int di_search(const DiCodes& c, int bits, double y) {   // boundaries below y (searchsorted, side = 'left')
  int m = 0;
#pragma unroll 1
  for (int b = 0; b < (1 << bits) - 1; ++b) m += c.bnd[b] < y ? 1 : 0;
  return m;
}
// Whole rows in fp64, sixteen at a time, by all row threads on the fp64 tensor cores: a warp has eight outputs of all sixteen.
struct DiPlain {
  static constexpr int PITCH = TQ_D + 8;   // (a load's rows 64 bytes apart modulo 128: no bank conflicts)
  double v[16][PITCH], part[DI_ROW_THREADS / 32][16];
  int row[16];
};
// c = rows g (c0, c1) and g + 8 (c2, c3) of s.v times m, rows of which are outputs: 8 warp + 2 t and the next
__device__ __forceinline__ void di_plain_product(double (&c)[4], const DiPlain& s, const double* __restrict__ m, int tid) {
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const double2* row = reinterpret_cast<const double2*>(m + (size_t)(8 * warp + g) * TQ_D + 2 * t);
  double2 b[8];   // (eight loads in flight; with sixteen the function's registers cost its callers theirs)
#pragma unroll
  for (int k = 0; k < 8; ++k) b[k] = __ldg(row + 4 * k);
  c[0] = c[1] = c[2] = c[3] = 0.0;
#pragma unroll
  for (int k = 0; k < 16; ++k) {   // slots t and t + 4 of a step carry elements 8 k + 2 t and the next
    const double2 lo = *reinterpret_cast<const double2*>(&s.v[g][8 * k + 2 * t]), hi = *reinterpret_cast<const double2*>(&s.v[g + 8][8 * k + 2 * t]);
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3]) : "d"(lo.x), "d"(hi.x), "d"(lo.y), "d"(hi.y), "d"(b[k & 7].x), "d"(b[k & 7].y));
    if (k < 8) b[k] = __ldg(row + 4 * (k + 8));
  }
}
// this warp's part of a sum over the outputs of rows g and g + 8, and the sums of all warps behind a barrier
__device__ __forceinline__ void di_plain_part(DiPlain& s, double lo, double hi, int tid) {
  const int lane = tid & 31, warp = tid >> 5;
  lo += __shfl_xor_sync(0xffffffffu, lo, 1);
  hi += __shfl_xor_sync(0xffffffffu, hi, 1);
  lo += __shfl_xor_sync(0xffffffffu, lo, 2);
  hi += __shfl_xor_sync(0xffffffffu, hi, 2);
  if ((lane & 3) == 0) s.part[warp][lane >> 2] = lo, s.part[warp][8 + (lane >> 2)] = hi;
}
__device__ __forceinline__ double di_plain_sum(const DiPlain& s, int r) {
  double sum = 0.0;
#pragma unroll
  for (int w = 0; w < DI_ROW_THREADS / 32; ++w) sum += s.part[w][r];
  return sum;
}
template <typename Tin>
__device__ __noinline__ void di_rows_plain(DiPlain& s, const TqDenseQuant& a, const DiCodes& c, const uint8_t* plain, const float* norms, const Tin* x,
                                           int64_t ld, int64_t v0, int64_t n, int tid) {
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3, out = 8 * warp + 2 * t;
  uint32_t in[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) in[j] = __ballot_sync(0xffffffffu, plain[32 * j + lane] && v0 + 32 * j + lane < n);
  unsigned long long lo = in[0] | (unsigned long long)in[1] << 32, hi = in[2] | (unsigned long long)in[3] << 32;
#pragma unroll 1
  while (lo | hi) {
    int mine = -1;   // this warp's row
#pragma unroll 1
    for (int k = 0; k < 16; ++k) {
      const int r = lo ? __ffsll(lo) - 1 : hi ? 63 + __ffsll(hi) : -1;
      if (lo) lo &= lo - 1;
      else hi &= hi - 1;
      if (k == warp) mine = r;
    }
    di_rows_sync();   // (the rows before have been read)
    if (lane == 0) s.row[warp] = mine;
    const float norm = mine >= 0 ? norms[mine] : 0.f, safe = norm > 0.f ? norm : 1.0f;
#pragma unroll
    for (int k = lane; k < TQ_D; k += 32) s.v[warp][k] = mine >= 0 ? (double)((float)di_d<Tin>(x[(v0 + mine) * ld + k]) / safe) : 0.0;
    di_rows_sync();
    const int row[2] = {s.row[g], s.row[g + 8]};
    double y[4];
    di_plain_product(y, s, a.rot, tid);
    int m[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) m[i] = di_search(c, a.bits, y[i]);
#pragma unroll
    for (int q = 0; q < 2; ++q)
      if (row[q] >= 0 && a.out_idx) *reinterpret_cast<uint16_t*>(a.out_idx + (v0 + row[q]) * TQ_D + out) = (uint16_t)(m[2 * q] | m[2 * q + 1] << 8);
    di_plain_part(s, c.cent[m[0]] * c.cent[m[0]] + c.cent[m[1]] * c.cent[m[1]], c.cent[m[2]] * c.cent[m[2]] + c.cent[m[3]] * c.cent[m[3]], tid);
    di_rows_sync();
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      double cn = sqrt(di_plain_sum(s, g + 8 * q));
      cn = cn > 1e-10 ? cn : 1.0;
      if (tid < 32 && t == 0 && row[q] >= 0) {
        const float nrm = norms[row[q]];
        if (a.out_norm) a.out_norm[v0 + row[q]] = nrm;
        if (a.out_scale) a.out_scale[v0 + row[q]] = (float)(a.norm_correction ? (double)nrm / cn : (double)nrm);
      }
      const double inv = a.norm_correction ? 1.0 / cn : 1.0;
      *reinterpret_cast<double2*>(&s.v[g + 8 * q][out]) = make_double2(c.cent[m[2 * q]] * inv, c.cent[m[2 * q + 1]] * inv);
    }
    if (!a.out_qjl && !a.out_rnorm) continue;
    di_rows_sync();
    di_plain_product(y, s, a.rot_t, tid);
    double e[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = row[i >> 1];
      e[i] = r >= 0 ? (double)(float)di_d<Tin>(x[(v0 + r) * ld + out + (i & 1)]) - y[i] * (double)norms[r] : 0.0;
    }
    di_plain_part(s, e[0] * e[0] + e[1] * e[1], e[2] * e[2] + e[3] * e[3], tid);
    di_rows_sync();
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      *reinterpret_cast<double2*>(&s.v[g + 8 * q][out]) = make_double2(e[2 * q], e[2 * q + 1]);
      if (tid < 32 && t == 0 && row[q] >= 0 && a.out_rnorm) a.out_rnorm[v0 + row[q]] = (float)sqrt(di_plain_sum(s, g + 8 * q));
    }
    if (!a.out_qjl) continue;
    di_rows_sync();
    di_plain_product(y, s, a.s, tid);
#pragma unroll
    for (int q = 0; q < 2; ++q) {   // (first output in the most significant bit)
      uint32_t z = (y[2 * q] < 0.0 ? 0u : 2u) << (6 - 2 * t) | (y[2 * q + 1] < 0.0 ? 0u : 1u) << (6 - 2 * t);
      z |= __shfl_xor_sync(0xffffffffu, z, 1);
      z |= __shfl_xor_sync(0xffffffffu, z, 2);
      if (t == 0 && row[q] >= 0) a.out_qjl[(v0 + row[q]) * 16 + warp] = (uint8_t)z;
    }
  }
}
template <typename T> __device__ __forceinline__ T di_from(double v) { return (T)v; }
template <> __device__ __forceinline__ __half di_from<__half>(double v) { return __float2half_rn((float)v); }
// A wait gave up: the results of this CTA's tiles from `t` on are not to come.  (Functions of their own: inlined, they cost the kernels registers.)
__device__ __noinline__ void di_give_up(const TqDenseQuant& a, int t, int mine, int row, int64_t n, int32_t* status) {
  const float nan = __int_as_float(0x7fffffff);
  for (; t < mine; ++t) {
    const int64_t v = (blockIdx.x + (int64_t)t * gridDim.x) * DI_ROWS + row;
    if (row < 0 || v >= n) continue;
    if (a.out_norm) a.out_norm[v] = nan;
    if (a.out_scale) a.out_scale[v] = nan;
    if (a.out_rnorm) a.out_rnorm[v] = nan;
  }
  if (status) *status = 1;
}
template <typename Tout> __device__ __noinline__ void di_give_up(const TqDenseDequant& a, int t, int mine, int row, int col, int64_t n, Tout* out, int32_t* status) {
  for (; t < mine; ++t) {
    const int64_t v = (blockIdx.x + (int64_t)t * gridDim.x) * DI_ROWS + row;
    for (int k = 0; k < DI_COLS && v < n; ++k) out[v * a.ld_out + col + k] = di_from<Tout>(__longlong_as_double(0x7ff8000000000000ll));
  }
  if (status) *status = 1;
}

template <typename Tin> constexpr int di_row_bytes() { return TQ_D * (int)sizeof(Tin) + 16; }   // (rows 4 banks apart: no conflicts)
// digits of a matrix in shared memory: of R in place for all tiles, or of R, R^T and S in turn
template <bool PROD> constexpr int di_quant_digits() { return PROD ? 6 : 4; }
template <typename Tin, bool PROD> constexpr int di_quant_smem() {
  return di_quant_digits<PROD>() * DI_TILE + DI_ROWS * di_row_bytes<Tin>() + 128 + (int)sizeof(DiPlain);
}

// Operand words of four indices below 8 (one a byte): a byte permute of eight digits picks a digit of all four.  words[p]: the digit p of
// centroids 0-3, 4-7
template <int COUNT> __device__ __forceinline__ void di_store_codes(uint32_t area, int col, const uint2 (&words)[DI_DIGITS], uint32_t q0, uint32_t q1) {
  const uint32_t s0 = __byte_perm(q0 | (q0 >> 4), 0, 0x4420), s1 = __byte_perm(q1 | (q1 >> 4), 0, 0x4420);
#pragma unroll
  for (int p = 0; p < COUNT; ++p) di_st2(area + 32 * p + col, di_prmt(words[p].x, words[p].y, s0), di_prmt(words[p].x, words[p].y, s1));
}

// R, R^T and S with 5, 6 and 6 digits, in turn: those among the first i matrices that have a digit p
__device__ __forceinline__ int di_uses(int i, int p) { return p < 5 ? i : p == 5 ? i - (i + 2) / 3 : 0; }

// Index of y: the boundaries below it, found bit by bit; near: the least distance of y + reach above one of those compared (the two
// next to y are among them), as an unsigned number: at most 2 `reach` if y is within `reach` of one
template <int BITS> __device__ __forceinline__ uint32_t di_index(const int32_t (&thr)[15], uint32_t reach, int32_t y, uint32_t& near) {
  const uint32_t yn = (uint32_t)y + reach;
  auto above = [&](int32_t t) {
    near = min(near, yn - (uint32_t)t);
    return y > t;
  };
  if constexpr (BITS == 1) {
    return above(thr[0]) ? 1u : 0u;
  } else if constexpr (BITS == 2) {
    const bool b1 = above(thr[1]), b0 = above(b1 ? thr[2] : thr[0]);
    return (b1 ? 2u : 0u) + (b0 ? 1u : 0u);
  } else if constexpr (BITS == 3) {
    const bool b2 = above(thr[3]), b1 = above(b2 ? thr[5] : thr[1]), b0 = above(b2 ? (b1 ? thr[6] : thr[4]) : (b1 ? thr[2] : thr[0]));
    return (b2 ? 4u : 0u) + (b1 ? 2u : 0u) + (b0 ? 1u : 0u);
  } else {
    const bool b3 = above(thr[7]), b2 = above(b3 ? thr[11] : thr[3]);
    const bool b1 = above(b3 ? (b2 ? thr[13] : thr[9]) : (b2 ? thr[5] : thr[1]));
    const bool b0 = above(b3 ? (b2 ? (b1 ? thr[14] : thr[12]) : (b1 ? thr[10] : thr[8])) : (b2 ? (b1 ? thr[6] : thr[4]) : (b1 ? thr[2] : thr[0])));
    return (b3 ? 8u : 0u) + (b2 ? 4u : 0u) + (b1 ? 2u : 0u) + (b0 ? 1u : 0u);
  }
}

// The same on the fp32 pipe: a boundary is a ramp from 0 to 1 over the values too close to it, the index the ramps' sum, in the low byte
// of the result; frac, at most 1/2: how far from a whole number.  Integer compares and selects, at half the rate, took 4,600 clocks of a
// tile's 14,300 with eight centroids.
template <int BITS> __device__ __forceinline__ uint32_t di_index_float(const DiQuant& A, int32_t y, float& frac) {
  const float z = (float)y;
  float m = 0.f;
#pragma unroll
  for (int b = 0; b < (1 << BITS) - 1; ++b) {
    const float ramp = __saturatef(fmaf(z, A.step, A.offset[b]));
    m = b == 0 ? ramp : m + ramp;
  }
  const float whole = m + 12582912.f;                          // 1.5 x 2^23
  frac = fmaxf(frac, fabsf(m - (whole - 12582912.f)));
  return __float_as_uint(whole);
}

// Outputs that are too close to a boundary, eight neighbouring columns an entry: the row warps add them once the indices are stored, the
// copier's warp, which has nothing else to do by then, decides them in fp64.  (By the row warps themselves, whose code for it is not in the
// instruction caches, a check cost 3 to 4 us, and some CTA of a large call had several.)  A random tile has less than one; where there are
// more than the ring holds, whole rows sixteen at a time are faster than one warp.
struct DiList {
  static constexpr int ROOM = 32;
  static constexpr uint32_t NONE = 0xffffffffu;
  volatile uint32_t entry[ROOM];   // in turn; row, column / 8 from bit 7, tile of the CTA from bit 11 on; written last
  float norm[ROOM];
  int count;                       // entries so far
  volatile int taken;              // ... of which the decider has read this many
  volatile int closed;             // no more to come
};
// One more, unless there is no room: the row is then for di_rows_plain
__device__ __forceinline__ bool di_add(DiList& list, uint32_t entry, float norm) {
  int at = *reinterpret_cast<volatile int*>(&list.count);
  while (at - list.taken < DiList::ROOM) {   // (another turn only where another thread has added one)
    const int seen = atomicCAS(&list.count, at, at + 1);
    if (seen == at) {
      __threadfence_block();
      list.norm[at % DiList::ROOM] = norm;
      __threadfence_block();
      list.entry[at % DiList::ROOM] = entry;
      return true;
    }
    at = seen;
  }
  return false;
}
// Indices of eight outputs of a row in fp64, by one warp: four lanes a column, 32 elements each, every load in flight
template <typename Tin>
__device__ __forceinline__ int di_check8(const TqDenseQuant& a, const DiCodes& c, const Tin* x, float nrm, int column, int lane) {
  const double2* r = reinterpret_cast<const double2*>(a.rot + (size_t)(column + (lane >> 2)) * TQ_D + 32 * (lane & 3));
  const uint8_t* xr = reinterpret_cast<const uint8_t*>(x + 32 * (lane & 3));
  const float inv = 1.0f / nrm;
  double2 rk[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) rk[k] = __ldg(r + k);
  double y = 0.0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float f[8];
    di_load8<Tin>(xr + 8 * k * sizeof(Tin), f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float w = f[j] * inv;
      w = fmaf(fmaf(-w, nrm, f[j]), inv, w);
      y = fma(j & 1 ? rk[4 * k + j / 2].y : rk[4 * k + j / 2].x, (double)w, y);
    }
  }
  y += __shfl_xor_sync(0xffffffffu, y, 1);
  y += __shfl_xor_sync(0xffffffffu, y, 2);
  return di_search(c, a.bits, y);
}
template <typename Tin, int SELFTEST>
__device__ __forceinline__ void di_decider(DiShared& s, DiList& list, const TqDenseQuant& a, const DiCodes& c, const Tin* x, int64_t ld, int lane,
                                           int32_t* status) {
  constexpr long long LIMIT = SELFTEST == DI_HASTY ? 0 : TC_WAIT_CYCLES;
  int done = 0;
  long long since = clock64();
#pragma unroll 1
  while (true) {
    const bool last = list.closed != 0;
    const uint32_t e = list.entry[done % DiList::ROOM];
    if (__any_sync(0xffffffffu, e == DiList::NONE)) {
      if (__any_sync(0xffffffffu, last)) break;
      if (__any_sync(0xffffffffu, clock64() - since > LIMIT)) {   // a wait as any other: what the rows still add is not decided
        if (lane == 0) {
          s.failed = 1;
          if (status) *status = 1;   // (the rows may have agreed on the end already)
        }
        break;
      }
      __nanosleep(100);
      continue;
    }
    since = clock64();
    __threadfence_block();
    const float nrm = list.norm[done % DiList::ROOM];
    __syncwarp();
    ++done;
    if (lane == 0) {
      list.entry[(done - 1) % DiList::ROOM] = DiList::NONE;
      __threadfence_block();
      list.taken = done;
    }
    const int64_t v = (blockIdx.x + (int64_t)(e >> 11) * gridDim.x) * DI_ROWS + (e & 127);
    const int column = 8 * ((e >> 7) & 15) + (lane >> 2);
    const int m = di_check8<Tin>(a, c, x + v * ld, nrm, 8 * ((e >> 7) & 15), lane);
    if ((lane & 3) == 0) a.out_idx[v * TQ_D + column] = (uint8_t)m;
  }
}

// PROD: residual, its norm and the sketch as well.  SELFTEST: see di_wait
template <typename Tin, int BITS, bool PROD, int SELFTEST = 0>
__global__ void __launch_bounds__(DI_THREADS, 1) k_dense_quantize_i8(const __grid_constant__ DiQuant A, const Tin* __restrict__ x, int64_t ld,
                                                                     int64_t n) {
  constexpr int ROWB = di_row_bytes<Tin>();
  extern __shared__ __align__(128) uint8_t di_raw[];
  __shared__ DiShared sh;
  __shared__ uint2 s_cdig[16];                  // digits of the centroids
  __shared__ DiCodes s_codes;
  __shared__ std::conditional_t<PROD, int, DiList> s_list;
  DiPlain& s_rows = *reinterpret_cast<DiPlain*>(di_raw + di_quant_smem<Tin, PROD>() - sizeof(DiPlain));
  __shared__ double s_part[4][DI_ROWS];
  __shared__ float s_norms[2][DI_ROWS];         // of two tiles in turn
  __shared__ uint8_t s_plains[2][DI_ROWS];      // rows for di_rows_plain
  const TqDenseQuant& a = A.q;
  uint8_t* tiles_b = di_raw + (((sptr(di_raw) + 127u) & ~127u) - sptr(di_raw));
  uint8_t* xs = tiles_b + di_quant_digits<PROD>() * DI_TILE;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) di_init(sh);
  if (tid < 16) {
    const double c = tid < (1 << BITS) ? a.cent[tid] : 0.0;
    s_codes.cent[tid] = c;
    s_codes.bnd[tid] = tid < (1 << BITS) - 1 ? a.bnd[tid] : 0.0;
    s_cdig[tid] = di_digits_f64(c / A.cent_scale);
  } else if (tid >= 32 && tid < 96) {
    const int i = tid - 32, lo = BITS < 4 ? i & 7 : i & 15, hi = BITS < 4 ? i >> 3 : 16;
    const double c0 = lo < (1 << BITS) ? a.cent[lo] : 0.0, c1 = hi < (1 << BITS) ? a.cent[hi] : 0.0;
    s_codes.square[i] = c0 * c0 + c1 * c1;
  }
  if constexpr (!PROD) {
    if (tid < DiList::ROOM) s_list.entry[tid] = DiList::NONE;
    if (tid == 0) s_list.count = 0, s_list.taken = 0, s_list.closed = 0;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sptr(&sh.tmem)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tb = sh.tmem;
  const int64_t tiles = (n + DI_ROWS - 1) / DI_ROWS, step = gridDim.x;
  const int mine = (int)((tiles - blockIdx.x + step - 1) / step);

  if (warp == DI_COPIER) {
    if (lane == 0) {
      if constexpr (PROD)
        di_copier<SELFTEST>(sh, tiles_b, 3 * mine, [&](int i) { return i % 3 == 0 ? A.r : i % 3 == 1 ? A.rt : A.s; },
                            [](int i) { return i % 3 == 0 ? 5 : 6; },
                            [](int i, int p) { return di_uses(i, p); });
      else
        di_copier<SELFTEST>(sh, tiles_b, mine > 0 ? 1 : 0, [&](int) { return A.r; }, [](int) { return 4; }, [](int i, int p) { return p < 4 ? i : 0; });
    }
    if constexpr (!PROD) {
      __syncwarp();
      di_decider<Tin, SELFTEST>(sh, s_list, a, s_codes, x, ld, lane, A.status);
    }
  } else if (warp == DI_MMA) {
    int item = 0, operands = 0;
    for (int i = 0; i < mine && !__any_sync(0xffffffffu, sh.failed); ++i) {
      if (SELFTEST == DI_LATE)
        for (const long long t0 = clock64(); clock64() - t0 < 1 << 16;) {}
      if constexpr (!PROD) {
        di_wait<SELFTEST>(sh, &sh.a_ready[i & 1], (uint32_t)((i >> 1) & 1));
        di_issue<4, 4, 3, SELFTEST>(sh, item, tiles_b, [](int) { return 0; }, [](int) {}, tb + 128 * (i & 1), tb + DI_ACC);
      } else {
        di_wait<SELFTEST>(sh, &sh.a_ready[0], (uint32_t)(operands++ & 1));
        di_issue<4, 5, 4, SELFTEST>(sh, item, tiles_b, [&](int q) { return di_uses(3 * i, q); }, [](int) {}, tb, tb + DI_ACC);
        di_wait<SELFTEST>(sh, &sh.a_ready[0], (uint32_t)(operands++ & 1));
        di_issue<6, 6, 5, SELFTEST>(sh, item, tiles_b, [&](int q) { return di_uses(3 * i + 1, q); }, [](int) {}, tb, tb + DI_ACC);
        di_wait<SELFTEST>(sh, &sh.a_ready[0], (uint32_t)(operands++ & 1));
        di_issue<6, 6, 5, SELFTEST>(sh, item, tiles_b, [&](int q) { return di_uses(3 * i + 2, q); }, [](int) {}, tb, tb + DI_ACC);
      }
    }
    di_drain(sh);
  } else {
    const int row = 32 * (warp & 3) + lane, h = warp >> 2;       // this thread's vector, and its columns 32 h .. + 31
    const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
    const uint32_t area = tb + lanes, myacc = tb + DI_ACC + lanes + DI_COLS * h;
    // A barrier for each half of the operand: without the sketch the rows are a tile ahead, and on one barrier nothing but their arithmetic's
    // time kept them from completing the phase behind the one that the MMA warp still waits for.  They come to a half again once they
    // have taken its sums, which the MMA warp issued behind that wait.
    auto operand_ready = [&](int half) {
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) di_arrive(&sh.a_ready[half]);
    };
    constexpr int CHUNKS = TQ_D * (int)sizeof(Tin) / 16;
    auto load_tile = [&](int64_t tile) {
      for (int i = tid; i < DI_ROWS * CHUNKS; i += DI_ROW_THREADS) {
        const int r = i / CHUNKS, c = i - r * CHUNKS;
        const uint32_t dst = sptr(xs + r * ROWB + 16 * c);
        if (tile * DI_ROWS + r < n)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst),
                       "l"(reinterpret_cast<const uint8_t*>(x + (tile * DI_ROWS + r) * ld) + 16 * c) : "memory");
        else
          *reinterpret_cast<uint4*>(xs + r * ROWB + 16 * c) = make_uint4(0u, 0u, 0u, 0u);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // Norms and the digits of w of a tile.  Without the sketch a tile ahead of the indices, into the other half of the operand: its
    // products are then done when the rows ask for them
    float nrm = 0.f, next_nrm = 0.f;
    bool plain = false, next_plain = false;
    auto prepare = [&](int t) {
      float* s_norm = s_norms[t & 1];
      // norms in the rows' own precision and NumPy's order (first term + pairwise sum of the rest), eight lanes a vector, two
      // vectors of a lane at once; the four vectors of a warp's load are two rows apart: no bank conflicts
      {
        const int j = tid & 7, i8 = tid >> 3, r0 = (i8 & ~7) | ((i8 & 3) << 1) | ((i8 >> 2) & 1);
        const Tin* xr[2] = {};
        float s[2];
        auto sq = [&](int q, int k) { const float f = di_f<Tin>(xr[q][k]); return __fmul_rn(f, f); };
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          xr[q] = reinterpret_cast<const Tin*>(xs + (r0 + 64 * q) * ROWB);
          s[q] = sq(q, 1 + j);
        }
#pragma unroll
        for (int i = 8; i < 120; i += 8)
#pragma unroll
          for (int q = 0; q < 2; ++q) s[q] = __fadd_rn(s[q], sq(q, 1 + i + j));
#pragma unroll
        for (int m = 1; m < 8; m <<= 1)
#pragma unroll
          for (int q = 0; q < 2; ++q) s[q] = __fadd_rn(s[q], __shfl_xor_sync(0xffffffffu, s[q], m));
#pragma unroll
        for (int i = 121; i < 128; ++i)
#pragma unroll
          for (int q = 0; q < 2; ++q) s[q] = __fadd_rn(s[q], sq(q, i));
#pragma unroll
        for (int q = 0; q < 2; ++q)
          if (j == 0) s_norm[r0 + 64 * q] = sqrtf(__fadd_rn(sq(q, 0), s[q]));
      }
      if (tid < DI_ROWS) s_plains[t & 1][tid] = 0;
      di_rows_sync();
      next_nrm = s_norm[row];
      const float safe = next_nrm > 0.f ? next_nrm : 1.0f;                // turboquant/polar_quant.py:74
      // w = x / ||x|| in the rows' precision (:75), times 2^30: the product with the reciprocal, corrected by its own exact remainder,
      // is the correctly rounded quotient (P. W. Markstein, IBM J. Res. Dev. 34 (1990), for a correctly rounded reciprocal of a divisor
      // that is not all ones).  Its digits: the nearest whole number, of which w may be off by half of one.
      const float inv = 1.0f / safe * 0x1p30f, back = safe * -0x1p-30f;
      const uint8_t* xr = xs + row * ROWB + DI_COLS * h * sizeof(Tin);
      float most = 0.f;
#pragma unroll 2
      for (int c = 0; c < DI_COLS / 8; ++c) {
        float f[8];
        di_load8<Tin>(xr + 8 * c * sizeof(Tin), f);
        uint2 u[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          float w = f[k] * inv;
          w = fmaf(fmaf(w, back, f[k]), inv, w);
          most = fmaxf(most, fabsf(w));
          u[k] = make_uint2(((uint32_t)__float2int_rn(w) + 0x00808080u) ^ 0x00808080u, 0u);
        }
        di_store8<4, 0>(area + (PROD ? 0 : 128 * (t & 1)), 8 * h + 2 * c, u);
      }
      // Norms that squares below or beyond the fp32 range have gone into (and w = x where all are below it), infinities and NaN; divisors
      // of all ones
      next_plain = next_nrm > 0.f ? !(next_nrm > 0x1p-60f && next_nrm < 0x1p63f && most < DI_LARGEST * 0x1p30f) || (__float_as_uint(next_nrm) & 0x7fffffu) == 0x7fffffu
                                  : next_nrm != 0.f || most != 0.f;
      operand_ready(PROD ? 0 : t & 1);
      if constexpr (!PROD) {
        di_rows_sync();                                            // (the rows have been read)
        if (t + 1 < mine) load_tile(blockIdx.x + (t + 1) * step);
      }
    };
    int item = 0, t = PROD ? 0 : -1;
    if (mine > 0) load_tile(blockIdx.x);
    for (; t < mine; ++t) {
      if (const int ahead = PROD ? t : t + 1; ahead < mine) {
        nrm = next_nrm;
        plain = next_plain;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (di_rows_any(sh.failed)) break;   // (in a tile before)
        prepare(ahead);
        if (!PROD && t < 0) continue;
      }
      if (PROD || t + 1 >= mine) {
        nrm = next_nrm;
        plain = next_plain;
      }
      const int64_t v0 = (blockIdx.x + t * step) * DI_ROWS, v = v0 + row;
      const bool live = v < n;
      const float* s_norm = s_norms[t & 1];
      uint8_t* s_plain = s_plains[t & 1];
      // ---- y = R w: indices, ||c[idx]||^2, the centroids as the next operand.  Without the sketch of the 34 products of all digits ten,
      // which leave at most 1.004 x 2^-21 of r_scale out (di_quant_args): one output in 90,000 of a rotation's with eight centroids is too close to a boundary
      // and is left to the decider.  With the sketch, where other outputs hang on it, 14 products: one in six million; its row is for
      // di_rows_plain.  Rows of zeros are on no boundary.
      uint32_t packed[DI_COLS / 4];
      uint32_t unsure = 0;   // groups of eight columns
      {
        int32_t y[DI_COLS];
        di_take32<PROD ? 4 : 3, SELFTEST>(sh, item, myacc, lane, PROD ? A.shift : 17, y);
        if constexpr (PROD) {
          uint32_t near = 0xffffffffu;
#pragma unroll
          for (int g = 0; g < DI_COLS / 4; ++g) {
            packed[g] = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) packed[g] |= di_index<BITS>(A.thr, A.near, y[4 * g + k], near) << (8 * k);
          }
          plain |= near <= 2 * A.near && nrm != 0.f;
        } else {
#pragma unroll
          for (int c = 0; c < DI_COLS / 8; ++c) {
            float frac = 0.f;
#pragma unroll
            for (int g = 2 * c; g < 2 * c + 2; ++g) {
              uint32_t m[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) m[k] = di_index_float<BITS>(A, y[4 * g + k], frac);
              packed[g] = __byte_perm(__byte_perm(m[0], m[1], 0x0040), __byte_perm(m[2], m[3], 0x0040), 0x5410);
            }
            unsure |= frac > 0.f ? 1u << c : 0u;
          }
          if (nrm == 0.f || !live) unsure = 0;
          if (a.out_scale && unsure) plain = true;
        }
#pragma unroll
        for (int g = 0; g < DI_COLS / 4; ++g)
          if (nrm == 0.f) packed[g] = 0x01010101u * (uint32_t)A.zero_idx;
      }
      if (PROD || a.out_scale) {
        double cc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int g = 0; g < DI_COLS / 4; ++g) {
          if constexpr (BITS < 4) {
            const uint32_t two = packed[g] | (packed[g] >> 5);
            cc[0] += s_codes.square[two & 63];
            cc[1] += s_codes.square[(two >> 16) & 63];
          } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) cc[k] += s_codes.square[(packed[g] >> (8 * k)) & 15];
          }
        }
        s_part[h][row] = (cc[0] + cc[1]) + (cc[2] + cc[3]);
      }
      if (live && a.out_idx) {
#pragma unroll
        for (int g = 0; g < DI_COLS / 4; g += 4)
          *reinterpret_cast<uint4*>(a.out_idx + v * TQ_D + DI_COLS * h + 4 * g) = make_uint4(packed[g], packed[g + 1], packed[g + 2], packed[g + 3]);
      }
      if constexpr (PROD) {
#pragma unroll
        for (int c = 0; c < DI_COLS / 8; ++c) {
          if constexpr (BITS < 4) {
            di_store_codes<6>(area, 8 * h + 2 * c, A.words, packed[2 * c], packed[2 * c + 1]);
          } else {
            uint2 u[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) u[k] = s_cdig[(packed[2 * c + (k >> 2)] >> (8 * (k & 3))) & 15];
            di_store8<6, 1>(area, 8 * h + 2 * c, u);
          }
        }
        operand_ready(0);
      }
      if constexpr (!PROD) {
        if (unsure && !plain && a.out_idx) {
          __threadfence_block();   // (the indices have been stored)
          for (; unsure && !plain; unsure &= unsure - 1)
            plain = !di_add(s_list, (uint32_t)row | (uint32_t)(4 * h + __ffs(unsure) - 1) << 7 | (uint32_t)t << 11, nrm);
        }
      }
      double cn = 1.0;
      if (PROD || a.out_scale) {
        di_rows_sync();
        cn = sqrt((s_part[0][row] + s_part[1][row]) + (s_part[2][row] + s_part[3][row]));
        cn = cn > 1e-10 ? cn : 1.0;                                               // turboquant/polar_quant.py:110-111
      }
      if (h == 0 && live) {
        if (a.out_norm) a.out_norm[v] = nrm;
        if (a.out_scale) a.out_scale[v] = (float)(a.norm_correction ? (double)nrm / cn : (double)nrm);
      }
      if constexpr (PROD) {
        // ---- x_hat = norm R^T c / ||c||, residual x - x_hat, with the norm that is returned and stored (fp32).  Six digits each:
        // what the 13 products left out would add to an element is below 2^-36.4 of r_scale cent_scale, to all 128 together 2^-32.9, in
        // practice 2^-44 of the vector's length (with five digits 2^-36, and one residual norm in 4,000 came out a neighbour).  Residuals
        // longer than 2^-6 of that unit, for a random rotation 2^-9 of the vector's length, are therefore within 2^-26.9 of their own, and
        // rounded to fp32.  Shorter ones, of vectors that are reconstructions, are for di_rows_plain (norms off by 2e-6 otherwise): rows none
        // of whose elements, of the columns of one thread, is above that (`least`) ----
        const double inv = a.norm_correction ? 1.0 / cn : 1.0;
        const double back = -0x1p-32 * A.r_scale * A.cent_scale * inv * (double)nrm;
        const double unit = nrm > 0.f && nrm < 1e38f ? ldexp(1.0, -(ilogbf(nrm) + 2)) : 1.0;   // |residual| x unit < 1 for a rotation
        const double unit46 = unit * 0x1p46;
        uint32_t over = 0;
        double rr[4] = {0.0, 0.0, 0.0, 0.0};
        long long acc[DI_COLS];
        di_take64<SELFTEST>(sh, item, myacc, lane, acc);
        const uint8_t* xr = xs + row * ROWB + DI_COLS * h * sizeof(Tin);
#pragma unroll
        for (int c = 0; c < DI_COLS / 8; ++c) {
          float f[8];
          di_load8<Tin>(xr + 8 * c * sizeof(Tin), f);
          uint2 u[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const double e = fma(di_double(acc[8 * c + k]), back, (double)f[k]);
            rr[k & 3] = fma(e, e, rr[k & 3]);
            // to a whole number of 2^-46, in balanced digits; the upper half tells what is too large, or too small in all elements
            const unsigned long long w = (unsigned long long)__double_as_longlong(fma(e, unit46, 6755399441055744.0));
            over = max(over, (uint32_t)(w >> 32) - 0x43380000u + 31000u);
            u[k] = di_split((w + 0x8080808080ull) ^ 0x8080808080ull);
          }
          di_store8<6, 0>(area, 8 * h + 2 * c, u);
        }
        // (too large, or too small in all elements; rows of zeros are neither)
        const uint32_t least = nrm != 0.f ? __float2uint_ru(fminf(A.least * (float)inv, 31000.f)) : 0u;
        plain |= over - 31000u - least > 31000u - least;
        operand_ready(0);
        di_rows_sync();   // (the sums of the squared centroids have been read, and the rows)
        const double part = (rr[0] + rr[1]) + (rr[2] + rr[3]);
        s_part[h][row] = part;
        if (t + 1 < mine) load_tile(blockIdx.x + (t + 1) * step);
        di_rows_sync();
        if (h == 0 && live && a.out_rnorm)
          a.out_rnorm[v] = (float)sqrt((s_part[0][row] + s_part[1][row]) + (s_part[2][row] + s_part[3][row]));
        // ---- sketch: sign(S r), zero counts as +1 (turboquant/qjl.py:89-90), first column in the most significant bit.  A projection
        // that what has been left out here (2^-36.3 s_scale) and of the residual may turn: di_rows_plain (with five digits each, three rows
        // of 64,000, each 20 us of a CTA) ----
        di_take64<SELFTEST>(sh, item, myacc, lane, acc);
        const long long band = (long long)fmin(256.0 + A.slack * (double)nrm * unit * inv, 0x1p60);
        uint32_t m = 0;
        bool close = false;
#pragma unroll
        for (int k = 0; k < DI_COLS; ++k) {
          m = (m << 1) | (acc[k] < 0 ? 0u : 1u);
          close |= (unsigned long long)(acc[k] + band) <= 2 * (unsigned long long)band;
        }
        plain |= close && nrm != 0.f;
        m = __byte_perm(m, 0, 0x0123);
        if (live && a.out_qjl) {
          uint8_t* z = a.out_qjl + v * 16 + 4 * h;
          if ((reinterpret_cast<uintptr_t>(a.out_qjl) & 3) == 0) *reinterpret_cast<uint32_t*>(z) = m;
          else z[0] = (uint8_t)m, z[1] = (uint8_t)(m >> 8), z[2] = (uint8_t)(m >> 16), z[3] = (uint8_t)(m >> 24);
        }
      }
      if (plain) s_plain[row] = 1;
      if (di_rows_any(plain)) {   // whole rows in plain arithmetic, over what has been stored
        di_rows_plain<Tin>(s_rows, a, s_codes, s_plain, s_norm, x, ld, v0, n, tid);
        di_rows_sync();
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    const bool failed = di_rows_any(sh.failed);
    if constexpr (!PROD)
      if (tid == 0) s_list.closed = 1;
    if (failed) {
      // The last tile begun and those behind it; without the sketch the one before it as well: the last turn prepares nothing, and does not
      // look at what the turn before it has seen (a barrier of 0.4 us)
      constexpr int BACK = PROD ? 1 : 2;
      di_give_up(a, t > BACK ? t - BACK : 0, mine, h == 0 ? row : -1, n, A.status);
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tb), "r"(512u) : "memory");
}

constexpr int DI_IDX_ROW = TQ_D + 16;   // bytes between staged rows: 16 bytes on, no bank conflicts
constexpr int DI_DEQUANT_SMEM = DI_DIGITS * DI_TILE + DI_ROW_THREADS * 128 + DI_ROWS * DI_IDX_ROW + 1024;

// x_hat = (norm / ||c[idx]||) R^T c[idx] + shrink sqrt(pi/2)/sqrt(d) rnorm S^T z.  The signs z are one digit, +-1: seven products.
// Once the sum s of a tile has been read, digit s of its operand is of no more use, and the rows write that digit of the next tile's: the MMAs
// go on from tile to tile, while the rows add up the last sums and store.
template <typename Tout, bool PROD, int SELFTEST = 0>
__global__ void __launch_bounds__(DI_THREADS, 1) k_dense_dequantize_i8(const __grid_constant__ DiDequant A, const __grid_constant__ CUtensorMap map,
                                                                       int64_t n, Tout* __restrict__ out) {
  extern __shared__ __align__(128) uint8_t di_raw[];
  __shared__ DiShared sh;
  __shared__ uint64_t s_digit[DI_DIGITS];       // digits of the operand, in place of a_ready, which is the signs'
  __shared__ uint32_t s_sign[16];               // four sketch bits, the first in bit 3, as +-1 digits
  __shared__ double s_sq[16], s_part[2][4][DI_ROWS];
  const TqDenseDequant& a = A.q;
  uint8_t* tiles_b = di_raw + (((sptr(di_raw) + 1023u) & ~1023u) - sptr(di_raw));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    for (int p = 0; p < DI_DIGITS; ++p)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sptr(&s_digit[p])), "r"(DI_ROW_THREADS / 32) : "memory");
    di_init(sh);
  }
  if (tid < 16) {
    const double c = tid < (1 << a.bits) ? a.cent[tid] : 0.0;
    s_sq[tid] = c * c;
    uint32_t w = 0;
    for (int k = 0; k < 4; ++k) w |= ((tid >> (3 - k)) & 1 ? 0x01u : 0xffu) << (8 * k);
    s_sign[tid] = w;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sptr(&sh.tmem)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tb = sh.tmem;
  const int64_t tiles = (n + DI_ROWS - 1) / DI_ROWS, step = gridDim.x;
  const int mine = (int)((tiles - blockIdx.x + step - 1) / step);
  constexpr int PHASES = PROD ? 2 : 1;   // (the signs' product last)

  if (warp == DI_COPIER) {
    // (without a sketch R^T stays in place)
    if (lane == 0)
      di_copier<SELFTEST>(sh, tiles_b, PROD ? mine * PHASES : mine > 0 ? 1 : 0, [&](int i) { return PROD && (i & 1) ? A.st : A.rt; },
                          [](int) { return DI_DIGITS; }, [](int i, int) { return i; });
  } else if (warp == DI_MMA) {
    int item = 0;
    for (int i = 0; i < mine && !__any_sync(0xffffffffu, sh.failed); ++i) {
      // (sum 7 takes digits 1 to 6, sum 6 the leading one as well)
      di_issue<DI_DIGITS, DI_DIGITS, DI_SUMS - 1, SELFTEST>(sh, item, tiles_b, [&](int) { return PROD ? 2 * i : 0; }, [&](int sum) {
        if (sum == DI_SUMS - 1)
          for (int p = 1; p < DI_DIGITS; ++p) di_wait<SELFTEST>(sh, &s_digit[p], (uint32_t)(i & 1));
        if (sum == DI_SUMS - 2) di_wait<SELFTEST>(sh, &s_digit[0], (uint32_t)(i & 1));
      }, tb, tb + DI_ACC);
      if constexpr (PROD) {
        di_wait<SELFTEST>(sh, &sh.a_ready[0], (uint32_t)(i & 1));
        di_issue<1, DI_DIGITS, DI_DIGITS - 1, SELFTEST>(sh, item, tiles_b, [&](int) { return 2 * i + 1; }, [](int) {}, tb + DI_SIGNS, tb + DI_ACC);
      }
    }
    di_drain(sh);
  } else {
    const int row = 32 * (warp & 3) + lane, h = warp >> 2;
    const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
    const uint32_t area = tb + lanes, myacc = tb + DI_ACC + lanes + DI_COLS * h;
    const bool wide = (a.ld_out * sizeof(Tout)) % 16 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    uint8_t* stage = tiles_b + DI_DIGITS * DI_TILE + warp * 4096;          // 32 rows x 128 bytes of this warp on their way out
    uint8_t* xi = tiles_b + DI_DIGITS * DI_TILE + DI_ROW_THREADS * 128;    // indices of a tile
    auto load_tile = [&](int64_t tile) {
      for (int i = tid; i < DI_ROWS * 8; i += DI_ROW_THREADS) {
        const int r = i >> 3, c = i & 7;
        if (tile * DI_ROWS + r < n)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sptr(xi + r * DI_IDX_ROW + 16 * c)),
                       "l"(a.idx + (tile * DI_ROWS + r) * TQ_D + 16 * c) : "memory");
        else
          *reinterpret_cast<uint4*>(xi + r * DI_IDX_ROW + 16 * c) = make_uint4(0u, 0u, 0u, 0u);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto ready = [&](uint64_t* bar) {   // what has been stored to tensor memory is there
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) di_arrive(bar);
    };
    // of the next tile: indices, a nibble each, norms and the sketch bits of this thread's columns
    uint32_t codes[4] = {}, signs = 0;
    bool high = false;                                                     // indices above 7
    float next_norm = 0.f, next_rnorm = 0.f;
    auto prepare = [&](int t) {
      const int64_t v = (blockIdx.x + t * step) * DI_ROWS + row;
      next_norm = v < n ? a.norm[v] : 0.f;
      if constexpr (PROD) {
        next_rnorm = v < n ? a.rnorm[v] : 0.f;
        signs = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) signs = (signs << 8) | (v < n ? a.qjl[v * 16 + 4 * h + k] : 0u);
      }
      double cc[4] = {0.0, 0.0, 0.0, 0.0};
      uint32_t any = 0;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const uint4 q = *reinterpret_cast<const uint4*>(xi + row * DI_IDX_ROW + DI_COLS * h + 16 * c);
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const uint32_t m = w[g] & 0x0f0f0f0fu, nibbles = __byte_perm(m | (m >> 4), 0, 0x4420);
          any |= m;
          if (g & 1) codes[2 * c + (g >> 1)] |= nibbles << 16; else codes[2 * c + (g >> 1)] = nibbles;
#pragma unroll
          for (int k = 0; k < 4; ++k) cc[k] += s_sq[(m >> (8 * k)) & 15];
        }
      }
      high = __any_sync(0xffffffffu, (any & 0x08080808u) != 0);
      s_part[t & 1][h][row] = (cc[0] + cc[1]) + (cc[2] + cc[3]);
    };
    // digit p of the 32 centroids of this thread; a byte permute picks four (where a selector's fourth bit is set it repeats a sign bit instead)
    auto write_digit = [&](int p) {
      uint32_t w[8];
      const uint32_t lo0 = A.words[p].x, lo1 = A.words[p].y, hi0 = A.words[p].z, hi1 = A.words[p].w;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t sel = i & 1 ? codes[i >> 1] >> 16 : codes[i >> 1];
        w[i] = di_prmt(lo0, lo1, sel);
        if (high) {
          const uint32_t above = (di_prmt(0x80808080u, 0x80808080u, sel) & 0x01010101u) * 255u;
          w[i] = (w[i] & ~above) | (di_prmt(hi0, hi1, sel & 0x7777u) & above);
        }
      }
      asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                   ::"r"(area + 32 * p + 8 * h), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
    };
    auto write_signs = [&]() {   // eight sketch bits a step, the first in the most significant place
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t z = (signs >> (24 - 8 * k)) & 255u;
        di_st2(area + DI_SIGNS + 8 * h + 2 * k, s_sign[z >> 4], s_sign[z & 15]);
      }
      ready(&sh.a_ready[0]);
    };
    int item = 0, t = 0;
    if (mine > 0) {
      load_tile(blockIdx.x);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      di_rows_sync();
      prepare(0);
      if constexpr (PROD) write_signs();
#pragma unroll 1
      for (int p = DI_DIGITS - 1; p >= 0; --p) write_digit(p);
      for (int p = DI_DIGITS - 1; p >= 0; --p) ready(&s_digit[p]);
      di_rows_sync();
      if (mine > 1) load_tile(blockIdx.x + step);
    }
    for (; t < mine; ++t) {
      const int64_t v0 = (blockIdx.x + t * step) * DI_ROWS, v = v0 + row;
      const bool live = v < n, more = t + 1 < mine;
      const float norm = next_norm, rnorm = next_rnorm;
      double acc[DI_COLS];
      double f = 0.0, g = 0.0;
      {
        // sums 7 to 4, whole numbers of 2^-68 below 2^48.  The next tile's indices and this one's factors while the MMAs, which have the most to do
        // here, are ahead; a digit is published after the sum behind the one that freed it: by then its store has come to an end
        long long y[DI_COLS];
        di_columns<SELFTEST>(sh, item++, myacc, lane, [&](int k, uint32_t x) { y[k] = (int32_t)x; });
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (di_rows_any(sh.failed)) break;
        if (live) {
          double cn = 1.0;
          if (a.norm_correction) {
            cn = sqrt((s_part[t & 1][0][row] + s_part[t & 1][1][row]) + (s_part[t & 1][2][row] + s_part[t & 1][3][row]));
            cn = cn > 1e-10 ? cn : 1.0;
          }
          f = (double)norm / cn;
          if constexpr (PROD) g = a.shrink * 1.2533141373155001 / sqrt((double)TQ_D) * (double)rnorm;   // turboquant/qjl.py:131-132
          // a factor that is not finite: sums of terms of both signs, not a number
          if (!(fabs(f) < 1e300)) f = __longlong_as_double(0x7ff8000000000000ll);
          if (!(fabs(g) < 1e300)) g = __longlong_as_double(0x7ff8000000000000ll);
          f *= A.r_scale * A.cent_scale;
          g *= A.s_scale;
        }
        if (more) prepare(t + 1);
        int32_t weight = 256;
#pragma unroll 1
        for (int sum = 6; sum > 3; --sum, weight <<= 8) {
          di_columns<SELFTEST>(sh, item++, myacc, lane, [&](int k, uint32_t x) { y[k] += (long long)(int32_t)x * weight; });
          if (more) {
            if (sum < 6) ready(&s_digit[sum + 1]);
            write_digit(sum);
          }
        }
        const double unit = f * 0x1p-56;
#pragma unroll
        for (int k = 0; k < DI_COLS; ++k) acc[k] = di_double(y[k]) * unit;
      }
      double unit = f * 0x1p-24;
#pragma unroll 1
      for (int sum = 3; sum > 0; sum -= 2, item += 2, unit *= 65536.0) {   // (256 times the sum s - 1 <= 2 plus the sum s is below 2^31)
        di_columns2<SELFTEST>(sh, item, myacc, lane, [&](int k, uint32_t x) { acc[k] = fma(di_double(x), unit, acc[k]); });
        if (more) {
          if (sum == 3) ready(&s_digit[4]);
          else ready(&s_digit[3]), di_arrive_warp(&s_digit[2], lane);
          write_digit(sum);
          write_digit(sum - 1);
        }
      }
      if (more) ready(&s_digit[1]), di_arrive_warp(&s_digit[0], lane);
      di_rows_sync();                      // (the indices have been read)
      if (t + 2 < mine) load_tile(blockIdx.x + (t + 2) * step);
      if constexpr (PROD) {   // seven sums, below 2^14
        unit = g * 0x1p-48;
        di_columns<SELFTEST>(sh, item++, myacc, lane, [&](int k, uint32_t x) { acc[k] = fma(di_double(x), unit, acc[k]); });
        unit *= 256.0;
#pragma unroll 1
        for (int sum = 5; sum > 0; sum -= 2, item += 2, unit *= 65536.0)
          di_columns2<SELFTEST>(sh, item, myacc, lane, [&](int k, uint32_t x) { acc[k] = fma(di_double(x), unit, acc[k]); });
        if (more) write_signs();
      }
      Tout* o = out + v * a.ld_out + DI_COLS * h;
      if (a.accumulate && live) {
#pragma unroll
        for (int k = 0; k < DI_COLS; ++k) acc[k] += di_d<Tout>(o[k]);
      }
      if (sizeof(Tout) == 8 && A.tiled) {
        // Sixteen columns at a time through shared memory, 16-byte chunks swizzled as the map has it, and out by a tiled copy that clips rows
        // past n (plain stores of whole lines took 5,800 clocks of a tile's 24,000)
        const int first = 32 * (warp & 3);
#pragma unroll
        for (int c = 0; c < DI_COLS / 16; ++c) {
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 8; ++k)
            *reinterpret_cast<double2*>(stage + 128 * lane + 16 * (k ^ (lane & 7))) = make_double2(acc[16 * c + 2 * k], acc[16 * c + 2 * k + 1]);
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0 && v0 + first < n) {
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(&map), "r"(DI_COLS * h + 16 * c),
                         "r"((int)(v0 + first)), "r"(sptr(stage)) : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
      } else if (live && wide) {
        constexpr int PER = 16 / (int)sizeof(Tout);
#pragma unroll
        for (int k = 0; k < DI_COLS; k += PER) {
          __align__(16) Tout r[PER];
#pragma unroll
          for (int j = 0; j < PER; ++j) r[j] = di_from<Tout>(acc[k + j]);
          *reinterpret_cast<uint4*>(o + k) = *reinterpret_cast<const uint4*>(r);
        }
      } else if (live) {
#pragma unroll
        for (int k = 0; k < DI_COLS; ++k) o[k] = di_from<Tout>(acc[k]);
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    if (di_rows_any(sh.failed)) {   // the last tile begun and those behind it
      di_give_up<Tout>(a, t > 0 ? t - 1 : 0, mine, row, DI_COLS * h, n, out, A.status);
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tb), "r"(512u) : "memory");
}

// Digits of 128 x 128 matrices (rows are outputs) as B operands: [digit][8-output group][16-element chunk][output][element]
// bytes, TQ_DENSE_DIGITS_BYTES in all; `scale` times a value is below 2^54.  A thread takes one element.
struct DiMatrices {
  const double* m[4];
  double scale[4];
  uint8_t* out[4];
};
__global__ void __launch_bounds__(128) k_dense_digits(const __grid_constant__ DiMatrices a) {
  const int n = blockIdx.x, k = threadIdx.x, i = blockIdx.y;
  const uint64_t u = di_digits(__double2ll_rn(a.m[i][n * TQ_D + k] * a.scale[i]));
  uint8_t* at = a.out[i] + (n >> 3) * 1024 + (k >> 4) * 128 + (n & 7) * 16 + (k & 15);
#pragma unroll
  for (int p = 0; p < DI_DIGITS; ++p) at[p * DI_TILE] = (uint8_t)(u >> (48 - 8 * p));
}

// The digits of a quantizer's matrices, behind which `st` may go on; false where they are not to be had now: the call then takes the
// fp64 kernels.  The first call makes them, on its own stream, so that quantizers which never see one do not pay for it
// (made with the quantizer they cost 30 to 90 us of its 1,100); later ones on any stream wait for its event until it
// has been seen.  A call that is being captured neither makes them nor waits: its graph could run before, or alone.
constexpr int32_t DI_MADE = 1, DI_SEEN = 2;
bool di_digits_ready(const tq_quantizer* q, cudaStream_t st) {
  if (__atomic_load_n(&q->digits_state, __ATOMIC_ACQUIRE) == DI_SEEN) return true;
  static std::mutex lock;
  const std::lock_guard<std::mutex> hold(lock);
  // (other threads may be capturing: nothing here touches their streams)
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) return false;
  auto prepare = [&]() -> cudaError_t {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(st, &capture);
    if (e != cudaSuccess) return e;
    if (q->digits_state >= DI_MADE) {
      e = cudaEventQuery(q->digits_event);
      if (e == cudaSuccess) __atomic_store_n(&q->digits_state, DI_SEEN, __ATOMIC_RELEASE);
      if (e != cudaErrorNotReady) return e;
      (void)cudaGetLastError();
      return capture == cudaStreamCaptureStatusNone ? cudaStreamWaitEvent(st, q->digits_event, 0) : cudaErrorNotReady;
    }
    if (capture != cudaStreamCaptureStatusNone) return cudaErrorNotReady;
    if (!q->digits_event && (e = cudaEventCreateWithFlags(&q->digits_event, cudaEventDisableTiming)) != cudaSuccess) return e;
    DiMatrices a;
    int count = 0;
    auto add = [&](const double* m, double scale, const uint8_t* out) {
      a.m[count] = m;
      a.scale[count] = 18014398509481984.0 / scale;
      a.out[count++] = const_cast<uint8_t*>(out);
    };
    const TqDenseDigits& g = q->dig;
    if (g.r_scale != 0.0) add(q->rot, g.r_scale, g.r), add(q->rot_t, g.r_scale, g.rt);
    if (g.s_scale != 0.0) add(q->s, g.s_scale, g.s), add(q->s_t, g.s_scale, g.st);
    k_dense_digits<<<dim3(TQ_D, count), TQ_D, 0, st>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess || (e = cudaEventRecord(q->digits_event, st)) != cudaSuccess) return e;
    __atomic_store_n(&q->digits_state, DI_MADE, __ATOMIC_RELEASE);
    return cudaSuccess;
  };
  const cudaError_t e = prepare();
  (void)cudaThreadExchangeStreamCaptureMode(&mode);
  if (e != cudaSuccess) (void)cudaGetLastError();
  return e == cudaSuccess;
}

template <auto kernel, typename... Args> int di_launch(int smem, int64_t n, cudaStream_t st, const char* what, const Args&... args) {
  static thread_local int configured_dev = -1;   // one per kernel: the kernel is a template argument
  int dev = 0;
  TQ_CUDA(cudaGetDevice(&dev));
  if (configured_dev != dev) {
    TQ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    configured_dev = dev;
  }
  const int64_t tiles = (n + DI_ROWS - 1) / DI_ROWS, sms = tq_num_sms();
  kernel<<<(unsigned)(tiles < sms ? tiles : sms), DI_THREADS, smem, st>>>(args...);
  return tq_launch_check(what);
}
template <typename Tin, int BITS> int di_quantize_bits(const DiQuant& A, const Tin* x, int64_t ld, int64_t n, cudaStream_t st) {
  if (A.q.out_qjl || A.q.out_rnorm)
    return di_launch<k_dense_quantize_i8<Tin, BITS, true>>(di_quant_smem<Tin, true>(), n, st, "k_dense_quantize_i8", A, x, ld, n);
  return di_launch<k_dense_quantize_i8<Tin, BITS, false>>(di_quant_smem<Tin, false>(), n, st, "k_dense_quantize_i8", A, x, ld, n);
}
template <typename Tin> int di_quantize(const DiQuant& A, const void* x, int64_t ld, int64_t n, cudaStream_t st) {
  const Tin* xt = reinterpret_cast<const Tin*>(x);
  switch (A.q.bits) {
    case 1: return di_quantize_bits<Tin, 1>(A, xt, ld, n, st);
    case 2: return di_quantize_bits<Tin, 2>(A, xt, ld, n, st);
    case 3: return di_quantize_bits<Tin, 3>(A, xt, ld, n, st);
    default: return di_quantize_bits<Tin, 4>(A, xt, ld, n, st);
  }
}
template <typename Tout, bool PROD, int SELFTEST = 0> int di_dequantize_launch(DiDequant& A, int64_t n, Tout* out, cudaStream_t st) {
  CUtensorMap map;
  memset(&map, 0, sizeof(map));
  A.tiled = sizeof(Tout) == 8 && tq_aligned(out, 16) && A.q.ld_out % 2 == 0 &&
            tc_map(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, out, TQ_D, n, A.q.ld_out * 8, 16, 32);
  return di_launch<k_dense_dequantize_i8<Tout, PROD, SELFTEST>>(DI_DEQUANT_SMEM, n, st, "k_dense_dequantize_i8", A, map, n, out);
}
template <typename Tout> int di_dequantize(DiDequant& A, int64_t n, void* out, cudaStream_t st) {
  Tout* o = reinterpret_cast<Tout*>(out);
  return A.q.qjl ? di_dequantize_launch<Tout, true>(A, n, o, st) : di_dequantize_launch<Tout, false>(A, n, o, st);
}

}  // namespace

// The power of two that a matrix's digits are relative to, or 0 for a matrix that stays with the fp64 kernels; rows, length: the largest
// sum of a row's magnitudes and the length of the longest row over it.
// The digits are fixed-point numbers of 2^-54 of the largest entry, where fp64 keeps every entry's own exponent.  No product may lose
// by that, so: every row and column is at least sqrt(2) times as long as the largest entry (the rounding of a row's digits is then
// 2^-55 of that row's length, below that of fp64 sums), and no entry is below 2^-30 of it (a row of x enters with 2^-54 of its length;
// an entry of zero would hide its large elements, and what an output then sees may be smaller than that).  Random rotations
// and Gaussian matrices are of this kind (their rows are three times and twice as long); uneven, diagonal or block matrices and what
// is not finite are not.
double tq_dense_digits_scale(const double* m, double* rows, double* length) {
  double most = 0.0, least = 1e300, row[TQ_D] = {}, col[TQ_D] = {}, sum[TQ_D] = {};
  for (int i = 0; i < TQ_D; ++i)
    for (int j = 0; j < TQ_D; ++j) {
      const double a = fabs(m[i * TQ_D + j]);
      most = a > most ? a : most;
      least = a < least ? a : least;
      row[i] += a * a;
      col[j] += a * a;
      sum[i] += a;
    }
  if (!(most > 1e-100 && most < 1e100 && least >= most * 0x1p-30)) return 0.0;
  for (int i = 0; i < TQ_D; ++i)
    if (!(row[i] >= 2.0 * most * most && col[i] >= 2.0 * most * most)) return 0.0;   // (also what is not a number)
  int e = 0;
  frexp(most, &e);   // most < 2^e
  *rows = *length = 0.0;
  for (int i = 0; i < TQ_D; ++i) *rows = fmax(*rows, ldexp(sum[i], -e)), *length = fmax(*length, ldexp(sqrt(row[i]), -e));
  return ldexp(1.0, e);
}
// A power of two above every centroid's magnitude, or 0 for a codebook whose centroids differ much in size: those of a row
// may all be small ones, whose digits would be short.  (Codebooks of one to four bits span a factor of 21 at most.)
double tq_dense_digits_centroids(const double* c, int n) {
  double most = 0.0;
  for (int i = 0; i < n; ++i) most = fabs(c[i]) > most ? fabs(c[i]) : most;
  if (!(most > 1e-100 && most < 1e100)) return 0.0;
  for (int i = 0; i < n; ++i)
    if (c[i] != 0.0 && !(fabs(c[i]) >= most / 64.0)) return 0.0;
  int e = 0;
  frexp(most, &e);
  return ldexp(1.0, e);
}

// The digits of the centroids, whole numbers of 2^-54 of the scale, as the kernels' operands are made from
void tq_dense_digits_words(const double* c, int n, double scale, uint32_t (&words)[7][4]) {
  memset(words, 0, sizeof(words));
  for (int i = 0; i < n; ++i) {
    const uint64_t u = ((uint64_t)llrint(c[i] / scale * 18014398509481984.0) + 0x808080808080ull) ^ 0x808080808080ull;
    for (int p = 0; p < 7; ++p) words[p][i >> 2] |= (uint32_t)(uint8_t)(u >> (48 - 8 * p)) << (8 * (i & 3));
  }
}

// Calls that come here, us here / in the fp64 kernels (which take tiles of 16, 32 or 64 vectors, two CTAs an SM, and step up at 32
// and 64 vectors per SM): quantize 4,096 vectors 14.6 / 14.6, 4,800 14.5 / 22.8, 9,472 14.6 / 22.8, 65,536 33 / 134; with the sketch 4,096
// 27 / 27, 4,800 27 / 43, 12,000 27 / 94, 65,536 90 / 302; dequantize 8,192 19 / 17, 12,000 19 / 29, 65,536 56 / 90; with the sketch 4,096
// 27 / 23, 6,000 27 / 31, 65,536 85 / 164.
static bool di_enough(int64_t n, bool dequantize, bool sketch) { return n > (dequantize && !sketch ? 64 : 32) * (int64_t)tq_num_sms(); }

// The kernels' arguments; false: not of these kernels' kind
static bool di_quant_args(const TqDenseQuant& a, const TqDenseDigits& g, const void* x, int32_t dtype, int64_t ld, DiQuant& A) {
  const bool prod = a.out_qjl || a.out_rnorm;
  if (a.d != TQ_D || g.r_scale == 0.0 || g.cent_scale == 0.0 || a.out_packed || a.out_res || (prod && g.s_scale == 0.0)) return false;
  if (dtype != TQ_F32 && dtype != TQ_F16) return false;
  if (!tq_aligned(x, 16) || ld * (dtype == TQ_F32 ? 4 : 2) % 16 || !tq_aligned(a.out_idx, 16)) return false;
  A.r = g.r; A.rt = g.rt; A.s = g.s;
  A.r_scale = g.r_scale / 4096.0;
  A.cent_scale = g.cent_scale;
  A.slack = 32768.0 * g.r_scale * g.cent_scale;
  A.least = (float)(128.0 * g.r_scale * g.cent_scale);
  A.status = tq_quantize_status_word();
  for (int p = 0; p < DI_DIGITS; ++p) A.words[p] = make_uint2(g.words[p][0], g.words[p][1]);
  // Boundaries as numbers of 2^-27 of r_scale (no y is beyond 16 of them: entries of R are below r_scale, rows of w shorter than 1 + 2^-20),
  // and what a y may be off by: the products left out (1.004 x 2^-21), half of 2^-30 of every element of w, two fields cut off, the
  // boundary's rounding; in fp32 also a rounding of y and one of the ramp's constant.  With the sketch numbers of 2^-29 where rows of R
  // are that short, products left out 2^-29, two or three fields.
  const double unit = !prod || g.r_length > 3.9 ? 0x1p27 : 0x1p29;
  A.shift = unit == 0x1p27 ? 17 : 15;
  double most = 0.0;
  for (int i = 0; i < 15; ++i) {
    const double t = fmin(fmax(rint(g.bnd[i] / g.r_scale * unit), -2147483000.0), 2147483000.0);
    A.thr[i] = (int32_t)t;
    if (i < (1 << a.bits) - 1) most = fmax(most, fabs(t));
  }
  A.near = (uint32_t)(A.shift == 15 ? ceil(g.r_rows * 0.25 + 3.6) : ceil(g.r_rows * 0.0625 + (prod ? 3.8 : 67.5)));
  const double reach = A.near + most * 0x1p-22;
  for (int i = 1; i < (1 << a.bits) - 1 && !prod; ++i)   // (ramps that overlap may add up to a whole number)
    if ((double)A.thr[i] - A.thr[i - 1] < 2.0 * reach + 8.0) return false;
  A.step = (float)(0.5 / reach);
  for (int i = 0; i < 15; ++i) A.offset[i] = (float)(0.5 - A.thr[i] * (double)A.step);
  A.zero_idx = 0;
  for (int i = 0; i < (1 << a.bits) - 1; ++i) A.zero_idx += g.bnd[i] < 0.0 ? 1 : 0;
  A.q = a;
  return true;
}
static bool di_dequant_args(const TqDenseDequant& a, const TqDenseDigits& g, DiDequant& A) {
  if (a.d != TQ_D || g.r_scale == 0.0 || g.cent_scale == 0.0 || !a.idx || (a.qjl && g.s_scale == 0.0)) return false;
  if (!tq_aligned(a.idx, 16)) return false;
  A.rt = g.rt; A.st = g.st;
  for (int p = 0; p < DI_DIGITS; ++p) A.words[p] = make_uint4(g.words[p][0], g.words[p][1], g.words[p][2], g.words[p][3]);
  A.r_scale = g.r_scale / 4096.0;
  A.s_scale = g.s_scale / 64.0;
  A.cent_scale = g.cent_scale;
  A.status = tq_quantize_status_word();
  A.q = a;
  return true;
}

// false: not of these kernels' kind, nothing launched
bool tq_dense_i8_quantize_try(const tq_quantizer* q, const TqDenseQuant& a, const void* x, int32_t dtype, int64_t ld, int64_t n, cudaStream_t st,
                              int* rc) {
  DiQuant A;
  if (!di_enough(n, false, a.out_qjl || a.out_rnorm) || !di_quant_args(a, q->dig, x, dtype, ld, A) || !di_digits_ready(q, st)) return false;
  *rc = dtype == TQ_F32 ? di_quantize<float>(A, x, ld, n, st) : di_quantize<__half>(A, x, ld, n, st);
  return true;
}

bool tq_dense_i8_dequantize_try(const tq_quantizer* q, const TqDenseDequant& a, int64_t n, void* out, int32_t dtype, cudaStream_t st, int* rc) {
  DiDequant A;
  if (dtype != TQ_F64 && dtype != TQ_F32 && dtype != TQ_F16) return false;
  if (!di_enough(n, true, a.qjl != nullptr) || !di_dequant_args(a, q->dig, A) || !di_digits_ready(q, st)) return false;
  switch (dtype) {
    case TQ_F64: *rc = di_dequantize<double>(A, n, out, st); return true;
    case TQ_F32: *rc = di_dequantize<float>(A, n, out, st); return true;
    default: *rc = di_dequantize<__half>(A, n, out, st); return true;
  }
}

// The self-tests' forms: fp32 rows of 2 bits, with a sketch (sum 18 is one of a CTA's second tile) or without (sum 10, of its third); fp64
// results with a sketch
int tq_dense_i8_quantize_selftest(const tq_quantizer* q, const TqDenseQuant& a, const void* x, int64_t ld, int64_t n, cudaStream_t st) {
  DiQuant A;
  TQ_REQUIRE(a.bits == 2 && !a.out_qjl == !a.out_rnorm && di_quant_args(a, q->dig, x, TQ_F32, ld, A) && di_digits_ready(q, st), TQ_ERR_UNSUPPORTED,
             "self-test of the dense quantizer: fp32 rows of 128 elements and 2 bits");
  const float* xt = reinterpret_cast<const float*>(x);
  if (a.out_qjl) return di_launch<k_dense_quantize_i8<float, 2, true, 18>>(di_quant_smem<float, true>(), n, st, "k_dense_quantize_i8", A, xt, ld, n);
  return di_launch<k_dense_quantize_i8<float, 2, false, 10>>(di_quant_smem<float, false>(), n, st, "k_dense_quantize_i8", A, xt, ld, n);
}
// fp32 rows of 2 bits without a sketch, in a run with a role out of step
int tq_dense_i8_quantize_role(const tq_quantizer* q, const TqDenseQuant& a, const void* x, int64_t ld, int64_t n, int role, cudaStream_t st) {
  DiQuant A;
  TQ_REQUIRE(a.bits == 2 && di_quant_args(a, q->dig, x, TQ_F32, ld, A) && di_digits_ready(q, st), TQ_ERR_UNSUPPORTED,
             "self-test of the dense quantizer: fp32 rows of 128 elements and 2 bits");
  const float* xt = reinterpret_cast<const float*>(x);
  if (role == 0) return di_launch<k_dense_quantize_i8<float, 2, false, DI_LATE>>(di_quant_smem<float, false>(), n, st, "k_dense_quantize_i8", A, xt, ld, n);
  return di_launch<k_dense_quantize_i8<float, 2, false, DI_HASTY>>(di_quant_smem<float, false>(), n, st, "k_dense_quantize_i8", A, xt, ld, n);
}
int tq_dense_i8_dequantize_selftest(const tq_quantizer* q, const TqDenseDequant& a, int64_t n, double* out, cudaStream_t st) {
  DiDequant A;
  TQ_REQUIRE(a.qjl && di_dequant_args(a, q->dig, A) && di_digits_ready(q, st), TQ_ERR_UNSUPPORTED, "self-test of the dense dequantizer: 128 elements and a sketch");
  return di_dequantize_launch<double, true, 26>(A, n, out, st);
}
