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
// One persistent CTA per SM, 128 vectors a tile:
//   warps 0-15 rows: warps w, w + 4, w + 8 and w + 12 share the 32 vectors that are lanes 32 (w & 3) .. of tensor memory, a thread
//              32 columns of a vector (64 in eight warps: their loads of sums waited behind the MMAs' own traffic).  They norm
//              the rows (in NumPy's order), write the digits of the first operand into tensor memory (7 x 32 columns, four
//              digits a word) and add up the sums of its product with R: indices, whose centroids' digits are the next
//              operand; then, with the sketch, the residual's digits, and the signs.
//   warp 16    bulk copies of the matrices' digits, 16 KB each (laid out by k_dense_digits).  The sums run from s = 7 to 0, so that
//              digit s of a matrix has been read for the last time after sum s, and the next matrix follows it.
//   warp 17    every MMA: one s of all 128 outputs is an accumulator of 128 columns, of which two take turns.
// Shapes by measurement: an MMA of 128 x N x 32 takes 44 clocks (its issue) for N = 32 and 64, 65 for N = 128.
//
// What bounds it: a product takes 18,600 clocks where its 136 MMAs take 8,800.  The rows' loads of sums (700 clocks each under
// MMAs, 120 without) and their fp64 additions, eight of each of 128 x 128 sums, run between the MMAs rather than under them.
// 65,536 fp32 vectors, before (fp64 tensor cores) / now: quantize 134 / 77 us, with the sketch 302 / 182, dequantize 90 / 63 and 164 / 93.
//
// A wait that gives up ends the waits of all roles; the results of its tile and of those behind it are then not numbers, and a
// status word is set (tq_quantize_status_sync).
//
// A row that this arithmetic does not carry -- values that are not finite or too small for a norm, residuals far beyond the
// vector's length, which an arbitrary matrix can produce -- is computed by one warp in plain fp64.
#include <mutex>
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
// the digits of an fp32 value below 2 in magnitude, from its bits: significand x 2^(exponent - 96); what a value below 2^-31 has
// beyond 2^-54 is cut off
__device__ __forceinline__ uint2 di_digits_f32(float v) {
  const uint32_t u = __float_as_uint(v), e = (u >> 23) & 255u, m = (u & 0x7fffffu) | (e ? 0x800000u : 0u);
  const uint32_t lo = e >= 96u ? m << ((e - 96u) & 31u) : e > 64u ? m >> (96u - e) : 0u, hi = e >= 96u ? __funnelshift_l(m, 0u, e - 96u) : 0u;
  const uint32_t neg = (uint32_t)((int)u >> 31);
  const uint64_t w = (((uint64_t)(hi ^ neg) << 32) | (lo ^ neg)) + (0x808080808080ull + (neg & 1u));   // -x = ~x + 1
  return make_uint2((uint32_t)w ^ 0x80808080u, (uint32_t)(w >> 32) ^ 0x8080u);
}
// of an fp64 value below 2 in magnitude: to a whole number of 2^-54 in two steps of a large constant's rounding
__device__ __forceinline__ uint2 di_digits_f64(double v) {
  constexpr double BIG = 6755399441055744.0;                            // 1.5 x 2^52: a sum's low bits are the whole number
  const double hi = fma(v, 4194304.0, BIG);                             // v x 2^22
  const double rest = fma(hi - BIG, -2.384185791015625e-07, v);         // exact
  const double lo = fma(rest, 18014398509481984.0, BIG);                // the rest x 2^54, at most 2^31
  const long long w = (__double_as_longlong(lo) - __double_as_longlong(BIG)) + ((long long)__double2loint(hi) << 32);
  return di_split(di_digits(w));
}
// digits of eight consecutive elements -> the seven operand words of each four of them, stored at column `col` of every digit
__device__ __forceinline__ void di_store8(uint32_t area, int col, const uint2 (&u)[8]) {
  uint32_t w[DI_DIGITS][2];
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    const uint2 a = u[4 * g], b = u[4 * g + 1], c = u[4 * g + 2], d = u[4 * g + 3];
    const uint32_t ab = __byte_perm(a.x, b.x, 0x5140), cd = __byte_perm(c.x, d.x, 0x5140);
    const uint32_t ab2 = __byte_perm(a.x, b.x, 0x7362), cd2 = __byte_perm(c.x, d.x, 0x7362);
    const uint32_t hab = __byte_perm(a.y, b.y, 0x5140), hcd = __byte_perm(c.y, d.y, 0x5140);
    w[6][g] = __byte_perm(ab, cd, 0x5410);
    w[5][g] = __byte_perm(ab, cd, 0x7632);
    w[4][g] = __byte_perm(ab2, cd2, 0x5410);
    w[3][g] = __byte_perm(ab2, cd2, 0x7632);
    w[2][g] = __byte_perm(hab, hcd, 0x5410);
    w[1][g] = __byte_perm(hab, hcd, 0x7632);
    w[0][g] = __byte_perm(__byte_perm(a.y, b.y, 0x0062), __byte_perm(c.y, d.y, 0x0062), 0x5410);
  }
#pragma unroll
  for (int p = 0; p < DI_DIGITS; ++p) di_st2(area + 32 * p + col, w[p][0], w[p][1]);
}

// int32 -> double: 2^52 + 2^31 + v has v ^ 0x80000000 in its low word
__device__ __forceinline__ double di_double(uint32_t v) { return __hiloint2double(0x43300000, (int)(v ^ 0x80000000u)) - 4503601774854144.0; }

// Barriers and the way of the roles through them; the row warps and the MMA warp count alike.
struct DiShared {
  uint64_t b_full[DI_DIGITS], b_free[DI_DIGITS], d_full[2], d_free[2], a_ready, drained;
  uint32_t tmem;
  volatile int failed;   // a wait gave up: nobody waits any more
};
// SELFTEST: waits are short, and one accumulator of the first CTA's second tile is never reported as full (di_issue)
template <bool SELFTEST> __device__ __forceinline__ void di_wait(DiShared& s, uint64_t* bar, uint32_t parity) {
  tc_wait(bar, parity, &s.failed, SELFTEST ? TC_SELFTEST_CYCLES : TC_WAIT_CYCLES);
}
__device__ __forceinline__ void di_init(DiShared& s) {
  auto init = [](uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sptr(bar)), "r"(count) : "memory");
  };
  for (int i = 0; i < DI_DIGITS; ++i) init(&s.b_full[i], 1), init(&s.b_free[i], 1);
  for (int i = 0; i < 2; ++i) init(&s.d_full[i], 1), init(&s.d_free[i], DI_ROW_THREADS / 32);
  init(&s.a_ready, DI_ROW_THREADS / 32);
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

// The copier's way: the digits of the matrices that `matrix(i)` gives, each into the place of the matrix before
template <bool SELFTEST, typename M> __device__ __forceinline__ void di_copier(DiShared& s, uint8_t* tiles, int count, M&& matrix) {
  int copies = 0;
  for (int i = 0; i < count && !s.failed; ++i) {
    const uint8_t* src = matrix(i);
    for (int p = DI_DIGITS - 1; p >= 0; --p, ++copies) {
      if (i > 0) di_wait<SELFTEST>(s, &s.b_free[p], (uint32_t)((i - 1) & 1));
      if (s.failed) break;
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sptr(&s.b_full[p])), "r"(DI_TILE) : "memory");
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sptr(tiles + p * DI_TILE)),
                   "l"(src + p * DI_TILE), "r"(DI_TILE), "r"(sptr(&s.b_full[p])) : "memory");
    }
  }
  for (int p = 0; p < DI_DIGITS; ++p) {   // none in flight at the end, also after a wait that gave up
    const int mine = (copies + p) / DI_DIGITS;
    if (mine > 0) tc_wait(&s.b_full[p], (uint32_t)((mine - 1) & 1));
  }
}

// The MMA warp: the operand at `area`, of DIGITS digits, against the `matrix`-th matrix; s from the last to the first
template <int DIGITS, bool SELFTEST>
__device__ __forceinline__ void di_issue(DiShared& s, int& item, const uint8_t* tiles, int matrix, uint32_t area, uint32_t acc_base) {
  constexpr int TOP = DI_DIGITS - 1, LAST = DIGITS == 1 ? TOP : DI_SUMS - 1;
  const uint32_t b = sptr(tiles), idesc = di_idesc();
#pragma unroll
  for (int sum = LAST; sum >= 0; --sum, ++item) {
    const int sl = item & 1;
    if (item >= 2) di_wait<SELFTEST>(s, &s.d_free[sl], (uint32_t)((item / 2 - 1) & 1));
#pragma unroll
    for (int q = 0; q < DI_DIGITS; ++q)   // digits used for the first time
      if (DIGITS == 1 ? q == sum : sum == LAST ? q > 0 : sum == LAST - 1 && q == 0) di_wait<SELFTEST>(s, &s.b_full[q], (uint32_t)(matrix & 1));
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
    for (int p = 0; p < DIGITS; ++p) {
      const int q = sum - p;
      if (q < 0 || q > TOP) continue;
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)
        di_mma(acc_base + 128 * sl, area + 32 * p + 8 * ks, umma_desc(b + q * DI_TILE + ks * 256, 128, 1024), idesc,
               p == (sum > TOP ? sum - TOP : 0) && ks == 0 ? 0u : 1u);
    }
    if (!(SELFTEST && blockIdx.x == 0 && item == 26)) di_commit(&s.d_full[sl]);   // (a tile with a sketch: 24 items, 15 to dequantize)
    if (sum < DI_DIGITS) di_commit(&s.b_free[sum]);
  }
}

// ... and nothing of its in flight at the end, also after a wait that gave up (else the rows have waited for every product)
__device__ __forceinline__ void di_drain(DiShared& s) {
  if (!__any_sync(0xffffffffu, s.failed)) return;
  __syncwarp();
  di_commit(&s.drained);
  tc_wait(&s.drained, 0);
}

// A row warp: acc += base x (the product's sums, 256^-s each), 32 columns of a thread
template <int DIGITS, bool SELFTEST>
__device__ __forceinline__ void di_take(DiShared& s, int& item, uint32_t acc_base, int lane, double base, double (&acc)[DI_COLS]) {
  constexpr int LAST = DIGITS == 1 ? DI_DIGITS - 1 : DI_SUMS - 1;
  double factor = base;
#pragma unroll
  for (int i = 0; i < LAST; ++i) factor *= 0.00390625;
#pragma unroll 1
  for (int sum = LAST; sum >= 0; --sum, ++item, factor *= 256.0) {
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
      for (int k = 0; k < 8; ++k) acc[8 * c + k] = fma(di_double(v[c & 1][k]), factor, acc[8 * c + k]);
    }
  }
}
__device__ __forceinline__ void di_zero(double (&acc)[DI_COLS]) {
#pragma unroll
  for (int k = 0; k < DI_COLS; ++k) acc[k] = 0.0;
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
  double r_scale;                     // R w = sums x this
  double cent_scale;                  // power of two above every centroid's magnitude
  double bnd[15];                     // boundaries (parameters: operands of the comparisons as they are)
  int32_t* status;                    // raised when a wait gives up
  TqDenseQuant q;
};
struct DiDequant {
  const uint8_t *rt, *st;
  double r_scale, s_scale, cent_scale;
  int32_t* status;
  TqDenseDequant q;
};

// A whole row in fp64, by one warp (four outputs a lane)
template <typename Tin>
__device__ void di_row_plain(const TqDenseQuant& a, const uint8_t* xrow, float nrm, int64_t v, int lane) {
  const Tin* x = reinterpret_cast<const Tin*>(xrow);
  const float safe = nrm > 0.f ? nrm : 1.0f;
  const int nb = (1 << a.bits) - 1;
  double y[4] = {0, 0, 0, 0};
  for (int k = 0; k < TQ_D; ++k) {
    const double w = (double)(di_f<Tin>(x[k]) / safe);
#pragma unroll
    for (int j = 0; j < 4; ++j) y[j] = fma(a.rot[(size_t)(4 * lane + j) * TQ_D + k], w, y[j]);
  }
  int m[4];
  double cc = 0.0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    m[j] = 0;
    for (int b = 0; b < nb; ++b) m[j] += a.bnd[b] < y[j] ? 1 : 0;
    cc += a.cent[m[j]] * a.cent[m[j]];
    if (a.out_idx) a.out_idx[v * TQ_D + 4 * lane + j] = (uint8_t)m[j];
  }
#pragma unroll
  for (int h = 16; h > 0; h >>= 1) cc += __shfl_xor_sync(0xffffffffu, cc, h);
  double cn = sqrt(cc);
  cn = cn > 1e-10 ? cn : 1.0;
  if (lane == 0) {
    if (a.out_norm) a.out_norm[v] = nrm;
    if (a.out_scale) a.out_scale[v] = (float)(a.norm_correction ? (double)nrm / cn : (double)nrm);
  }
  if (!a.out_qjl && !a.out_rnorm) return;
  const double inv = a.norm_correction ? 1.0 / cn : 1.0;
  double e[4] = {0, 0, 0, 0}, rr = 0.0;
  for (int k = 0; k < TQ_D; ++k) {
    const int mk = __shfl_sync(0xffffffffu, (k & 2) ? ((k & 1) ? m[3] : m[2]) : ((k & 1) ? m[1] : m[0]), k >> 2);
    const double c = a.cent[mk] * inv;
#pragma unroll
    for (int j = 0; j < 4; ++j) e[j] = fma(a.rot_t[(size_t)(4 * lane + j) * TQ_D + k], c, e[j]);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    e[j] = (double)di_f<Tin>(x[4 * lane + j]) - e[j] * (double)nrm;
    rr += e[j] * e[j];
  }
#pragma unroll
  for (int h = 16; h > 0; h >>= 1) rr += __shfl_xor_sync(0xffffffffu, rr, h);
  if (lane == 0 && a.out_rnorm) a.out_rnorm[v] = (float)sqrt(rr);
  if (!a.out_qjl) return;
  double p[4] = {0, 0, 0, 0};
  for (int k = 0; k < TQ_D; ++k) {
    const double ek = __shfl_sync(0xffffffffu, (k & 2) ? ((k & 1) ? e[3] : e[2]) : ((k & 1) ? e[1] : e[0]), k >> 2);
#pragma unroll
    for (int j = 0; j < 4; ++j) p[j] = fma(a.s[(size_t)(4 * lane + j) * TQ_D + k], ek, p[j]);
  }
  uint32_t nib = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) nib = (nib << 1) | (p[j] < 0.0 ? 0u : 1u);
  const uint32_t up = __shfl_down_sync(0xffffffffu, nib, 1);
  if ((lane & 1) == 0) a.out_qjl[v * 16 + (lane >> 1)] = (uint8_t)((nib << 4) | up);
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
template <typename Tin> constexpr int di_quant_smem() { return DI_DIGITS * DI_TILE + DI_ROWS * di_row_bytes<Tin>() + 128; }

// PROD: residual, its norm and the sketch as well
template <typename Tin, int BITS, bool PROD, bool SELFTEST = false>
__global__ void __launch_bounds__(DI_THREADS, 1) k_dense_quantize_i8(const __grid_constant__ DiQuant A, const Tin* __restrict__ x, int64_t ld,
                                                                     int64_t n) {
  constexpr int ROWB = di_row_bytes<Tin>();
  extern __shared__ __align__(128) uint8_t di_raw[];
  __shared__ DiShared sh;
  __shared__ uint2 s_cdig[16];                  // digits of the centroids
  __shared__ double s_sq[16], s_part[4][DI_ROWS];
  __shared__ float s_norm[DI_ROWS];
  __shared__ uint8_t s_plain[DI_ROWS];          // rows for di_row_plain
  const TqDenseQuant& a = A.q;
  uint8_t* tiles_b = di_raw + (((sptr(di_raw) + 127u) & ~127u) - sptr(di_raw));
  uint8_t* xs = tiles_b + DI_DIGITS * DI_TILE;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) di_init(sh);
  if (tid < 16) {
    const double c = tid < (1 << BITS) ? a.cent[tid] : 0.0;
    s_sq[tid] = c * c;
    s_cdig[tid] = di_digits_f64(c / A.cent_scale);
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
  constexpr int PHASES = PROD ? 3 : 1;

  if (warp == DI_COPIER) {
    if (lane == 0) di_copier<SELFTEST>(sh, tiles_b, mine * PHASES, [&](int i) { return !PROD || i % 3 == 0 ? A.r : i % 3 == 1 ? A.rt : A.s; });
  } else if (warp == DI_MMA) {
    int item = 0;
    for (int i = 0; i < mine * PHASES && !__any_sync(0xffffffffu, sh.failed); ++i) {
      di_wait<SELFTEST>(sh, &sh.a_ready, (uint32_t)(i & 1));
      di_issue<DI_DIGITS, SELFTEST>(sh, item, tiles_b, i, tb, tb + DI_ACC);
    }
    di_drain(sh);
  } else {
    const int row = 32 * (warp & 3) + lane, h = warp >> 2;       // this thread's vector, and its columns 32 h .. + 31
    const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
    const uint32_t area = tb + lanes, myacc = tb + DI_ACC + lanes + DI_COLS * h;
    auto operand_ready = [&]() {
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) di_arrive(&sh.a_ready);
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
    int item = 0, t = 0;
    if (mine > 0) load_tile(blockIdx.x);
    for (; t < mine; ++t) {
      const int64_t v0 = (blockIdx.x + t * step) * DI_ROWS, v = v0 + row;
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      if (di_rows_any(sh.failed)) break;   // (in the tile before)
      // norms in the rows' own precision and NumPy's order (first term + pairwise sum of the rest), eight lanes a vector, two
      // vectors of a lane at once
      {
        const int j = tid & 7;
        const Tin* xr[2] = {};
        float s[2];
        auto sq = [&](int q, int k) { const float f = di_f<Tin>(xr[q][k]); return __fmul_rn(f, f); };
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          xr[q] = reinterpret_cast<const Tin*>(xs + ((tid >> 3) + 64 * q) * ROWB);
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
          if (j == 0) s_norm[(tid >> 3) + 64 * q] = sqrtf(__fadd_rn(sq(q, 0), s[q]));
      }
      if (tid < DI_ROWS) s_plain[tid] = 0;
      di_rows_sync();
      const float nrm = s_norm[row], safe = nrm > 0.f ? nrm : 1.0f;                // turboquant/polar_quant.py:74
      bool plain = false;
      {
        // w = x / ||x|| in the rows' precision (:75).  As x times the fp64 reciprocal, rounded once to fp32: the quotient of two 24-bit
        // significands is never within 2^-49 of a rounding boundary, and the fp64 product is off by 2^-52 at most, so this is the
        // correctly rounded quotient, without the branch of a division.
        const double inv = 1.0 / (double)safe;
        const uint8_t* xr = xs + row * ROWB + DI_COLS * h * sizeof(Tin);
#pragma unroll 1
        for (int c = 0; c < DI_COLS / 8; ++c) {
          float f[8];
          di_load8<Tin>(xr + 8 * c * sizeof(Tin), f);
          uint2 u[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const float w = (float)((double)f[k] * inv);
            plain |= !(fabsf(w) < DI_LARGEST) || (nrm == 0.f && f[k] != 0.f);   // (squares below the fp32 range: w = x)
            u[k] = di_digits_f32(w);
          }
          di_store8(area, 8 * h + 2 * c, u);
        }
      }
      if (plain) s_plain[row] = 1;
      operand_ready();
      // rows for the plain arithmetic: whole ones, while the rows are in shared memory; their results otherwise are dropped
      auto plain_rows = [&]() {
        if (!di_rows_any(plain)) return;
        for (int r = warp; r < DI_ROWS; r += DI_ROW_THREADS / 32)
          if (s_plain[r] && v0 + r < n) di_row_plain<Tin>(a, xs + r * ROWB, s_norm[r], v0 + r, lane);
        plain = s_plain[row] != 0;
        di_rows_sync();
      };
      if constexpr (!PROD) {
        plain_rows();
        if (t + 1 < mine) load_tile(blockIdx.x + (t + 1) * step);
      }
      bool live = v < n && !plain;
      // ---- y = R w: indices, ||c[idx]||^2, the centroids as the next operand ----
      double acc[DI_COLS], cc[4] = {0.0, 0.0, 0.0, 0.0};
      di_zero(acc);
      di_take<DI_DIGITS, SELFTEST>(sh, item, myacc, lane, A.r_scale, acc);
      uint32_t packed[DI_COLS / 4];
#pragma unroll
      for (int g = 0; g < DI_COLS / 4; ++g) {
        packed[g] = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          uint32_t m = 0;                                  // boundaries below y (searchsorted, side = 'left')
#pragma unroll
          for (int b = 0; b < (1 << BITS) - 1; ++b) m += A.bnd[b] < acc[4 * g + k] ? 1u : 0u;
          packed[g] |= m << (8 * k);
          cc[k] += s_sq[m];
        }
      }
      if (live && a.out_idx) {
#pragma unroll
        for (int g = 0; g < DI_COLS / 4; g += 4)
          *reinterpret_cast<uint4*>(a.out_idx + v * TQ_D + DI_COLS * h + 4 * g) = make_uint4(packed[g], packed[g + 1], packed[g + 2], packed[g + 3]);
      }
      s_part[h][row] = (cc[0] + cc[1]) + (cc[2] + cc[3]);
      if constexpr (PROD) {
#pragma unroll
        for (int c = 0; c < DI_COLS / 8; ++c) {
          uint2 u[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) u[k] = s_cdig[(packed[2 * c + (k >> 2)] >> (8 * (k & 3))) & 15];
          di_store8(area, 8 * h + 2 * c, u);
        }
        operand_ready();
      }
      di_rows_sync();
      double cn = sqrt((s_part[0][row] + s_part[1][row]) + (s_part[2][row] + s_part[3][row]));
      cn = cn > 1e-10 ? cn : 1.0;                                                 // turboquant/polar_quant.py:110-111
      if (h == 0 && live) {
        if (a.out_norm) a.out_norm[v] = nrm;
        if (a.out_scale) a.out_scale[v] = (float)(a.norm_correction ? (double)nrm / cn : (double)nrm);
      }
      if constexpr (PROD) {
        // ---- x_hat = norm R^T c / ||c||, residual x - x_hat, with the norm that is returned and stored (fp32) ----
        const double back = A.r_scale * A.cent_scale * (a.norm_correction ? 1.0 / cn : 1.0) * (double)nrm;
        const double unit = nrm > 0.f && nrm < 1e38f ? ldexp(1.0, -(ilogbf(nrm) + 2)) : 1.0;   // |residual| x unit < 1 for a rotation
        double rr[4] = {0.0, 0.0, 0.0, 0.0};
        di_zero(acc);
        di_take<DI_DIGITS, SELFTEST>(sh, item, myacc, lane, back, acc);
        const uint8_t* xr = xs + row * ROWB + DI_COLS * h * sizeof(Tin);
#pragma unroll
        for (int c = 0; c < DI_COLS / 8; ++c) {
          float f[8];
          di_load8<Tin>(xr + 8 * c * sizeof(Tin), f);
          uint2 u[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const double e = (double)f[k] - acc[8 * c + k], es = e * unit;
            rr[k & 3] = fma(e, e, rr[k & 3]);
            plain |= !(fabs(es) < (double)DI_LARGEST);
            u[k] = di_digits_f64(es);
          }
          di_store8(area, 8 * h + 2 * c, u);
        }
        di_rows_sync();   // (the sums of the squared centroids have been read)
        s_part[h][row] = (rr[0] + rr[1]) + (rr[2] + rr[3]);
        if (plain) s_plain[row] = 1;
        operand_ready();
        plain_rows();
        live = v < n && !plain;
        if (h == 0 && live && a.out_rnorm)
          a.out_rnorm[v] = (float)sqrt((s_part[0][row] + s_part[1][row]) + (s_part[2][row] + s_part[3][row]));
        if (t + 1 < mine) load_tile(blockIdx.x + (t + 1) * step);
        // ---- sketch: sign(S r), zero counts as +1 (turboquant/qjl.py:89-90), first column in the most significant bit ----
        di_zero(acc);
        di_take<DI_DIGITS, SELFTEST>(sh, item, myacc, lane, 1.0, acc);
        uint32_t m = 0;
#pragma unroll
        for (int k = 0; k < DI_COLS; ++k) m = (m << 1) | (acc[k] < 0.0 ? 0u : 1u);
        m = __byte_perm(m, 0, 0x0123);
        if (live && a.out_qjl) {
          uint8_t* z = a.out_qjl + v * 16 + 4 * h;
          if ((reinterpret_cast<uintptr_t>(a.out_qjl) & 3) == 0) *reinterpret_cast<uint32_t*>(z) = m;
          else z[0] = (uint8_t)m, z[1] = (uint8_t)(m >> 8), z[2] = (uint8_t)(m >> 16), z[3] = (uint8_t)(m >> 24);
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (di_rows_any(sh.failed)) {   // the last tile begun and those behind it
      di_give_up(a, t > 0 ? t - 1 : 0, mine, h == 0 ? row : -1, n, A.status);
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tb), "r"(512u) : "memory");
}

constexpr int DI_IDX_ROW = TQ_D + 16, DI_OUT_ROW = 16 * 8 + 16;   // bytes between staged rows: 16 bytes on, no bank conflicts
constexpr int DI_DEQUANT_SMEM = DI_DIGITS * DI_TILE + DI_ROWS * DI_IDX_ROW + DI_ROW_THREADS * DI_OUT_ROW + 128;

// x_hat = (norm / ||c[idx]||) R^T c[idx] + shrink sqrt(pi/2)/sqrt(d) rnorm S^T z.  The signs z are one digit, +-1: seven products.
template <typename Tout, bool PROD, bool SELFTEST = false>
__global__ void __launch_bounds__(DI_THREADS, 1) k_dense_dequantize_i8(const __grid_constant__ DiDequant A, int64_t n, Tout* __restrict__ out) {
  extern __shared__ __align__(128) uint8_t di_raw[];
  __shared__ DiShared sh;
  __shared__ uint2 s_cdig[16];
  __shared__ uint32_t s_sign[16];               // four sketch bits, the first in bit 3, as +-1 digits
  __shared__ double s_sq[16], s_part[4][DI_ROWS];
  const TqDenseDequant& a = A.q;
  uint8_t* tiles_b = di_raw + (((sptr(di_raw) + 127u) & ~127u) - sptr(di_raw));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) di_init(sh);
  if (tid < 16) {
    const double c = tid < (1 << a.bits) ? a.cent[tid] : 0.0;
    s_sq[tid] = c * c;
    s_cdig[tid] = di_digits_f64(c / A.cent_scale);
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
  constexpr int PHASES = PROD ? 2 : 1;   // (the signs' product first)

  if (warp == DI_COPIER) {
    if (lane == 0) di_copier<SELFTEST>(sh, tiles_b, mine * PHASES, [&](int i) { return PROD && (i & 1) == 0 ? A.st : A.rt; });
  } else if (warp == DI_MMA) {
    int item = 0;
    for (int i = 0; i < mine && !__any_sync(0xffffffffu, sh.failed); ++i) {
      di_wait<SELFTEST>(sh, &sh.a_ready, (uint32_t)(i & 1));
      if constexpr (PROD) di_issue<1, SELFTEST>(sh, item, tiles_b, 2 * i, tb + DI_SIGNS, tb + DI_ACC);
      di_issue<DI_DIGITS, SELFTEST>(sh, item, tiles_b, PROD ? 2 * i + 1 : i, tb, tb + DI_ACC);
    }
    di_drain(sh);
  } else {
    const int row = 32 * (warp & 3) + lane, h = warp >> 2;
    const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
    const uint32_t area = tb + lanes, myacc = tb + DI_ACC + lanes + DI_COLS * h;
    const bool wide = (a.ld_out * sizeof(Tout)) % 16 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    uint8_t* xi = tiles_b + DI_DIGITS * DI_TILE;                           // indices of a tile
    uint8_t* stage = xi + DI_ROWS * DI_IDX_ROW + warp * 32 * DI_OUT_ROW;   // 32 rows x 16 columns of this warp on their way out
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
    int item = 0, t = 0;
    if (mine > 0) load_tile(blockIdx.x);
    for (; t < mine; ++t) {
      const int64_t v0 = (blockIdx.x + t * step) * DI_ROWS, v = v0 + row;
      const bool live = v < n;
      const float norm = live ? a.norm[v] : 0.f, rnorm = PROD && live ? a.rnorm[v] : 0.f;
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      if (di_rows_any(sh.failed)) break;   // (in the tile before)
      // ---- digits of the centroids, ||c||^2, signs ----
      double cc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
      for (int c = 0; c < DI_COLS / 8; ++c) {
        const uint2 q = *reinterpret_cast<const uint2*>(xi + row * DI_IDX_ROW + DI_COLS * h + 8 * c);
        uint2 u[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int m = ((k < 4 ? q.x : q.y) >> (8 * (k & 3))) & 15;
          u[k] = s_cdig[m];
          cc[k & 3] += s_sq[m];
        }
        di_store8(area, 8 * h + 2 * c, u);
        if constexpr (PROD) {   // eight sketch bits, the first in the most significant place
          const uint32_t z = live ? a.qjl[v * 16 + 4 * h + c] : 0u;
          di_st2(area + DI_SIGNS + 8 * h + 2 * c, s_sign[z >> 4], s_sign[z & 15]);
        }
      }
      s_part[h][row] = (cc[0] + cc[1]) + (cc[2] + cc[3]);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) di_arrive(&sh.a_ready);
      di_rows_sync();
      if (t + 1 < mine) load_tile(blockIdx.x + (t + 1) * step);
      double f = 0.0, g = 0.0;
      if (live) {
        double cn = 1.0;
        if (a.norm_correction) {
          cn = sqrt((s_part[0][row] + s_part[1][row]) + (s_part[2][row] + s_part[3][row]));
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
      double acc[DI_COLS];
      di_zero(acc);
      if constexpr (PROD) di_take<1, SELFTEST>(sh, item, myacc, lane, g, acc);
      di_take<DI_DIGITS, SELFTEST>(sh, item, myacc, lane, f, acc);
      Tout* o = out + v * a.ld_out + DI_COLS * h;
      if (a.accumulate && live) {
#pragma unroll
        for (int k = 0; k < DI_COLS; ++k) acc[k] += di_d<Tout>(o[k]);
      }
      if (sizeof(Tout) == 8 && wide) {
        // Sixteen columns at a time through shared memory: a warp then stores whole lines, four rows an instruction (straight from
        // the registers every store touched 32 lines: 4,400 clocks a tile)
#pragma unroll
        for (int c = 0; c < DI_COLS / 16; ++c) {
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 16; k += 2) *reinterpret_cast<double2*>(stage + lane * DI_OUT_ROW + 8 * k) = make_double2(acc[16 * c + k], acc[16 * c + k + 1]);
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int r = 4 * i + (lane >> 3);
            const double2 p = *reinterpret_cast<const double2*>(stage + r * DI_OUT_ROW + 16 * (lane & 7));
            const int64_t vr = v0 + 32 * (warp & 3) + r;
            if (vr < n) *reinterpret_cast<double2*>(out + vr * a.ld_out + DI_COLS * h + 16 * c + 2 * (lane & 7)) = p;
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
    return di_launch<k_dense_quantize_i8<Tin, BITS, true>>(di_quant_smem<Tin>(), n, st, "k_dense_quantize_i8", A, x, ld, n);
  return di_launch<k_dense_quantize_i8<Tin, BITS, false>>(di_quant_smem<Tin>(), n, st, "k_dense_quantize_i8", A, x, ld, n);
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
template <typename Tout> int di_dequantize(const DiDequant& A, int64_t n, void* out, cudaStream_t st) {
  Tout* o = reinterpret_cast<Tout*>(out);
  if (A.q.qjl) return di_launch<k_dense_dequantize_i8<Tout, true>>(DI_DEQUANT_SMEM, n, st, "k_dense_dequantize_i8", A, n, o);
  return di_launch<k_dense_dequantize_i8<Tout, false>>(DI_DEQUANT_SMEM, n, st, "k_dense_dequantize_i8", A, n, o);
}

}  // namespace

// The power of two that a matrix's digits are relative to, or 0 for a matrix that stays with the fp64 kernels.
// The digits are fixed-point numbers of 2^-54 of the largest entry, where fp64 keeps every entry's own exponent.  No product may lose
// by that, so: every row and column is at least sqrt(2) times as long as the largest entry (the rounding of a row's digits is then
// 2^-55 of that row's length, below that of fp64 sums), and no entry is below 2^-30 of it (a row of x enters with 2^-54 of its length;
// an entry of zero would hide its large elements, and what an output then sees may be smaller than that).  Random rotations
// and Gaussian matrices are of this kind (their rows are three times and twice as long); uneven, diagonal or block matrices and what
// is not finite are not.
double tq_dense_digits_scale(const double* m) {
  double most = 0.0, least = 1e300, row[TQ_D] = {}, col[TQ_D] = {};
  for (int i = 0; i < TQ_D; ++i)
    for (int j = 0; j < TQ_D; ++j) {
      const double a = fabs(m[i * TQ_D + j]);
      most = a > most ? a : most;
      least = a < least ? a : least;
      row[i] += a * a;
      col[j] += a * a;
    }
  if (!(most > 1e-100 && most < 1e100 && least >= most * 0x1p-30)) return 0.0;
  for (int i = 0; i < TQ_D; ++i)
    if (!(row[i] >= 2.0 * most * most && col[i] >= 2.0 * most * most)) return 0.0;   // (also what is not a number)
  int e = 0;
  frexp(most, &e);   // most < 2^e
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

// Calls that come here, us here / in the fp64 kernels (which take tiles of 16, 32 or 64 vectors, two CTAs an SM, and step up at 32
// and 64 vectors per SM): quantize 8,192 vectors 23.2 / 23.2, 12,000 23.2 / 39.6, 65,536 77 / 134; with the sketch 4,096 50 / 34, 8,192
// 52 / 52, 12,000 56 / 94, 65,536 182 / 302; dequantize 8,192 19 / 17, 12,000 19 / 29, 65,536 63 / 90; with the sketch 4,096 28 / 23,
// 6,000 29 / 31, 65,536 93 / 164.
static bool di_enough(int64_t n, bool sketched_dequantize) { return n > (sketched_dequantize ? 32 : 64) * (int64_t)tq_num_sms(); }

// The kernels' arguments; false: not of these kernels' kind
static bool di_quant_args(const TqDenseQuant& a, const TqDenseDigits& g, const void* x, int32_t dtype, int64_t ld, DiQuant& A) {
  const bool prod = a.out_qjl || a.out_rnorm;
  if (a.d != TQ_D || g.r_scale == 0.0 || g.cent_scale == 0.0 || a.out_packed || a.out_res || (prod && g.s_scale == 0.0)) return false;
  if (dtype != TQ_F32 && dtype != TQ_F16) return false;
  if (!tq_aligned(x, 16) || ld * (dtype == TQ_F32 ? 4 : 2) % 16 || !tq_aligned(a.out_idx, 16)) return false;
  A.r = g.r; A.rt = g.rt; A.s = g.s;
  A.r_scale = g.r_scale / 4096.0;
  A.cent_scale = g.cent_scale;
  A.status = tq_quantize_status_word();
  for (int i = 0; i < 15; ++i) A.bnd[i] = g.bnd[i];
  A.q = a;
  return true;
}
static bool di_dequant_args(const TqDenseDequant& a, const TqDenseDigits& g, DiDequant& A) {
  if (a.d != TQ_D || g.r_scale == 0.0 || g.cent_scale == 0.0 || !a.idx || (a.qjl && g.s_scale == 0.0)) return false;
  if (!tq_aligned(a.idx, 16)) return false;
  A.rt = g.rt; A.st = g.st;
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
  if (!di_enough(n, false) || !di_quant_args(a, q->dig, x, dtype, ld, A) || !di_digits_ready(q, st)) return false;
  *rc = dtype == TQ_F32 ? di_quantize<float>(A, x, ld, n, st) : di_quantize<__half>(A, x, ld, n, st);
  return true;
}

bool tq_dense_i8_dequantize_try(const tq_quantizer* q, const TqDenseDequant& a, int64_t n, void* out, int32_t dtype, cudaStream_t st, int* rc) {
  DiDequant A;
  if (dtype != TQ_F64 && dtype != TQ_F32 && dtype != TQ_F16) return false;
  if (!di_enough(n, a.qjl != nullptr) || !di_dequant_args(a, q->dig, A) || !di_digits_ready(q, st)) return false;
  switch (dtype) {
    case TQ_F64: *rc = di_dequantize<double>(A, n, out, st); return true;
    case TQ_F32: *rc = di_dequantize<float>(A, n, out, st); return true;
    default: *rc = di_dequantize<__half>(A, n, out, st); return true;
  }
}

// The self-tests' forms: fp32 rows of 2 bits and a sketch; fp64 results with a sketch
int tq_dense_i8_quantize_selftest(const tq_quantizer* q, const TqDenseQuant& a, const void* x, int64_t ld, int64_t n, cudaStream_t st) {
  DiQuant A;
  TQ_REQUIRE(a.bits == 2 && a.out_qjl && di_quant_args(a, q->dig, x, TQ_F32, ld, A) && di_digits_ready(q, st), TQ_ERR_UNSUPPORTED,
             "self-test of the dense quantizer: fp32 rows of 128 elements, 2 bits and a sketch");
  return di_launch<k_dense_quantize_i8<float, 2, true, true>>(di_quant_smem<float>(), n, st, "k_dense_quantize_i8", A,
                                                              reinterpret_cast<const float*>(x), ld, n);
}
int tq_dense_i8_dequantize_selftest(const tq_quantizer* q, const TqDenseDequant& a, int64_t n, double* out, cudaStream_t st) {
  DiDequant A;
  TQ_REQUIRE(a.qjl && di_dequant_args(a, q->dig, A) && di_digits_ready(q, st), TQ_ERR_UNSUPPORTED, "self-test of the dense dequantizer: 128 elements and a sketch");
  return di_launch<k_dense_dequantize_i8<double, true, true>>(DI_DEQUANT_SMEM, n, st, "k_dense_dequantize_i8", A, n, out);
}
