// d = 128 sign-WHT quantizer for long appends: 128 vectors a tcgen05 tile, a thread a vector.
//
//   k_quantize_tc<Tin, BITS, NORMC>   Tin = __half or __nv_bfloat16, symmetric codebook, packed output.
//
// The 16-point stage of the rotation, H128 = H8 (x) H16, is eight 128 x 16 x 16 products whose second operand is +-1: exact
// products, fp32 sums.  With the sums in tensor memory a thread owns one vector (lane = vector): the 8-point stage, norms,
// and level counts are sums in its own registers and the packed indices are its own 16 b bytes: no exchanges between lanes,
// no staging.  The warp-level kernel (tq_quantize_mma.cu) deals a vector to four lanes: quad reductions and a 4 x 4 word
// transpose, 72 warp-instructions per turbo3 vector.  Every sum that decides an index is formed in that kernel's order (the whole
// 128-point rotation as one product rounds otherwise, and a handful of indices in a million vectors then differ).
//
//   * One CTA per SM: a warp issues the tiled copies of the rows (a ring of operand tiles), a warp the MMAs (a ring of
//     accumulators in tensor memory), and four groups of four warps take the accumulators in turn: 96 registers a thread, one
//     piece of 32 columns at a time.  Three groups with 128 are a sixth slower; loads and MMAs issued by the groups themselves a half.
//   * the last stage of the 8-point transform gives minus the value, (-a) - b and b - a, as in the warp-level kernel: the sign bit
//     of a sum alone decides the centre boundary.  A zero by cancellation is not above it; one from two zeros comes out as -0 and
//     takes the upper central index -- in both kernels, so that a record does not depend on its append's length.
//   * thresholds are scaled by the vector's norm; a magnitude level is found bit by bit, the threshold of the next bit picked
//     arithmetically; eight indices are an exact fp32 Horner sum; sign2 mirrors an index, an XOR of the packed words; level
//     counts, exact small integers, give the norm correction.
//   * PROD keys (2 or 3 index bits): the residual and the two 128-point transforms of the sign sketch are butterflies in a thread's registers,
//     64 values at a time and back to tensor memory in between (qt_sketch), every sum in the warp-level kernel's order, so that a
//     key's record is the same at every length.  (The two transforms as one product with an integer matrix are a third faster, but round
//     otherwise: of 33.6 M sketch bits some four then differ, which a key that a softmax rests on shows.)  The warp-level kernel does the
//     same butterflies with 128 lane exchanges a vector and 134 warp-instructions: 1,048,576 keys with 2 index bits 228 -> 165 us.
//   * a wait that gives up ends the other roles' waits too; the vectors whose indices were not found then have norms and factors that
//     are not a number, and a status word is set (tq_quantize_status_sync).
//   * loops over the columns stay loops: unrolled, a tile's code misses the instruction caches.
//
// 1,048,576 fp16 vectors of turbo3: 106 -> 87 us (3.7 TB/s; HBM would take 49); the arithmetic on the coordinates bounds it, most of it
// on the half-rate compare and packed fp32 pipes.  Scales are within 4e-7 of 64 bits, as the warp-level kernel's.
#include <type_traits>
#include "tq_quantize_math.cuh"
#include "tq_tcgen05.cuh"

namespace {

// Which appends come here; the warp-level kernel's tiles of 16 vectors spread fewer of them over more warps, its CTAs leave room
// beside them for the V rows of the same append and for the call behind, and this one's first tile takes 3 us.  Measured with 8
// heads of fp16, graph replays one after the other, us here / there:
//   K and V in one launch, by vectors of one: turbo3 16,384 7.2 / 6.2, 24,576 9.3 / 9.3, 32,768 10.9 / 11.1, 65,536 15.3 / 16.9;
//     turbo4 24,576 12.5 / 13.1, 65,536 23.4 / 25.1; turbo2 24,576 7.7 / 8.1, 65,536 13.6 / 14.2
//   one tensor beside another kernel: q8_0 / turbo3 131,072 27.2 / 27.7, 262,144 51.2 / 51.4, 1,048,576 171 / 190; q8_0 / turbo2
//     131,072 25.7 / 24.7, 262,144 45.8 / 45.7, 1,048,576 147 / 168
//   PROD keys and the V rows beside them: prod3 / turbo3 32,768 15.1 / 13.8, 49,152 19.3 / 19.7, 65,536 23.6 / 25.5, 1,048,576 250 / 302;
//     prod4 / turbo4 32,768 19.5 / 17.4, 49,152 25.0 / 25.1, 65,536 31.0 / 32.6, 1,048,576 382 / 451
// In vectors per SM (148), so that a device with fewer SMs takes the step earlier.
inline int64_t qt_min_vectors(bool pair, bool sketch) { return (int64_t)tq_num_sms() * (pair ? 166 : sketch ? 332 : 1776); }

struct QtJob {
  CUtensorMap map;   // of the rows: 64 elements x 128 rows a box, 128-byte swizzle
  TqFast f;
  TqQuantDst dst;
};

constexpr int QT_GROUPS = 4, QT_TMA_WARP = 4 * QT_GROUPS, QT_MMA_WARP = QT_TMA_WARP + 1, QT_THREADS = 32 * (QT_MMA_WARP + 1);
constexpr int QT_SLOTS = 4;                            // 128-column accumulators
constexpr int QT_STAGES = 6;                           // row tiles in flight
constexpr int QT_TILE = TQ_D * TQ_D * 2;               // bytes of a row tile
constexpr int QT_OFF_B = QT_STAGES * QT_TILE;          // the eight 16 x 16 matrices
constexpr int QT_BYTES = QT_OFF_B + 8 * 512 + 1024;    // + alignment (128-byte swizzle: 1,024)

template <typename T> struct QtIn;
template <> struct QtIn<__half> { static constexpr uint32_t ONES = 0x3C003C00u, FMT = 0; };
template <> struct QtIn<__nv_bfloat16> { static constexpr uint32_t ONES = 0x3F803F80u, FMT = (1u << 7) | (1u << 10); };

// row a of the 8-point Hadamard matrix as bits: bit j = parity(a & j)
__device__ __forceinline__ uint32_t qt_had8(uint32_t a) { return (uint32_t)(0x963C5AF066CCAA00ull >> (8 * a)) & 0xffu; }

// D = A B^T (128 x 16 x 16, one CTA)
__device__ __forceinline__ void qt_mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
               ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void qt_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(sptr(bar)) : "memory");
}

// Per-vector thresholds and what selects among them.  Level bits p4 p2 p1 (most significant first; BITS - 1 of them).
template <int BITS> struct QtLevels {
  float thr[(1 << (BITS - 1)) - 1], d31;
  __device__ __forceinline__ void init(const float (&bnd)[15], float ts) {
    constexpr int H = 1 << (BITS - 1);   // bnd[H .. ]: the positive boundaries
#pragma unroll
    for (int j = 0; j < H - 1; ++j) thr[j] = bnd[H + j] * ts;
    d31 = BITS == 3 ? thr[BITS == 3 ? 2 : 0] - thr[0] : 0.f;
  }
  // p is 1 or 0, q 1 - p: one of two thresholds, exactly
  static __device__ __forceinline__ float2 pick(float2 p, float2 q, float2 hi, float2 lo) { return qm_fma2(p, hi, qm_mul2(q, lo)); }
  // level bits of two magnitudes
  __device__ __forceinline__ void test(float2 a, float2& p4, float2& p2, float2& p1) const {
    auto gt = [](float2 x, float2 t) { return make_float2(qm_gt(x.x, t.x), qm_gt(x.y, t.y)); };
    auto other = [](float2 p) { return qm_sub2(qm_dup(1.0f), p); };
    if constexpr (BITS == 2) {
      p1 = gt(a, qm_dup(thr[0]));
    } else if constexpr (BITS == 3) {
      p2 = gt(a, qm_dup(thr[1]));
      p1 = gt(a, qm_fma2(p2, qm_dup(d31), qm_dup(thr[0])));   // (within an ulp of thr[2], as in the warp-level kernel)
    } else {
      p4 = gt(a, qm_dup(thr[3]));
      const float2 q4 = other(p4);
      p2 = gt(a, pick(p4, q4, qm_dup(thr[5]), qm_dup(thr[1])));
      p1 = gt(a, pick(p2, other(p2), pick(p4, q4, qm_dup(thr[6]), qm_dup(thr[2])), pick(p4, q4, qm_dup(thr[4]), qm_dup(thr[0]))));
    }
  }
};

// sums of the level bits and their products over a vector: exact integers, from which the counts #{level >= j} follow
template <int BITS> struct QtCounts {
  float2 s1, s2, s21, s4, s42, s41, s421;
  __device__ __forceinline__ void zero() { s1 = s2 = s21 = s4 = s42 = s41 = s421 = make_float2(0.f, 0.f); }
  __device__ __forceinline__ void add(int, float2 p4, float2 p2, float2 p1) {
    s1 = qm_add2(s1, p1);
    if constexpr (BITS >= 3) {
      s2 = qm_add2(s2, p2);
      s21 = qm_fma2(p2, p1, s21);
    }
    if constexpr (BITS == 4) {
      const float2 p42 = qm_mul2(p4, p2);
      s4 = qm_add2(s4, p4);
      s42 = qm_add2(s42, p42);
      s41 = qm_fma2(p4, p1, s41);
      s421 = qm_fma2(p42, p1, s421);
    }
  }
  // sum over the vector of the squared centroids less 128 times the smallest
  __device__ __forceinline__ float squares(const float (&cent)[16]) const {
    constexpr int H = 1 << (BITS - 1);
    auto step = [&](int j) { return cent[H + j] * cent[H + j] - cent[H + j - 1] * cent[H + j - 1]; };
    const float a1 = s1.x + s1.y;
    if constexpr (BITS == 2) {
      return a1 * step(1);
    } else {
      const float a2 = s2.x + s2.y, a21 = s21.x + s21.y;
      if constexpr (BITS == 3) {
        return fmaf(a2, step(2), fmaf(a21, step(3), (a2 + a1 - a21) * step(1)));
      } else {
        const float a4 = s4.x + s4.y, a42 = s42.x + s42.y, a41 = s41.x + s41.y, a421 = s421.x + s421.y;
        float cc = (a4 + a2 + a1 - a42 - a41 - a21 + a421) * step(1);
        cc = fmaf(a4 + a2 - a42, step(2), cc);
        cc = fmaf(a4 + a21 - a421, step(3), cc);
        cc = fmaf(a4, step(4), cc);
        cc = fmaf(a42 + a41 - a421, step(5), cc);
        cc = fmaf(a42, step(6), cc);
        return fmaf(a421, step(7), cc);
      }
    }
  }
};

// The same for keys with a sketch (2 or 3 bits), where the factor goes into the residual and with it into signs: a sum for each of the four
// lanes that share a vector in the warp-level kernel (every fourth group of four columns), joined as there.  The three counts of three
// bits, at most 32 each, are digits of one exact fp32 number.
template <int BITS> struct QtLaneCounts {
  float2 s[4];
  __device__ __forceinline__ void zero() { s[0] = s[1] = s[2] = s[3] = make_float2(0.f, 0.f); }
  __device__ __forceinline__ void add(int e, float2, float2 p2, float2 p1) {
    float2& t = s[(e & 15) >> 2];
    t = qm_add2(t, p1);
    if constexpr (BITS == 3) t = qm_fma2(p2, qm_fma2(p1, qm_dup(4096.f), qm_dup(64.f)), t);
  }
  __device__ __forceinline__ float squares(const float (&cent)[16]) const {
    constexpr int H = 1 << (BITS - 1);
    auto step = [&](int j) { return cent[H + j] * cent[H + j] - cent[H + j - 1] * cent[H + j - 1]; };
    float part[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float v = s[t].x + s[t].y;
      if constexpr (BITS == 2) {
        part[t] = __fmul_rn(v, step(1));   // (not part of the sums below)
      } else {
        const uint32_t n = __float2uint_rn(v), a1 = n & 63u, a2 = (n >> 6) & 63u, a21 = n >> 12;
        part[t] = fmaf((float)a2, step(2), fmaf((float)a21, step(3), (float)(a1 + a2 - a21) * step(1)));
      }
    }
    return (part[0] + part[1]) + (part[2] + part[3]);
  }
};

// 32 coordinates (minus the rotated values) -> BITS words of the packed stream, most significant bit first
template <int BITS, bool COUNT, class CNT>
__device__ __forceinline__ void qt_pack32(const uint32_t (&nu)[32], const QtLevels<BITS>& lv, CNT& cnt, uint32_t (&out)[BITS]) {
  constexpr int NC = 1 << BITS, HG = BITS == 4 ? 4 : 8;   // digits per exact fp32 Horner sum (at most 24 bits)
  constexpr float RADIX = (float)NC, HALF = (float)(NC / 2);
  constexpr float OFF = (HALF - 0.5f) * (float)(((1u << (HG * BITS)) - 1) / (NC - 1));
  uint32_t w[32 / HG];
#pragma unroll
  for (int q = 0; q < 32 / HG; ++q) {
    float2 ch = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < HG; k += 2) {
      const uint32_t u0 = nu[q * HG + k], u1 = nu[q * HG + k + 1];
      float2 p4, p2, p1;
      lv.test(make_float2(fabsf(__uint_as_float(u0)), fabsf(__uint_as_float(u1))), p4, p2, p1);
      if constexpr (COUNT) cnt.add(q * HG + k, p4, p2, p1);
      float2 m5 = qm_add2(p1, qm_dup(0.5f));
      if constexpr (BITS >= 3) m5 = qm_fma2(p2, qm_dup(2.0f), m5);
      if constexpr (BITS == 4) m5 = qm_fma2(p4, qm_dup(4.0f), m5);
      // index = HALF - 1/2 + sign * (level + 1/2), sign = -1 where the value is <= 0, i.e. where nu's sign bit is clear
      const float2 digit = make_float2(__uint_as_float(__float_as_uint(m5.x) | (~u0 & 0x80000000u)),
                                       __uint_as_float(__float_as_uint(m5.y) | (~u1 & 0x80000000u)));
      ch = k == 0 ? digit : qm_fma2(ch, qm_dup(RADIX * RADIX), digit);
    }
    w[q] = __float2uint_rn(fmaf(ch.x, RADIX, ch.y) + OFF);
  }
  if constexpr (BITS == 2) {          // 16 bits a word
    out[0] = __byte_perm(w[0], w[1], 0x4501);
    out[1] = __byte_perm(w[2], w[3], 0x4501);
  } else if constexpr (BITS == 3) {   // 24 bits a word
    out[0] = __byte_perm(w[0], w[1], 0x6012);
    out[1] = __byte_perm(w[1], w[2], 0x5601);
    out[2] = __byte_perm(w[2], w[3], 0x4560);
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) out[q] = __byte_perm(w[2 * q], w[2 * q + 1], 0x4501);
  }
}

// K-major operand in 128-byte swizzle atoms of 8 rows x 64 elements (what the tiled copies write)
__device__ __forceinline__ uint64_t qt_desc_sw128(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// 32 columns into u, no wait; qt_ld_wait orders every use of u behind the loads' completion
__device__ __forceinline__ void qt_ld32(uint32_t addr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(addr) : "memory");
}
__device__ __forceinline__ void qt_ld_wait(uint32_t (&v)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
      : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]),
        "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]), "+r"(v[16]),
        "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]), "+r"(v[24]),
        "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]), "+r"(v[30]), "+r"(v[31]) :: "memory");
}
// 128 columns as two turns of two pieces of 32: use(half, turn, values) twice, then done(turn).  A loop, not unrolled: the code of
// a tile then fits the instruction caches.
template <typename U, typename D> __device__ __forceinline__ void qt_columns(uint32_t addr, U&& use, D&& done) {
  uint32_t u[32];
#pragma unroll 1
  for (int turn = 0; turn < 2; ++turn) {
    qt_ld32(addr + 64 * turn, u);
    qt_ld_wait(u);
    use(std::integral_constant<int, 0>{}, turn, u);
    qt_ld32(addr + 64 * turn + 32, u);
    qt_ld_wait(u);
    use(std::integral_constant<int, 1>{}, turn, u);
    done(turn);
  }
}
// eight columns
__device__ __forceinline__ void qt_ld8(uint32_t addr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void qt_ld8_wait(uint32_t (&v)[8][8]) {   // (every use of v behind the wait)
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i)
    asm volatile("" : "+r"(v[i][0]), "+r"(v[i][1]), "+r"(v[i][2]), "+r"(v[i][3]), "+r"(v[i][4]), "+r"(v[i][5]), "+r"(v[i][6]), "+r"(v[i][7]));
}
__device__ __forceinline__ void qt_st8(uint32_t addr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
// sixteen columns at v[at ..], no wait, and back; qt_wait64 orders every use of v behind the loads
__device__ __forceinline__ void qt_ld16(uint32_t addr, float* v) {
  uint32_t* u = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]),
                 "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void qt_st16(uint32_t addr, const float* v) {
  const uint32_t* u = reinterpret_cast<const uint32_t*>(v);
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(addr), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(u[8]), "r"(u[9]), "r"(u[10]),
               "r"(u[11]), "r"(u[12]), "r"(u[13]), "r"(u[14]), "r"(u[15]) : "memory");
}
__device__ __forceinline__ void qt_wait64(float (&v)[64]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 64; i += 8)
    asm volatile("" : "+f"(v[i]), "+f"(v[i + 1]), "+f"(v[i + 2]), "+f"(v[i + 3]), "+f"(v[i + 4]), "+f"(v[i + 5]), "+f"(v[i + 6]), "+f"(v[i + 7]));
}
// the butterfly of distance H: a + b and a - b
template <int H> __device__ __forceinline__ void qt_butterfly(float (&v)[64]) {
#pragma unroll
  for (int i = 0; i < 64; i += H == 1 ? 2 : 1)
    if constexpr (H == 1) {
      const float a = v[i], b = v[i + 1];
      v[i] = a + b;
      v[i + 1] = a - b;
    } else if ((i & H) == 0 && (i & 1) == 0) {
      const float2 a = make_float2(v[i], v[i + 1]), b = make_float2(v[i + H], v[i + H + 1]);
      const float2 p = qm_add2(a, b), m = qm_sub2(a, b);
      v[i] = p.x; v[i + 1] = p.y;
      v[i + H] = m.x; v[i + H + 1] = m.y;
    }
}

// Keys with a sketch: the residual -(u - c cs) of the values (minus u) at `tm`, its squares' sum, and the sketch words (the first column in
// the most significant bit, before the last signs) -- two 128-point transforms with the signs `mid` between them, all in the order of the
// warp-level kernel, whose bits these are: butterflies of distances 1 to 64, of which 64 registers hold six; the seventh, and the last two
// of the second transform, take the columns from tensor memory again, 32 (or 16) of either half (quarter).
template <int BITS>
__device__ __forceinline__ float qt_sketch(uint32_t tm, const QtLevels<BITS>& lv, const float (&cent)[16], float cs, const float* mid, uint32_t (&words)[4]) {
  constexpr int H = 1 << (BITS - 1);
  float2 ee[4];
#pragma unroll
  for (int t = 0; t < 4; ++t) ee[t] = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    float v[64];
#pragma unroll
    for (int c = 0; c < 64; c += 16) qt_ld16(tm + 64 * half + c, v + c);
    qt_wait64(v);
#pragma unroll
    for (int k = 0; k < 64; k += 2) {
      const float2 nu = make_float2(v[k], v[k + 1]);
      float2 p4, p2, p1, cm;
      lv.test(make_float2(fabsf(nu.x), fabsf(nu.y)), p4, p2, p1);
      if constexpr (BITS == 3) {   // level 2 p2 + p1
        const float2 base = qm_fma2(p2, qm_dup(cent[6] - cent[4]), qm_dup(cent[4]));
        const float2 slope = qm_fma2(p2, qm_dup((cent[7] - cent[6]) - (cent[5] - cent[4])), qm_dup(cent[5] - cent[4]));
        cm = qm_fma2(p1, slope, base);
      } else {
        cm = qm_fma2(p1, qm_dup(cent[H + 1] - cent[H]), qm_dup(cent[H]));
      }
      cm.x = __int_as_float(__float_as_int(cm.x) | (~__float_as_int(nu.x) & 0x80000000));
      cm.y = __int_as_float(__float_as_int(cm.y) | (~__float_as_int(nu.y) & 0x80000000));
      const float2 r = qm_fma2(cm, qm_dup(cs), nu);
      ee[(k & 15) >> 2] = qm_fma2(r, r, ee[(k & 15) >> 2]);
      v[k] = r.x; v[k + 1] = r.y;
    }
    qt_butterfly<1>(v); qt_butterfly<2>(v); qt_butterfly<4>(v); qt_butterfly<8>(v); qt_butterfly<16>(v); qt_butterfly<32>(v);
#pragma unroll
    for (int c = 0; c < 64; c += 16) qt_st16(tm + 64 * half + c, v + c);
  }
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
#pragma unroll 1
  for (int part = 0; part < 2; ++part) {   // columns 32 part .. + 31 of both halves
    float v[64];
#pragma unroll
    for (int c = 0; c < 32; c += 16) qt_ld16(tm + 32 * part + c, v + c), qt_ld16(tm + 64 + 32 * part + c, v + 32 + c);
    qt_wait64(v);
    qt_butterfly<32>(v);
#pragma unroll
    for (int k = 0; k < 64; k += 4) {
      const float4 m = *reinterpret_cast<const float4*>(mid + 32 * part + (k & 31) + 2 * (k & 32));
      const float2 a = qm_mul2(make_float2(v[k], v[k + 1]), make_float2(m.x, m.y)), b = qm_mul2(make_float2(v[k + 2], v[k + 3]), make_float2(m.z, m.w));
      v[k] = a.x; v[k + 1] = a.y; v[k + 2] = b.x; v[k + 3] = b.y;
    }
    qt_butterfly<1>(v); qt_butterfly<2>(v); qt_butterfly<4>(v); qt_butterfly<8>(v); qt_butterfly<16>(v);
#pragma unroll
    for (int c = 0; c < 32; c += 16) qt_st16(tm + 32 * part + c, v + c), qt_st16(tm + 64 + 32 * part + c, v + 32 + c);
  }
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
#pragma unroll 1
  for (int part = 0; part < 2; ++part) {   // columns 16 part .. + 15 of the four quarters
    float v[64];
#pragma unroll
    for (int c = 0; c < 4; ++c) qt_ld16(tm + 32 * c + 16 * part, v + 16 * c);
    qt_wait64(v);
    qt_butterfly<16>(v); qt_butterfly<32>(v);
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int k = 0; k < 16; ++k) words[c] = __funnelshift_l(__float_as_uint(v[16 * c + k]), words[c], 1);
  }
  return ((ee[0].x + ee[0].y) + (ee[1].x + ee[1].y)) + ((ee[2].x + ee[2].y) + (ee[3].x + ee[3].y));
}
__device__ __forceinline__ void qt_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sptr(bar)) : "memory");
}

// A wait gave up: a group's tiles from the i-th of this CTA's on are not to come.  (A function of its own: inlined, it costs the kernel registers.)
__device__ __noinline__ void qt_give_up(const TqQuantDst& dst, int i, int mine, int gtid, int64_t n, int32_t* status) {
  const float nan = __int_as_float(0x7fffffff);
  for (; i < mine; i += QT_GROUPS) {
    const int64_t v = (blockIdx.x + (int64_t)i * gridDim.x) * TQ_D + gtid;
    if (v >= n) continue;
    bool good = true;
    int64_t within = 0;
    const int64_t rec = tq_dst_record(dst, v, within, good);
    if (good && dst.scale) *reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(dst.scale) + rec + within * 4) = nan;
    if (dst.norm) dst.norm[v] = nan;
    if (good && dst.rnorm) *reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(dst.rnorm) + rec + within * 4) = nan;
  }
  if (status) *status = 1;
}

// SELFTEST: the first CTA's second tile is never reported as multiplied, and waits are short
template <typename Tin, int BITS, bool NORMC, bool SELFTEST = false, bool QJLS = false>
__global__ void __launch_bounds__(QT_THREADS, 1) k_quantize_tc(const __grid_constant__ QtJob j0, const __grid_constant__ QtJob j1,
                                                                         int64_t n, int32_t* status) {
  constexpr long long LIMIT = SELFTEST ? TC_SELFTEST_CYCLES : TC_WAIT_CYCLES;
  constexpr int IDXB = 16 * BITS, NC = 1 << BITS, HALF = NC / 2, SLOTS = QT_SLOTS, STAGES = QT_STAGES;
  extern __shared__ __align__(128) uint8_t qt_raw[];
  __shared__ uint64_t a_full[STAGES], a_free[STAGES], d_full[SLOTS], d_free[SLOTS];
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_failed;   // a wait gave up: nobody waits any more
  __shared__ __align__(16) uint32_t s_flip[4 * BITS];
  __shared__ __align__(16) float s_mid[QJLS ? TQ_D : 4];   // signs between the transforms of the sketch
  __shared__ __align__(16) uint32_t s_last[4];             // ... and behind them, as bits in the order of the sketch words
  const QtJob& job = blockIdx.y == 0 ? j0 : j1;
  const TqFast& f = job.f;
  const TqQuantDst& dst = job.dst;
  if (dst.beside) TQ_PDL_TRIGGER();
  uint8_t* sm = qt_raw + (((sptr(qt_raw) + 1023u) & ~1023u) - sptr(qt_raw));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, group = warp >> 2, gtid = tid & 127;

  // ---- tables: they need the parameters only ----
  if (tid == 0) {
    auto init = [](uint64_t* bar, int count) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sptr(bar)), "r"(count) : "memory");
    };
    for (int i = 0; i < STAGES; ++i) init(&a_full[i], 1), init(&a_free[i], 1);
    for (int i = 0; i < SLOTS; ++i) init(&d_full[i], 1), init(&d_free[i], 4);
    s_failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  {
    // H16 D1 of block i as +-1, 16-byte chunk c of it: outputs 8 (c >> 4) + (c & 7), inputs 8 ((c >> 3) & 1) ..
    if (tid < 256) {
      const int i = tid >> 5, c = tid & 31, out = 8 * (c >> 4) + (c & 7), k8 = (c >> 3) & 1, e = 16 * i + 8 * k8;
      uint32_t m = qt_had8(out & 7) ^ ((f.s1[e >> 5] >> (e & 31)) & 0xffu);
      if ((out >> 3) & k8) m ^= 0xffu;
      uint32_t w[4];
#pragma unroll
      for (int p = 0; p < 4; ++p)
        w[p] = QtIn<Tin>::ONES ^ (((m >> (2 * p)) & 1u) << 15) ^ (((m >> (2 * p + 1)) & 1u) << 31);
      *reinterpret_cast<uint4*>(sm + QT_OFF_B + tid * 16) = make_uint4(w[0], w[1], w[2], w[3]);
    } else if (tid < 256 + 4 * BITS) {   // sign2 mirrors an index (i -> 2^b - 1 - i): all bits of its field in the packed stream
      uint32_t w = 0;
#pragma unroll
      for (int k = 0; k < 32; ++k) w |= qm_bit(f.s2, (32 * (tid - 256) + k) / BITS) << (8 * (k >> 3) + 7 - (k & 7));
      s_flip[tid - 256] = w;
    } else if (QJLS && tid >= 288 && tid < 288 + TQ_D) {
      const int e = tid - 288;
      s_mid[e] = qm_bit(f.s1, e) ^ qm_bit(f.j1, e) ? -1.f : 1.f;
    } else if (QJLS && tid >= 416 && tid < 420) {
      s_last[tid - 416] = __brev(f.j2[tid - 416]);
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (!dst.beside) TQ_PDL_WAIT();
  // Tensor memory only now: the kernel in front may hold it, and would never finish if this one kept it waiting.
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sptr(&s_tmem)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tb = s_tmem;
  const int64_t tiles = (n + TQ_D - 1) / TQ_D, step = gridDim.x;
  const int mine = (int)((tiles - blockIdx.x + step - 1) / step);   // tiles of this CTA: blockIdx.x + i step

  if (warp == QT_TMA_WARP) {
    if (lane == 0) {
      int i = 0;
      for (; i < mine && !s_failed; ++i) {
        const int st = i % STAGES;
        if (i >= STAGES && !tc_wait(&a_free[st], (uint32_t)((i / STAGES - 1) & 1), &s_failed, LIMIT)) break;
        const uint32_t dsts = sptr(sm) + st * QT_TILE;
        const int row = (int)((blockIdx.x + i * step) * TQ_D);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sptr(&a_full[st])), "r"(QT_TILE) : "memory");
#pragma unroll
        for (int h = 0; h < 2; ++h)   // (rows past n come as zeros)
          asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                           dsts + h * (QT_TILE / 2)), "l"(&job.map), "r"(64 * h), "r"(row), "r"(sptr(&a_full[st])) : "memory");
      }
      for (int k = i < STAGES ? 0 : i - STAGES; k < i; ++k) tc_wait(&a_full[k % STAGES], (uint32_t)((k / STAGES) & 1));   // none in flight at the end
    }
  } else if (warp == QT_MMA_WARP) {
    if (lane == 0) {
      const uint32_t idesc = umma_idesc(128, 16, false) | QtIn<Tin>::FMT, b = sptr(sm) + QT_OFF_B;
      int i = 0;
      for (; i < mine && !s_failed; ++i) {
        const int st = i % STAGES, sl = i % SLOTS;
        if (!tc_wait(&a_full[st], (uint32_t)((i / STAGES) & 1), &s_failed, LIMIT) ||
            (i >= SLOTS && !tc_wait(&d_free[sl], (uint32_t)((i / SLOTS - 1) & 1), &s_failed, LIMIT)))
          break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a = sptr(sm) + st * QT_TILE;
#pragma unroll
        for (int i16 = 0; i16 < 8; ++i16)
          qt_mma_ss(tb + 128 * sl + 16 * i16, qt_desc_sw128(a + (i16 >> 2) * (QT_TILE / 2) + (i16 & 3) * 32),
                    umma_desc(b + i16 * 512, 128, 256), idesc, 0);
        qt_commit(&a_free[st]);
        if (!(SELFTEST && blockIdx.x == 0 && i == 1)) qt_commit(&d_full[sl]);
      }
      if (s_failed && i > 0) tc_wait(&a_free[(i - 1) % STAGES], (uint32_t)(((i - 1) / STAGES) & 1));   // none in flight at the end
    }
  } else if (warp < QT_TMA_WARP) {
  const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;   // this warp's 32 lanes
  const uint32_t zero_idx = 0.f > f.bnd[HALF - 1] ? HALF : HALF - 1;   // index of the value 0
  int i = group;
  for (; i < mine; i += QT_GROUPS) {
    const int sl = i % SLOTS;
    const uint32_t tm = tb + 128 * sl + lanes;
    const int64_t v = (blockIdx.x + i * step) * TQ_D + gtid;
    bool good = v < n;
    int64_t within = 0;
    const int64_t rec = good ? tq_dst_record(dst, v, within, good) : 0;   // (the slot's load flies under the MMAs)
    if (!__all_sync(0xffffffffu, tc_wait(&d_full[sl], (uint32_t)((i / SLOTS) & 1), &s_failed, LIMIT))) break;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // ---- the 8-point stage over the blocks, in place, eight columns of every block a turn, and ||x||: ||H x||^2 = 128 ||x||^2.
    // Sums in the warp-level kernel's order (four columns of all blocks, then those four sums in pairs): both kernels then
    // find the same indices ----
    float ss = 0.f;
#pragma unroll 1
    for (int turn = 0; turn < 2; ++turn) {
      uint32_t u[8][8];   // [block][column]
#pragma unroll
      for (int i16 = 0; i16 < 8; ++i16) qt_ld8(tm + 16 * i16 + 8 * turn, u[i16]);
      qt_ld8_wait(u);
#pragma unroll
      for (int h = 1; h < 8; h <<= 1)
#pragma unroll
        for (int i16 = 0; i16 < 8; ++i16)
          if ((i16 & h) == 0)
#pragma unroll
            for (int c = 0; c < 8; c += 2) {
              const float2 a = make_float2(__uint_as_float(u[i16][c]), __uint_as_float(u[i16][c + 1]));
              const float2 b = make_float2(__uint_as_float(u[i16 + h][c]), __uint_as_float(u[i16 + h][c + 1]));
              // (the last stage costs no more: the negation is part of the subtraction)
              const float2 sum = h < 4 ? qm_add2(a, b) : qm_sub2(make_float2(-a.x, -a.y), b);
              const float2 dif = h < 4 ? qm_sub2(a, b) : qm_sub2(b, a);
              u[i16][c] = __float_as_uint(sum.x);
              u[i16][c + 1] = __float_as_uint(sum.y);
              u[i16 + h][c] = __float_as_uint(dif.x);
              u[i16 + h][c + 1] = __float_as_uint(dif.y);
            }
      float part[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        float2 s2 = make_float2(0.f, 0.f);
#pragma unroll
        for (int i16 = 0; i16 < 8; ++i16)
#pragma unroll
          for (int c = 4 * q; c < 4 * q + 4; c += 2) {
            const float2 y = make_float2(__uint_as_float(u[i16][c]), __uint_as_float(u[i16][c + 1]));
            s2 = qm_fma2(y, y, s2);
          }
        part[q] = s2.x + s2.y;
      }
      ss = turn == 0 ? part[0] + part[1] : ss + (part[0] + part[1]);
#pragma unroll
      for (int i16 = 0; i16 < 8; ++i16) qt_st8(tm + 16 * i16 + 8 * turn, u[i16]);
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    const float nrm = sqrtf(ss) * TQ_RSQRT_D;           // ||H x|| = sqrt(d) ||x||
    const float safe = nrm > 0.f ? nrm : 1.0f;          // turboquant/polar_quant.py:74
    const float ts = safe * TQ_SQRT_D;                  // the sums are y * ||x|| * sqrt(d), y the rotated unit vector
    QtLevels<BITS> lv;
    lv.init(f.bnd, ts);
    std::conditional_t<QJLS, QtLaneCounts<BITS>, QtCounts<BITS>> cnt;
    cnt.zero();
    // ---- indices: 64 coordinates a turn, 8 BITS bytes ----
    // a zero vector takes the index of the value 0 in every coordinate
    const uint32_t zero24 = zero_idx * 0x249249u;
    const uint32_t zero0 = BITS == 2 ? zero_idx * 0x55555555u : BITS == 4 ? zero_idx * 0x11111111u : __byte_perm(zero24, zero24, 0x6012);
    const uint32_t zero1 = BITS == 3 ? __byte_perm(zero24, zero24, 0x5601) : zero0, zero2 = BITS == 3 ? __byte_perm(zero24, zero24, 0x4560) : zero0;
    uint32_t w[2 * BITS];
    qt_columns(tm, [&](auto half, int turn, const uint32_t (&u)[32]) {
      uint32_t o[BITS];
      qt_pack32<BITS, NORMC>(u, lv, cnt, o);
#pragma unroll
      for (int k = 0; k < BITS; ++k) w[BITS * decltype(half)::value + k] = nrm > 0.f ? o[k] ^ s_flip[2 * BITS * turn + BITS * decltype(half)::value + k] : k % 3 == 0 ? zero0 : k % 3 == 1 ? zero1 : zero2;
    }, [&](int turn) {
      if (!good) return;
      uint8_t* p = dst.idx + rec + within * IDXB + 8 * BITS * turn;
#pragma unroll
      for (int k = 0; k < 2 * BITS; k += 2) {
        if constexpr (BITS == 3) reinterpret_cast<uint2*>(p)[k / 2] = make_uint2(w[k], w[k + 1]);
        else if (k % 4 == 0) reinterpret_cast<uint4*>(p)[k / 4] = make_uint4(w[k], w[k + 1], w[k + 2], w[k + 3]);
      }
    });
    float invn = 1.0f;
    auto free_slot = [&]() {
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) qt_arrive(&d_free[sl]);
    };
    if constexpr (!QJLS) free_slot();
    if constexpr (NORMC) {
      float cn = sqrtf(fmaf((float)TQ_D, f.cent[HALF] * f.cent[HALF], cnt.squares(f.cent)));
      cn = cn > 1e-10f ? cn : 1.0f;                      // turboquant/polar_quant.py:110-111
      invn = 1.0f / cn;
    }
    if (good && dst.scale) {
      *reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(dst.scale) + rec + within * 4) = nrm * invn;
    }
    if constexpr (QJLS) {
      uint32_t words[4] = {};
      const float ee = qt_sketch<BITS>(tm, lv, f.cent, invn * ts, s_mid, words);
      free_slot();
      const float rn = nrm > 0.f ? sqrtf(ee) * TQ_RSQRT_D : 0.f;   // ||r|| = ||x|| * ||y - yhat'||
      // (the values were minus the projections: a sign bit is a sketch bit; a zero input has no residual: all +1)
      uint4 z;
      z.x = nrm > 0.f ? __byte_perm(words[0] ^ s_last[0], 0, 0x0123) : 0xffffffffu;
      z.y = nrm > 0.f ? __byte_perm(words[1] ^ s_last[1], 0, 0x0123) : 0xffffffffu;
      z.z = nrm > 0.f ? __byte_perm(words[2] ^ s_last[2], 0, 0x0123) : 0xffffffffu;
      z.w = nrm > 0.f ? __byte_perm(words[3] ^ s_last[3], 0, 0x0123) : 0xffffffffu;
      if (good && dst.qjl) *reinterpret_cast<uint4*>(dst.qjl + rec + within * 16) = z;
      if (good && dst.rnorm)   // sqrt(pi/2)/sqrt(d): turboquant/qjl.py:32,131
        *reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(dst.rnorm) + rec + within * 4) = dst.rscale_const ? rn * (1.2533141373155001f * TQ_RSQRT_D) : rn;
    }
    if (v < n && dst.norm) dst.norm[v] = nrm;
  }
  if (i < mine) qt_give_up(dst, i, mine, gtid, n, status);
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem), "r"(512u) : "memory");
  if (dst.beside) TQ_PDL_WAIT(); else TQ_PDL_TRIGGER();
}

// the rows as a tensor of n x 128 16-bit elements, copied in boxes of 128 x 64; false where no such map can be made
bool qt_map(CUtensorMap* map, const void* x, int32_t dtype, int64_t ld, int64_t n) {
  return tc_map(map, dtype == TQ_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, x, TQ_D, n, ld * 2, 64, TQ_D);
}

template <typename Tin, int BITS, bool NORMC, bool SELFTEST = false, bool QJLS = false>
int launch_tc(const QtJob& j0, const QtJob& j1, int jobs, int64_t n, cudaStream_t st) {
  auto kernel = k_quantize_tc<Tin, BITS, NORMC, SELFTEST, QJLS>;
  static thread_local int configured_dev = -1;   // one per kernel
  int dev = 0;
  TQ_CUDA(cudaGetDevice(&dev));
  if (configured_dev != dev) {
    TQ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, QT_BYTES));
    configured_dev = dev;
  }
  const int64_t tiles = (n + TQ_D - 1) / TQ_D, places = tq_num_sms() / jobs > 0 ? tq_num_sms() / jobs : 1;
  const dim3 grid((unsigned)(tiles < places ? tiles : places), jobs);   // one CTA per SM; few tiles: one group of each
  TQ_CUDA(tq_launch_early(kernel, grid, QT_THREADS, QT_BYTES, st, j0, j1, n, tq_quantize_status_word()));
  return tq_launch_check("k_quantize_tc");
}

template <typename Tin>
int launch_tc_bits(const QtJob& j0, const QtJob& j1, int jobs, bool normc, bool want_qjl, int64_t n, cudaStream_t st) {
  if (want_qjl) {   // (the residual needs the norm correction whether or not the factor is stored)
#define TQ_TC(B) \
  if (j0.f.bits == B) return j0.f.norm_correction ? launch_tc<Tin, B, true, false, true>(j0, j1, 1, n, st) : launch_tc<Tin, B, false, false, true>(j0, j1, 1, n, st);
    TQ_TC(2) TQ_TC(3)
#undef TQ_TC
    return TQ_ERR_UNSUPPORTED;
  }
#define TQ_TC(B) \
  if (j0.f.bits == B) return normc ? launch_tc<Tin, B, true>(j0, j1, jobs, n, st) : launch_tc<Tin, B, false>(j0, j1, jobs, n, st);
  TQ_TC(2) TQ_TC(3) TQ_TC(4)
#undef TQ_TC
  return TQ_ERR_UNSUPPORTED;
}

}  // namespace

// One tensor, or two of the same shape and format (x1 != nullptr), whose requests the warp-level kernel serves: false where that
// kernel is to take them.
bool tq_quantize_tc_try(const TqFast& f0, const void* x0, const TqQuantDst& d0, const TqFast* f1, const void* x1, const TqQuantDst* d1,
                        int32_t dtype, int64_t ld, int64_t n, bool normc, bool want_qjl, cudaStream_t st, int* rc) {
  if (dtype != TQ_F16 && dtype != TQ_BF16) return false;
  if (n < qt_min_vectors(x1 != nullptr, want_qjl) || (want_qjl && f0.bits == 4)) return false;
  // a thread stores its vector's indices up to 16 bytes at a time
  auto aligned = [](const TqQuantDst& d) {
    return tq_aligned(d.idx, 16) && tq_aligned(d.qjl, 16) && d.page_stride % 16 == 0 && d.head_stride % 16 == 0;
  };
  if (!tq_aligned(x0, 16) || !aligned(d0) || (x1 && (!tq_aligned(x1, 16) || !aligned(*d1)))) return false;
  QtJob j0, j1;
  j0.f = f0; j0.dst = d0;
  if (!qt_map(&j0.map, x0, dtype, ld, n)) return false;
  if (x1) {
    j1.f = *f1; j1.dst = *d1;
    if (!qt_map(&j1.map, x1, dtype, ld, n)) return false;
  } else {
    j1 = j0;
  }
  const int jobs = x1 ? 2 : 1;
  *rc = dtype == TQ_F16 ? launch_tc_bits<__half>(j0, j1, jobs, normc, want_qjl, n, st)
                        : launch_tc_bits<__nv_bfloat16>(j0, j1, jobs, normc, want_qjl, n, st);
  return true;
}

// fp16 rows of a 3-bit quantizer with norm correction, plain arrays
int tq_quantize_tc_selftest(const TqFast& f, const void* x, const TqQuantDst& d, int64_t ld, int64_t n, cudaStream_t st) {
  QtJob j;
  j.f = f; j.dst = d;
  TQ_REQUIRE(f.bits == 3 && f.norm_correction && tq_aligned(x, 16) && ld % 8 == 0 && qt_map(&j.map, x, TQ_F16, ld, n), TQ_ERR_UNSUPPORTED,
             "self-test of the long append: fp16 rows of a 3-bit quantizer with norm correction");
  return launch_tc<__half, 3, true, true>(j, j, 1, n, st);
}
