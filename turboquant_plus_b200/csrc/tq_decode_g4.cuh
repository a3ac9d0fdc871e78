// Decode attention on 128-token pages for at most four (NH = 4) or eight (NH = 8) query heads per KV head: the shape of
// the headline workload (Llama-3-8B: 32 query / 8 KV heads, turbo3 K and V), of the other decode configurations (q8_0 keys
// with turbo2 values, PROD keys -- PolarQuant + QJL sign sketch -- with turbo3 values) and of Llama-3-70B's 64 / 8 heads.
// Same pipeline and the same split / ticket protocol as k_decode_attn (tq_attention.cu); what changes is how the 8
// columns of the MMA tiles are spent, and that everything the page loop needs is a compile-time constant:
//   * S = K q^T: columns 0..3 carry the fp16 "hi" halves of the four query heads, columns 4..7 the "lo" halves,
//     so one m16n8k16 per 16 dims instead of two; the halves meet through one lane exchange (lane ^ 2), after
//     which thread (g, t) owns one token (g + 8 (t >> 1)) and two heads (2 (t & 1), + 1).
//   * O^T += V^T P^T: a k-slot pair is (token, dim parity) instead of (token, token'), column n is
//     (head n >> 1, parity n & 1), and the P operand is p on the matching parity, 0 on the other.  A pair-table
//     word (two dims of one token) is then an A-operand register as it comes: no re-pairing permutes, 32 dims per
//     MMA, and O takes 16 accumulator registers per thread: o[blk] = head t, dims 16 g + 4 blk .. + 3.
//   * the running maxima are only reduced across the warp when some score exceeds them.
//   * page size (128 tokens = one 16-token tile per warp and page), pipeline depth (3 records) and every offset
//     inside a record are template constants; record bytes are read through 32-bit shared-memory addresses with
//     immediate offsets; only the last page of a sequence runs the variant that masks tokens past the end.
//   * q8_0 operands are int8 -> fp16 by byte permute + one subtract (exact), the per-block scales applied to the
//     partial scores of each 32-dim block in fp32 (keys) or to the operand pairs (values); the sign sketch of PROD
//     keys becomes operands by one logic op per pair: dims d and d + 16 of a 32-bit word pair up, and the masked word is a
//     pair of fp16 numbers of one set bit each (or zero), against the S-projected query divided by them.
//   * eight heads: the columns of S are the heads, hi and lo halves are two MMAs into two accumulators and no exchange is
//     needed (thread (g, t) owns tokens g and g + 8, heads 2t and 2t + 1); O^T takes two MMAs per operand, heads 0..3 and
//     4..7, for the same dequantized words.  Dequantization is the cost, and eight heads share it: dealt to two CTAs of
//     four heads each it was done twice, and the general kernel, with its re-pairing permutes, ran at a quarter of the
//     rate (2 x 131,072 tokens of turbo4, 8 KV heads: 256 us).
//   * 4-bit tables (256 pairs) are replicated per lane like the smaller ones where 32 KB fit (eight-warp CTAs): with one
//     copy the lanes of a lookup collide in 3.4 wavefronts on average.
#pragma once
#include "tq_attention.cuh"

namespace {

using namespace tqatt;

// What the kernel needs of a quantizer, packed into 112 bytes so that the whole parameter block is a handful of
// 64-byte lines: parameters live in the constant bank, every line misses once per launch, and the misses of one
// warp are serial.  The warps therefore touch one line each before anything else happens.
struct AttnQuant {
  uint32_t s1[4], s2[4];   // rotation signs
  uint32_t j1[4], j2[4];   // QJL sign-WHT signs (PROD keys)
  uint16_t cent16[16];
  float alpha;
  uint32_t pad[3];
};
static_assert(sizeof(AttnQuant) == 112, "AttnQuant layout");

constexpr int G4_HSTRIDE = TQ_D + 4;  // floats between heads in the warp-merge buffer: 16-byte stores stay conflict-free
constexpr int G4_PT = 128;            // tokens per page

// One 256-thread CTA per (KV head, split), two CTAs per SM.  (One 512-thread CTA running two such groups keeps the
// two in step inside a single launch and is 3 % faster there at 32K tokens; but in a chain of launches with
// programmatic dependent launch the half-SM CTAs of the next call take the place of finished ones one by one, so
// that one CTA's latency-bound prologue and tail run under the other's page loop: 11.4 against 13.2 us per call.)

constexpr int up128(int x) { return (x + 127) / 128 * 128; }


// Record layout of a (page, head) for 128-token pages, as tq_cache_layout_init lays it out, and the carve-up of
// the CTA's shared memory: the two pair tables, the query buffer(s), the mbarriers and flags, and the pipeline stages
// (reused as the warp-merge buffer after the page loop).
// KK / VK: 2,3,4 = turbo bits; 8 = q8_0; 18,19,20 = PROD with 1,2,3 PolarQuant bits + sign sketch (keys only).
// Pair table of this kernel: 16-bit-pair entries replicated per lane (see PairLut), the 256-entry one only where REPL4.
// Tables up to 8 KB start on a multiple of their size and the address of an entry is (field | base); the 32 KB one would
// waste a quarter of the CTA's shared memory on that, its base is added.
template <int BITS, bool REPL4> struct G4Lut {
  static constexpr int ENTRIES = PairLut<BITS>::ENTRIES;
  static constexpr bool BIG = BITS == 4 && REPL4;
  static constexpr bool REPL = BIG || PairLut<BITS>::REPL;
  static constexpr int SHIFT = REPL ? 7 : 2;
  static constexpr int BYTES = BITS ? ENTRIES << SHIFT : 0;
  static constexpr int ALIGN = BIG ? 512 : BYTES;
  // `base`: (aligned start | lane part), BIG: lane part; `start`: BIG: start of the table
  static __device__ __forceinline__ uint32_t load(uint32_t field, uint32_t base, uint32_t start) {
    return lds32(BIG ? (field | base) + start : field | base);
  }
};

// lut_fill for any of these tables
template <class LUT, int BITS>
__device__ __forceinline__ void g4_lut_fill(uint8_t* lut, const uint16_t* c16, int tid, int nthreads) {
  if constexpr (LUT::BIG) {
    for (int i = tid; i < LUT::ENTRIES * 8; i += nthreads) {
      const int e = i >> 3;
      const uint32_t v = (uint32_t)c16[e >> BITS] | ((uint32_t)c16[e & ((1 << BITS) - 1)] << 16);
      reinterpret_cast<uint4*>(lut)[i] = make_uint4(v, v, v, v);
    }
  } else {
    lut_fill<BITS>(lut, c16, tid, nthreads);
  }
}

template <int KK, int VK, int NW = ATT_WARPS, int NH = 4> struct G4 {
  using KT = Kind<KK>;
  using VT = Kind<VK>;
  static constexpr int KB = KT::BITS, VB = VT::BITS;
  static constexpr int KIDXB = KT::Q8 ? TQ_D : 16 * KB, VIDXB = VT::Q8 ? TQ_D : 16 * VB;  // index bytes per token
  static constexpr int KSCB = KT::Q8 ? 8 : 4, VSCB = VT::Q8 ? 8 : 4;                      // scale bytes per token
  static constexpr int K_IDX = 0;
  static constexpr int K_SCALE = K_IDX + G4_PT * KIDXB;
  static constexpr int K_QJL = K_SCALE + G4_PT * KSCB;        // PROD keys: sign sketch, then residual scales
  static constexpr int K_RSCALE = K_QJL + G4_PT * 16;
  static constexpr int V_IDX = KT::PROD ? K_RSCALE + G4_PT * 4 : K_QJL;
  static constexpr int V_SCALE = V_IDX + G4_PT * VIDXB;
  static constexpr int REC = V_SCALE + G4_PT * VSCB;
  static constexpr bool REPL4 = NW == 8;   // two CTAs per SM: room for the replicated 4-bit tables
  using KLut = G4Lut<KB, REPL4>;
  using VLut = G4Lut<VB, REPL4>;
  static constexpr int LK = KLut::BYTES, LV = VLut::BYTES;
  static constexpr int TALIGN = KLut::ALIGN > VLut::ALIGN ? KLut::ALIGN : VLut::ALIGN;
  static constexpr int ALIGN = TALIGN > 512 ? TALIGN : 512;
  static constexpr bool K_FIRST = KLut::ALIGN >= VLut::ALIGN;   // the stricter alignment first: each keeps its own
  static constexpr int OFF_K = K_FIRST ? 0 : LV;
  static constexpr int OFF_V = K_FIRST ? LK : 0;
  static constexpr int OFF_GROUPS = up128(LK + LV);
  static constexpr int G_Q = 0;                                   // float [4 heads][128] (PROD: + the projected queries)
  // PROD keys, eight heads: the lo halves of the query fragments (64 registers otherwise), uint2[2][8 k-steps][32 lanes]
  static constexpr bool LO_SMEM = KT::PROD && NH == 8;
  static constexpr int G_LO = G_Q + (KT::PROD ? 2 : 1) * NH * TQ_D * 4;
  static constexpr int G_BAR = G_LO + (LO_SMEM ? 4096 : 0);                       // 3 mbarriers, two flag words at + 64
  static constexpr int G_STAGE = G_BAR + 128;
  // page records in flight: 3 (4 and 5 measured: no faster); 2 for the four-warp CTAs, four of which share an SM, and
  // where two large tables and three records exceed half an SM
  static constexpr int NS = NW == 4 || 3 * REC + LK + LV > 104 * 1024 ? 2 : 3;
  static constexpr int MERGE = NW * NH * (G4_HSTRIDE + 2) * 4;
  static constexpr int GROUP_BYTES = up128(G_STAGE + (NS * REC > MERGE ? NS * REC : MERGE));
  static constexpr int SMEM = ALIGN + OFF_GROUPS + GROUP_BYTES;
};

// ---- shared-memory loads through 32-bit addresses with immediate offsets ----------------------------------------
// Not volatile: the compiler may schedule and combine them.  What keeps a load of a pipeline stage behind the wait
// for that stage is a data dependency: the stage address is formed from a value the wait produces.
template <int OFF> __device__ __forceinline__ uint32_t lds_u32(uint32_t a) {
  uint32_t v;
  asm("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(a), "n"(OFF));
  return v;
}
template <int OFF> __device__ __forceinline__ uint32_t lds_u16(uint32_t a) {
  uint16_t v;
  asm("ld.shared.u16 %0, [%1+%2];" : "=h"(v) : "r"(a), "n"(OFF));
  return v;
}
template <int OFF> __device__ __forceinline__ float lds_f32(uint32_t a) {
  float v;
  asm("ld.shared.f32 %0, [%1+%2];" : "=f"(v) : "r"(a), "n"(OFF));
  return v;
}
template <int OFF> __device__ __forceinline__ uint2 lds_u64(uint32_t a) {
  uint2 v;
  asm("ld.shared.v2.u32 {%0,%1}, [%2+%3];" : "=r"(v.x), "=r"(v.y) : "r"(a), "n"(OFF));
  return v;
}
template <int OFF> __device__ __forceinline__ uint4 lds_u128(uint32_t a) {
  uint4 v;
  asm("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4+%5];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a), "n"(OFF));
  return v;
}

// One row chunk of K indices (a thread's 32 dims of one token: 4 KB bytes at a 4 KB-byte-aligned address) as
// big-endian words: word k holds stream bits 32 k .. 32 k + 31, first bit in the most significant position.
template <int KB, int OFF> __device__ __forceinline__ void load_k_words(uint32_t a, uint32_t (&w)[KB]) {
  if constexpr (KB == 1) {
    w[0] = __byte_perm(lds_u32<OFF>(a), 0, 0x0123);
  } else if constexpr (KB == 2) {
    const uint2 v = lds_u64<OFF>(a);
    w[0] = __byte_perm(v.x, 0, 0x0123);
    w[1] = __byte_perm(v.y, 0, 0x0123);
  } else if constexpr (KB == 3) {
    w[0] = __byte_perm(lds_u32<OFF>(a), 0, 0x0123);
    w[1] = __byte_perm(lds_u32<OFF + 4>(a), 0, 0x0123);
    w[2] = __byte_perm(lds_u32<OFF + 8>(a), 0, 0x0123);
  } else {
    const uint4 v = lds_u128<OFF>(a);
    w[0] = __byte_perm(v.x, 0, 0x0123);
    w[1] = __byte_perm(v.y, 0, 0x0123);
    w[2] = __byte_perm(v.z, 0, 0x0123);
    w[3] = __byte_perm(v.w, 0, 0x0123);
  }
}

// A thread's 16 dims of one V token (2 VB bytes at byte offset 2 VB g of the token's row) as two big-endian words.
// Three-bit rows put that chunk on a 2-byte boundary: two aligned words that cover it are loaded from `a` (the
// chunk's address rounded down to 4 bytes) and the six bytes are picked out with selectors that depend on whether
// the chunk starts the word (even g) or sits in its upper half (odd g).
template <int VB, int OFF> __device__ __forceinline__ void load_v_words(uint32_t a, uint32_t sel0, uint32_t sel1, uint32_t (&w)[2]) {
  if constexpr (VB == 2) {
    w[0] = __byte_perm(lds_u32<OFF>(a), 0, 0x0123);
    w[1] = 0;
  } else if constexpr (VB == 3) {
    const uint32_t x0 = lds_u32<OFF>(a), x1 = lds_u32<OFF + 4>(a);
    w[0] = __byte_perm(x0, x1, sel0);
    w[1] = __byte_perm(x0, x1, sel1);
  } else {
    const uint2 v = lds_u64<OFF>(a);
    w[0] = __byte_perm(v.x, 0, 0x0123);
    w[1] = __byte_perm(v.y, 0, 0x0123);
  }
}

// Splits that a cluster holds at most, its barrier, and eight bytes out of the shared memory of its CTA `rank`, at the same place as `addr` here
constexpr int CLUSTER_MOST = 8;
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ float2 lds_remote2(uint32_t addr, int rank) {
  float2 v;
  asm volatile("{\n .reg .b32 a;\n mapa.shared::cluster.u32 a, %2, %3;\n ld.shared::cluster.v2.f32 {%0,%1}, [a];\n}\n"
               : "=f"(v.x), "=f"(v.y) : "r"(addr), "r"(rank) : "memory");
  return v;
}

// DPT elements of a head's row out of the `ns` CTAs of the cluster: (maximum, sum) at `ml`, the elements at `row` in each.
template <int DPT> __device__ __forceinline__ void cluster_fold(uint32_t ml, uint32_t row, int ns, float alpha, float* out, float* lse) {
  float2 mls[CLUSTER_MOST], part[CLUSTER_MOST][DPT / 2];
#pragma unroll
  for (int r = 0; r < CLUSTER_MOST; ++r) mls[r] = r < ns ? lds_remote2(ml, r) : make_float2(-INFINITY, 0.f);
#pragma unroll
  for (int r = 0; r < CLUSTER_MOST; ++r)
#pragma unroll
    for (int k = 0; k < DPT / 2; ++k) part[r][k] = r < ns ? lds_remote2(row + 8 * k, r) : make_float2(0.f, 0.f);
  float M = -INFINITY, sum = 0.f, a[DPT];
#pragma unroll
  for (int r = 0; r < CLUSTER_MOST; ++r) M = fmaxf(M, mls[r].x);
#pragma unroll
  for (int k = 0; k < DPT; ++k) a[k] = 0.f;
#pragma unroll
  for (int r = 0; r < CLUSTER_MOST; ++r) {
    const float f = fast_exp2(mls[r].x - M);
    sum = fmaf(mls[r].y, f, sum);
#pragma unroll
    for (int k = 0; k < DPT / 2; ++k) {
      a[2 * k] = fmaf(part[r][k].x, f, a[2 * k]);
      a[2 * k + 1] = fmaf(part[r][k].y, f, a[2 * k + 1]);
    }
  }
  const float inv = 1.0f / (sum * alpha);
#pragma unroll
  for (int k = 0; k < DPT; ++k) out[k] = a[k] * inv;
  if (lse) *lse = (M + log2f(sum)) * 0.6931471805599453f;
}

// Per-thread state of the page loop: o[set][blk] = head 4 set + t, dims 16 g + 4 blk .. + 3; maxima and sums of heads
// 2 (t & 1), + 1 (NH 4) or 2 t, + 1 (NH 8).
template <int NH> struct G4State {
  float o[NH / 4][4][4];
  float m0, m1, l0, l1;
};

// What a thread needs to find its part of a page record: byte offsets inside the record of the data of its warp's
// tile (tokens 16 warp .. + 15), and the lane roles of the two exchanges.
struct G4Thr {
  uint32_t k_thr;    // K indices (or int8 values) of row g: its 32 dims (q8_0: its 8 dims of block 0)
  uint32_t ks_thr;   // K scale of the token this thread keeps after the exchange (PROD, q8_0: of row g)
  uint32_t z_thr;    // PROD: sign-sketch word of row g; residual scales follow at rs_thr
  uint32_t rs_thr;
  uint32_t v_thr;    // V indices of token t, dims 16 g .. (rounded down to 4 bytes; q8_0: the 16 int8 values)
  uint32_t vs_thr;   // V scale of the kept token (q8_0: fp16 scale of token t, block g >> 1)
  uint32_t vsel0, vsel1;
  uint32_t psel;
  int src0, rsrc;
  bool upper;
  int t, tok_in_page, vtok_in_page;
};

__device__ __forceinline__ uint32_t s8x2_to_h2(uint32_t biased, uint32_t sel) {
  // two int8 values, stored as value ^ 0x80 = value + 128, as exact fp16: (b | 0x6400) is 1024 + b; subtract 1152
  return hsub2_u32(__byte_perm(biased, 0x64646464u, sel), 0x64806480u);
}

// Sign sketch: where a half of a pair word has the bit of dim i (of 0..15), and what fp16 number that is, inverted
__device__ __forceinline__ constexpr int g4_sketch_bit(int i) { return 13 - (i & 7); }
__device__ __forceinline__ constexpr float g4_sketch_scale(int i) {
  const int b = g4_sketch_bit(i);   // 13, 12, 11, 10: exponents 8, 4, 2, 1; below: subnormal
  return (float)(1 << (b == 13 ? 7 : b == 12 ? 11 : b == 11 ? 13 : b == 10 ? 14 : 24 - b));
}
// The queries as B operands, and what goes with the tables
template <int KK, int NH> struct G4Q {
  static constexpr bool PROD = Kind<KK>::PROD;
  uint32_t qf[8][2];                                  // NH 4: columns 0-3 the hi halves, 4-7 the lo halves; NH 8: hi
  uint32_t ql[NH == 8 && !PROD ? 8 : 1][2];           // NH 8: lo
  uint32_t qp[PROD ? 8 : 1][2];                       // PROD: the projected query, as qf, over the sketch operands' values
  float zs0, zs1, zc0, zc1;                           // PROD: <S q, z> of columns 2t, 2t + 1 = sums x zs - zc
  uint32_t lo;                                        // PROD, NH 8: shared-memory address of this lane's lo fragments
  uint32_t lk_base, lk_start, lv_base, lv_start;
};

__device__ __forceinline__ uint2 lds_u64_at(uint32_t a) {
  uint2 v;   // volatile: loaded where it is used, not kept in 32 registers
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}

// Scores of one 16-token tile, per thread the MMA accumulator fragment (rows g and g + 8, columns 2t and 2t + 1).  NH 4:
// hi halves in columns 0-3, lo halves in 4-7, still to be joined; NH 8: finished, column = head.  LUT keys return raw
// sums (the caller applies the K scales); q8_0 and PROD keys have their scales applied.
template <int KK, int VK, bool NODEQ, int NW, int NH, int TOK0>
__device__ __forceinline__ void g4_scores(float (&s)[4], uint32_t st, const G4Thr& T, const G4Q<KK, NH>& Q) {
  using C = G4<KK, VK, NW, NH>;
  using KT = Kind<KK>;
  constexpr int KB = KT::BITS;
  s[0] = s[1] = s[2] = s[3] = 0.f;
  // lo halves of eight heads: accumulators of their own (two chains instead of one twice as long)
  auto lo_half = [&](float (&sl)[4], int j, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, bool projected) {
    if constexpr (NH == 8) {
      if constexpr (KT::PROD) {
        const uint2 f = lds_u64_at(Q.lo + (projected ? 2048 : 0) + j * 256);
        mma16816(sl, a0, a1, a2, a3, f.x, f.y);
      } else {
        mma16816(sl, a0, a1, a2, a3, Q.ql[j][0], Q.ql[j][1]);
      }
    }
  };
  if constexpr (KT::Q8) {
    // a 32-value block has one scale: k-steps 2b and 2b+1 cover block b (this thread supplies its dims 8t .. 8t+7 of
    // the block), and the block's partial scores are scaled in fp32 -- the operands carry no rounding
    const uint2 sc0 = lds_u64<TOK0 * C::KSCB>(st + T.ks_thr), sc1 = lds_u64<(TOK0 + 8) * C::KSCB>(st + T.ks_thr);
    const uint32_t scw0[2] = {sc0.x, sc0.y}, scw1[2] = {sc1.x, sc1.y};
#pragma unroll
    for (int blk = 0; blk < 4; ++blk) {
      uint2 u0, u1;
      constexpr int R0 = TOK0 * TQ_D, R1 = (TOK0 + 8) * TQ_D;   // rows g and g + 8 of this tile
      if (blk == 0) { u0 = lds_u64<R0>(st + T.k_thr); u1 = lds_u64<R1>(st + T.k_thr); }
      if (blk == 1) { u0 = lds_u64<R0 + 32>(st + T.k_thr); u1 = lds_u64<R1 + 32>(st + T.k_thr); }
      if (blk == 2) { u0 = lds_u64<R0 + 64>(st + T.k_thr); u1 = lds_u64<R1 + 64>(st + T.k_thr); }
      if (blk == 3) { u0 = lds_u64<R0 + 96>(st + T.k_thr); u1 = lds_u64<R1 + 96>(st + T.k_thr); }
      const uint32_t x0[2] = {u0.x ^ 0x80808080u, u0.y ^ 0x80808080u};
      const uint32_t x1[2] = {u1.x ^ 0x80808080u, u1.y ^ 0x80808080u};
      float sb[4] = {0.f, 0.f, 0.f, 0.f}, sl[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int h2 = 0; h2 < 2; ++h2) {
        const int j = 2 * blk + h2;
        const uint32_t a0 = s8x2_to_h2(x0[h2], 0x4140), a1 = s8x2_to_h2(x1[h2], 0x4140);
        const uint32_t a2 = s8x2_to_h2(x0[h2], 0x4342), a3 = s8x2_to_h2(x1[h2], 0x4342);
        mma16816(sb, a0, a1, a2, a3, Q.qf[j][0], Q.qf[j][1]);
        lo_half(sl, j, a0, a1, a2, a3, false);
      }
      if constexpr (NH == 8) { sb[0] += sl[0]; sb[1] += sl[1]; sb[2] += sl[2]; sb[3] += sl[3]; }
      const __half2 hs0 = *reinterpret_cast<const __half2*>(&scw0[blk >> 1]);
      const __half2 hs1 = *reinterpret_cast<const __half2*>(&scw1[blk >> 1]);
      const float f0 = (blk & 1) ? __high2float(hs0) : __low2float(hs0);
      const float f1 = (blk & 1) ? __high2float(hs1) : __low2float(hs1);
      s[0] = fmaf(sb[0], f0, s[0]); s[1] = fmaf(sb[1], f0, s[1]);
      s[2] = fmaf(sb[2], f1, s[2]); s[3] = fmaf(sb[3], f1, s[3]);
    }
  } else {
    uint32_t w0[KB], w1[KB];
    load_k_words<KB, TOK0 * C::KIDXB>(st + T.k_thr, w0);
    load_k_words<KB, (TOK0 + 8) * C::KIDXB>(st + T.k_thr, w1);
    using Lut = typename C::KLut;
    constexpr int SH = Lut::SHIFT;
    float sl[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      uint32_t a0, a1, a2, a3;
      if constexpr (NODEQ) {
        a0 = w0[j % KB]; a1 = w1[j % KB]; a2 = w0[(j + 1) % KB]; a3 = w1[(j + 1) % KB];
      } else {
        const uint2 f0 = field_pair<2 * KB, SH, KB>(w0, 2 * j), f1 = field_pair<2 * KB, SH, KB>(w1, 2 * j);
        a0 = Lut::load(f0.x, Q.lk_base, Q.lk_start);
        a1 = Lut::load(f1.x, Q.lk_base, Q.lk_start);
        a2 = Lut::load(f0.y, Q.lk_base, Q.lk_start);
        a3 = Lut::load(f1.y, Q.lk_base, Q.lk_start);
      }
      mma16816(s, a0, a1, a2, a3, Q.qf[j][0], Q.qf[j][1]);
      lo_half(sl, j, a0, a1, a2, a3, false);
    }
    if constexpr (NH == 8) { s[0] += sl[0]; s[1] += sl[1]; s[2] += sl[2]; s[3] += sl[3]; }
    if constexpr (KT::PROD) {
      // + sqrt(pi/2)/sqrt(d) * ||r|| * <S q, z>, as 2 sum over the set bits minus the sum over all.  Word t of a row holds its 32 dims
      // 32t .. 32t+31, first dim in the most significant bit; dims i and i + 16 form a pair, whose bits sit at the same place of
      // the word's two halves.  A half with one of the bits 6..13 set is the fp16 number 2^-18 .. 2^-7 (g4_sketch_scale), by which the
      // projected query is divided beforehand: after two shifts a pair is one logic operation.  +-1 operands took a shift and a
      // logic operation, on the half-rate integer pipe that bounds the loop: 256 ragged sequences of prod3 / turbo3 1,349 us, so 1,244.
      const uint32_t z0 = __byte_perm(lds_u32<TOK0 * 16>(st + T.z_thr), 0, 0x0123);
      const uint32_t z1 = __byte_perm(lds_u32<(TOK0 + 8) * 16>(st + T.z_thr), 0, 0x0123);
      float s2[4] = {0.f, 0.f, 0.f, 0.f}, sl2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t m0 = 0x00010001u << g4_sketch_bit(2 * j), m1 = 0x00010001u << g4_sketch_bit(2 * j + 1);
        const uint32_t x0 = j < 4 ? z0 >> 2 : z0 << 6, x1 = j < 4 ? z1 >> 2 : z1 << 6;
        const uint32_t a0 = x0 & m0, a1 = x1 & m0, a2 = x0 & m1, a3 = x1 & m1;
        mma16816(s2, a0, a1, a2, a3, Q.qp[j][0], Q.qp[j][1]);
        lo_half(sl2, j, a0, a1, a2, a3, true);
      }
      if constexpr (NH == 8) { s2[0] += sl2[0]; s2[1] += sl2[1]; s2[2] += sl2[2]; s2[3] += sl2[3]; }
      s2[0] = fmaf(s2[0], Q.zs0, -Q.zc0); s2[1] = fmaf(s2[1], Q.zs1, -Q.zc1);
      s2[2] = fmaf(s2[2], Q.zs0, -Q.zc0); s2[3] = fmaf(s2[3], Q.zs1, -Q.zc1);
      const float k0 = lds_f32<TOK0 * 4>(st + T.ks_thr), k1 = lds_f32<TOK0 * 4 + 32>(st + T.ks_thr);
      const float r0 = lds_f32<TOK0 * 4>(st + T.rs_thr), r1 = lds_f32<TOK0 * 4 + 32>(st + T.rs_thr);
      s[0] = fmaf(s2[0], r0, s[0] * k0); s[1] = fmaf(s2[1], r0, s[1] * k0);
      s[2] = fmaf(s2[2], r1, s[2] * k1); s[3] = fmaf(s2[3], r1, s[3] * k1);
    }
  }
}

// One 16-token tile of one warp: scores against the four query heads, online softmax, O^T += V^T P^T.
//   st      shared-memory address of the page record
//   MASKED  the page may end inside or before this tile (`valid` tokens of the page exist)
//   NODEQ   measurement variant: the table lookups are left out and the packed words themselves are fed to the
//           tensor cores (copies, barriers, MMAs, softmax and merges as in the real kernel; results meaningless)
//   TOK0    first token of the tile relative to the warp's first tile of the page (a multiple of 16)
template <int KK, int VK, bool MASKED, bool SPARSE, bool NODEQ, int NW, int NH, int TOK0>
__device__ __forceinline__ void g4_tile(G4State<NH>& S, uint32_t st, const G4Thr& T, const G4Q<KK, NH>& Q, int valid) {
  using C = G4<KK, VK, NW, NH>;
  using KT = Kind<KK>;
  using VT = Kind<VK>;
  constexpr int VB = VT::BITS;
  constexpr bool K_LUT = !KT::Q8 && !KT::PROD;   // raw sums, one scale per row
  constexpr float MAX_SLACK = 4.0f;
  const int t = T.t;
  // ---------------- S = K_tile (16 tokens x 128) . [q_hi | q_lo] ----------------
  float ks = 1.0f, ks_b = 1.0f;   // (NH 8: rows g and g + 8)
  if constexpr (K_LUT) ks = lds_f32<TOK0 * 4>(st + T.ks_thr);
  if constexpr (K_LUT && NH == 8) ks_b = lds_f32<TOK0 * 4 + 32>(st + T.ks_thr);
  float s[4];
  g4_scores<KK, VK, NODEQ, NW, NH, TOK0>(s, st, T, Q);
  // the V words and scale of this tile are fetched here, ahead of the softmax arithmetic that separates them from
  // their use: the loads then wait under it instead of in front of the table lookups
  uint32_t vw[4][VT::Q8 ? 4 : 2];
  uint32_t vsc16[4];   // q8_0 values: fp16 block scale of the thread's four tokens, both halves alike
  float vs_raw = 1.0f, vs_raw_b = 1.0f;
  if constexpr (VT::Q8) {
#pragma unroll
    for (int q4 = 0; q4 < 4; ++q4) {
      uint4 v;
      uint32_t sc;
      if (q4 == 0) { v = lds_u128<TOK0 * TQ_D>(st + T.v_thr); sc = lds_u16<TOK0 * C::VSCB>(st + T.vs_thr); }
      if (q4 == 1) { v = lds_u128<(TOK0 + 4) * TQ_D>(st + T.v_thr); sc = lds_u16<(TOK0 + 4) * C::VSCB>(st + T.vs_thr); }
      if (q4 == 2) { v = lds_u128<(TOK0 + 8) * TQ_D>(st + T.v_thr); sc = lds_u16<(TOK0 + 8) * C::VSCB>(st + T.vs_thr); }
      if (q4 == 3) { v = lds_u128<(TOK0 + 12) * TQ_D>(st + T.v_thr); sc = lds_u16<(TOK0 + 12) * C::VSCB>(st + T.vs_thr); }
      vw[q4][0] = v.x ^ 0x80808080u; vw[q4][1] = v.y ^ 0x80808080u;
      vw[q4][2] = v.z ^ 0x80808080u; vw[q4][3] = v.w ^ 0x80808080u;
      if constexpr (MASKED) sc = (T.vtok_in_page + TOK0 + 4 * q4 < valid) ? sc : 0u;   // a stale scale must not meet p = 0
      vsc16[q4] = __byte_perm(sc, 0, 0x1010);
    }
  } else {
    load_v_words<VB, TOK0 * C::VIDXB>(st + T.v_thr, T.vsel0, T.vsel1, vw[0]);
    load_v_words<VB, (TOK0 + 4) * C::VIDXB>(st + T.v_thr, T.vsel0, T.vsel1, vw[1]);
    load_v_words<VB, (TOK0 + 8) * C::VIDXB>(st + T.v_thr, T.vsel0, T.vsel1, vw[2]);
    load_v_words<VB, (TOK0 + 12) * C::VIDXB>(st + T.v_thr, T.vsel0, T.vsel1, vw[3]);
    vs_raw = lds_f32<TOK0 * 4>(st + T.vs_thr);
    if constexpr (NH == 8) vs_raw_b = lds_f32<TOK0 * 4 + 32>(st + T.vs_thr);
  }
  using VLut = typename C::VLut;
  constexpr int SHV = VLut::SHIFT;
  auto v_half = [&](uint32_t (&h)[2][8], int u) {
#pragma unroll
    for (int q2 = 0; q2 < 2; ++q2) {
#pragma unroll
      for (int jj = 0; jj < 8; ++jj) {
        if constexpr (VT::Q8) {
          h[q2][jj] = hmul2_u32(s8x2_to_h2(vw[2 * u + q2][jj >> 1], (jj & 1) ? 0x4342 : 0x4140), vsc16[2 * u + q2]);
        } else if constexpr (NODEQ) {
          h[q2][jj] = vw[2 * u + q2][jj & 1] ^ (uint32_t)jj;
        } else {
          if ((jj & 1) == 0) {
            const uint2 f = field_pair<2 * VB, SHV, 2>(vw[2 * u + q2], jj);
            h[q2][jj] = VLut::load(f.x, Q.lv_base, Q.lv_start);
            h[q2][jj + 1] = VLut::load(f.y, Q.lv_base, Q.lv_start);
          }
        }
      }
    }
  };
  // ---------------- online softmax (log2 domain) ----------------
  // The running maxima move only when a score exceeds them by more than 2^MAX_SLACK, so that almost every tile skips
  // the warp reduction and the rescaling of O.  What is tracked is the maximum of score + log2(V scale), not of the
  // score alone: the P operand of the second product is p * (V scale) in fp16, and with this reference it never
  // exceeds 2^MAX_SLACK whatever the norms of the values are (a reference that is too high only scales p, the
  // softmax sums and O by the same factor, which the final division removes).
  uint32_t pb[NH / 4][4];
  if constexpr (NH == 4) {
    // hi + lo: the partner lane (t ^ 2) holds the other half of the same heads
    const bool upper = T.upper;
    const float give0 = upper ? s[0] : s[2], give1 = upper ? s[1] : s[3];
    const float keep0 = upper ? s[2] : s[0], keep1 = upper ? s[3] : s[1];
    const float sum0 = keep0 + __shfl_xor_sync(0xffffffffu, give0, 2);
    const float sum1 = keep1 + __shfl_xor_sync(0xffffffffu, give1, 2);
    bool ok = true;
    float vs = vs_raw;
    float d0 = fmaf(sum0, ks, -S.m0), d1 = fmaf(sum1, ks, -S.m1);   // score - running reference
    if constexpr (MASKED) {
      ok = T.tok_in_page + TOK0 < valid;
      vs = ok ? vs_raw : 0.f;                                       // a stale scale must not meet p = 0
      d0 = ok ? d0 : -INFINITY;
      d1 = ok ? d1 : -INFINITY;
    }
    const float lvs = VT::Q8 ? 0.f : fmaxf(fast_log2(vs), -100.0f);  // zero vectors have scale 0
    if (__any_sync(0xffffffffu, (d0 + lvs > MAX_SLACK) || (d1 + lvs > MAX_SLACK))) {
      float sc0 = sum0 * ks, sc1 = sum1 * ks;
      if constexpr (MASKED) {
        sc0 = ok ? sc0 : -INFINITY;
        sc1 = ok ? sc1 : -INFINITY;
      }
      float mx0 = sc0 + lvs, mx1 = sc1 + lvs;
#pragma unroll
      for (int sh = 2; sh < 32; sh <<= 1) {
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, sh));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, sh));
      }
      const float mn0 = fmaxf(S.m0, mx0), mn1 = fmaxf(S.m1, mx1);  // finite: the tile's first token exists
      const float r0 = fast_exp2(S.m0 - mn0), r1 = fast_exp2(S.m1 - mn1);
      S.m0 = mn0;
      S.m1 = mn1;
      S.l0 *= r0;
      S.l1 *= r1;
      d0 = sc0 - mn0;
      d1 = sc1 - mn1;
      const float ra = __shfl_sync(0xffffffffu, r0, T.rsrc), rb = __shfl_sync(0xffffffffu, r1, T.rsrc);
      const float r = (t & 1) ? rb : ra;                        // O of this thread belongs to head t
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        S.o[0][j][0] *= r; S.o[0][j][1] *= r; S.o[0][j][2] *= r; S.o[0][j][3] *= r;
      }
    }
    const float p0 = fast_exp2(d0), p1 = fast_exp2(d1);
    S.l0 += p0;
    S.l1 += p1;
    // a template parameter, not a run-time flag: the possible jump keeps the V loads below it from being issued early
    // (the threshold is applied to p * V scale, the token's weight in the output relative to the largest one)
    if (SPARSE && !__any_sync(0xffffffffu, fmaxf(p0, p1) * vs >= SPARSE_V_TAU)) return;
    const uint32_t hp = pack_h2(p0 * vs, p1 * vs);
#pragma unroll
    for (int q4 = 0; q4 < 4; ++q4)
      pb[0][q4] = __byte_perm(__shfl_sync(0xffffffffu, hp, T.src0 + 16 * (q4 & 1) + 2 * (q4 >> 1)), 0, T.psel);
  } else {
    bool ok0 = true, ok1 = true;
    float vs0 = vs_raw, vs1 = vs_raw_b;
    float d00 = fmaf(s[0], ks, -S.m0), d01 = fmaf(s[1], ks, -S.m1), d10 = fmaf(s[2], ks_b, -S.m0), d11 = fmaf(s[3], ks_b, -S.m1);
    if constexpr (MASKED) {
      ok0 = T.tok_in_page + TOK0 < valid;
      ok1 = T.tok_in_page + TOK0 + 8 < valid;
      vs0 = ok0 ? vs_raw : 0.f;                                       // a stale scale must not meet p = 0
      vs1 = ok1 ? vs_raw_b : 0.f;
      d00 = ok0 ? d00 : -INFINITY;
      d01 = ok0 ? d01 : -INFINITY;
      d10 = ok1 ? d10 : -INFINITY;
      d11 = ok1 ? d11 : -INFINITY;
    }
    const float lv0 = VT::Q8 ? 0.f : fmaxf(fast_log2(vs0), -100.0f), lv1 = VT::Q8 ? 0.f : fmaxf(fast_log2(vs1), -100.0f);
    if (__any_sync(0xffffffffu, fmaxf(fmaxf(d00, d01) + lv0, fmaxf(d10, d11) + lv1) > MAX_SLACK)) {
      float sc00 = s[0] * ks, sc01 = s[1] * ks, sc10 = s[2] * ks_b, sc11 = s[3] * ks_b;
      if constexpr (MASKED) {
        sc00 = ok0 ? sc00 : -INFINITY;
        sc01 = ok0 ? sc01 : -INFINITY;
        sc10 = ok1 ? sc10 : -INFINITY;
        sc11 = ok1 ? sc11 : -INFINITY;
      }
      float mx0 = fmaxf(sc00 + lv0, sc10 + lv1), mx1 = fmaxf(sc01 + lv0, sc11 + lv1);
#pragma unroll
      for (int sh = 4; sh < 32; sh <<= 1) {
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, sh));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, sh));
      }
      const float mn0 = fmaxf(S.m0, mx0), mn1 = fmaxf(S.m1, mx1);  // finite: the tile's first token exists
      const float r0 = fast_exp2(S.m0 - mn0), r1 = fast_exp2(S.m1 - mn1);
      S.m0 = mn0;
      S.m1 = mn1;
      S.l0 *= r0;
      S.l1 *= r1;
      d00 = sc00 - mn0;
      d01 = sc01 - mn1;
      d10 = sc10 - mn0;
      d11 = sc11 - mn1;
#pragma unroll
      for (int set = 0; set < NH / 4; ++set) {                      // O of this thread: heads t and 4 + t
        const float ra = __shfl_sync(0xffffffffu, r0, T.rsrc + 2 * set), rb = __shfl_sync(0xffffffffu, r1, T.rsrc + 2 * set);
        const float r = (t & 1) ? rb : ra;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          S.o[set][j][0] *= r; S.o[set][j][1] *= r; S.o[set][j][2] *= r; S.o[set][j][3] *= r;
        }
      }
    }
    const float p00 = fast_exp2(d00), p01 = fast_exp2(d01), p10 = fast_exp2(d10), p11 = fast_exp2(d11);
    S.l0 += p00 + p10;
    S.l1 += p01 + p11;
    if (SPARSE && !__any_sync(0xffffffffu, fmaxf(fmaxf(p00, p01) * vs0, fmaxf(p10, p11) * vs1) >= SPARSE_V_TAU)) return;
    const uint32_t hp0 = pack_h2(p00 * vs0, p01 * vs0), hp1 = pack_h2(p10 * vs1, p11 * vs1);
#pragma unroll
    for (int set = 0; set < NH / 4; ++set)
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4)   // token t + 4 q4: row t + 4 (q4 & 1), of the upper eight for q4 >= 2
        pb[set][q4] = __byte_perm(__shfl_sync(0xffffffffu, q4 < 2 ? hp0 : hp1, T.src0 + 16 * (q4 & 1) + 2 * set), 0, T.psel);
  }
  // ---------------- O^T += V_tile^T . P^T : tokens t, t+4, t+8, t+12 of the tile, dims 16g .. 16g+15 ----------------
  // (neighbouring lanes read neighbouring token rows: rows are 16 VB bytes apart, which spreads a quad of lanes over
  // the shared-memory banks; a stride of four rows put lanes t and t+2 on the same banks)
  // two halves of eight tokens: the table words of one half (16 registers) are live at a time, which leaves the
  // compiler room to keep more loads in flight (all four token rows at once: 5 % slower at 256K tokens; forming
  // the first half ahead of the softmax arithmetic: no gain)
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    uint32_t h[2][8];
    v_half(h, u);
#pragma unroll
    for (int blk = 0; blk < 4; ++blk)
#pragma unroll
      for (int set = 0; set < NH / 4; ++set)
        mma16816(S.o[set][blk], h[0][2 * blk], h[0][2 * blk + 1], h[1][2 * blk], h[1][2 * blk + 1], pb[set][2 * u], pb[set][2 * u + 1]);
  }
}

// the warp's tiles of one page: tile TT covers tokens 16 (warp + NW TT) .. + 15
template <int KK, int VK, bool SPARSE, bool NODEQ, int NW, int NH, int TT>
__device__ __forceinline__ void g4_page(G4State<NH>& S, uint32_t st, const G4Thr& T, const G4Q<KK, NH>& Q, bool full,
                                        int last_valid, int warp) {
  constexpr int TOK0 = 16 * NW * TT;
  if (full) g4_tile<KK, VK, false, SPARSE, NODEQ, NW, NH, TOK0>(S, st, T, Q, G4_PT);
  else if (16 * warp + TOK0 < last_valid) g4_tile<KK, VK, true, SPARSE, NODEQ, NW, NH, TOK0>(S, st, T, Q, last_valid);
  if constexpr (TT + 1 < ATT_WARPS / NW) g4_page<KK, VK, SPARSE, NODEQ, NW, NH, TT + 1>(S, st, T, Q, full, last_valid, warp);
}

// NW warps per CTA: 8 (two CTAs per SM), or 4 (four per SM, two tiles per warp and page) for chains of calls that may
// overlap completely: the CTAs of two consecutive calls then share an SM four at a time, each in a phase of its own,
// and the SM's warps are in a page loop 80 % of the time instead of 67 %.
// TAIL: the call follows the append of the step's token (TQ_DECODE_OVERLAP_APPEND).  A template parameter, so that the
// page loop of every other instantiation carries nothing for it.
// CL: the splits of a (sequence, KV head) are a cluster.  A template parameter: with the cluster's instructions in it, every other launch
// of the kernel was 0.1 to 0.4 us longer.
template <int KK, int VK, bool SPARSE, bool NODEQ, int NW, bool TAIL, int NH, bool CL>
__global__ void __launch_bounds__(32 * NW, 16 / NW) k_decode_attn_g4(const __grid_constant__ AttnParams P, const __grid_constant__ AttnQuant fk,
                                                                      const __grid_constant__ AttnQuant fv) {
  using C = G4<KK, VK, NW, NH>;
  constexpr int NT = 32 * NW;          // threads
  constexpr int G4_NS = C::NS;
  using KT = Kind<KK>;
  using VT = Kind<VK>;
  constexpr int KB = KT::BITS, VB = VT::BITS;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  int split, kvh, b;
  split_index(P, split, kvh, b);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  constexpr int bar_id = 0;
  {  // one parameter line per warp, all misses in flight together
    const uint32_t* pp = reinterpret_cast<const uint32_t*>(&P);
    uint32_t touch;
    if (warp < 4) touch = pp[min(16 * warp, (int)(sizeof(AttnParams) / 4) - 1)];
    else if (warp < 6) touch = warp == 4 ? fk.s1[0] : fk.pad[2];   // first and last word of the 112-byte blocks
    else touch = warp == 6 ? fv.s1[0] : fv.pad[2];
    asm volatile("" ::"r"(touch));
  }
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* sm = smem_raw + (((raw + C::ALIGN - 1) & ~(uint32_t)(C::ALIGN - 1)) - raw);
  // Programmatic dependent launch (every launch has the attribute, see TQ_PDL_ENTER).  In stream order the CTA fills the
  // pair tables, waits for the preceding kernel, lets the next one start and only then reads anything.
  // With an overlap mode the next kernel may start as soon as SMs free up, and everything before this kernel's
  // griddepcontrol.wait reads only the cache, the block table and the sequence lengths -- and, when the caller says that
  // the preceding kernel does not write the queries either (q_early), the queries.  What comes after the wait runs after
  // the preceding kernel has completed and its writes are visible: the workspace and the output are only ever touched
  // there.  Without q_early the wait stands in front of the query load; with it, in front of the first write (after the
  // page loop).
  if (P.overlap) {
    TQ_PDL_TRIGGER();
  } else {
    if constexpr (KB > 0) g4_lut_fill<typename C::KLut, KB>(sm + C::OFF_K, fk.cent16, tid, NT);
    if constexpr (VB > 0) g4_lut_fill<typename C::VLut, VB>(sm + C::OFF_V, fv.cent16, tid, NT);
    TQ_PDL_ENTER();
  }
  const int chunk = split_chunk(P, G4_PT, lane), page_lo = split * chunk;
  const size_t row0 = (size_t)b * P.hq + (size_t)kvh * P.group;
  int seq;
  const int seq_len = row_length(P, b, G4_PT, seq);
  const int32_t* bt = P.block_table + (size_t)seq * P.max_pages;
  uint8_t* smg = sm + C::OFF_GROUPS;
  float* qbuf = reinterpret_cast<float*>(smg + C::G_Q);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smg + C::G_BAR);
  volatile int* s_flags = reinterpret_cast<volatile int*>(smg + C::G_BAR + 64);
  uint8_t* stage0 = smg + C::G_STAGE;
  constexpr int PRODUCER = NT - 32;  // lane 0 of the last warp issues every bulk copy
  const uint8_t* pool_head = P.pool + (int64_t)kvh * P.L.head_stride;

  auto issue = [&](int stage, int64_t page) {
    uint64_t* bar = &bars[stage];
    mbar_expect_tx(bar, C::REC);
    bulk_g2s(stage0 + stage * C::REC, pool_head + page * P.L.page_stride, C::REC, bar);
  };

  // The warps take different roles so that their global-load latencies (and their instruction fetches, which are
  // cold in every launch) overlap: the producer sends the first pages on their way as early as it can, the first
  // `group` warps rotate one query head each, the others fill the pair tables.
  const int n_pages = (seq_len + G4_PT - 1) / G4_PT;
  const int np = min(n_pages, page_lo + chunk) - page_lo;   // pages of this CTA (<= 0: none)
  int pg_ahead = 0;  // producer: block-table entry of the page issued in the next iteration
  if (tid == PRODUCER) {   // (where every warp rotates a query, this one does so afterwards)
    int pg_next[G4_NS];
#pragma unroll
    for (int i = 0; i < G4_NS; ++i) pg_next[i] = bt[min(page_lo + i, P.max_pages - 1)];
#pragma unroll
    for (int s = 0; s < G4_NS; ++s) mbar_init(&bars[s], 1);
    s_flags[0] = 0;
    s_flags[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
#pragma unroll
    for (int s = 0; s < G4_NS - 1; ++s)
      if (np > s) {
        // after an append the last page of the sequence is what the preceding kernel writes: it is fetched once that
        // kernel has completed (the wait costs nothing when it already has), every other page right away
        if (TAIL && page_lo + s == n_pages - 1) asm volatile("griddepcontrol.wait;" ::: "memory");
        issue(s, pg_next[s]);
      }
    pg_ahead = pg_next[G4_NS - 1];
  }
  if (warp < P.group && P.overlap && !P.q_early) asm volatile("griddepcontrol.wait;" ::: "memory");
  for (int hd = warp; hd < P.group; hd += NW) {
    float x[4], y[4];
    if (P.k_pre) {   // dense rotations: rotated (and, for PROD keys, projected) queries come from k_prepare_queries
      load_q4(P.qrot, TQ_F32, (row0 + hd) * TQ_D + 4 * lane, x);
      if constexpr (KT::PROD) load_q4(P.qproj, TQ_F32, (row0 + hd) * TQ_D + 4 * lane, y);
    } else {
      load_q4(P.q, P.q_dtype, (row0 + hd) * TQ_D + 4 * lane, x);
      if constexpr (KT::PROD) {
#pragma unroll
        for (int k = 0; k < 4; ++k) y[k] = x[k];
        warp_wht128(y, fk.j1, fk.j2, lane);
      }
      if (!KT::Q8) warp_wht128(x, fk.s1, fk.s2, lane);   // q8_0 tensors are stored unrotated
      const float sk = P.qscale / fk.alpha;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        x[k] *= sk;
        if constexpr (KT::PROD) y[k] *= P.qscale;
      }
    }
    // 16-byte chunk c = 8 t + j of head h sits at 8 t + (j ^ (t + 4 (h & 1))): the fragment reads below (fixed j,
    // all t and h) then touch every bank group instead of one
    const int tq = lane >> 3, jq = lane & 7;
    *reinterpret_cast<float4*>(qbuf + hd * TQ_D + 4 * (8 * tq + (jq ^ (tq + 4 * (hd & 1))))) =
        make_float4(x[0], x[1], x[2], x[3]);
    if constexpr (KT::PROD) {
      // projected queries behind the rotated ones, dim 32 t + c of head h at (c NH + h) 4 + t: the fragment reads below (one
      // c, all t and h) then are 32 neighbouring floats.  As plain rows they all fell into one bank, 32 reads of 32
      // wavefronts in every warp: with eight heads this cost more than the general kernel's whole lead (prod3 / turbo3, one
      // sequence of 4,096 tokens, 64/8 heads: general kernel 16.6 us, 19.0 -> 11.4; 32/8 heads 12.7 -> 9.0)
#pragma unroll
      for (int k = 0; k < 4; ++k)
        qbuf[NH * TQ_D + ((4 * (lane & 7) + k) * NH + hd) * 4 + (lane >> 3)] = y[k];
    }
    if constexpr (NH <= NW) break;
  }
  __syncwarp();
  if (!P.overlap) {   // filled above
  } else if (NW == 4 || NH == 8) {   // every warp may have rotated a query: all of them fill the tables afterwards
    if constexpr (KB > 0) g4_lut_fill<typename C::KLut, KB>(sm + C::OFF_K, fk.cent16, tid, NT);
    if constexpr (VB > 0) g4_lut_fill<typename C::VLut, VB>(sm + C::OFF_V, fv.cent16, tid, NT);
  } else if (warp >= P.group) {
    const int fh = NT - 32 * P.group;   // table-filling threads
    if constexpr (KB > 0) g4_lut_fill<typename C::KLut, KB>(sm + C::OFF_K, fk.cent16, tid - 32 * P.group, fh);
    if constexpr (VB > 0) g4_lut_fill<typename C::VLut, VB>(sm + C::OFF_V, fv.cent16, tid - 32 * P.group, fh);
  }
  if (P.overlap && !P.q_early) asm volatile("griddepcontrol.wait;" ::: "memory");   // the query warps already have
  if (n_pages == 0 && split == 0) {  // empty sequence: zeros (split 0 exists for every kv head)
    if (P.overlap && P.q_early) asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int e = tid; e < P.group * TQ_D; e += NT) store_out(P.out, P.out_dtype, row0 * TQ_D + e, 0.f);
    if (P.lse && tid < P.group) P.lse[row0 + tid] = -INFINITY;
  }
  const int ns = (n_pages + chunk - 1) / chunk;
  __syncthreads();               // tables, query buffer and mbarriers are ready
  if (np <= 0) return;           // this CTA has no pages (its split lies beyond the sequence)

  // B operand of S = K q^T: column g is head g & 3, hi half for g < 4, lo half otherwise (NH 8: head g, hi and lo apart)
  G4Q<KK, NH> Q;
  {
    const int head = NH == 8 ? g : g & 3;
    const bool hv = head < P.group, lo = NH == 4 && g >= 4;
    const float* qh = qbuf + (hv ? head : 0) * TQ_D;
    uint2* lo_frag = reinterpret_cast<uint2*>(smg + C::G_LO) + lane;   // (LO_SMEM: the same in every warp, written by the first)
    Q.lo = smem_u32(lo_frag);
    // PROD: the projected query's largest element is brought to 2^-4 .. 2^-3, so that 2^18 times it is an fp16 number
    float zscale = 1.f;
    if constexpr (KT::PROD) {
      const float* ph = qbuf + NH * TQ_D + (hv ? head : 0) * 4 + t;
      float most = 0.f, total = 0.f;
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        const float y = hv ? ph[c * (4 * NH)] : 0.f;
        most = fmaxf(most, fabsf(y));
        total += y;
      }
#pragma unroll
      for (int m = 1; m <= 2; m <<= 1) {   // the quad's four parts of the row
        most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, m));
        total += __shfl_xor_sync(0xffffffffu, total, m);
      }
      const int e = max((int)((__float_as_uint(most) >> 23) & 255u), 14);   // most < 2^(e - 126); from 14: 2^18 zscale is a finite number
      zscale = e < 240 ? __uint_as_float((uint32_t)(250 - e) << 23) : 1.f;  // 2^(123 - e): most x zscale < 2^-3
      const float back = 2.f / zscale, take = lo ? 0.f : total;             // (the lo halves are part of the same sum)
      Q.zs0 = __shfl_sync(0xffffffffu, back, 8 * t);                        // column 2t is that of the lanes g = 2t
      Q.zs1 = __shfl_sync(0xffffffffu, back, 8 * t + 4);
      Q.zc0 = __shfl_sync(0xffffffffu, take, 8 * t);
      Q.zc1 = __shfl_sync(0xffffffffu, take, 8 * t + 4);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      // dims this thread supplies in k-step j: 32t + 4j .. +3 (packed formats), or, for q8_0 keys, its 8 dims of
      // block j/2: 32(j/2) + 8t + 4(j%2) .. +3; as the 16-byte chunk (row, col) of the staged query
      const int crow = KT::Q8 ? (j >> 1) : t, ccol = KT::Q8 ? 2 * t + (j & 1) : j;
      float4 v = hv ? *reinterpret_cast<const float4*>(qh + 4 * (8 * crow + (ccol ^ (crow + 4 * (head & 1)))))
                    : make_float4(0.f, 0.f, 0.f, 0.f);
      const __half2 h0 = __floats2half2_rn(v.x, v.y), h1 = __floats2half2_rn(v.z, v.w);
      const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
      const uint32_t l0 = pack_h2(v.x - f0.x, v.y - f0.y), l1 = pack_h2(v.z - f1.x, v.w - f1.y);
      Q.qf[j][0] = lo ? l0 : *reinterpret_cast<const uint32_t*>(&h0);
      Q.qf[j][1] = lo ? l1 : *reinterpret_cast<const uint32_t*>(&h1);
      if constexpr (NH == 8 && !KT::PROD) {
        Q.ql[j][0] = l0;
        Q.ql[j][1] = l1;
      }
      if constexpr (C::LO_SMEM)
        if (warp == 0) lo_frag[32 * j] = make_uint2(l0, l1);
      if constexpr (KT::PROD) {
        // sign-sketch operands pair dims i and i + 16 of the thread's 32 (i = 2j for the first register of the
        // k-step, 2j + 1 for the second), dim i + 16 in the low half
        const float* ph = qbuf + NH * TQ_D + (hv ? head : 0) * 4 + t;
        auto proj = [&](int c) { return hv ? ph[c * (4 * NH)] : 0.f; };
        const float za = zscale * g4_sketch_scale(2 * j), zb = zscale * g4_sketch_scale(2 * j + 1);
        const float a0 = proj(16 + 2 * j) * za, a1 = proj(2 * j) * za, b0 = proj(16 + 2 * j + 1) * zb, b1 = proj(2 * j + 1) * zb;
        const __half2 e0 = __floats2half2_rn(a0, a1), e1 = __floats2half2_rn(b0, b1);
        const float2 r0 = __half22float2(e0), r1 = __half22float2(e1);
        const uint32_t m0 = pack_h2(a0 - r0.x, a1 - r0.y), m1 = pack_h2(b0 - r1.x, b1 - r1.y);
        Q.qp[j][0] = lo ? m0 : *reinterpret_cast<const uint32_t*>(&e0);
        Q.qp[j][1] = lo ? m1 : *reinterpret_cast<const uint32_t*>(&e1);
        if constexpr (C::LO_SMEM)
          if (warp == 0) lo_frag[256 + 32 * j] = make_uint2(m0, m1);
      }
    }
  }
  if constexpr (C::LO_SMEM) group_sync<NT>(bar_id);
  Q.lk_start = smem_u32(sm + C::OFF_K);
  Q.lv_start = smem_u32(sm + C::OFF_V);
  Q.lk_base = (C::KLut::BIG ? 0u : Q.lk_start) + (C::KLut::REPL ? lane * 4 : 0);
  Q.lv_base = (C::VLut::BIG ? 0u : Q.lv_start) + (C::VLut::REPL ? lane * 4 : 0);
  // P operand: this thread's column is (head g >> 1, parity g & 1); the owner of p[token][head] is lane
  // 4 (token & 7) + 2 (token >> 3) + (head >> 1), half (head & 1) of its packed pair
  const int src0 = 4 * t + (g >> 2);                                  // token t; token 4 i + t: + 16 (i & 1) + 2 (i >> 1)
  const uint32_t psel = ((g >> 1) & 1) ? ((g & 1) ? 0x3244u : 0x4432u) : ((g & 1) ? 0x1044u : 0x4410u);
  const int rsrc = (lane & ~3) | (t >> 1);                             // a lane that tracks head t's running maximum (4 + t: + 2)
  const bool upper = NH == 4 && t >= 2;                                // keeps token g + 8 after the exchange

  G4State<NH> S;
#pragma unroll
  for (int set = 0; set < NH / 4; ++set)
#pragma unroll
    for (int j = 0; j < 4; ++j) S.o[set][j][0] = S.o[set][j][1] = S.o[set][j][2] = S.o[set][j][3] = 0.f;
  S.m0 = S.m1 = -INFINITY;
  S.l0 = S.l1 = 0.f;

  // byte offsets inside a page record of what this thread reads in its warp's tile (tokens 16 warp .. + 15)
  G4Thr T;
  T.t = t;
  T.upper = upper;
  T.src0 = src0;
  T.rsrc = rsrc;
  T.psel = psel;
  T.tok_in_page = 16 * warp + g + (upper ? 8 : 0);
  T.vtok_in_page = 16 * warp + t;
  T.k_thr = C::K_IDX + (16 * warp + g) * C::KIDXB + (KT::Q8 ? 8 * t : t * (C::KIDXB / 4));
  // the row this thread keeps (packed keys: the scale is applied after the exchange), or row g (q8_0 and PROD keys
  // finish the scores of both rows before the exchange)
  T.ks_thr = C::K_SCALE + C::KSCB * ((KT::Q8 || KT::PROD) ? 16 * warp + g : T.tok_in_page);
  T.z_thr = C::K_QJL + (16 * warp + g) * 16 + 4 * t;
  T.rs_thr = C::K_RSCALE + 4 * (16 * warp + g);
  const uint32_t v_chunk = C::V_IDX + (16 * warp + t) * C::VIDXB + g * (VT::Q8 ? 16 : 2 * VB);
  T.v_thr = v_chunk & ~3u;
  T.vs_thr = VT::Q8 ? C::V_SCALE + (16 * warp + t) * C::VSCB + 2 * (g >> 1) : C::V_SCALE + 4 * T.tok_in_page;
  const bool v_odd = (v_chunk & 2u) != 0;
  T.vsel0 = v_odd ? 0x2345u : 0x0123u;
  T.vsel1 = v_odd ? 0x6744u : 0x4544u;
  const uint32_t stage_addr = smem_u32(stage0);
  // pages 0 .. np-2 of the CTA are full; the last one is full unless the sequence ends inside it
  const int last_valid = seq_len - (page_lo + np - 1) * G4_PT;          // >= 1
  const int n_full = last_valid >= G4_PT ? np : np - 1;

  int stage = 0;
  uint32_t parity = 0;
  for (int i = 0; i < np; ++i) {
    if (tid == PRODUCER && i + G4_NS - 1 < np) {
      if (TAIL && page_lo + i + G4_NS - 1 == n_pages - 1) asm volatile("griddepcontrol.wait;" ::: "memory");
      issue(stage == 0 ? G4_NS - 1 : stage - 1, pg_ahead);            // the stage the page before this one has left
      pg_ahead = bt[min(page_lo + i + G4_NS, P.max_pages - 1)];
    }
    // (the page the preceding kernel writes is only fetched once that kernel has completed: the bounded wait for it
    // starts then, however long that kernel runs)
    if (TAIL && page_lo + i == n_pages - 1) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (!s_flags[0] && !mbar_wait_bounded(&bars[stage], parity)) s_flags[0] = 1;
    // the stage address carries a value the wait above produced (always zero), so that no load of the stage can
    // be scheduled ahead of the wait
    uint32_t dep;
    asm volatile("mov.u32 %0, 0;" : "=r"(dep)::"memory");
    const uint32_t st = stage_addr + stage * C::REC + dep;
    g4_page<KK, VK, SPARSE, NODEQ, NW, NH, 0>(S, st, T, Q, i < n_full, last_valid, warp);
    group_sync<NT>(bar_id);  // every warp is done with this stage before it is refilled
    if (++stage == G4_NS) {
      stage = 0;
      parity ^= 1u;
    }
  }
  // from here on the workspace and the output are written
  if (P.overlap && P.q_early) asm volatile("griddepcontrol.wait;" ::: "memory");
  // ---------------- merge the eight warps, write the split partial ----------------
#pragma unroll
  for (int sh = NH == 4 ? 2 : 4; sh < 32; sh <<= 1) {
    S.l0 += __shfl_xor_sync(0xffffffffu, S.l0, sh);
    S.l1 += __shfl_xor_sync(0xffffffffu, S.l1, sh);
  }
  float* so = reinterpret_cast<float*>(stage0);                    // [warp][head][G4_HSTRIDE]
  float* sml = so + NW * NH * G4_HSTRIDE;                    // [warp][head][2]
#pragma unroll
  for (int set = 0; set < NH / 4; ++set)
#pragma unroll
    for (int blk = 0; blk < 4; ++blk)
      *reinterpret_cast<float4*>(so + (size_t)(warp * NH + 4 * set + t) * G4_HSTRIDE + 16 * g + 4 * blk) =
          make_float4(S.o[set][blk][0], S.o[set][blk][1], S.o[set][blk][2], S.o[set][blk][3]);
  if (g == 0 && t < NH / 2) {
    *reinterpret_cast<float4*>(sml + (warp * NH + 2 * t) * 2) = make_float4(S.m0, S.l0, S.m1, S.l1);
  }
  group_sync<NT>(bar_id);
  float* rows = qbuf;   // of the finished output, in V's rotated space
  {
    // thread (head, DPT consecutive dims): NH heads x 128 dims over the CTA's threads; the warps' rows are added in
    // warp order
    constexpr int DPT = NH * TQ_D / NT;     // 2, 4 or 8
    const int head = tid / (TQ_D / DPT), dim = DPT * (tid % (TQ_D / DPT));
    // Four warps (chains, many CTAs): the partial of several splits is stored where its values are added up, the single split's way behind
    // it; eight warps the other way round.  The order alone is worth this much (us; 32/8 heads; single splits in front / behind): 40 chained
    // layers over 32,768 tokens 416.0 / 413.3 a step, 256 ragged sequences of prod3 / turbo3 1,268 / 1,264; one sequence of 128 tokens of
    // turbo3 4.09 / 4.23, of 1,500 of turbo4 6.83 / 6.96.
    constexpr bool EARLY = NW == 4;
    static_assert(!(EARLY && CL), "clusters are of eight-warp CTAs");
    float a[DPT], M = -INFINITY, Lsum = 0.f;
    const bool several = ns != 1;
    auto store_partial = [&]() {
      const size_t slot = (row0 + head) * P.num_splits + split;
#pragma unroll
      for (int k = 0; k < DPT; k += 2)
        *reinterpret_cast<float2*>(P.part_o + slot * TQ_D + dim + k) = make_float2(a[k], a[k + 1]);
      if (dim == 0) *reinterpret_cast<float2*>(P.part_ml + slot * 2) = make_float2(M, Lsum);
    };
    if (head < P.group) {
      float mw[NW];
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        mw[w] = sml[(w * NH + head) * 2];
        M = fmaxf(M, mw[w]);
      }
#pragma unroll
      for (int k = 0; k < DPT; ++k) a[k] = 0.f;
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        const float f = mw[w] == -INFINITY ? 0.f : fast_exp2(mw[w] - M);
        const float* v = so + (size_t)(w * NH + head) * G4_HSTRIDE + dim;
#pragma unroll
        for (int k = 0; k < DPT; ++k) a[k] = fmaf(v[k], f, a[k]);
        Lsum = fmaf(sml[(w * NH + head) * 2 + 1], f, Lsum);
      }
      if (EARLY && several) store_partial();
    }
    // The only split is finished here, as the fold of one would (its partial, a ticket and the way back were 2 us of each CTA; turbo3,
    // 32/8 heads, 128 sequences of 100 tokens 15.4 -> 11.1 us, one of 128 5.8 -> 3.8).  Splits in a cluster: the first CTA takes the
    // others' rows out of their shared memory.  One copy of the code that stores rows: with one per way here, long contexts took 0.06 us
    // a call longer.
    auto merge = [&]() { return merge_splits<VT::Q8, NT, NH>(P, fv.alpha, qbuf, s_flags, row0, ns, b, kvh, tid, bar_id); };
    if (EARLY && several) {
      if (!merge()) return;
    } else if (EARLY || CL || !several) {
      if (tid == 0 && s_flags[0]) atomicExch(P.status, 1);
      if (CL && several) {
        float2* ml = reinterpret_cast<float2*>(stage0);   // (the warps' rows there have been read)
        group_sync<NT>(bar_id);
        if (head < P.group) {
#pragma unroll
          for (int k = 0; k < DPT; k += 2) *reinterpret_cast<float2*>(qbuf + head * TQ_D + dim + k) = make_float2(a[k], a[k + 1]);
          if (dim == 0) ml[head] = make_float2(M, Lsum);
        }
        cluster_arrive();
        cluster_wait();
        if (split != 0) {   // this CTA's memory stays until it has been read
          cluster_arrive();
          cluster_wait();
          return;
        }
        rows = reinterpret_cast<float*>(stage0 + 1024);
        if (head < P.group)
          cluster_fold<DPT>(smem_u32(ml + head), smem_u32(qbuf + head * TQ_D + dim), ns, VT::Q8 ? 1.0f : fv.alpha, rows + head * TQ_D + dim,
                            P.lse && dim == 0 ? P.lse + row0 + head : nullptr);
        cluster_arrive();
      } else if (head < P.group) {
        const float inv = 1.0f / (Lsum * (VT::Q8 ? 1.0f : fv.alpha));
#pragma unroll
        for (int k = 0; k < DPT; ++k) qbuf[head * TQ_D + dim + k] = a[k] * inv;
        if (P.lse && dim == 0) P.lse[row0 + head] = (M + log2f(Lsum)) * 0.6931471805599453f;
      }
      group_sync<NT>(bar_id);
    } else {
      if (head < P.group) store_partial();
      if (!merge()) return;
    }
  }
  store_rows<NT, NH>(P, fv.s1, fv.s2, rows, row0, tid);
  if (CL && ns != 1) cluster_wait();
}

template <int KK, int VK, bool SPARSE, bool NODEQ, int NW, bool TAIL, int NH, bool CL>
int launch_attn_form(const AttnParams& P, const TqFast& fk, const TqFast& fv, cudaStream_t st) {
  using C = G4<KK, VK, NW, NH>;
  static_assert((16 / NW) * (C::SMEM + 1024) <= 228 * 1024, "CTAs of the specialised decode kernel per SM");
  constexpr auto kernel = k_decode_attn_g4<KK, VK, SPARSE, NODEQ, NW, TAIL, NH, CL>;
  static thread_local int configured_dev = -1;  // per instantiation
  int dev = 0;
  TQ_CUDA(cudaGetDevice(&dev));
  if (configured_dev != dev) {
    TQ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
    configured_dev = dev;
  }
  AttnQuant ak, av;
  memset(&ak, 0, sizeof(ak));
  memset(&av, 0, sizeof(av));
  memcpy(ak.s1, fk.s1, 16); memcpy(ak.s2, fk.s2, 16); memcpy(ak.j1, fk.j1, 16); memcpy(ak.j2, fk.j2, 16);
  memcpy(ak.cent16, fk.cent16, 32); ak.alpha = fk.lut_alpha;
  memcpy(av.s1, fv.s1, 16); memcpy(av.s2, fv.s2, 16); memcpy(av.cent16, fv.cent16, 32); av.alpha = fv.lut_alpha;
  TQ_CUDA(tq_launch_cluster(kernel, split_grid(P), 32 * NW, C::SMEM, st, CL ? P.num_splits : 1, P, ak, av));
  return tq_launch_check("k_decode_attn_g4");
}

template <int KK, int VK, bool SPARSE, bool NODEQ, int NW = ATT_WARPS, bool TAIL = false, int NH = 4>
int launch_attn_g4(const AttnParams& P_in, const SplitPlan& plan, const TqFast& fk, const TqFast& fv, cudaStream_t st) {
  const AttnParams P = with_splits(P_in, plan, NW == 4);
  // Splits that are a cluster, in calls of few CTAs that no chain overlaps: the merge's way through memory, a ticket and two fences, made
  // them 1 us longer (turbo3, 32/8 heads, behind the append of the step's token: one sequence of 517 tokens 9.3 -> 8.2 us, four 10.4 -> 9.3,
  // eight of 500 10.8 -> 9.6; 16/2 heads, four of 1,000 10.0 -> 9.7).  Clusters of eight do not find their places where CTAs share SMs (four
  // of 1,000, without appends between: 7.4 -> 8.9), clusters of sixteen not at all (16 of 2,000, 4/1 heads: 7.6 -> 10.8).
  if constexpr (!SPARSE && !NODEQ && NW == ATT_WARPS) {
    const int64_t ctas = (int64_t)P.num_splits * P.hkv * P.batch, sms = tq_num_sms();
    if (P.num_splits > 1 && P.num_splits <= CLUSTER_MOST && !P.chunk_spread && (TAIL || (!P.q_early && !P.chain_head)) &&
        ctas <= (P.num_splits <= 6 ? 2 * sms : sms))
      return launch_attn_form<KK, VK, SPARSE, NODEQ, NW, TAIL, NH, true>(P, fk, fv, st);
  }
  return launch_attn_form<KK, VK, SPARSE, NODEQ, NW, TAIL, NH, false>(P, fk, fv, st);
}

template <int KK, int VK>
bool layout_matches(const tq_cache_layout& L) {
  using C = G4<KK, VK>;
  if (Kind<KK>::PROD && (L.k_qjl_off != C::K_QJL || L.k_rscale_off != C::K_RSCALE)) return false;
  return L.page_tokens == G4_PT && L.k_idx_off == C::K_IDX && L.k_scale_off == C::K_SCALE && L.v_idx_off == C::V_IDX &&
         L.v_scale_off == C::V_SCALE && L.record_bytes == C::REC && L.k_idx_bytes == C::KIDXB && L.v_idx_bytes == C::VIDXB;
}

// The form of a call: four-warp CTAs, four per SM, or eight-warp CTAs, two per SM.
// Four warps pay where CTAs in different phases share an SM -- one in its latency-bound prologue or merge while the others
// stream pages: in a chain of attention calls (TQ_DECODE_OVERLAP_Q, and the call in front of them when the caller says so,
// TQ_DECODE_CHAIN_HEAD), and inside a call of more CTAs than one round at two per SM (256 sequences of 8,192 tokens of
// turbo3: 529 us with eight warps, 457 with four).  A call of one round on its own takes the eight-warp form (16 sequences:
// 43 against 47 us).
// 4-bit tables: only the eight-warp form has room for lane-replicated ones (32 KB each), which is worth more where a CTA
// streams pages (turbo4 / turbo4, 16 sequences of 8,192 tokens, per call of a chain: 62 us with four warps and one copy of the
// tables, 37 with eight), but they are filled anew by every CTA: a chain of calls with one or two pages per CTA is ahead with
// four warps (32/8 heads, 32 sequences of 100 tokens 7.5 -> 5.5 us, 16 of 256 6.9 -> 5.6, 8 of 1,024 7.4 -> 7.1; 16 of 1,024,
// four pages: 9.9 against 11.0), unless many splits leave a long fold to the four (32 splits of a page: 5.8 against 6.1).  So are
// single calls of more than one round (turbo4 / turbo4, 32/8 heads, 128 sequences of 100 tokens 27.2 -> 19.5 us, 214 of 147 46.1 -> 33.7,
// ragged ones up to 147 42.2 -> 27.0; 64/8 heads 51.4 -> 41.7; with four pages, 256 of 512, 75.2 against 77.6).
// Five to eight heads: four warps rotate and fold two heads each, 0.6 us and, with several splits, 0.8 us and 0.045 us per
// split of a chained call, against 0.55 us saved per page of a CTA (64/8 heads of turbo3, eight warps / four: one sequence
// of 4,096 tokens, 32 x 1 pages 6.7 / 9.8 us, of 65,536, 37 x 14, 23.7 / 21.2; 4 of 4,096, 8 x 4, 9.6 / 9.1; 16/2 heads, one
// of 65,536, 128 x 4, 11.8 / 17.3).
inline bool four_warps(const AttnParams& P, const SplitPlan& plan) {
  const bool wide = P.L.k_format == TQ_FMT_TURBO4 || P.L.v_format == TQ_FMT_TURBO4;   // (prod4: 3 bits and the sketch)
  if ((P.q_early || P.chain_head) && !P.tail_late) {
    if (P.group > 4) return !wide && 12 * plan.chunk_pages > (plan.num_splits > 1 ? 31 : 13) + plan.num_splits;
    return !wide || (plan.chunk_pages <= 2 && plan.num_splits <= 16);
  }
  return (!wide || plan.chunk_pages <= 2) && (int64_t)plan.num_splits * P.hkv * P.batch > 2 * (int64_t)tq_num_sms();
}

}  // namespace
