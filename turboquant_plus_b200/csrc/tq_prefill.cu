// Chunked-prefill attention over the packed paged cache on the 5th-generation tensor cores (tcgen05).
//
// One CTA = 128 rows of (query token, query head) pairs that share a KV head; row r is lane r of tensor memory.
// Per 128-token page: the packed page record arrives by a bulk async copy; producer warps turn the K and V indices
// (2b-bit pairs -> fp16 centroid pairs through a lane-replicated table) into unswizzled tcgen05 operand tiles in
// shared memory (K-major for K, MN-major for V); S = Q K^T and O += P V run as tcgen05.mma with the rotated queries
// (fp16 hi + lo halves), S, P and O all in tensor memory; the row warps do the online softmax between the two
// products.  The kernel, its roles, its tensor-memory map and its hand-offs are described above k_prefill_attn2.
// Every wait is bounded in time; a CTA that gives up sets the status word and still frees its tensor memory.
#include <type_traits>
#include "tq_tcgen05.cuh"

namespace {

constexpr int PF_ROWS = 128, PF_PAGE = 128;   // rows of a CTA, tokens of a page
// CG CTAs on one tile: with two, the accumulator's rows 0-127 are the even CTA's tensor memory and 128-255 the odd one's,
// A likewise, and each CTA's shared memory holds its half of B's columns (N) at the same offsets.
// A pair's are executed by a whole warp of the even CTA, one elected thread of which issues them: the warp stays converged, so
// that addresses and descriptors live in uniform registers, which is where the instruction wants them (issued from a branch
// of one thread, every MMA spent some 75 cycles moving its operands there).  A CTA on its own issues them from a branch of
// one thread all the same: it is bound by its shared-memory pipe, and the 18th warp's elections cost more than they save
// (nine row blocks of 32 query tokens, 8 KV heads, 1,024 pages of turbo3: 838 us with one thread in an earlier form of
// the kernel, 895 with elections, 851 with one thread now).
template <int CG> __device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
  if constexpr (CG == 1)
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
                 ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
  else
    asm volatile("{\n .reg .pred p, q;\n elect.sync _|q, 0xffffffff;\n setp.ne.b32 p, %4, 0;\n @q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
                 ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}
// arrival on `bar` of every CTA of the pair once the MMAs issued so far have completed
template <int CG> __device__ __forceinline__ void umma_commit(uint64_t* bar) {
  if constexpr (CG == 1)
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(sptr(bar)) : "memory");
  else
    asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n @q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n}\n"
                 ::"r"(sptr(bar)), "h"((uint16_t)3) : "memory");
}
// all 512 columns of tensor memory, by one warp of each CTA of the pair
template <int CG> __device__ __forceinline__ void tmem_alloc_all(uint32_t* where) {
  if constexpr (CG == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sptr(where)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  } else {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sptr(where)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
}
template <int CG> __device__ __forceinline__ void tmem_free_all(uint32_t base) {
  if constexpr (CG == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(512u) : "memory");
  else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(512u) : "memory");
}
// every thread of the CTA, or of both CTAs of the pair
template <int CG> __device__ __forceinline__ void pf_sync_all() {
  if constexpr (CG == 1) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  }
}
__device__ __forceinline__ float pf_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// two fp32 operations per instruction (sm_100 packed fp32), and the three-input maximum
__device__ __forceinline__ float2 pf_mul2(float2 a, float2 b) {
  float2 d;
  asm("{\n .reg .b64 ra, rb, rd;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %5};\n mul.rn.f32x2 rd, ra, rb;\n mov.b64 {%0, %1}, rd;\n}\n"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 pf_add2(float2 a, float2 b) {
  float2 d;
  asm("{\n .reg .b64 ra, rb, rd;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %5};\n add.rn.f32x2 rd, ra, rb;\n mov.b64 {%0, %1}, rd;\n}\n"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float pf_max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ uint32_t pf_pack(float lo, float hi) {
  __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t pf_lds(uint32_t addr) {
  uint32_t v;
  asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}

// 128-point sign * Walsh-Hadamard of a row, y = post (H/sqrt d) pre x, held by two threads, 64 elements each: thread `half` comes with
// elements 64 half ... 64 half + 63 and leaves with 32 half ... + 31 (x[0..31]) and 64 + 32 half ... + 31 (x[32..63]).  A 64-point transform
// in registers, then the last butterfly: each thread forms both results of half of the pairs and passes the other's 32 elements through `xs`
// ([element][row] floats, 32 KB of shared memory that nothing else uses meanwhile).  Called by all 256 row threads (named barrier 2).
constexpr int PF_HALF = TQ_D / 2;
__device__ __forceinline__ void rows_sync() { asm volatile("bar.sync 2, 256;" ::: "memory"); }
// element that x[j] of such a thread is, before (or without) a transform and after it
template <bool ROTATED> __device__ __forceinline__ int pf_dim(int half, int j) {
  return ROTATED ? 64 * (j >> 5) + 32 * half + (j & 31) : PF_HALF * half + j;
}
__device__ __forceinline__ void row_wht128_pair(float (&x)[PF_HALF], const uint32_t (&pre)[4], const uint32_t (&post)[4],
                                                int half, float* xs, int r) {
  const uint32_t pre0 = half ? pre[2] : pre[0], pre1 = half ? pre[3] : pre[1];
  const uint32_t post0 = half ? post[1] : post[0], post1 = half ? post[3] : post[2];
#pragma unroll
  for (int e = 0; e < PF_HALF; ++e) x[e] = (((e < 32 ? pre0 : pre1) >> (e & 31)) & 1u) ? -x[e] : x[e];
#pragma unroll
  for (int h = 1; h < PF_HALF; h <<= 1) {
#pragma unroll
    for (int i = 0; i < PF_HALF; ++i) {
      if ((i & h) == 0) {
        const float a = x[i], b = x[i + h];
        x[i] = a + b;
        x[i + h] = a - b;
      }
    }
  }
#pragma unroll
  for (int e = 0; e < 32; ++e) {
    xs[(32 * half + e) * PF_ROWS + r] = half ? x[e] : x[32 + e];
    x[e] = half ? x[32 + e] : x[e];
  }
  rows_sync();
#pragma unroll
  for (int e = 0; e < 32; ++e) {
    const float y = xs[(32 * (half ^ 1) + e) * PF_ROWS + r];   // thread 0 has the pair's first element, thread 1 its second
    const float s = x[e] + y, d = half ? y - x[e] : x[e] - y;
    x[e] = (((post0 >> e) & 1u) ? -s : s) * TQ_RSQRT_D;
    x[32 + e] = (((post1 >> e) & 1u) ? -d : d) * TQ_RSQRT_D;
  }
}

struct PrefillParams {
  const uint8_t* pool;
  const int32_t* block_table;
  const int32_t* kv_lens;   // cached tokens per sequence, the chunk's own tokens included
  const void* q;            // [B][Tq][Hq][128]
  void* out;                // same shape
  const float* k_s_t;       // dense sketch matrix transposed (PROD keys of a dense quantizer), or nullptr
  const float* k_rot_t;     // dense K rotation transposed (R x)_j = sum_k rot_t[k][j] x_k, or nullptr
  const float* v_rot;       // dense V rotation row-major (R^T y)_j = sum_k rot[k][j] y_k, or nullptr
  int32_t* status;
  float qscale;             // softmax scale * log2(e)
  int32_t q_dtype, out_dtype;
  int32_t max_pages, batch, tq, hq, hkv, group;
  // split of the page range over several CTAs (flash-decoding style), merged by the last CTA to finish
  float* part_o;            // [slot][16 four-element groups][2 halves][128 rows][4]
  float* part_ml;           // [slot][128 rows][2]
  int32_t* tickets;         // [(b * hkv + kvh) * row_blocks + rb], zero between calls
  int32_t chunk_pages, num_splits, row_blocks;
  tq_cache_layout L;
};

// KK / VK: 2,3,4 = turbo bits; 8 = q8_0; 18,19,20 = PROD with 1,2,3 PolarQuant bits + sign sketch (keys only).
template <int KIND> struct PfKind {
  static constexpr bool Q8 = KIND == 8, PROD = KIND >= 18;
  static constexpr int BITS = Q8 ? 0 : (PROD ? KIND - 17 : KIND);
  // K operand tiles of a page.  turbo: centroids (the row scale is applied to the scores in fp32).  q8_0: int8 x block
  // scale is 19 bits, so its fp16 rounding and the rest, exactly; of a token with a block scale of 512 or more, whose
  // products may exceed the fp16 range, divided by 128, which the scores get back in fp32 (what falls below fp16's
  // smallest number then is under 2^-32 of the token's largest element).  PROD: centroids, then +-ratio for the sketch, ratio =
  // residual scale / row scale (one row scale then serves both parts), as its fp16 rounding and the rest of it.
  static constexpr int TILES = PROD ? 3 : (Q8 ? 2 : 1);
  // PROD queries (rotated and projected, hi and lo) take 256 tensor-memory columns: one score buffer instead of two
  static constexpr int SBUF = PROD ? 1 : 2;
};

// Pair tables, replicated per lane (a lookup then hits the lane's own bank) up to 8 KB; the 256 pairs of a 4-bit codebook
// only where 32 KB are to be had (REPL4: with one copy a lookup takes 3.4 wavefronts on average).  Tables up to 8 KB start on
// a multiple of their size, the address of an entry is (field | base); the 32 KB one's start is added.
template <int BITS, bool REPL4> struct PfLut {
  static constexpr int ENTRIES = BITS ? 1 << (2 * BITS) : 0;
  static constexpr bool BIG = BITS == 4 && REPL4;
  static constexpr bool REPL = BIG || ENTRIES <= 64;
  static constexpr int SHIFT = REPL ? 7 : 2;
  static constexpr int BYTES = ENTRIES << SHIFT;
  static __device__ __forceinline__ uint32_t load(uint32_t field, uint32_t base, uint32_t start) {
    return pf_lds(BIG ? (field | base) + start : field | base);
  }
  static __device__ __forceinline__ uint32_t base(uint32_t start, int lane) { return (BIG ? 0u : start) + (REPL ? lane * 4 : 0); }
  static __device__ __forceinline__ void fill(uint8_t* lut, const uint16_t* c16, int tid, int threads) {
    if constexpr (BITS > 0)
      for (int i = tid; i < BYTES / 16; i += threads) {
        uint32_t v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int e = REPL ? i >> 3 : 4 * i + k;
          v[k] = (uint32_t)c16[e >> BITS] | ((uint32_t)c16[e & ((1 << BITS) - 1)] << 16);
        }
        reinterpret_cast<uint4*>(lut)[i] = make_uint4(v[0], v[1], v[2], v[3]);
      }
  }
};

// DIMS of one token's packed indices (DIMS * BITS / 8 bytes at `src`) -> fp16 values written as 16-byte rows of the operand
// tile: chunk c (8 dims) goes to dst + c*128.  SCALED: every pair is multiplied by `scale2` (one fp16 factor in both halves).
template <int BITS, class LUT, int DIMS, bool SCALED = false>
__device__ __forceinline__ void pf_dequant_token(const uint8_t* src, uint8_t* dst, uint32_t lut_base, uint32_t lut_start,
                                                 uint32_t scale2 = 0) {
  constexpr int SH = LUT::SHIFT;
  constexpr uint32_t MASK = ((1u << (2 * BITS)) - 1) << SH;
  constexpr int NW = DIMS * BITS / 32;  // 32-bit words
  uint32_t w[NW];
  if constexpr (DIMS == 128) {
#pragma unroll
    for (int i = 0; i < BITS; ++i) {
      const uint4 v = reinterpret_cast<const uint4*>(src)[i];
      w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < BITS; ++i) {
      const uint2 v = reinterpret_cast<const uint2*>(src)[i];
      w[2 * i] = v.x; w[2 * i + 1] = v.y;
    }
  }
#pragma unroll
  for (int i = 0; i < NW; ++i) w[i] = __byte_perm(w[i], 0, 0x0123);
#pragma unroll
  for (int c = 0; c < DIMS / 8; ++c) {
    uint32_t o4[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int start = (4 * c + p) * 2 * BITS, k = start >> 5, o = start & 31;
      uint32_t f;
      if (o + 2 * BITS <= 32) {
        const int sr = 32 - 2 * BITS - o;
        f = sr > SH ? (w[k] >> (sr - SH)) : (sr < SH ? (w[k] << (SH - sr)) : w[k]);
      } else {
        f = __funnelshift_l(w[k + 1 < NW ? k + 1 : k], w[k], o) >> (32 - 2 * BITS - SH);
      }
      o4[p] = LUT::load(f & MASK, lut_base, lut_start);
      if constexpr (SCALED) asm("mul.f16x2 %0, %0, %1;" : "+r"(o4[p]) : "r"(scale2));
    }
    *reinterpret_cast<uint4*>(dst + c * 128) = make_uint4(o4[0], o4[1], o4[2], o4[3]);
  }
}

// q8_0 keys: whether one of a token's four block scales (fp16, not negative) is 512 or more, i.e. has its two upper exponent
// bits set.  Below, every product int8 x scale is at most 127 x 511.75 = 64,992, above, 127 x 65,504 / 128 = 64,992.
__device__ __forceinline__ bool pf_q8_big(uint2 sc) {
  return (((sc.x & (sc.x << 1)) | (sc.y & (sc.y << 1))) & 0x40004000u) != 0;
}
__device__ __forceinline__ uint32_t pf_div128(uint32_t h2) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(h2), "r"(0x20002000u));
  return d;
}

__device__ __forceinline__ uint32_t pf_s8x2(uint32_t biased, uint32_t sel) {
  // two int8 values, stored as value ^ 0x80 = value + 128, as exact fp16: (b | 0x6400) is 1024 + b; subtract 1152
  uint32_t d;
  asm("sub.f16x2 %0, %1, %2;" : "=r"(d) : "r"(__byte_perm(biased, 0x64646464u, sel)), "r"(0x64806480u));
  return d;
}

// One token's DIMS int8 values at `src` with their block scales (sc01, sc23: two fp16 each) -> fp16 products in the
// operand tile at `dst`, and, SPLIT, what the fp16 rounding left of them (exact: 8 x 11 bits) in the tile at dst + TILE.
// Rows are 128 bytes apart, so a lane starts at a chunk of its own: the lanes of a load then touch every bank.
template <bool SPLIT, int DIMS, int TILE>
__device__ __forceinline__ void pf_q8_token(const uint8_t* src, uint8_t* dst, uint32_t sc01, uint32_t sc23, int lane) {
#pragma unroll
  for (int i = 0; i < DIMS / 16; ++i) {
    const int c = (i + lane) & (DIMS / 16 - 1);   // 16 values: dims 16 c .. 16 c + 15, half of block c >> 1
    const uint4 v = *reinterpret_cast<const uint4*>(src + 16 * c);
    const uint32_t w[4] = {v.x ^ 0x80808080u, v.y ^ 0x80808080u, v.z ^ 0x80808080u, v.w ^ 0x80808080u};
    const uint32_t s2 = __byte_perm(c & 4 ? sc23 : sc01, 0, c & 2 ? 0x3232 : 0x1010);
    uint32_t hi[8], lo[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t x = pf_s8x2(w[j >> 1], (j & 1) ? 0x4342 : 0x4140);
      asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(hi[j]) : "r"(x), "r"(s2));
      if constexpr (SPLIT) asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(lo[j]) : "r"(x), "r"(s2), "r"(hi[j] ^ 0x80008000u));
    }
    uint8_t* d = dst + c * 256;
    *reinterpret_cast<uint4*>(d) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(d + 128) = make_uint4(hi[4], hi[5], hi[6], hi[7]);
    if constexpr (SPLIT) {
      *reinterpret_cast<uint4*>(d + TILE) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      *reinterpret_cast<uint4*>(d + TILE + 128) = make_uint4(lo[4], lo[5], lo[6], lo[7]);
    }
  }
}

// One token's sign sketch, DIMS bits (first dim in the most significant bit, set = +1) -> +-ratio in the tile at `dst`, as
// the fp16 rounding of the ratio there and the rest of it in the tile behind.
template <int DIMS, int TILE>
__device__ __forceinline__ void pf_sketch_token(const uint8_t* src, uint8_t* dst, float ratio) {
  const __half h = __float2half_rn(ratio);
  const __half2 h2 = __half2half2(h), e2 = __float2half2_rn(ratio - __half2float(h));
  const uint32_t hw = *reinterpret_cast<const uint32_t*>(&h2), ew = *reinterpret_cast<const uint32_t*>(&e2);
  uint32_t zw[DIMS / 32];
#pragma unroll
  for (int k = 0; k < DIMS / 64; ++k) {
    const uint2 v = reinterpret_cast<const uint2*>(src)[k];
    zw[2 * k] = v.x;
    zw[2 * k + 1] = v.y;
  }
#pragma unroll
  for (int k = 0; k < DIMS / 32; ++k) {
    const uint32_t n = ~__byte_perm(zw[k], 0, 0x0123);   // set = negative; dim 32 k + i in bit 31 - i
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t m[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) {   // dims 2 j, 2 j + 1 of the word: bits 31 - 2 j and 30 - 2 j -> the two sign positions
        const int j = 4 * c + p;
        const uint32_t lo = j < 8 ? n >> (16 - 2 * j) : n << (2 * j - 16);
        m[p] = (lo & 0x8000u) | ((n << (2 * j + 1)) & 0x80000000u);
      }
      uint8_t* d = dst + (4 * k + c) * 128;
      *reinterpret_cast<uint4*>(d) = make_uint4(hw ^ m[0], hw ^ m[1], hw ^ m[2], hw ^ m[3]);
      *reinterpret_cast<uint4*>(d + TILE) = make_uint4(ew ^ m[0], ew ^ m[1], ew ^ m[2], ew ^ m[3]);
    }
  }
}

// ------------------------------------------------------------------------------------------
// k_prefill_attn2: the work split over specialised warps, one CTA per SM.
//
// Two CTAs of a cluster take two neighbouring row blocks over one range of pages (CG = 2): tcgen05.mma.cta_group::2 multiplies
// both blocks with one operand tile of which each CTA holds half, so that each dequantizes half of every page.  Alone (CG =
// 1: a single row block, PROD keys) a CTA dequantizes the whole page, and the shared-memory pipe -- tiles written, read by
// the tensor core, table lookups -- is busy 92 % of a page's ~3,000 cycles.  In a pair it is half as busy, and a page takes
// ~2,500 cycles: the row warps' softmax (2,250: 16 KB of scores read, maxima exchanged, 64 exponentials per thread) and the
// MMAs (1,536 at the tensor core's rate, ~2,100 as issued) are the two limits.  Measured per page and CTA: turbo3 / turbo3
// 1.64 -> 1.37 us, turbo4 / turbo3 2.1 -> 1.4 (with lane-replicated 4-bit tables, for which a pair has room), turbo4 /
// turbo4 2.5 -> 1.4, q8_0 / turbo2 2.1 -> 1.7.
//   warps 0-7  rows: two threads per row r = lane r of tensor memory (warps w and w + 4 reach the same 32 lanes), one
//              per half of a page's 128 score columns: reads S, online softmax (the halves exchange their maxima
//              through shared memory), writes P, rescales its half of O (lazily: only when the row maximum grows by
//              more than 2^4); both threads share the query rotation, the split partial, the merge and the output
//              (64 elements each; query and output rows pass through shared memory and the partials are laid out
//              by warp, so that every global access of a warp covers whole lines);
//   PW warps   K producers: a thread dequantizes the K row of one token of the page into a double-buffered operand tile;
//              they wait for the score MMA of page i - 2 only, one page ahead of
//   PW warps   V producers: V rows times the V scale; their tile is free after the product of page i - 2;
//   one warp   issues every tcgen05.mma (the even CTA's, for both): S_{i+1} = Q K_{i+1}^T is queued before O += P_i V_i, so
//              that the tensor core works on the next page while the row warps are in the softmax of this one;
//   one warp   issues the bulk copies of the page records.
// Tensor memory, all 512 columns: Q hi 0-63 | Q lo 64-127 | S0 128-255 | S1 256-383 | O 384-511 (fp32, accumulated
// by the MMAs across pages); PROD keys: the projected queries' hi and lo in 128-255 and one score buffer in 256-383.
// P overlays the first 64 columns of its S buffer.
// q8_0 and PROD keys have two and three K tiles per page (PfKind) and sum 3 and 5 products into S: their queries' chunk runs
// here instead of one decode call per query, which read and dequantized the cache once per query (2 x 128 queries x 32
// heads over 8,192 tokens of q8_0 / turbo2: 650 us).
// Hand-offs are mbarriers (counts in brackets, times the CTAs of a pair where they count for both): k_ready/v_ready [PW
// producer warps], s_full/o_done [tcgen05.commit, to both CTAs], p_ready [8 row warps], rec_free [2 PW producer warps];
// buffer b of page i completes each of the first five for the (i >> 1)-th time, which fixes the parity to wait for.  No
// generic-proxy data crosses the CTAs (scales, maxima and records are each CTA's own), so arrivals at the other CTA carry
// no cluster-wide fence: with acquire and release at cluster scope a page took 0.4 us longer.  Every wait is bounded; a
// role that gives up raises the CTA's fail flag, the others see it or run out of time themselves, and the tensor memory
// is released on every path.
// Tried without gain: probabilities formed ahead of the exchanged maximum; a part of the exponentials as polynomials on the
// fp32 pipe (one pair in two to one in six).
// ------------------------------------------------------------------------------------------
constexpr float PF2_SLACK = 4.0f;

// CG: CTAs per operand tile (1, or a pair of 2)
template <int KK, int VK, int CG> struct PfSmem2 {
  using KT = PfKind<KK>;
  using VT = PfKind<VK>;
  // Producer warps of K and of V.  A pair's CTA dequantizes half as much and gets by with two each: 14 warps then, at most
  // four per scheduler, which leaves the row warps 128 registers (96 with 17 to 20 warps).
  static constexpr int PW = CG == 2 ? 2 : 4;
  static constexpr int K_AT = 256, V_AT = K_AT + 32 * PW, MMA_AT = V_AT + 32 * PW, COPIER = MMA_AT + 32, THREADS = COPIER + 32;
  static constexpr bool REPL4 = CG == 2;
  using KLut = PfLut<KT::BITS, REPL4>;
  using VLut = PfLut<VT::BITS, REPL4>;
  static constexpr int TILE = 32768 / CG;               // one operand tile: this CTA's half of it in a pair
  static constexpr int KBUF = CG == 2 || KT::TILES == 1 ? 2 : 1;   // buffers of K tiles
  static constexpr int REC = 128 * ((KT::Q8 ? 136 : 16 * KT::BITS + 4) + (KT::PROD ? 20 : 0) + (VT::Q8 ? 136 : 16 * VT::BITS + 4));
  static constexpr int ALIGN = 8192;                    // each table starts on a multiple of its size (or of 8 KB)
  static constexpr int OFF_K = 0;
  static constexpr int OFF_V = KLut::BYTES > 8192 ? KLut::BYTES : 8192;
  static constexpr int OFF_BAR = OFF_V + (VLut::BYTES > 8192 ? VLut::BYTES : 8192);   // mbarriers, tensor-memory base, fail flag
  static constexpr int OFF_SC = OFF_BAR + 256;          // float K scales[4 slots][128 tokens], then the row halves'
                                                        // exchange area float[2 buffers][2 halves][128 rows], then
                                                        // their parts of the row sum float[2 halves][128 rows]
  static constexpr int OFF_KT = OFF_SC + 5120;          // K operand tiles (the first 64 KB from here also stage the output rows)
  static constexpr int OFF_VT = OFF_KT + KBUF * KT::TILES * TILE;   // V operand tiles, two
  static constexpr int OFF_ST = OFF_VT + 2 * TILE;      // page records in flight: as many as fit, at most four
  static constexpr int LIMIT = 227 * 1024;
  static constexpr int NST_FIT = (LIMIT - ALIGN - OFF_ST) / REC;
  static constexpr int NST = CG == 1 ? 2 : NST_FIT > 4 ? 4 : NST_FIT;
  static constexpr int BYTES = ALIGN + OFF_ST + NST * REC;
  static_assert(NST >= 2 && BYTES <= LIMIT && OFF_ST - OFF_KT >= 65536, "shared memory of the prefill kernel");
};

// One arrival for a whole warp: its lanes' earlier accesses are ordered in front of it by the warp barrier.  (An arrival
// per thread is an operation of the shared-memory pipe per thread, 768 per page.)
__device__ __forceinline__ void pf_arrive_warp(uint64_t* bar, int lane) {
  __syncwarp();
  if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sptr(bar)) : "memory");
}
// ... on the barrier of the CTA that issues the MMAs: the even one of a pair
template <int CG> __device__ __forceinline__ void pf_arrive_leader(uint64_t* bar, int lane) {
  if constexpr (CG == 1) {
    pf_arrive_warp(bar, lane);
  } else {
    __syncwarp();
    if (lane == 0) {
      uint32_t addr;
      asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(addr) : "r"(sptr(bar)));
      asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
    }
  }
}
// bounded wait whose verdict is the same in every lane of the warp (warp-collective tcgen05 instructions follow)
__device__ __forceinline__ bool pf_wait_warp(uint64_t* bar, uint32_t parity) {
  return __all_sync(0xffffffffu, tc_wait(bar, parity));
}
template <int KK, int VK, int CG>
__global__ void __launch_bounds__(PfSmem2<KK, VK, CG>::THREADS, 1) k_prefill_attn2(const __grid_constant__ PrefillParams P,
                                                                  const __grid_constant__ TqFast fk, const __grid_constant__ TqFast fv) {
  using SP = PfSmem2<KK, VK, CG>;
  using KT = PfKind<KK>;
  using VT = PfKind<VK>;
  constexpr int KB = KT::BITS, VB = VT::BITS, NST = SP::NST;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t raw = sptr(smem_raw);
  uint8_t* sm = smem_raw + (((raw + SP::ALIGN - 1) & ~(uint32_t)(SP::ALIGN - 1)) - raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + SP::OFF_BAR);
  // (k_ready, v_ready, p_ready and q_ready count in the even CTA of a pair)
  uint64_t *rec_full = bars, *rec_free = bars + 4, *k_ready = bars + 8, *v_ready = bars + 10, *s_full = bars + 12,
           *p_ready = bars + 14, *o_done = bars + 16, *q_ready = bars + 18;
  uint64_t* xbar = bars + 19;   // one per row quarter: both halves' maxima of a page are in shared memory [2 warps]
  uint32_t* tbase = reinterpret_cast<uint32_t*>(sm + SP::OFF_BAR + 224);
  volatile int* fail = reinterpret_cast<volatile int*>(sm + SP::OFF_BAR + 232);
  uint32_t* q8_big = reinterpret_cast<uint32_t*>(sm + SP::OFF_BAR + 236);   // [4 slots], a byte per K producer warp: its tokens
                                                                            // have factors (see PfKind) in `scales`
  if (tid == SP::COPIER) {   // lane 0 of the last warp issues the record copies
    auto init = [](uint64_t* bar, int count) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sptr(bar)), "r"(count) : "memory");
    };
    for (int i = 0; i < NST; ++i) {
      init(&rec_full[i], 1);
      init(&rec_free[i], 2 * SP::PW);
    }
    for (int i = 0; i < 2; ++i) {
      init(&k_ready[i], SP::PW * CG);
      init(&v_ready[i], SP::PW * CG);
      init(&p_ready[i], 8 * CG);
      init(&s_full[i], 1);
      init(&o_done[i], 1);
    }
    for (int i = 0; i < 4; ++i) init(&xbar[i], 2);
    init(q_ready, 8 * CG);
    *fail = 0;
    for (int i = 0; i < 4; ++i) q8_big[i] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  TQ_PDL_ENTER();   // so far only the parameters have been read

  // Row blocks from the last to the first: the later ones of a causal chunk see more pages, and what is left when the SMs
  // run dry should be short.  A pair's CTAs take two neighbouring blocks over one range of pages.
  const int unit = blockIdx.x / CG, per = P.batch * P.hkv * P.num_splits, crank = CG == 2 ? (int)(blockIdx.x & 1) : 0;
  const int rbp = (P.row_blocks + CG - 1) / CG - 1 - unit / per, item = unit % per;
  const int split = item % P.num_splits, kvh = item / P.num_splits % P.hkv, b = item / (P.num_splits * P.hkv);
  const int rb = rbp * CG + crank;
  const int PT = P.L.page_tokens;  // 128 (checked on the host)
  const int kv_len = P.kv_lens[b];
  const int nrows = P.tq * P.group;
  const int rtid = tid & 127;                        // row of a row thread
  const int row = rb * PF_ROWS + rtid;
  const bool is_row = tid < SP::K_AT;
  const bool is_prim = tid < 128;
  const int hf = (tid >> 7) & 1;                     // row threads: half of a page's columns
  const bool row_ok = is_row && row < nrows;
  const int qi = row_ok ? row / P.group : 0;
  const int pos = row_ok ? kv_len - P.tq + qi : -1;
  const int last_row = min(nrows, (rbp + 1) * CG * PF_ROWS) - 1;
  const int pos_max = kv_len - P.tq + last_row / P.group;
  const int np_all = min(P.max_pages, pos_max >= 0 ? pos_max / PT + 1 : 0);
  const int ns = np_all > 0 ? (np_all + P.chunk_pages - 1) / P.chunk_pages : 1;
  if (split >= ns) return;                           // nothing to do (for both CTAs of a pair), and no tensor memory taken yet
  const int page_lo = split * P.chunk_pages;
  const int np = max(0, min(np_all, page_lo + P.chunk_pages) - page_lo);
  float* scales = reinterpret_cast<float*>(sm + SP::OFF_SC);
  uint8_t* ktile = sm + SP::OFF_KT;
  uint8_t* vtile = sm + SP::OFF_VT;
  uint8_t* stage0 = sm + SP::OFF_ST;
  if (warp == SP::K_AT / 32) tmem_alloc_all<CG>(tbase);   // all 512 columns of the SM (one CTA per SM)

  auto issue = [&](int i) {
    const int64_t page = P.block_table[(size_t)b * P.max_pages + page_lo + i];
    const uint8_t* src = P.pool + page * P.L.page_stride + (int64_t)kvh * P.L.head_stride;
    const int st = i % NST;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sptr(&rec_full[st])), "r"(SP::REC) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     sptr(stage0 + st * SP::REC)), "l"(src), "r"(SP::REC), "r"(sptr(&rec_full[st])) : "memory");
  };
  if (tid == SP::COPIER)
    for (int i = 0; i < NST && i < np; ++i) issue(i);

  // ---- prologue (row warps): this row's query, rotated by the K rotation (q8_0 keys: as it is), scaled, fp16 hi + lo
  // into tensor memory; PROD keys: its projection by the sketch's transform as well.  Each of the row's two threads holds
  // one half of its elements ----
  float o[PF_HALF];
  const uint32_t TQc = 0, TQLc = 64, TPc = 128, TPLc = 192, TOc = 384;
  // score buffer of page i; P overlays its first 64 columns
  auto s_col = [](int bf) { return KT::SBUF == 2 ? 128u + 128u * bf : 256u; };
  const int q_esz = P.q_dtype == TQ_F32 ? 4 : 2;
  // The rows' staging and exchange area ends where the records begin: 64 KB, or 32 in a pair whose 16-bit queries are rotated by
  // transforms.  So the first page's K tile is another memory, and its producers fill their tables and dequantize it while the rows are
  // rotated (7,000 clocks); one before and one behind them, the two were another 4,000.  With the append, 32 / 8 heads: a prompt of 3,999
  // tokens, turbo4 / turbo3, 273 -> 268 us, the last 128 of 8,192 positions of two sequences, q8_0 / turbo2, 82 -> 78 (64 / 8 heads, the
  // last 128 of 131,072: 1 to 2 % of some 830 with the copies below, no more than its runs differ by).  A pair's `wide` rows need that tile too.
  const bool wide = CG == 2 && !KT::Q8 && (q_esz == 4 || P.k_rot_t != nullptr);
  uint8_t* const rows_at = sm + SP::OFF_ST - (CG == 2 && !KT::Q8 && !wide ? 32768 : 65536);
  // Rows pass through shared memory: accessed directly, a thread's own half row would put the lanes of a load 256 or 512
  // bytes apart (one line per lane and instruction); staged, a warp moves whole rows.  16-byte chunk w of row r sits at
  // chunk w ^ (r & 7) of its row, so that the accesses of consecutive rows fall into different banks.
  auto chunk_at = [](uint8_t* area, int r, int w, int esz) { return area + r * (TQ_D * esz) + ((w ^ (r & 7)) << 4); };
  // Row threads, between q or out and the staged rows: move(chunk in shared memory, whether the chunk of rows has this row, byte offset in
  // q or out) for each 16-byte chunk that this thread moves.  A row's number is divided by the group with a shift where that is a power of
  // two, and the queries come by asynchronous copies: divided out for every chunk and loaded through registers, they took 8,000 clocks of a
  // CTA's 28,000 beside its pages (with the append, 32 / 8 heads: a prompt of 3,999 tokens, turbo4 / turbo3, 306 -> 273 us; the last 128 of
  // 8,192 positions of two sequences, q8_0 / turbo2, 90 -> 82).
  const int group_log = (P.group & (P.group - 1)) == 0 ? 31 - __clz(P.group) : -1;
  auto move_rows = [&](uint8_t* area, int esz, auto&& move) {
    const int per_log = esz == 4 ? 5 : 4, w = tid & ((1 << per_log) - 1);
    const size_t first = (size_t)b * P.tq * P.hq + (size_t)kvh * P.group;
#pragma unroll 4
    for (int it = 0; it < (1 << (per_log - 1)); ++it) {
      const int r = (it * 256 + tid) >> per_log, grow = rb * PF_ROWS + r;
      const int gq = group_log >= 0 ? grow >> group_log : grow / P.group, gh = grow - gq * P.group;
      move(chunk_at(area, r, w, esz), grow < nrows, (first + (size_t)gq * P.hq + gh) * (TQ_D * esz) + w * 16);
    }
  };
  auto stage_rows = [&]() {
    move_rows(rows_at, q_esz, [&](uint8_t* to, bool there, size_t off) {   // (rows past the chunk come as zeros)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sptr(to)), "l"(reinterpret_cast<const uint8_t*>(P.q) + (there ? off : 0)),
                   "r"(there ? 16 : 0) : "memory");
    });
  };
  auto rows_staged = [&]() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    rows_sync();
  };
  auto read_row = [&]() {
    if (P.q_dtype == TQ_F32) {
#pragma unroll
      for (int e = 0; e < PF_HALF; e += 4) {
        const float4 v = *reinterpret_cast<const float4*>(chunk_at(rows_at, rtid, (PF_HALF * hf + e) / 4, 4));
        o[e] = v.x; o[e + 1] = v.y; o[e + 2] = v.z; o[e + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int e = 0; e < PF_HALF; e += 8) {
        const uint4 w4 = *reinterpret_cast<const uint4*>(chunk_at(rows_at, rtid, (PF_HALF * hf + e) / 8, 2));
        const uint32_t ww[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 f = P.q_dtype == TQ_F16 ? __half22float2(*reinterpret_cast<const __half2*>(&ww[k]))
                                               : __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ww[k]));
          o[e + 2 * k] = f.x; o[e + 2 * k + 1] = f.y;
        }
      }
    }
  };
  auto rotate = [&](const float* dense_t, const uint32_t (&pre)[4], const uint32_t (&post)[4]) {
    float* xs = reinterpret_cast<float*>(rows_at);
    if (dense_t) {
      // dense rotation: the rows staged transposed ([k][row], 64 KB), then this thread's 64 elements of y = R x
#pragma unroll
      for (int k = 0; k < PF_HALF; ++k) xs[(PF_HALF * hf + k) * PF_ROWS + rtid] = o[k];
      rows_sync();
#pragma unroll
      for (int j = 0; j < PF_HALF; ++j) o[j] = 0.f;
      for (int k = 0; k < TQ_D; ++k) {
        const float xv = xs[k * PF_ROWS + rtid];
        const float4* rr = reinterpret_cast<const float4*>(dense_t + (size_t)k * TQ_D + 32 * hf);
#pragma unroll
        for (int j = 0; j < PF_HALF; j += 4) {
          const float4 r4 = __ldg(rr + pf_dim<true>(0, j) / 4);
          o[j] = fmaf(r4.x, xv, o[j]); o[j + 1] = fmaf(r4.y, xv, o[j + 1]);
          o[j + 2] = fmaf(r4.z, xv, o[j + 2]); o[j + 3] = fmaf(r4.w, xv, o[j + 3]);
        }
      }
    } else {
      row_wht128_pair(o, pre, post, hf, xs, rtid);
    }
  };
  auto to_tmem = [&](uint32_t tmem, float sk, uint32_t hi_col, uint32_t lo_col) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint32_t u[16], ul[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float a = o[32 * c + 2 * j] * sk, bq = o[32 * c + 2 * j + 1] * sk;
        const __half2 h = __floats2half2_rn(a, bq);
        const float2 hv = __half22float2(h);
        u[j] = *reinterpret_cast<const uint32_t*>(&h);
        ul[j] = pf_pack(a - hv.x, bq - hv.y);
      }
      tmem_st16(tmem + hi_col + pf_dim<!KT::Q8>(hf, 32 * c) / 2, u);
      tmem_st16(tmem + lo_col + pf_dim<!KT::Q8>(hf, 32 * c) / 2, ul);
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  };
  if (is_row) stage_rows();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  pf_sync_all<CG>();  // tensor-memory base and barriers visible
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tb = *tbase;
  // rows done with their area (named barriers 3 and 4, at which the V and a pair's K producers wait before they write there)
  constexpr int FREE_V = 256 + 32 * SP::PW, FREE_K = 256 + 32 * SP::PW;

  if (is_row) {
    // =========================== row warps ===========================
    const uint32_t tm = tb + ((uint32_t)((warp & 3) * 32) << 16);  // this warp's 32 lanes
    float* xch = scales + 512;                                     // [buffer][half][row]
    rows_staged();
    read_row();
    if constexpr (!KT::Q8) {
      rows_sync();                          // the staged rows are read: the rotation's exchange area is the same memory
      rotate(P.k_rot_t, fk.s1, fk.s2);
    }
    if constexpr (KT::PROD) {   // both transforms of a row share registers and staging: the first goes to tensor memory first
      to_tmem(tm, P.qscale / fk.lut_alpha, TQc, TQLc);
      rows_sync();                          // the exchange area has been read
      stage_rows();
      rows_staged();
      read_row();
      rows_sync();
      rotate(P.k_s_t, fk.j1, fk.j2);
    }
    asm volatile("bar.arrive 3, %0;" ::"n"(FREE_V) : "memory");
    if constexpr (CG == 2) asm volatile("bar.arrive 4, %0;" ::"n"(FREE_K) : "memory");
    if constexpr (KT::PROD) to_tmem(tm, P.qscale, TPc, TPLc);
    else to_tmem(tm, P.qscale / fk.lut_alpha, TQc, TQLc);
    pf_arrive_leader<CG>(q_ready, lane);             // the queries are in tensor memory

    float m_run = -INFINITY, l_run = 0.f;   // l_run: this half's part of the row sum
    for (int i = 0; i < np; ++i) {
      if (__any_sync(0xffffffffu, *fail != 0)) break;
      const int bf = i & 1;
      const uint32_t ph = (uint32_t)((i >> 1) & 1);
      if (!pf_wait_warp(&s_full[bf], ph)) { *fail = 1; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float4* ksc4 = reinterpret_cast<const float4*>(scales + (i & 3) * PF_ROWS + 64 * hf);
      const uint32_t ts = tm + s_col(bf);
      const int t0 = (page_lo + i) * PT;
      // a page that every row of this warp sees completely needs no causal mask (rows without a query count as
      // seeing everything: nothing of theirs is stored)
      // (q8_0: neither does one without factors, which nearly all are: both are the business of the other copy of pass 1)
      uint32_t big = 0;
      if constexpr (KT::Q8) big = *reinterpret_cast<volatile uint32_t*>(q8_big + (i & 3));
      const bool masked = !__all_sync(0xffffffffu, !row_ok || t0 + PT - 1 <= pos) || big != 0;
      // pass 1: this half's scaled scores into registers, row maximum
      float sv[64];
      float mx = -INFINITY;
      uint32_t raw[64];   // the four loads fly together; each score replaces its raw value (same registers)
      tmem_ld16_nowait<0>(ts + 64 * hf, raw);
      tmem_ld16_nowait<16>(ts + 64 * hf + 16, raw);
      tmem_ld16_nowait<32>(ts + 64 * hf + 32, raw);
      tmem_ld16_nowait<48>(ts + 64 * hf + 48, raw);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      auto pass1 = [&](auto masked_c) {   // two copies behind a warp-uniform branch: only the diagonal pages pay for the mask
        constexpr bool MASKED = decltype(masked_c)::value;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint32_t* v = raw + 16 * c;
#pragma unroll
          for (int j = 0; j < 16; j += 4) {
            float2 x01 = make_float2(__uint_as_float(v[j]), __uint_as_float(v[j + 1]));
            float2 x23 = make_float2(__uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
            if constexpr (!KT::Q8) {   // (q8_0 operands carry their block scales)
              const float4 k4 = ksc4[4 * c + (j >> 2)];
              x01 = pf_mul2(x01, make_float2(k4.x, k4.y));
              x23 = pf_mul2(x23, make_float2(k4.z, k4.w));
            } else if (MASKED) {   // (columns 32 c .. + 31 are producer warp c's, of a pair's two warps c & 1)
              if ((big >> (8 * ((2 * hf + (c >> 1)) & (SP::PW - 1)))) & 1u) {
                const float4 k4 = ksc4[4 * c + (j >> 2)];
                x01 = pf_mul2(x01, make_float2(k4.x, k4.y));
                x23 = pf_mul2(x23, make_float2(k4.z, k4.w));
              }
            }
            if (MASKED) {
              const int tt = t0 + 64 * hf + 16 * c + j;
              x01.x = tt <= pos ? x01.x : -INFINITY;
              x01.y = tt + 1 <= pos ? x01.y : -INFINITY;
              x23.x = tt + 2 <= pos ? x23.x : -INFINITY;
              x23.y = tt + 3 <= pos ? x23.y : -INFINITY;
            }
            sv[16 * c + j] = x01.x; sv[16 * c + j + 1] = x01.y;
            sv[16 * c + j + 2] = x23.x; sv[16 * c + j + 3] = x23.y;
            mx = pf_max3(mx, x01.x, x01.y);
            mx = pf_max3(mx, x23.x, x23.y);
          }
        }
      };
      if (masked) pass1(std::true_type{}); else pass1(std::false_type{});
      // the other half's maximum: both threads of a row then take the same decisions below.  (The arrival also tells
      // the other half that this one has read its scores: the P columns that half writes overlay them.)
      xch[(bf * 2 + hf) * PF_ROWS + rtid] = mx;
      pf_arrive_warp(&xbar[warp & 3], lane);
      if (!pf_wait_warp(&xbar[warp & 3], (uint32_t)(i & 1))) { *fail = 1; break; }
      mx = fmaxf(mx, xch[(bf * 2 + (hf ^ 1)) * PF_ROWS + rtid]);
      // The row maximum moves only when it grows by more than 2^PF2_SLACK (probabilities stay below 2^PF2_SLACK).
      // O lives in tensor memory and is being accumulated by the MMAs: a rescale waits for the product of the
      // page before, multiplies the row in place, and only then lets this page's product start (p_ready below).
      float resc = 1.0f;
      if (i == 0) {
        // the reference starts PF2_SLACK above the first page's maximum: a later page then moves it only when it
        // beats that maximum by 2^(2 PF2_SLACK), which is rare -- and every move stalls the row on the tensor core
        m_run = mx + PF2_SLACK;
      } else if (mx > m_run + PF2_SLACK) {
        resc = pf_exp2(m_run - mx);   // m_run == -inf (nothing seen yet) gives 0: the row of O is zero anyway
        m_run = mx;
        l_run *= resc;
      }
      if (i > 0 && __any_sync(0xffffffffu, resc != 1.0f)) {
        if (!pf_wait_warp(&o_done[(i - 1) & 1], (uint32_t)(((i - 1) >> 1) & 1))) { *fail = 1; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {   // this half's 64 columns of O
          uint32_t v[32];
          tmem_ld32(tm + TOc + 64 * hf + 32 * c, v);
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * resc);
          tmem_st32(tm + TOc + 64 * hf + 32 * c, v);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      }
      // pass 2: probabilities (masked scores are -inf and give 0), row sum, P as packed fp16 (the V scales are in the
      // V operand tile)
      const float m_use = m_run == -INFINITY ? 0.f : m_run;
      const float2 nm2 = make_float2(-m_use, -m_use);
      float2 ls2 = make_float2(0.f, 0.f);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t u[16];
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          float2 p = pf_add2(make_float2(sv[32 * c + j], sv[32 * c + j + 1]), nm2);
          p.x = pf_exp2(p.x);
          p.y = pf_exp2(p.y);
          ls2 = pf_add2(ls2, p);
          u[j >> 1] = pf_pack(p.x, p.y);
        }
        tmem_st16(ts + 32 * hf + 16 * c, u);  // P overlays S columns 0-63, which the first half has consumed
      }
      l_run += ls2.x + ls2.y;
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      pf_arrive_leader<CG>(&p_ready[bf], lane);
    }
    // this thread's half of the accumulated row of O, once the last product has completed
    scales[(8 + hf) * PF_ROWS + rtid] = l_run;   // the halves' parts of the row sum
#pragma unroll
    for (int j = 0; j < PF_HALF; ++j) o[j] = 0.f;
    if (np > 0 && !*fail) {
      if (!pf_wait_warp(&o_done[(np - 1) & 1], (uint32_t)(((np - 1) >> 1) & 1))) {
        *fail = 1;
      } else {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t v[32];
          tmem_ld32(tm + TOc + PF_HALF * hf + 32 * c, v);
#pragma unroll
          for (int j = 0; j < 32; ++j) o[32 * c + j] = __uint_as_float(v[j]);
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    pf_sync_all<CG>();  // every role, of both CTAs, is done with tensor memory and the operand tiles
    if (CG == 2 && rb >= P.row_blocks) return;   // the pair's second block of an odd number
    l_run = scales[8 * PF_ROWS + rtid] + scales[9 * PF_ROWS + rtid];
    // A CTA that gave up a wait reports it, writes no partial and merges nothing, but still takes its ticket below:
    // the counter of its (sequence, KV head, row block) then returns to zero like after a clean call, and a later
    // call on the same workspace cannot elect its merger too early.
    const bool failed = *fail != 0;   // stable: every role has passed the barrier above
    if (failed && tid == 0) atomicExch(P.status, 1);
    if (failed && ns <= 1) return;
    // ---- split partial / merge by the last split / epilogue: the 256 row threads only ----
    if (ns > 1) {
      const size_t slot0 = (((size_t)b * P.hkv + kvh) * P.row_blocks + rb) * P.num_splits;
      if (!failed) {
        // partial of a slot: [16 four-element groups][half][128 rows] float4 -- a warp's stores and loads are contiguous
        float4* po = reinterpret_cast<float4*>(P.part_o + (slot0 + split) * PF_ROWS * TQ_D) + hf * PF_ROWS + rtid;
#pragma unroll
        for (int j = 0; j < PF_HALF; j += 4) po[(j >> 2) * 2 * PF_ROWS] = make_float4(o[j], o[j + 1], o[j + 2], o[j + 3]);
        if (is_prim) reinterpret_cast<float2*>(P.part_ml)[(slot0 + split) * PF_ROWS + rtid] = make_float2(m_run, l_run);
      }
      __threadfence();
      rows_sync();
      if (tid == 0) {
        int* tk = P.tickets + ((size_t)b * P.hkv + kvh) * P.row_blocks + rb;
        const int prev = atomicAdd(tk, 1);
        int last = 0;
        if (prev == ns - 1) {
          *tk = 0;  // zero again for the next call
          last = 1;
        }
        *fail = last;  // reuse the flag word as "this CTA merges"
      }
      rows_sync();
      if (!*fail || failed) return;
      __threadfence();
      float M = -INFINITY;
      for (int s_i = 0; s_i < ns; ++s_i)
        M = fmaxf(M, __ldcg(reinterpret_cast<const float2*>(P.part_ml) + (slot0 + s_i) * PF_ROWS + rtid).x);
#pragma unroll
      for (int j = 0; j < PF_HALF; ++j) o[j] = 0.f;
      l_run = 0.f;
      for (int s_i = 0; s_i < ns; ++s_i) {
        const float2 ml = __ldcg(reinterpret_cast<const float2*>(P.part_ml) + (slot0 + s_i) * PF_ROWS + rtid);
        const float f = ml.x == -INFINITY ? 0.f : exp2f(ml.x - M);
        l_run = fmaf(ml.y, f, l_run);
        const float4* po = reinterpret_cast<const float4*>(P.part_o + (slot0 + s_i) * PF_ROWS * TQ_D) + hf * PF_ROWS + rtid;
#pragma unroll
        for (int j = 0; j < PF_HALF; j += 4) {
          const float4 v = __ldcg(po + (j >> 2) * 2 * PF_ROWS);
          o[j] = fmaf(v.x, f, o[j]); o[j + 1] = fmaf(v.y, f, o[j + 1]);
          o[j + 2] = fmaf(v.z, f, o[j + 2]); o[j + 3] = fmaf(v.w, f, o[j + 3]);
        }
      }
    }
    {
      const float inv = l_run > 0.f ? 1.0f / (l_run * fv.lut_alpha) : 0.f;
#pragma unroll
      for (int j = 0; j < PF_HALF; ++j) o[j] *= inv;
      float* ys = reinterpret_cast<float*>(ktile);  // the operand tiles are idle by now
      if (P.v_rot) {
#pragma unroll
        for (int k = 0; k < PF_HALF; ++k) ys[(PF_HALF * hf + k) * PF_ROWS + rtid] = o[k];
        rows_sync();
#pragma unroll
        for (int j = 0; j < PF_HALF; ++j) o[j] = 0.f;
        for (int k = 0; k < TQ_D; ++k) {
          const float yv = ys[k * PF_ROWS + rtid];
          const float4* rr = reinterpret_cast<const float4*>(P.v_rot + (size_t)k * TQ_D + 32 * hf);
#pragma unroll
          for (int j = 0; j < PF_HALF; j += 4) {
            const float4 r4 = __ldg(rr + pf_dim<true>(0, j) / 4);
            o[j] = fmaf(r4.x, yv, o[j]); o[j + 1] = fmaf(r4.y, yv, o[j + 1]);
            o[j + 2] = fmaf(r4.z, yv, o[j + 2]); o[j + 3] = fmaf(r4.w, yv, o[j + 3]);
          }
        }
      } else if constexpr (!VT::Q8) {
        row_wht128_pair(o, fv.s2, fv.s1, hf, ys, rtid);  // R^T = D1 (H/sqrt d) D2
      }
      // The rows leave through shared memory like they came in: staged, a warp writes whole rows.
      rows_sync();   // the exchange area of the rotation is read: the staging below is the same memory
      {
        const int esz = P.out_dtype == TQ_F32 ? 4 : 2;
        if (P.out_dtype == TQ_F32) {
#pragma unroll
          for (int j = 0; j < PF_HALF; j += 4)
            *reinterpret_cast<float4*>(chunk_at(ktile, rtid, pf_dim<!VT::Q8>(hf, j) / 4, 4)) = make_float4(o[j], o[j + 1], o[j + 2], o[j + 3]);
        } else if (P.out_dtype == TQ_F16) {
#pragma unroll
          for (int j = 0; j < PF_HALF; j += 8)
            *reinterpret_cast<uint4*>(chunk_at(ktile, rtid, pf_dim<!VT::Q8>(hf, j) / 8, 2)) = make_uint4(pf_pack(o[j], o[j + 1]), pf_pack(o[j + 2], o[j + 3]),
                                                                 pf_pack(o[j + 4], o[j + 5]), pf_pack(o[j + 6], o[j + 7]));
        } else {
#pragma unroll
          for (int j = 0; j < PF_HALF; j += 8) {
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const __nv_bfloat162 h = __floats2bfloat162_rn(o[j + 2 * k], o[j + 2 * k + 1]);
              w[k] = *reinterpret_cast<const uint32_t*>(&h);
            }
            *reinterpret_cast<uint4*>(chunk_at(ktile, rtid, pf_dim<!VT::Q8>(hf, j) / 8, 2)) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
        rows_sync();
        move_rows(ktile, esz, [&](uint8_t* from, bool there, size_t off) {
          if (there) *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(P.out) + off) = *reinterpret_cast<const uint4*>(from);
        });
      }
    }
    return;
  }

  if (tid < SP::MMA_AT) {
    // =========================== producer warps ===========================
    // In a pair a CTA dequantizes K of its 64 tokens (its half of the columns of S) and, of all 128 tokens, its 64 dims of V
    // (its half of the columns of O).
    constexpr int TILE = SP::TILE;
    const uint32_t lk_start = sptr(sm + SP::OFF_K), lv_start = sptr(sm + SP::OFF_V);
    const uint32_t lk_base = SP::KLut::base(lk_start, lane), lv_base = SP::VLut::base(lv_start, lane);
    if (tid < SP::V_AT) {
      // K producers, a token per thread.  The K tiles are free once S of the page that used them before is complete (page
      // i - 2 with two buffers, i - 1 with one), and so is the scale slot i & 3 (the rows finished page i - 4 long before):
      // they run one page ahead of the V producers, whose tile is free only after the product of page i - 2, and S of the
      // next page is ready before the rows ask for it.
      const int tl = tid - SP::K_AT, tok = 64 * crank + tl;
      uint8_t* drow = ktile + (tl >> 3) * 2048 + (tl & 7) * 16;
      uint32_t marked = 0;   // q8_0: slots whose q8_big byte of this warp is set
      bool waited = CG == 1;   // for the rows
      if constexpr (KB > 0) {
        SP::KLut::fill(sm + SP::OFF_K, fk.cent16, tl, 32 * SP::PW);
        asm volatile("bar.sync 5, %0;" ::"n"(32 * SP::PW) : "memory");
      }
      for (int i = 0; i < np; ++i) {
        const int bf = i & 1, st_i = i % NST;
        if constexpr (CG == 2) {
          if (i == (wide ? 0 : 1)) {
            __syncwarp();
            asm volatile("bar.sync 4, %0;" ::"n"(FREE_K) : "memory");
            waited = true;
          }
        }
        bool ok = !*fail;
        if constexpr (SP::KBUF == 2) {
          if (ok && i >= 2) ok = tc_wait(&s_full[bf], (uint32_t)(((i - 2) >> 1) & 1));
        } else {
          if (ok && i >= 1) ok = tc_wait(&s_full[bf ^ 1], (uint32_t)(((i - 1) >> 1) & 1));
        }
        if (ok) ok = tc_wait(&rec_full[st_i], (uint32_t)((i / NST) & 1));
        if (!__all_sync(0xffffffffu, ok)) { *fail = 1; break; }   // a warp goes on or gives up as a whole
        const uint8_t* st = stage0 + st_i * SP::REC;
        uint8_t* dst = drow + (SP::KBUF == 2 ? bf * KT::TILES * TILE : 0);
        if constexpr (KT::Q8) {
          uint2 sc = *reinterpret_cast<const uint2*>(st + P.L.k_scale_off + tok * 8);
          // (a pair's CTA has the columns of both: this thread's other token is the other CTA's)
          const bool own = pf_q8_big(sc);
          bool other = false;
          if constexpr (CG == 2) other = pf_q8_big(*reinterpret_cast<const uint2*>(st + P.L.k_scale_off + (tok ^ 64) * 8));
          const uint32_t slot = 1u << (i & 3);
          if (__any_sync(0xffffffffu, own || other)) {   // not on most pages: nothing is written for them
            scales[(i & 3) * PF_ROWS + tok] = own ? 128.f : 1.f;
            if constexpr (CG == 2) scales[(i & 3) * PF_ROWS + (tok ^ 64)] = other ? 128.f : 1.f;
            if (own) sc = make_uint2(pf_div128(sc.x), pf_div128(sc.y));
            if (lane == 0) *(reinterpret_cast<volatile uint8_t*>(q8_big + (i & 3)) + (tl >> 5)) = 1;
            marked |= slot;
          } else if (marked & slot) {
            if (lane == 0) *(reinterpret_cast<volatile uint8_t*>(q8_big + (i & 3)) + (tl >> 5)) = 0;
            marked &= ~slot;
          }
          pf_q8_token<true, TQ_D, TILE>(st + P.L.k_idx_off + tok * TQ_D, dst, sc.x, sc.y, lane);
        } else {
          pf_dequant_token<KB, typename SP::KLut, TQ_D>(st + P.L.k_idx_off + tok * (16 * KB), dst, lk_base, lk_start);
          for (int t = tl; t < PF_PAGE; t += 32 * SP::PW)   // the scales of all columns of S
            scales[(i & 3) * PF_ROWS + t] = reinterpret_cast<const float*>(st + P.L.k_scale_off)[t];
          if constexpr (KT::PROD) {   // (a zero vector has two zero scales)
            const float ks = reinterpret_cast<const float*>(st + P.L.k_scale_off)[tok];
            const float rs = reinterpret_cast<const float*>(st + P.L.k_rscale_off)[tok];
            pf_sketch_token<TQ_D, TILE>(st + P.L.k_qjl_off + tok * 16, dst + TILE, ks != 0.f ? rs / ks : 0.f);
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        pf_arrive_leader<CG>(&k_ready[bf], lane);
        pf_arrive_warp(&rec_free[st_i], lane);
      }
      __syncwarp();
      if (!waited) asm volatile("bar.arrive 4, %0;" ::"n"(FREE_K) : "memory");
    } else {
      // V producers
      constexpr int DIMS = TQ_D / CG;
      if constexpr (VB > 0) SP::VLut::fill(sm + SP::OFF_V, fv.cent16, tid - SP::V_AT, 32 * SP::PW);
      asm volatile("bar.sync 3, %0;" ::"n"(FREE_V) : "memory");
      for (int i = 0; i < np; ++i) {
        const int bf = i & 1, st_i = i % NST;
        bool ok = !*fail;
        if (ok && i >= 2) ok = tc_wait(&o_done[bf], (uint32_t)(((i - 2) >> 1) & 1));
        if (ok) ok = tc_wait(&rec_full[st_i], (uint32_t)((i / NST) & 1));
        if (!__all_sync(0xffffffffu, ok)) { *fail = 1; break; }
        const uint8_t* st = stage0 + st_i * SP::REC;
        // The token's V scale goes into its row of the operand tile (fp16 product, rounding 2^-11 per element), so
        // that the P operand is the bare probability, bounded by 2^(2 PF2_SLACK) whatever the norms of the values
        // are; a token past the end of the sequence may hold anything: its row is zeroed (its P is zero too, but
        // 0 x inf would not be).  Scales beyond the fp16 range saturate.
#pragma unroll
        for (int k = 0; k < PF_PAGE / (32 * SP::PW); ++k) {
          const int tok = tid - SP::V_AT + k * 32 * SP::PW;
          const bool exists = (page_lo + i) * PT + tok < kv_len;
          uint8_t* dst = vtile + bf * TILE + (tok >> 3) * (2048 / CG) + (tok & 7) * 16;
          if constexpr (VT::Q8) {
            const uint2 sc = exists ? *reinterpret_cast<const uint2*>(st + P.L.v_scale_off + tok * 8) : make_uint2(0u, 0u);
            pf_q8_token<false, DIMS, TILE>(st + P.L.v_idx_off + tok * TQ_D + crank * DIMS, dst, crank ? sc.y : sc.x, sc.y, lane);
          } else {
            const float vsc = exists ? reinterpret_cast<const float*>(st + P.L.v_scale_off)[tok] : 0.f;
            const __half2 s2 = __float2half2_rn(fminf(vsc, 65504.0f));
            pf_dequant_token<VB, typename SP::VLut, DIMS, true>(st + P.L.v_idx_off + tok * (16 * VB) + crank * (DIMS * VB / 8), dst,
                                                                lv_base, lv_start, *reinterpret_cast<const uint32_t*>(&s2));
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        pf_arrive_leader<CG>(&v_ready[bf], lane);
        pf_arrive_warp(&rec_free[st_i], lane);
      }
    }
  } else if (tid == SP::COPIER) {
    // =========================== record copies ===========================
    int issued = min(np, NST);
    while (issued < np && !*fail) {   // the stage of page issued - NST, once all producer warps have read it
      if (!tc_wait(&rec_free[issued % NST], (uint32_t)((issued / NST - 1) & 1))) { *fail = 1; break; }
      issue(issued++);
    }
    for (int i = max(0, issued - NST); i < issued; ++i) tc_wait(&rec_full[i % NST], (uint32_t)((i / NST) & 1));   // none in flight at the end
  } else if (warp == SP::MMA_AT / 32 && crank == 0 && np > 0) {
    // =========================== MMA warp ===========================
    // (all 512 columns are this CTA's: its tensor memory starts at address 0)
    bool okay = pf_wait_warp(q_ready, 0) && __all_sync(0xffffffffu, tb == 0);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t idesc_s = umma_idesc(128 * CG, 128, false), idesc_o = umma_idesc(128 * CG, 128, true);
    const bool issues = CG == 2 || lane == 0;
    auto qk = [&](int i) {   // S_i = Q K_i^T (fp16 hi and lo halves of Q), into the score buffer of page i
      if (!issues) return;
      const int bf = i & 1;
      const uint32_t kt = sptr(ktile) + (SP::KBUF == 2 ? bf * KT::TILES * SP::TILE : 0), d = s_col(bf);
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        const uint64_t kd = umma_desc(kt + ks * 256, 128, 2048);
        umma_ts<CG>(d, TQc + ks * 8, kd, idesc_s, ks > 0);
        umma_ts<CG>(d, TQLc + ks * 8, kd, idesc_s, 1);
        if constexpr (KT::TILES > 1) {   // q8_0: what the fp16 products left; PROD: the sketch against the projected query
          const uint64_t k1 = umma_desc(kt + SP::TILE + ks * 256, 128, 2048);
          umma_ts<CG>(d, (KT::PROD ? TPc : TQc) + ks * 8, k1, idesc_s, 1);
          if constexpr (KT::PROD) {
            umma_ts<CG>(d, TPLc + ks * 8, k1, idesc_s, 1);
            umma_ts<CG>(d, TPc + ks * 8, umma_desc(kt + 2 * SP::TILE + ks * 256, 128, 2048), idesc_s, 1);
          }
        }
      }
      umma_commit<CG>(&s_full[bf]);
    };
    if (okay) okay = pf_wait_warp(&k_ready[0], 0);
    if (okay) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      qk(0);
    }
    for (int i = 0; okay && i < np; ++i) {
      if (__any_sync(0xffffffffu, *fail != 0)) break;
      const int bf = i & 1;
      const uint32_t ph = (uint32_t)((i >> 1) & 1);
      if (KT::SBUF == 2 && i + 1 < np) {
        if (!pf_wait_warp(&k_ready[(i + 1) & 1], (uint32_t)(((i + 1) >> 1) & 1))) { okay = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        qk(i + 1);
      }
      if (!pf_wait_warp(&p_ready[bf], ph) || !pf_wait_warp(&v_ready[bf], ph)) { okay = false; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (issues) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)   // O += P_i V_i: P from tensor memory, V tile MN-major, N = 128
          umma_ts<CG>(TOc, s_col(bf) + ks * 8,
                      umma_desc(sptr(vtile + bf * SP::TILE) + ks * (4096 / CG), 2048 / CG, 128), idesc_o, (i > 0 || ks > 0) ? 1u : 0u);
        umma_commit<CG>(&o_done[bf]);
      }
      __syncwarp();
      if (KT::SBUF == 1 && i + 1 < np) {
        // one score buffer: the next page's scores follow once this page's product, which reads P out of it, is done
        if (!pf_wait_warp(&o_done[bf], ph) || !pf_wait_warp(&k_ready[(i + 1) & 1], (uint32_t)(((i + 1) >> 1) & 1))) { okay = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        qk(i + 1);
      }
    }
    if (!okay) *fail = 1;
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  pf_sync_all<CG>();  // matches the row warps' barrier
  if (warp == SP::K_AT / 32) tmem_free_all<CG>(tb);
}

}  // namespace

template <int KK, int VK, int CG>
static int launch_prefill_cg(const PrefillParams& P, const TqFast& fk, const TqFast& fv, cudaStream_t st) {
  using SP = PfSmem2<KK, VK, CG>;
  TQ_REQUIRE(P.L.record_bytes == SP::REC, TQ_ERR_UNSUPPORTED, "prefill attention: page record of %d bytes, expected %d",
             P.L.record_bytes, SP::REC);
  static thread_local int configured_dev = -1;
  int dev = 0;
  TQ_CUDA(cudaGetDevice(&dev));
  if (configured_dev != dev) {
    TQ_CUDA(cudaFuncSetAttribute(k_prefill_attn2<KK, VK, CG>, cudaFuncAttributeMaxDynamicSharedMemorySize, SP::BYTES));
    configured_dev = dev;
  }
  const int64_t grid = (int64_t)CG * ((P.row_blocks + CG - 1) / CG) * P.batch * P.hkv * P.num_splits;
  TQ_REQUIRE(grid < (1LL << 31), TQ_ERR_TOO_LARGE, "prefill attention: %lld CTAs", (long long)grid);
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(SP::THREADS);
  cfg.dynamicSmemBytes = SP::BYTES;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = CG;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CG == 1 ? 1 : 2;
  TQ_CUDA(cudaLaunchKernelEx(&cfg, k_prefill_attn2<KK, VK, CG>, P, fk, fv));
  return tq_launch_check("k_prefill_attn2");
}

template <int KK, int VK>
static int launch_prefill(const PrefillParams& P, int cg, const TqFast& fk, const TqFast& fv, cudaStream_t st) {
  if constexpr (!PfKind<KK>::PROD)
    if (cg == 2) return launch_prefill_cg<KK, VK, 2>(P, fk, fv, st);
  return launch_prefill_cg<KK, VK, 1>(P, fk, fv, st);
}

struct PfPlan {
  int row_blocks, chunk_pages, num_splits;
  long waves;   // of CTAs
  size_t part_o, part_ml, total;
};
static const size_t PF_TAIL = 65536 * 4 + 256;  // tickets + status word, at the end of the workspace
static const long PF_CTA_COST_PAGES = 12;  // prologue, partial and merge of a CTA, in units of one page of the main loop

// The plan of a form: cg CTAs per operand tile.  coarse: at least eight pages per split, for workspaces that the finer one does not fit
// (sized for a prompt's largest chunk, of few splits, they have to do for its last one).
static PfPlan pf_plan(int batch, int chunk_tokens, int hq, int hkv, int max_pages, int cg, bool coarse = false) {
  PfPlan p;
  p.row_blocks = (chunk_tokens * (hq / hkv) + PF_ROWS - 1) / PF_ROWS;
  const long base = (long)((p.row_blocks + cg - 1) / cg) * hkv * batch;
  const int slots = tq_num_sms() / cg;  // one CTA per SM
  // Splits per row block: the count that minimises (waves of CTAs) x (pages per split + fixed cost of a CTA) + the CTA's work that merges
  // them, 0.8 of a page each (without that, and down to three pages a split, 22 queries over 16,000 tokens of one KV head went from 55 to
  // 69 us).  At least three pages per split: where eight were the least, 26 queries over 2,300 tokens of turbo3, 32 / 8 heads, took 37 us
  // and take 31; 32 over 1,500 of turbo4 43 and 29; 128 over 4,000 of prod3 / turbo3, 16 / 4 heads, 74 and 63.
  const int least = coarse ? 8 : 3, cap = max_pages / least > 1 ? max_pages / least : 1;
  int s = 1;
  long best = -1;
  for (int c = 1; c <= cap && c <= 64; ++c) {
    const long waves = (base * c + slots - 1) / slots;
    const long cost = 10 * waves * ((max_pages + c - 1) / c + PF_CTA_COST_PAGES) + (c > 1 && !coarse ? 8 * c : 0);
    if (best < 0 || cost < best) {
      best = cost;
      s = c;
    }
  }
  p.chunk_pages = (max_pages + s - 1) / s;
  p.num_splits = (max_pages + p.chunk_pages - 1) / p.chunk_pages;
  p.waves = (base * p.num_splits + slots - 1) / slots;
  const size_t slots_total = (size_t)p.row_blocks * hkv * batch * p.num_splits;
  p.part_o = 0;
  p.part_ml = slots_total * PF_ROWS * TQ_D * 4;
  p.total = p.part_ml + slots_total * PF_ROWS * 2 * 4 + PF_TAIL;
  p.total = (p.total + 255) & ~(size_t)255;
  return p;
}

// Time of a plan, by which the form of a call is chosen.  A pair's page takes less (its CTAs dequantize half of it each), but
// an odd last row block occupies a whole pair, and the plan rounds on 74 places instead of 148: three row blocks x 8 KV heads
// x 256 pages of turbo3 are 144 CTAs of 43 pages alone and 64 of 64 as pairs, 99 us against 113; nine x 16 x 32 one wave alone
// and three as pairs, 71 against 113; at 2, 5, 7 and 11 row blocks pairs are ahead (5 x 8 x 1,024: 495 against 540).  Page
// times are what long chunks measure; a CTA is taken to cost 18 us beside its pages (it was 15 and is 10 now; counted as 11, and as 8 pages
// instead of 12 in the plan, none of 34 shapes of 16 to 4,096 queries over up to 65,000 positions took another time), a split its partial
// and its part of the merge.  PROD keys have no pairs: their
// one score buffer puts scores, softmax and product of a page one after the other, 4 us a page in either form.
static long pf_time_ns(const PfPlan& p, int k_format, int v_format, int cg) {
  const int wide = (k_format == TQ_FMT_TURBO4) + (v_format == TQ_FMT_TURBO4);   // tables of 256 pairs
  long page;
  if (k_format == TQ_FMT_Q8_0) page = cg == 1 ? 2280 : v_format == TQ_FMT_Q8_0 ? 1940 : 1790;
  else if (cg == 2) page = 1430 + 20 * wide;
  else page = wide == 0 ? 1620 : wide == 1 ? 1830 : 2200;
  return p.waves * (p.chunk_pages * page + 18000) + p.num_splits * (cg == 2 ? 700 : 1300);
}

// A short chunk over q8_0 or PROD tensors: every query as a row of the decode kernel, which reads a page per row and KV head
// where the kernel here multiplies 128 rows whatever the chunk has, converts every key to two or three operand tiles, and
// splits no finer than three pages.  Rows x KV heads x pages, and 12 ns a row and KV head, bound the one; pages of a wave, the
// splits' merge and a start the other (q8_0 / turbo2, 32/8 heads, rows | tiles: 1 query over 256 pages 17 | 77 us, 4 47 | 78,
// 8 over 32 pages 18 | 35, over 256 some 90 | 78; 48 over 2 pages 12 | 16; prod3 / turbo3, 4 over 256 53 | 109).  (turbo2/3/4
// K and V always take the kernel here.)
static const int64_t PF_MOST_ROW_PAGES = 49152;   // above: tiles, for any pair of formats
static int64_t pf_row_pages(int32_t batch, int32_t chunk_tokens, int32_t hq, int32_t hkv, int32_t max_pages) {
  const int64_t rows = (int64_t)batch * chunk_tokens;
  if (hq / hkv > 8 || rows > 65535 || rows * hkv > 65536) return PF_MOST_ROW_PAGES + 1;   // the decode kernel's limits
  return rows * hkv * max_pages;
}
static bool pf_takes_rows(const PfPlan& single, int64_t row_pages, int64_t row_heads, bool prod, int group) {
  if (row_pages > PF_MOST_ROW_PAGES) return false;
  const int64_t rows_ns = 8000 + row_pages * (prod ? (group > 4 ? 9500 : 7000) : (group > 4 ? 8000 : 6500)) / 1000 + 12 * row_heads;
  const int64_t tiles_ns = single.waves * (single.chunk_pages * (prod ? 4100L : 2200L) + (prod ? 19000 : 8000)) + 1900L * single.num_splits;
  return rows_ns < tiles_ns;
}

extern "C" int64_t tq_prefill_workspace_bytes(int32_t batch, int32_t chunk_tokens, int32_t num_q_heads,
                                              int32_t num_kv_heads, int32_t max_pages_per_seq) {
  if (batch < 1 || chunk_tokens < 1 || num_q_heads < 1 || num_kv_heads < 1 || max_pages_per_seq < 1 ||
      num_q_heads % num_kv_heads)
    return TQ_ERR_INVALID;
  const size_t a = pf_plan(batch, chunk_tokens, num_q_heads, num_kv_heads, max_pages_per_seq, 1).total;
  const size_t b = pf_plan(batch, chunk_tokens, num_q_heads, num_kv_heads, max_pages_per_seq, 2).total;
  int64_t most = (int64_t)(a > b ? a : b);   // enough for every pair of formats
  if (pf_row_pages(batch, chunk_tokens, num_q_heads, num_kv_heads, max_pages_per_seq) <= PF_MOST_ROW_PAGES) {
    const int64_t c = tq_decode_workspace_bytes(batch * chunk_tokens, num_q_heads, num_kv_heads, max_pages_per_seq);
    if (c > most) most = c;
  }
  return most;
}

extern "C" int tq_prefill_attn(const tq_quantizer* kq, const tq_quantizer* vq, const tq_cache_layout* L,
                               const uint8_t* pool_dev, const int32_t* block_table_dev, int32_t max_pages_per_seq,
                               const int32_t* kv_lens_dev, const void* q_dev, int32_t q_dtype, int32_t batch,
                               int32_t chunk_tokens, int32_t num_q_heads, float scale, void* workspace_dev,
                               int64_t workspace_bytes, void* out_dev, int32_t out_dtype, void* stream) {
  TQ_REQUIRE(L, TQ_ERR_INVALID, "tq_prefill_attn: layout missing");
  TQ_REQUIRE(batch >= 0 && chunk_tokens >= 1 && num_q_heads >= 1 && max_pages_per_seq >= 1, TQ_ERR_INVALID, "bad sizes");
  if (batch == 0) return TQ_OK;
  TQ_REQUIRE(pool_dev && block_table_dev && kv_lens_dev && q_dev && out_dev && workspace_dev, TQ_ERR_INVALID,
             "tq_prefill_attn: null buffer");
  TQ_REQUIRE(workspace_bytes % 256 == 0 && tq_aligned(workspace_dev, 256), TQ_ERR_ALIGN,
             "workspace must be 256-byte aligned and a multiple of 256 bytes");
  TQ_REQUIRE(L->d == TQ_D && L->page_tokens == 128, TQ_ERR_UNSUPPORTED,
             "prefill attention is built for d == 128 and 128-token pages");
  const bool k_q8 = L->k_format == TQ_FMT_Q8_0, v_q8 = L->v_format == TQ_FMT_Q8_0, k_prod = L->k_format >= TQ_FMT_PROD2;
  TQ_REQUIRE(k_q8 || kq, TQ_ERR_INVALID, "tq_prefill_attn: K quantizer missing");
  TQ_REQUIRE(v_q8 || vq, TQ_ERR_INVALID, "tq_prefill_attn: V quantizer missing");
  TQ_REQUIRE((k_q8 || (kq->d == TQ_D && kq->bits == (k_prod ? L->k_format - 17 : L->k_format))) &&
                 (v_q8 || (vq->d == TQ_D && vq->bits == L->v_format)),
             TQ_ERR_INVALID, "quantizer bit widths do not match the cache formats");
  TQ_REQUIRE(!k_prod || kq->qjl, TQ_ERR_INVALID, "PROD cache format needs a K quantizer with a QJL stage");
  TQ_REQUIRE(num_q_heads % L->num_kv_heads == 0, TQ_ERR_INVALID, "num_q_heads must be a multiple of num_kv_heads");
  TQ_REQUIRE(q_dtype == TQ_F16 || q_dtype == TQ_BF16 || q_dtype == TQ_F32, TQ_ERR_UNSUPPORTED, "bad query dtype %d", q_dtype);
  TQ_REQUIRE(out_dtype == TQ_F16 || out_dtype == TQ_BF16 || out_dtype == TQ_F32, TQ_ERR_UNSUPPORTED, "bad output dtype %d", out_dtype);
  TQ_REQUIRE(tq_aligned(pool_dev, 128) && tq_aligned(q_dev, 16) && tq_aligned(out_dev, 16), TQ_ERR_ALIGN,
             "pool (128), q and out (16) must be aligned");
  TQ_REQUIRE(batch <= 65535 && L->num_kv_heads <= 65535, TQ_ERR_TOO_LARGE, "batch and KV heads are grid dimensions");
  PrefillParams P;
  memset(&P, 0, sizeof(P));
  P.pool = pool_dev;
  P.block_table = block_table_dev;
  P.kv_lens = kv_lens_dev;
  P.q = q_dev;
  P.out = out_dev;
  P.k_rot_t = !k_q8 && kq->rotation == TQ_ROT_DENSE ? kq->rot32_t : nullptr;
  P.k_s_t = k_prod && kq->rotation == TQ_ROT_DENSE ? kq->s32_t : nullptr;
  P.v_rot = !v_q8 && vq->rotation == TQ_ROT_DENSE ? vq->rot32 : nullptr;
  P.status = reinterpret_cast<int32_t*>((uint8_t*)workspace_dev + workspace_bytes - 256);
  if (scale <= 0.f) scale = TQ_RSQRT_D;
  P.qscale = scale * 1.4426950408889634f;
  P.q_dtype = q_dtype;
  P.out_dtype = out_dtype;
  P.max_pages = max_pages_per_seq;
  P.batch = batch;
  P.tq = chunk_tokens;
  P.hq = num_q_heads;
  P.hkv = L->num_kv_heads;
  P.group = num_q_heads / L->num_kv_heads;
  PfPlan plan;
  int cg = 1;
  for (const bool coarse : {false, true}) {
    plan = pf_plan(batch, chunk_tokens, num_q_heads, L->num_kv_heads, max_pages_per_seq, cg = 1, coarse);
    if ((k_q8 || k_prod || v_q8) &&
        pf_takes_rows(plan, pf_row_pages(batch, chunk_tokens, num_q_heads, L->num_kv_heads, max_pages_per_seq),
                      (int64_t)batch * chunk_tokens * L->num_kv_heads, k_prod, P.group) &&
        tq_decode_workspace_bytes(batch * chunk_tokens, num_q_heads, L->num_kv_heads, max_pages_per_seq) <= workspace_bytes)
      return tq_decode_chunk(kq, vq, L, pool_dev, block_table_dev, max_pages_per_seq, kv_lens_dev, q_dev, q_dtype, batch, chunk_tokens,
                             num_q_heads, scale, workspace_dev, workspace_bytes, out_dev, out_dtype, stream);
    if (plan.row_blocks > 1 && !k_prod) {
      const PfPlan pair = pf_plan(batch, chunk_tokens, num_q_heads, L->num_kv_heads, max_pages_per_seq, 2, coarse);
      if (pf_time_ns(pair, L->k_format, L->v_format, 2) < pf_time_ns(plan, L->k_format, L->v_format, 1)) plan = pair, cg = 2;
    }
    if ((int64_t)plan.total <= workspace_bytes) break;
  }
  TQ_REQUIRE((int64_t)plan.total <= workspace_bytes, TQ_ERR_TOO_LARGE,
             "prefill workspace of %lld bytes is smaller than the %lld needed (tq_prefill_workspace_bytes)",
             (long long)workspace_bytes, (long long)plan.total);
  TQ_REQUIRE((int64_t)batch * L->num_kv_heads * plan.row_blocks <= 65536, TQ_ERR_TOO_LARGE,
             "batch x KV heads x row blocks beyond 65536");
  P.part_o = reinterpret_cast<float*>((uint8_t*)workspace_dev + plan.part_o);
  P.part_ml = reinterpret_cast<float*>((uint8_t*)workspace_dev + plan.part_ml);
  P.tickets = reinterpret_cast<int32_t*>((uint8_t*)workspace_dev + workspace_bytes - PF_TAIL);
  P.chunk_pages = plan.chunk_pages;
  P.num_splits = plan.num_splits;
  P.row_blocks = plan.row_blocks;
  P.L = *L;
  cudaStream_t st = (cudaStream_t)stream;
  TqFast none;
  memset(&none, 0, sizeof(none));
  none.lut_alpha = 1.0f;
  const TqFast &fk = k_q8 ? none : kq->fast, &fv = v_q8 ? none : vq->fast;
  int rc = TQ_ERR_UNSUPPORTED;
#define TQ_PF(K, V) \
  if (L->k_format == K && L->v_format == V) rc = launch_prefill<K, V>(P, cg, fk, fv, st);
  TQ_PF(2, 2) TQ_PF(3, 3) TQ_PF(4, 4) TQ_PF(3, 2) TQ_PF(4, 2) TQ_PF(4, 3)
  TQ_PF(8, 2) TQ_PF(8, 3) TQ_PF(8, 4) TQ_PF(8, 8)
  TQ_PF(18, 2) TQ_PF(18, 3) TQ_PF(19, 2) TQ_PF(19, 3) TQ_PF(19, 4) TQ_PF(20, 3) TQ_PF(20, 4)
#undef TQ_PF
  if (rc == TQ_ERR_UNSUPPORTED) tq_set_error("prefill attention: K format %d with V format %d is not instantiated", L->k_format, L->v_format);
  return rc;
}
