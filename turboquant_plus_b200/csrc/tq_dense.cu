// Dense-rotation quantize and dequantize (fp64, any d <= 256) on the fp64 tensor cores.
//
// The reference multiplies every vector by a d x d matrix in fp64 (turboquant/polar_quant.py:56-119,
// turboquant/turboquant.py:79-124): one product to quantize, two more for the residual and its sketch, one or two to
// dequantize.  A CTA takes MT vectors through all of them: the vectors sit in shared memory, the matrices stream from L2
// as B operands, and mma.sync m16n8k8.f64 does the products -- a warp holds 32 vectors x 32 outputs, so that a step of
// eight MMAs (1,024 multiply-adds each) needs 8 KB of operands and the fp64 units are the limit, not the loads (one
// thread per output and eight vectors read five shared-memory operands per eight multiply-adds).  Arithmetic is the
// reference's: inputs normalised in their own precision, fp64 products and sums, boundaries counted from below.  Rows
// and columns past d are zeros (the matrices are uploaded padded to a multiple of eight).
#include "tq_internal.cuh"

namespace {

constexpr int DN_THREADS = 256, DN_WARPS = 8;

__device__ __forceinline__ void dmma(double (&c)[4], const double (&a)[4], double b0, double b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
               : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}

template <typename T> __device__ __forceinline__ double dn_d(T v) { return (double)v; }
template <> __device__ __forceinline__ double dn_d<__half>(__half v) { return (double)__half2float(v); }

// A CTA's eight warps: WM along the vectors, WN along the outputs; a warp holds 16 MF vectors x 8 NF outputs.
template <int MF_, int NF_, int WM_> struct DnTile {
  static constexpr int MF = MF_, NF = NF_, WM = WM_, WN = DN_WARPS / WM, MT = 16 * MF * WM;
  static constexpr int DP = 8 * NF * WN;   // largest padded d
};

template <int MF, int NF> __device__ __forceinline__ void dn_zero(double (&c)[MF][NF][4]) {
#pragma unroll
  for (int mf = 0; mf < MF; ++mf)
#pragma unroll
    for (int nf = 0; nf < NF; ++nf)
#pragma unroll
      for (int r = 0; r < 4; ++r) c[mf][nf][r] = 0.0;
}

// c += (16 MF vectors from row m0 of the CTA) x (8 NF outputs from column n0): c[mf][nf] = rows m0 + 16 mf + g (c0, c1) and
// + 8 (c2, c3), columns n0 + 8 nf + 2 t, + 1.  `bmat` rows are outputs, contiguous over k (dp of them); a_pair(row, k)
// gives the operand values (k, k + 1).  Slots t and t + 4 of a k-step carry k = 2 t and 2 t + 1, in A and B alike.
template <int MF, int NF, typename A>
__device__ __forceinline__ void dn_product(double (&c)[MF][NF][4], A a_pair, const double* __restrict__ bmat, int dp, int m0,
                                           int n0, int lane) {
  const int g = lane >> 2, t = lane & 3;
  const double* brow[NF];
#pragma unroll
  for (int nf = 0; nf < NF; ++nf) brow[nf] = bmat + (size_t)min(n0 + 8 * nf + g, dp - 1) * dp + 2 * t;   // (past dp: unused)
  double2 b[NF], bn[NF];
#pragma unroll
  for (int nf = 0; nf < NF; ++nf) bn[nf] = __ldg(reinterpret_cast<const double2*>(brow[nf]));
  for (int k = 0; k < dp; k += 8) {
#pragma unroll
    for (int nf = 0; nf < NF; ++nf) b[nf] = bn[nf];
    if (k + 8 < dp) {   // the next step's operands are on their way while this one multiplies
#pragma unroll
      for (int nf = 0; nf < NF; ++nf) bn[nf] = __ldg(reinterpret_cast<const double2*>(brow[nf] + k + 8));
    }
#pragma unroll
    for (int mf = 0; mf < MF; ++mf) {
      const double2 lo = a_pair(m0 + 16 * mf + g, k + 2 * t), hi = a_pair(m0 + 16 * mf + g + 8, k + 2 * t);
      const double a[4] = {lo.x, hi.x, lo.y, hi.y};
#pragma unroll
      for (int nf = 0; nf < NF; ++nf) dmma(c[mf][nf], a, b[nf].x, b[nf].y);
    }
  }
}

// each vector's sum over this warp's outputs into part[warp column][vector]; the columns are then added in order
template <int MT, int MF>
__device__ __forceinline__ void dn_row_parts(const double (&rowsum)[MF][2], double* part, int wn, int m0, int lane) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int mf = 0; mf < MF; ++mf)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      double v = rowsum[mf][h];
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      if (t == 0) part[wn * MT + m0 + 16 * mf + 8 * h + g] = v;
    }
}

// ---- norms in NumPy's order (first term + pairwise sum of the rest), as in k_quantize_dense ----------------------------
__device__ __forceinline__ float dn_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double dn_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float dn_sq(float a) { return __fmul_rn(a, a); }
__device__ __forceinline__ double dn_sq(double a) { return __dmul_rn(a, a); }

// NumPy's pairwise sum of squares by eight lanes: fewer than 8 terms in order; up to 128 terms in eight interleaved sums
// (lane j has terms j, j + 8, ...) combined pairwise, the remaining n % 8 added in order; more in halves, the first a
// multiple of eight (n <= 255: a half holds at most 135 terms, its halves fewer than 128).
template <typename E, int DEPTH = 2>
__device__ __forceinline__ E dn_pairwise(const E* xs, int n, int j) {
  if (n < 8) {
    E r = (E)0;
    for (int i = 0; i < n; ++i) r = dn_add(r, dn_sq(xs[i]));
    return r;
  }
  if constexpr (DEPTH > 0) {
    if (n > 128) {
      int n2 = n / 2;
      n2 -= n2 % 8;
      const E lo = dn_pairwise<E, DEPTH - 1>(xs, n2, j);
      return dn_add(lo, dn_pairwise<E, DEPTH - 1>(xs + n2, n - n2, j));
    }
  }
  E r = dn_sq(xs[j]);
  const int full = n - (n % 8);
  for (int i = 8; i < full; i += 8) r = dn_add(r, dn_sq(xs[i + j]));
#pragma unroll
  for (int m = 1; m < 8; m <<= 1) r = dn_add(r, __shfl_xor_sync(0xffffffffu, r, m));   // ((0+1)+(2+3))+((4+5)+(6+7))
  for (int i = full; i < n; ++i) r = dn_add(r, dn_sq(xs[i]));
  return r;
}

// elements between rows of a staged array: the rows that the lanes of a load touch start in different banks (float rows
// 32 bytes apart modulo 64, double rows 64 modulo 128)
__host__ __device__ constexpr int dn_stride(int dp) { return (dp + 15) / 16 * 16 + 8; }
__host__ __device__ constexpr int dn_istride(int d) { return (d + 15) / 16 * 16; }

template <typename E, int MT> __host__ __device__ constexpr size_t dn_stage_bytes(int dp) {
  const size_t two = 2 * (size_t)MT * dn_stride(dp) * sizeof(E), res = (size_t)MT * dn_stride(dp) * 8;
  return two > res ? two : res;
}

}  // namespace

namespace {

template <typename Tin, typename E, class TL>
__global__ void __launch_bounds__(DN_THREADS, sizeof(E) == 4 ? 2 : 1)
    k_dense_quantize(const TqDenseQuant a, const Tin* __restrict__ x, int64_t ld, int64_t n) {
  constexpr int MF = TL::MF, NF = TL::NF, WN = TL::WN, MT = TL::MT;
  extern __shared__ __align__(16) uint8_t dn_mem[];
  __shared__ double s_cent[16], s_bnd[16], s_part[DN_WARPS * MT];
  __shared__ float s_norm[MT];
  __shared__ double s_inv[MT];        // 1 / ||c[idx]|| with norm correction, else 1
  const int d = a.d, dp = a.dp, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int wn = warp / TL::WM, m0 = 16 * MF * (warp % TL::WM), n0 = 8 * NF * wn;   // dp <= 8 NF WN: dn_pick
  const int st = dn_stride(dp), ist = dn_istride(d);
  E* xs = reinterpret_cast<E*>(dn_mem);                // inputs
  E* ws = xs + (size_t)MT * st;                        // normalised inputs
  double* rs = reinterpret_cast<double*>(dn_mem);      // later: the residual, over both
  uint8_t* s_idx = dn_mem + dn_stage_bytes<E, MT>(dp); // [MT][ist] indices, later the sketch bits
  const int64_t v0 = (int64_t)blockIdx.x * MT;
  const int nv = (int)(n - v0 < MT ? n - v0 : MT);
  if (tid < 16) {
    s_cent[tid] = tid < (1 << a.bits) ? a.cent[tid] : 0.0;
    s_bnd[tid] = tid < (1 << a.bits) - 1 ? a.bnd[tid] : 0.0;
  }
  for (int v = warp; v < MT; v += DN_WARPS)
    for (int k = lane; k < dp; k += 32) xs[v * st + k] = v < nv && k < d ? (E)dn_d<Tin>(x[(v0 + v) * ld + k]) : (E)0;
  __syncthreads();
  // norms in the input's own precision, eight lanes per vector
  for (int v = tid >> 3; v < MT; v += DN_THREADS / 8) {
    const int j = tid & 7;
    const E s0 = dn_sq(xs[v * st]);
    const E ss = d > 1 ? dn_add(s0, dn_pairwise<E>(xs + v * st + 1, d - 1, j)) : s0;
    const E nrm = sizeof(E) == 4 ? (E)sqrtf((float)ss) : (E)sqrt((double)ss);
    const E safe = nrm > (E)0 ? nrm : (E)1;                                    // turboquant/polar_quant.py:74
    if (j == 0) s_norm[v] = (float)nrm;
    for (int k = j; k < dp; k += 8) ws[v * st + k] = xs[v * st + k] / safe;    // in the input's precision: :75
  }
  __syncthreads();

  double c[MF][NF][4];
  // ---- y = R x / ||x||, indices, ||c[idx]||^2 ----
  {
    double cc[MF][2] = {};
    const int nb = (1 << a.bits) - 1;
    if (n0 < dp) {
      dn_zero(c);
      dn_product(c, [&](int row, int k) {
        if constexpr (sizeof(E) == 4) {
          const float2 v = *reinterpret_cast<const float2*>(ws + row * st + k);
          return make_double2((double)v.x, (double)v.y);
        } else {
          return *reinterpret_cast<const double2*>(ws + row * st + k);
        }
      }, a.rot, dp, m0, n0, lane);
#pragma unroll
      for (int mf = 0; mf < MF; ++mf)
#pragma unroll
        for (int nf = 0; nf < NF; ++nf)
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const int col = n0 + 8 * nf + 2 * t + (r & 1), row = m0 + 16 * mf + g + 8 * (r >> 1);
            if (col < d) {
              int m = 0;
              for (int b = 0; b < nb; ++b) m += s_bnd[b] < c[mf][nf][r] ? 1 : 0;   // searchsorted, side = 'left'
              s_idx[row * ist + col] = (uint8_t)m;
              cc[mf][r >> 1] += s_cent[m] * s_cent[m];
            }
          }
    }
    dn_row_parts<MT>(cc, s_part, wn, m0, lane);
  }
  __syncthreads();
  if (tid < MT) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < WN; ++w) s += s_part[w * MT + tid];
    double cn = sqrt(s);
    cn = cn > 1e-10 ? cn : 1.0;                                                 // turboquant/polar_quant.py:110-111
    s_inv[tid] = a.norm_correction ? 1.0 / cn : 1.0;
    if (tid < nv) {
      if (a.out_norm) a.out_norm[v0 + tid] = s_norm[tid];
      if (a.out_scale) a.out_scale[v0 + tid] = (float)(a.norm_correction ? (double)s_norm[tid] / cn : (double)s_norm[tid]);
    }
  }
  // outputs that only need the indices
  if (a.out_idx) {
    if (d % 16 == 0 && (reinterpret_cast<uintptr_t>(a.out_idx) & 15) == 0) {
      const int per = d / 16;
      for (int i = tid; i < nv * per; i += DN_THREADS) {
        const int v = i / per, o = i - v * per;
        *reinterpret_cast<uint4*>(a.out_idx + (v0 + v) * d + 16 * o) = *reinterpret_cast<const uint4*>(s_idx + v * ist + 16 * o);
      }
    } else {
      for (int v = warp; v < nv; v += DN_WARPS)
        for (int k = lane; k < d; k += 32) a.out_idx[(v0 + v) * d + k] = s_idx[v * ist + k];
    }
  }
  if (a.out_packed) {
    const int bpv = d * a.bits / 8;
    for (int i = tid; i < nv * bpv; i += DN_THREADS) {
      const int v = i / bpv, o = i - v * bpv;
      uint32_t byte = 0;
      for (int bit = 0; bit < 8; ++bit) {
        const int pos = o * 8 + bit, e = pos / a.bits, r = pos - e * a.bits;
        byte = (byte << 1) | ((s_idx[v * ist + e] >> (a.bits - 1 - r)) & 1u);
      }
      a.out_packed[v0 * bpv + i] = (uint8_t)byte;
    }
  }
  if (a.out_qjl == nullptr && a.out_rnorm == nullptr && a.out_res == nullptr) return;
  __syncthreads();

  // ---- residual x - x_hat, x_hat = norm R^T c[idx] / ||c[idx]||.  The norm is the one that is returned and stored (fp32):
  // the residual is then exactly x - dequantize(indices, norms) for the norms the caller holds
  // (turboquant/polar_quant.py:121-132) ----
  double rr[MF][2] = {};
  if (n0 < dp) {
    dn_zero(c);
    dn_product(c, [&](int row, int k) {   // (columns past d: the matrix is zero there, any index will do)
      const uint32_t pair = *reinterpret_cast<const uint16_t*>(s_idx + row * ist + (k < d ? k : 0));
      const double f = s_inv[row];
      return make_double2(s_cent[pair & 15] * f, s_cent[(pair >> 8) & 15] * f);
    }, a.rot_t, dp, m0, n0, lane);
#pragma unroll
    for (int mf = 0; mf < MF; ++mf)
#pragma unroll
      for (int nf = 0; nf < NF; ++nf)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int col = n0 + 8 * nf + 2 * t + (r & 1), row = m0 + 16 * mf + g + 8 * (r >> 1);
          const double e = col < d ? (double)xs[row * st + col] - c[mf][nf][r] * (double)s_norm[row] : 0.0;
          c[mf][nf][r] = e;
          rr[mf][r >> 1] += e * e;
          if (a.out_res && row < nv && col < d) a.out_res[(v0 + row) * a.ld_res + col] = e;
        }
  }
  dn_row_parts<MT>(rr, s_part, wn, m0, lane);
  __syncthreads();   // (also: nobody reads the inputs any more)
  if (tid < nv && a.out_rnorm) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < WN; ++w) s += s_part[w * MT + tid];
    a.out_rnorm[v0 + tid] = (float)sqrt(s);
  }
  if (a.out_qjl == nullptr) return;
  if (n0 < dp) {
#pragma unroll
    for (int mf = 0; mf < MF; ++mf)
#pragma unroll
      for (int nf = 0; nf < NF; ++nf)
        if (n0 + 8 * nf < dp) {
          const int col = n0 + 8 * nf + 2 * t, row = m0 + 16 * mf + g;
          *reinterpret_cast<double2*>(rs + row * st + col) = make_double2(c[mf][nf][0], c[mf][nf][1]);
          *reinterpret_cast<double2*>(rs + (row + 8) * st + col) = make_double2(c[mf][nf][2], c[mf][nf][3]);
        }
  }
  __syncthreads();
  // ---- sketch: sign(S r), zero counts as +1 (turboquant/qjl.py:89-90) ----
  if (n0 < dp) {
    dn_zero(c);
    dn_product(c, [&](int row, int k) { return *reinterpret_cast<const double2*>(rs + row * st + k); }, a.s, dp, m0, n0, lane);
#pragma unroll
    for (int mf = 0; mf < MF; ++mf)
#pragma unroll
      for (int nf = 0; nf < NF; ++nf)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int col = n0 + 8 * nf + 2 * t + (r & 1), row = m0 + 16 * mf + g + 8 * (r >> 1);
          if (col < d) s_idx[row * ist + col] = c[mf][nf][r] < 0.0 ? 0 : 1;
        }
  }
  __syncthreads();
  const int rb = (d + 7) / 8;
  for (int i = tid; i < nv * rb; i += DN_THREADS) {
    const int v = i / rb, o = i - v * rb;
    uint32_t byte = 0;
    for (int bit = 0; bit < 8; ++bit) {
      const int e = o * 8 + bit;
      byte = (byte << 1) | (e < d ? s_idx[v * ist + e] : 0u);
    }
    a.out_qjl[v0 * rb + i] = (uint8_t)byte;
  }
}

template <typename T> __device__ __forceinline__ T dn_from(double v);
template <> __device__ __forceinline__ double dn_from<double>(double v) { return v; }
template <> __device__ __forceinline__ float dn_from<float>(double v) { return (float)v; }
template <> __device__ __forceinline__ __half dn_from<__half>(double v) { return __float2half_rn((float)v); }

// x_hat = (norm / ||c[idx]||) R^T c[idx] + shrink sqrt(pi/2)/sqrt(d) rnorm S^T z, both products into one set of sums: the
// factors of a vector go into its operand values
template <typename Tout, class TL>
__global__ void __launch_bounds__(DN_THREADS, 2) k_dense_dequantize(const TqDenseDequant a, int64_t n, Tout* __restrict__ out) {
  constexpr int MF = TL::MF, NF = TL::NF, MT = TL::MT;
  extern __shared__ __align__(16) uint8_t dn_mem[];
  __shared__ double s_cent[16], s_f[MT], s_g[MT];
  const int d = a.d, dp = a.dp, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int m0 = 16 * MF * (warp % TL::WM), n0 = 8 * NF * (warp / TL::WM);
  const int ist = dn_istride(d), rb = (d + 7) / 8;
  uint8_t* s_idx = dn_mem;                       // [MT][ist]
  uint8_t* s_z = dn_mem + (size_t)MT * ist;      // [MT][rb]
  const int64_t v0 = (int64_t)blockIdx.x * MT;
  const int nv = (int)(n - v0 < MT ? n - v0 : MT);
  if (tid < 16) s_cent[tid] = tid < (1 << a.bits) ? a.cent[tid] : 0.0;
  if (a.packed) {
    const int bpv = d * a.bits / 8;
    for (int v = warp; v < MT; v += DN_WARPS)
      for (int k = lane; k < ist; k += 32) {
        uint32_t m = 0;
        if (v < nv && k < d)
          for (int r = 0; r < a.bits; ++r) {
            const int pos = k * a.bits + r;
            m = (m << 1) | ((a.packed[(v0 + v) * bpv + (pos >> 3)] >> (7 - (pos & 7))) & 1u);
          }
        s_idx[v * ist + k] = (uint8_t)m;
      }
  } else if (d % 16 == 0 && (reinterpret_cast<uintptr_t>(a.idx) & 15) == 0) {
    const int per = d / 16;
    for (int i = tid; i < MT * per; i += DN_THREADS) {
      const int v = i / per, o = i - v * per;
      *reinterpret_cast<uint4*>(s_idx + v * ist + 16 * o) =
          v < nv ? *reinterpret_cast<const uint4*>(a.idx + (v0 + v) * d + 16 * o) : make_uint4(0u, 0u, 0u, 0u);
    }
  } else {
    for (int v = warp; v < MT; v += DN_WARPS)
      for (int k = lane; k < ist; k += 32) s_idx[v * ist + k] = v < nv && k < d ? a.idx[(v0 + v) * d + k] : (uint8_t)0;
  }
  if (a.qjl)
    for (int i = tid; i < MT * rb; i += DN_THREADS) s_z[i] = i < nv * rb ? a.qjl[v0 * rb + i] : (uint8_t)0;
  __syncthreads();
  for (int v = tid >> 3; v < MT; v += DN_THREADS / 8) {   // eight lanes per vector
    double cc = 0.0;
    for (int k = tid & 7; k < d; k += 8) {
      const double cv = s_cent[s_idx[v * ist + k] & 15];
      cc += cv * cv;
    }
    cc += __shfl_xor_sync(0xffffffffu, cc, 1);
    cc += __shfl_xor_sync(0xffffffffu, cc, 2);
    cc += __shfl_xor_sync(0xffffffffu, cc, 4);
    if ((tid & 7) == 0) {
      double cn = 1.0;
      if (a.norm_correction) {
        cn = sqrt(cc);
        cn = cn > 1e-10 ? cn : 1.0;
      }
      s_f[v] = v < nv ? (double)a.norm[v0 + v] / cn : 0.0;
      s_g[v] = a.qjl && v < nv ? a.shrink * 1.2533141373155001 / sqrt((double)d) * (double)a.rnorm[v0 + v] : 0.0;  // qjl.py:131-132
    }
  }
  __syncthreads();
  if (n0 >= dp) return;
  double c[MF][NF][4];
  dn_zero(c);
  dn_product(c, [&](int row, int k) {
    const uint32_t pair = *reinterpret_cast<const uint16_t*>(s_idx + row * ist + (k < d ? k : 0));
    const double f = s_f[row];
    return make_double2(s_cent[pair & 15] * f, s_cent[(pair >> 8) & 15] * f);
  }, a.rot_t, dp, m0, n0, lane);
  if (a.qjl)
    dn_product(c, [&](int row, int k) {
      const uint32_t z = (uint32_t)s_z[row * rb + (k < d ? k >> 3 : 0)] << (k & 7);   // bit 7: k, bit 6: k + 1
      const double f = s_g[row];
      return make_double2(z & 0x80u ? f : -f, z & 0x40u ? f : -f);
    }, a.s_t, dp, m0, n0, lane);
  const bool wide = sizeof(Tout) == 8 && (a.ld_out & 1) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0 && (d & 1) == 0;
#pragma unroll
  for (int mf = 0; mf < MF; ++mf)
#pragma unroll
    for (int nf = 0; nf < NF; ++nf)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int row = m0 + 16 * mf + 8 * h + g, col = n0 + 8 * nf + 2 * t;
        if (row >= nv || col >= d) continue;
        double y0 = c[mf][nf][2 * h], y1 = c[mf][nf][2 * h + 1];
        Tout* o = out + (v0 + row) * a.ld_out + col;
        if (a.accumulate) {
          y0 += dn_d<Tout>(o[0]);
          if (col + 1 < d) y1 += dn_d<Tout>(o[1]);
        }
        if (wide) {
          *reinterpret_cast<double2*>(o) = make_double2(y0, y1);
        } else {
          o[0] = dn_from<Tout>(y0);
          if (col + 1 < d) o[1] = dn_from<Tout>(y1);
        }
      }
}

// Raises the kernel's limit to `most`, what it takes at its largest d whatever this call's d is: the limit belongs to the
// process, and a thread that set it to the size of its own call would lower it under the others'.
template <auto kernel> int dn_configure(size_t most) {
  static thread_local int configured_dev = -1;   // one per kernel: the kernel is a template argument
  int dev = 0;
  TQ_CUDA(cudaGetDevice(&dev));
  if (configured_dev != dev) {
    TQ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    configured_dev = dev;
  }
  return TQ_OK;
}

// Tile of a call.  Every CTA streams the matrices once, so more vectors per CTA are cheaper while the SMs are full (two
// CTAs each); fewer fill more SMs: 100 vectors in tiles of 32 keep four SMs busy for 25 us.
template <typename F> int dn_pick(int dp, int64_t n, F&& launch) {
  const int64_t full = 2 * (int64_t)tq_num_sms();
  if (dp > 128) return launch(DnTile<2, 4, 1>{});            // 32 vectors x 256 outputs
  if (n > 32 * full) return launch(DnTile<2, 4, 2>{});       // 64 x 128
  if (n > 16 * full) return launch(DnTile<1, 4, 2>{});       // 32 x 128
  return launch(DnTile<1, 2, 1>{});                          // 16 x 128
}

template <typename Tin, typename E>
int dn_launch_quantize(const TqDenseQuant& a, const void* x, int64_t ld, int64_t n, cudaStream_t st) {
  return dn_pick(a.dp, n, [&](auto tile) {
    using TL = decltype(tile);
    auto bytes = [](int d, int dp) { return dn_stage_bytes<E, TL::MT>(dp) + (size_t)TL::MT * dn_istride(d); };
    const size_t smem = bytes(a.d, a.dp);
    const int rc = dn_configure<k_dense_quantize<Tin, E, TL>>(bytes(TL::DP, TL::DP));
    if (rc != TQ_OK) return rc;
    k_dense_quantize<Tin, E, TL><<<(unsigned)((n + TL::MT - 1) / TL::MT), DN_THREADS, smem, st>>>(a, (const Tin*)x, ld, n);
    return tq_launch_check("k_dense_quantize");
  });
}

template <typename Tout>
int dn_launch_dequantize(const TqDenseDequant& a, int64_t n, void* out, cudaStream_t st) {
  return dn_pick(a.dp, n, [&](auto tile) {
    using TL = decltype(tile);
    const size_t smem = (size_t)TL::MT * (dn_istride(a.d) + (a.qjl ? (a.d + 7) / 8 : 0));
    const int rc = dn_configure<k_dense_dequantize<Tout, TL>>((size_t)TL::MT * (dn_istride(TL::DP) + TL::DP / 8));
    if (rc != TQ_OK) return rc;
    k_dense_dequantize<Tout, TL><<<(unsigned)((n + TL::MT - 1) / TL::MT), DN_THREADS, smem, st>>>(a, n, (Tout*)out);
    return tq_launch_check("k_dense_dequantize");
  });
}

}  // namespace

// false: not of this kernel's shape (d > 256), nothing launched
bool tq_dense_quantize_try(const TqDenseQuant& a, const void* x, int32_t dtype, int64_t ld, int64_t n, cudaStream_t st, int* rc) {
  if (a.dp > 256) return false;
  switch (dtype) {
    case TQ_F32: *rc = dn_launch_quantize<float, float>(a, x, ld, n, st); return true;
    case TQ_F16: *rc = dn_launch_quantize<__half, float>(a, x, ld, n, st); return true;
    case TQ_F64: *rc = dn_launch_quantize<double, double>(a, x, ld, n, st); return true;
    default: return false;
  }
}

bool tq_dense_dequantize_try(const TqDenseDequant& a, int64_t n, void* out, int32_t dtype, cudaStream_t st, int* rc) {
  if (a.dp > 256) return false;
  switch (dtype) {
    case TQ_F64: *rc = dn_launch_dequantize<double>(a, n, out, st); return true;
    case TQ_F32: *rc = dn_launch_dequantize<float>(a, n, out, st); return true;
    case TQ_F16: *rc = dn_launch_dequantize<__half>(a, n, out, st); return true;
    default: return false;
  }
}
