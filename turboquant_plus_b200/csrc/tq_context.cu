// Quantizer constants, error reporting and the paged-cache layout arithmetic.
#include <math.h>
#include <stdarg.h>
#include <stdlib.h>

#include <vector>

#include "tq_internal.cuh"

static thread_local char g_err[512] = "";

void tq_set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

int tq_cuda_fail(cudaError_t e, const char* what) {
  tq_set_error("CUDA error %d (%s) in %s", (int)e, cudaGetErrorString(e), what);
  return (e == cudaErrorNoKernelImageForDevice || e == cudaErrorInvalidDeviceFunction) ? TQ_ERR_DEVICE
                                                                                       : TQ_ERR_CUDA;
}

int tq_launch_check(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return tq_cuda_fail(e, what);
  return TQ_OK;
}

int tq_num_sms() {
  static thread_local int cached_dev = -1, cached = 0;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  if (dev != cached_dev) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached = n;
    cached_dev = dev;
  }
  return cached;
}

extern "C" const char* tq_version(void) { return "tq_b200 0.1 (sm_100a)"; }

extern "C" const char* tq_error_string(int code) {
  switch (code) {
    case TQ_OK: return "ok";
    case TQ_ERR_INVALID: return "invalid argument";
    case TQ_ERR_UNSUPPORTED: return "unsupported combination";
    case TQ_ERR_ALIGN: return "misaligned pointer or stride";
    case TQ_ERR_CUDA: return "CUDA runtime error";
    case TQ_ERR_TOO_LARGE: return "size beyond the supported maximum";
    case TQ_ERR_DEVICE: return "no kernel image for this device (needs sm_100a)";
    default: return "unknown error";
  }
}

extern "C" const char* tq_last_error(void) { return g_err; }

static bool is_pm1(const double* v, int n) {
  for (int i = 0; i < n; ++i)
    if (v[i] != 1.0 && v[i] != -1.0) return false;
  return true;
}

static void sign_bits(const double* v, uint32_t (&out)[4]) {
  for (int w = 0; w < 4; ++w) out[w] = 0;
  for (int e = 0; e < TQ_D; ++e)
    if (v[e] < 0) out[e >> 5] |= 1u << (e & 31);
}

// The device arrays of a quantizer are parts of one allocation, filled by one copy: every allocation and every pageable
// copy synchronises with the device, and a quantizer that is built inside a program pays for each of them.
struct DeviceImage {
  std::vector<uint8_t> bytes;
  size_t add(const void* src, size_t n) {
    const size_t at = (bytes.size() + 255) & ~(size_t)255;
    bytes.resize(at + n);
    memcpy(bytes.data() + at, src, n);
    return at;
  }
};

struct MatrixParts {
  size_t m, t, m32, t32, mp, tp;   // mp, tp: padded with zeros to dp x dp (m and t themselves when d is a multiple of 8)
  double scale;                    // d = 128: what the digits of tq_dense_i8.cu are relative to (0: it has none)
  double rows, length;             // the largest sum of magnitudes of a row, and the longest row's length, over that
};
static MatrixParts add_matrix(DeviceImage& im, const double* m, int d) {
  std::vector<double> t((size_t)d * d);
  std::vector<float> a32((size_t)d * d), t32((size_t)d * d);
  for (int i = 0; i < d; ++i)
    for (int j = 0; j < d; ++j) {
      t[(size_t)j * d + i] = m[(size_t)i * d + j];
      a32[(size_t)i * d + j] = (float)m[(size_t)i * d + j];
      t32[(size_t)j * d + i] = (float)m[(size_t)i * d + j];
    }
  MatrixParts p{};
  p.m = im.add(m, t.size() * 8);
  p.t = im.add(t.data(), t.size() * 8);
  p.mp = p.m;
  p.tp = p.t;
  if (d % 8) {
    const int dp = (d + 7) / 8 * 8;
    std::vector<double> mp((size_t)dp * dp, 0.0), tp((size_t)dp * dp, 0.0);
    for (int i = 0; i < d; ++i)
      for (int j = 0; j < d; ++j) {
        mp[(size_t)i * dp + j] = m[(size_t)i * d + j];
        tp[(size_t)j * dp + i] = m[(size_t)i * d + j];
      }
    p.mp = im.add(mp.data(), mp.size() * 8);
    p.tp = im.add(tp.data(), tp.size() * 8);
  }
  p.scale = d == TQ_D ? tq_dense_digits_scale(m, &p.rows, &p.length) : 0.0;
  p.m32 = im.add(a32.data(), a32.size() * 4);
  p.t32 = im.add(t32.data(), t32.size() * 4);
  return p;
}

// (tq_quantize_status_word; this file has no kernels)
static __device__ int32_t quantize_status;

int32_t* tq_quantize_status_word() {
  static thread_local int word_dev = -1;
  static thread_local int32_t* word = nullptr;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  if (word_dev != dev) {
    if (cudaGetSymbolAddress((void**)&word, quantize_status) != cudaSuccess) {
      (void)cudaGetLastError();
      return nullptr;
    }
    word_dev = dev;
  }
  return word;
}

extern "C" int tq_quantize_status_sync(int32_t* status_out) {
  TQ_REQUIRE(status_out, TQ_ERR_INVALID, "tq_quantize_status_sync: status_out is null");
  int32_t* word = tq_quantize_status_word();
  TQ_REQUIRE(word, TQ_ERR_CUDA, "tq_quantize_status_sync: no status word on this device");
  TQ_CUDA(cudaMemcpy(status_out, word, 4, cudaMemcpyDeviceToHost));
  if (*status_out != 0) TQ_CUDA(cudaMemset(word, 0, 4));
  return TQ_OK;
}

extern "C" int tq_quantizer_destroy(tq_quantizer* q) {
  if (!q) return TQ_OK;
  if (q->mem) cudaFree(q->mem);
  if (q->digits_event) cudaEventDestroy(q->digits_event);
  free(q);
  return TQ_OK;
}

extern "C" int tq_quantizer_create(const tq_quantizer_desc* desc, tq_quantizer** out) {
  TQ_REQUIRE(desc && out, TQ_ERR_INVALID, "tq_quantizer_create: null argument");
  *out = nullptr;
  TQ_REQUIRE(desc->bits >= 1 && desc->bits <= 4, TQ_ERR_INVALID, "bits must be 1..4, got %d", desc->bits);
  TQ_REQUIRE(desc->centroids, TQ_ERR_INVALID, "centroids missing");
  TQ_REQUIRE(desc->rotation == TQ_ROT_DENSE || desc->rotation == TQ_ROT_WHT, TQ_ERR_INVALID,
             "rotation kind %d unknown", desc->rotation);
  const int nc = 1 << desc->bits;
  for (int i = 1; i < nc; ++i)
    TQ_REQUIRE(desc->centroids[i] > desc->centroids[i - 1], TQ_ERR_INVALID, "centroids must be strictly increasing");
  if (desc->rotation == TQ_ROT_WHT) {
    TQ_REQUIRE(desc->d == TQ_D, TQ_ERR_UNSUPPORTED, "WHT mode is built for d == 128, got d = %d", desc->d);
    TQ_REQUIRE(desc->signs1 && desc->signs2, TQ_ERR_INVALID, "WHT mode needs signs1 and signs2");
    TQ_REQUIRE(is_pm1(desc->signs1, TQ_D) && is_pm1(desc->signs2, TQ_D), TQ_ERR_INVALID, "signs must be +-1");
    if (desc->qjl) {
      TQ_REQUIRE(desc->qjl_signs1 && desc->qjl_signs2, TQ_ERR_INVALID, "WHT mode QJL needs qjl_signs1/2");
      TQ_REQUIRE(is_pm1(desc->qjl_signs1, TQ_D) && is_pm1(desc->qjl_signs2, TQ_D), TQ_ERR_INVALID,
                 "qjl signs must be +-1");
    }
  } else {
    TQ_REQUIRE(desc->d >= 1 && desc->d <= 1024, TQ_ERR_UNSUPPORTED, "dense mode supports d in 1..1024, got %d", desc->d);
    TQ_REQUIRE(desc->rot || desc->qjl, TQ_ERR_INVALID, "dense mode needs rot (or only a QJL matrix)");
    if (desc->qjl) TQ_REQUIRE(desc->qjl_s, TQ_ERR_INVALID, "dense mode QJL needs qjl_s");
  }
  tq_quantizer* q = (tq_quantizer*)calloc(1, sizeof(tq_quantizer));
  TQ_REQUIRE(q, TQ_ERR_INVALID, "out of host memory");
  q->d = desc->d;
  q->bits = desc->bits;
  q->rotation = desc->rotation;
  q->norm_correction = desc->norm_correction ? 1 : 0;
  q->qjl = desc->qjl ? 1 : 0;
  (void)tq_quantize_status_word();   // its module is loaded here, not by a call that may be captured
  cudaError_t e = cudaGetDevice(&q->device);
  if (e != cudaSuccess) {
    free(q);
    return tq_cuda_fail(e, "cudaGetDevice");
  }
  std::vector<double> c(desc->centroids, desc->centroids + nc), b(nc - 1);
  for (int i = 0; i < nc - 1; ++i) b[i] = (c[i] + c[i + 1]) / 2.0;  // turboquant/codebook.py:133
  for (int i = 0; i < nc; ++i) q->host_cent[i] = c[i];

  TqFast& f = q->fast;
  memset(&f, 0, sizeof(f));
  f.bits = desc->bits;
  f.norm_correction = q->norm_correction;
  f.has_qjl = q->qjl;
  for (int i = 0; i < nc; ++i) f.cent[i] = (float)c[i];
  for (int i = 0; i < nc - 1; ++i) f.bnd[i] = (float)b[i];
  // symmetric codebook: positive boundaries mirror negative ones, centre boundary is (almost) zero
  bool sym = fabs(b[nc / 2 - 1]) < 1e-12;
  for (int i = 0; i < nc; ++i) sym = sym && (f.cent[i] == -f.cent[nc - 1 - i]);
  for (int i = 0; i < nc - 1; ++i)
    if (i != nc / 2 - 1) sym = sym && (f.bnd[i] == -f.bnd[nc - 2 - i]);
  f.symmetric = sym ? 1 : 0;
  // The attention kernels feed centroids to the tensor cores as fp16.  A common factor alpha in
  // [1, 2) is picked so that alpha * c_i all round to fp16 with the smallest worst relative error
  // (the factor is divided out of the query / output once), instead of taking alpha = 1.
  {
    double best = 1e30;
    float best_a = 1.0f;
    for (int i = 0; i < 65536; ++i) {
      const float a = 1.0f + (float)i / 65536.0f;
      double worst = 0.0;
      for (int k = 0; k < nc && worst < best; ++k) {   // (a factor already beaten needs no further centroids)
        const double want = (double)a * c[k];
        const double got = (double)__half2float(__float2half_rn((float)want));
        const double rel = want != 0.0 ? fabs(got / want - 1.0) : 0.0;
        if (rel > worst) worst = rel;
      }
      if (worst < best) {
        best = worst;
        best_a = a;
      }
    }
    f.lut_alpha = best_a;
    for (int k = 0; k < nc; ++k) {
      const __half h = __float2half_rn((float)((double)best_a * c[k]));
      f.cent16[k] = *reinterpret_cast<const uint16_t*>(&h);
    }
  }

  DeviceImage im;
  MatrixParts mr{}, ms{};
  const bool dense_rot = desc->rotation == TQ_ROT_DENSE && desc->rot, dense_s = desc->rotation == TQ_ROT_DENSE && desc->qjl;
  if (desc->rotation == TQ_ROT_WHT) {
    sign_bits(desc->signs1, f.s1);
    sign_bits(desc->signs2, f.s2);
    if (desc->qjl) {
      sign_bits(desc->qjl_signs1, f.j1);
      sign_bits(desc->qjl_signs2, f.j2);
    }
  }
  if (dense_rot) mr = add_matrix(im, desc->rot, q->d);
  if (dense_s) ms = add_matrix(im, desc->qjl_s, q->d);
  const size_t cent_at = im.add(c.data(), c.size() * 8), bnd_at = im.add(b.data(), b.size() * 8);
  // room for the digits of R, R^T, S, S^T, which the first call of many vectors makes (tq_dense_i8.cu)
  const size_t digits_at = (im.bytes.size() + 255) & ~(size_t)255;
  const size_t total = digits_at + ((mr.scale != 0.0 ? 2 : 0) + (ms.scale != 0.0 ? 2 : 0)) * (size_t)TQ_DENSE_DIGITS_BYTES;
  e = cudaMalloc((void**)&q->mem, total);
  if (e == cudaSuccess) e = cudaMemcpy(q->mem, im.bytes.data(), im.bytes.size(), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    tq_quantizer_destroy(q);
    return tq_cuda_fail(e, "quantizer constants");
  }
  auto f64 = [&](size_t at) { return reinterpret_cast<double*>(q->mem + at); };
  auto f32 = [&](size_t at) { return reinterpret_cast<float*>(q->mem + at); };
  if (dense_rot) q->rot = f64(mr.m), q->rot_t = f64(mr.t), q->rot32 = f32(mr.m32), q->rot32_t = f32(mr.t32), q->rotp = f64(mr.mp), q->rotp_t = f64(mr.tp);
  if (dense_s) q->s = f64(ms.m), q->s_t = f64(ms.t), q->s32 = f32(ms.m32), q->s32_t = f32(ms.t32), q->sp = f64(ms.mp), q->sp_t = f64(ms.tp);
  uint8_t* digits = q->mem + digits_at;
  auto digits_place = [&]() {
    uint8_t* at = digits;
    digits += TQ_DENSE_DIGITS_BYTES;
    return at;
  };
  if (mr.scale != 0.0) q->dig.r = digits_place(), q->dig.rt = digits_place(), q->dig.r_scale = mr.scale, q->dig.r_rows = mr.rows, q->dig.r_length = mr.length;
  if (ms.scale != 0.0) q->dig.s = digits_place(), q->dig.st = digits_place(), q->dig.s_scale = ms.scale;
  q->dig.cent_scale = tq_dense_digits_centroids(c.data(), nc);
  if (q->dig.cent_scale != 0.0) tq_dense_digits_words(c.data(), nc, q->dig.cent_scale, q->dig.words);
  for (size_t i = 0; i < b.size(); ++i) q->dig.bnd[i] = b[i];
  q->cent64 = f64(cent_at);
  q->bnd64 = f64(bnd_at);
  *out = q;
  return TQ_OK;
}

// ------------------------------------------------------------------------------------------
static int fmt_idx_bits(int fmt) {
  switch (fmt) {
    case TQ_FMT_TURBO2: return 2;
    case TQ_FMT_TURBO3: return 3;
    case TQ_FMT_TURBO4: return 4;
    case TQ_FMT_PROD2: return 1;
    case TQ_FMT_PROD3: return 2;
    case TQ_FMT_PROD4: return 3;
    default: return -1;
  }
}

static inline int32_t up128(int32_t v) { return (v + 127) & ~127; }

extern "C" int tq_cache_layout_init(tq_cache_layout* L, int32_t d, int32_t page_tokens, int32_t num_kv_heads,
                                    int32_t k_format, int32_t v_format) {
  TQ_REQUIRE(L, TQ_ERR_INVALID, "layout is null");
  TQ_REQUIRE(d == TQ_D, TQ_ERR_UNSUPPORTED, "the paged cache is built for d == 128, got %d", d);
  TQ_REQUIRE(page_tokens >= 32 && page_tokens <= 256 && page_tokens % 32 == 0, TQ_ERR_INVALID,
             "page_tokens must be a multiple of 32 in 32..256, got %d", page_tokens);
  TQ_REQUIRE(num_kv_heads >= 1, TQ_ERR_INVALID, "num_kv_heads must be >= 1");
  const bool k_q8 = k_format == TQ_FMT_Q8_0, v_q8 = v_format == TQ_FMT_Q8_0;
  TQ_REQUIRE(k_q8 || fmt_idx_bits(k_format) > 0, TQ_ERR_INVALID, "unknown K format %d", k_format);
  TQ_REQUIRE(v_q8 || (fmt_idx_bits(v_format) > 0 && v_format < TQ_FMT_PROD2), TQ_ERR_INVALID,
             "V format %d must be turbo2/3/4 or q8_0", v_format);
  memset(L, 0, sizeof(*L));
  L->d = d;
  L->page_tokens = page_tokens;
  L->num_kv_heads = num_kv_heads;
  L->k_format = k_format;
  L->v_format = v_format;
  int32_t off = 0;
  L->k_idx_bytes = k_q8 ? d : d * fmt_idx_bits(k_format) / 8;
  L->k_idx_off = off;
  off = up128(off + page_tokens * L->k_idx_bytes);
  L->k_scale_off = off;
  off = up128(off + page_tokens * (k_q8 ? (d / 32) * 2 : 4));
  L->k_qjl_off = L->k_rscale_off = -1;
  if (k_format >= TQ_FMT_PROD2 && k_format <= TQ_FMT_PROD4) {
    L->k_qjl_off = off;
    off = up128(off + page_tokens * (d / 8));
    L->k_rscale_off = off;
    off = up128(off + page_tokens * 4);
  }
  L->v_idx_bytes = v_q8 ? d : d * fmt_idx_bits(v_format) / 8;
  L->v_idx_off = off;
  off = up128(off + page_tokens * L->v_idx_bytes);
  L->v_scale_off = off;
  off = up128(off + page_tokens * (v_q8 ? (d / 32) * 2 : 4));
  L->record_bytes = off;
  L->head_stride = off;
  L->page_stride = (int64_t)off * num_kv_heads;
  return TQ_OK;
}
