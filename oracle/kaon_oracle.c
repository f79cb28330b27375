/*
 * kaon_oracle.c — CPU restatement of the kaon (Koronos/K-Optimizers 0.7.4) fused optimizer step.
 *
 * TEST INFRASTRUCTURE ONLY.  This file is what the CUDA kernels are compared against and the
 * timed CPU baseline.  Nothing in the shipped package may import, link or call it; the product path
 * has no CPU fallback and fails loudly when the CUDA library is missing.
 *
 * Every function cites the reference lines (path within the reference project) whose arithmetic it
 * restates.  The arithmetic contract is that of torch-CPU fp32 kernels: scalars are Python doubles
 * cast to fp32 at use, lerp and add(alpha) are FMA forms, divisions are true IEEE divisions, rounding
 * to integer is half-to-even, rsqrt is 1/sqrtf.  Order-dependent reductions (row/col means, norms,
 * the GC row mean) are accumulated in double here; torch accumulates in fp32 in a vectorised order,
 * so those agree with the reference to ~1e-7 relative, not bit for bit.
 *
 * Pinned against the reference by tests/golden/ (vectors generated by importing the reference;
 * generator committed beside them).
 *
 * Build: see oracle/Makefile (gcc -O2 -ffp-contract=off -mfma -fopenmp).
 */
#include <math.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#define KO_F32 0
#define KO_BF16 1

#define KO_M_F32 0
#define KO_M_BF16 1
#define KO_M_INT8 2
#define KO_M_4BIT 3

#define KO_W_NONE 0 /* bf16_method="none": p - bf16(delta), rounded to nearest even */
#define KO_W_SR 1   /* bf16_method="stochastic_rounding" with the Philox stream below */
#define KO_W_SR_NOISE 2 /* stochastic rounding with caller-supplied 16-bit noise (validation only) */
#define KO_W_KAHAN 3    /* bf16_method="kahan": compensated write through the tensor's shift buffer */

/* ------------------------------------------------------------------ scalar helpers */

static inline float bf16_to_f32(uint16_t h) {
  uint32_t u = (uint32_t)h << 16;
  float f;
  memcpy(&f, &u, 4);
  return f;
}

/* round-to-nearest-even fp32 -> bf16 (what torch's .to(bfloat16) does) */
static inline uint16_t f32_to_bf16(float f) {
  uint32_t u;
  memcpy(&u, &f, 4);
  if ((u & 0x7fffffffu) > 0x7f800000u) return (uint16_t)((u >> 16) | 0x40u);
  u += 0x7fffu + ((u >> 16) & 1u);
  return (uint16_t)(u >> 16);
}

static inline float rbf16(float f) { return bf16_to_f32(f32_to_bf16(f)); }

static inline float ld(const void* a, int dtype, int64_t i) {
  return dtype == KO_BF16 ? bf16_to_f32(((const uint16_t*)a)[i]) : ((const float*)a)[i];
}

/* torch lerp_(end, w) on fp32: FMA forms of  start + w*(end-start)  /  end - (end-start)*(1-w)
 * (ATen/native/Lerp.h; probe-verified bit for bit on this torch build). */
static inline float ko_lerp(float start, float end, float w) {
  float diff = end - start;
  return (w < 0.5f) ? fmaf(w, diff, start) : fmaf(w - 1.0f, diff, end);
}

/* ------------------------------------------------------------------ Philox4x32-R (Salmon et al. 2011) */

/* The round function and key schedule are pinned by the published 10-round known-answer vectors
 * (ko_philox4x32); the stochastic-rounding stream runs the same function with KO_SR_ROUNDS = 7 rounds,
 * the smallest round count the Random123 authors report as passing BigCrush (Philox4x32-7). */
#define KO_SR_ROUNDS 7

void ko_philox4x32_r(const uint32_t ctr[4], const uint32_t key[2], int rounds, uint32_t out[4]) {
  uint32_t c0 = ctr[0], c1 = ctr[1], c2 = ctr[2], c3 = ctr[3];
  uint32_t k0 = key[0], k1 = key[1];
  for (int r = 0; r < rounds; ++r) {
    if (r) {
      k0 += 0x9E3779B9u;
      k1 += 0xBB67AE85u;
    }
    uint64_t p0 = (uint64_t)0xD2511F53u * c0;
    uint64_t p1 = (uint64_t)0xCD9E8D57u * c2;
    uint32_t n0 = (uint32_t)(p1 >> 32) ^ c1 ^ k0;
    uint32_t n1 = (uint32_t)p1;
    uint32_t n2 = (uint32_t)(p0 >> 32) ^ c3 ^ k1;
    uint32_t n3 = (uint32_t)p0;
    c0 = n0; c1 = n1; c2 = n2; c3 = n3;
  }
  out[0] = c0; out[1] = c1; out[2] = c2; out[3] = c3;
}

void ko_philox4x32(const uint32_t ctr[4], const uint32_t key[2], uint32_t out[4]) {
  ko_philox4x32_r(ctr, key, 10, out);
}

/* The stochastic-rounding noise stream of this framework (no reference counterpart: the reference
 * draws from torch's global RNG, _stochastic_rounding.py:88-96).  One Philox4x32-7 call serves the eight
 * consecutive elements 8q..8q+7:  counter = (q_lo, tensor_id, step, tag | q_hi<<8), key = seed.
 * Element e takes 16-bit lane (e & 7): word (e&7)>>1, low half for even e, high half for odd e. */
static inline uint32_t ko_sr_noise(uint64_t seed, uint32_t step, uint32_t tensor_id, uint32_t tag,
                                   int64_t e) {
  uint64_t q = (uint64_t)e >> 3;
  uint32_t ctr[4] = {(uint32_t)q, tensor_id, step, (tag & 0xffu) | ((uint32_t)(q >> 32) << 8)};
  uint32_t key[2] = {(uint32_t)seed, (uint32_t)(seed >> 32)};
  uint32_t out[4];
  ko_philox4x32_r(ctr, key, KO_SR_ROUNDS, out);
  uint32_t w = out[(e & 7) >> 1];
  return (e & 1) ? (w >> 16) : (w & 0xffffu);
}

void ko_sr_noise_fill(uint64_t seed, uint32_t step, uint32_t tensor_id, uint32_t tag, int64_t n,
                      uint16_t* out) {
  for (int64_t e = 0; e < n; ++e) out[e] = (uint16_t)ko_sr_noise(seed, step, tensor_id, tag, e);
}

/* ------------------------------------------------------------------ a1: gradient centralization */

/* _backend.py:147-177.  For an ndim>=2 grad viewed as [R, C]: g -= mean(g over the row), in the
 * grad's own dtype.  bf16: the fp32-accumulated mean is rounded to bf16, the difference is computed
 * in fp32 and rounded to bf16.  fp32: plain fp32 mean and subtract.  Writes fp32 values to out. */
void ko_centralize(const void* g, int dtype, int64_t R, int64_t C, float* out) {
#pragma omp parallel for schedule(static)
  for (int64_t r = 0; r < R; ++r) {
    double s = 0.0;
    for (int64_t c = 0; c < C; ++c) s += (double)ld(g, dtype, r * C + c);
    float mean = (float)s / (float)C;
    if (dtype == KO_BF16) mean = rbf16(mean);
    for (int64_t c = 0; c < C; ++c) {
      float d = ld(g, dtype, r * C + c) - mean;
      out[r * C + c] = (dtype == KO_BF16) ? rbf16(d) : d;
    }
  }
}

/* ------------------------------------------------------------------ a4/a5: momentum codec */

/* _momentum_codec.py:72-97  per-row absmax int8.  rows==0 means a 1-D tensor: one scalar scale. */
void ko_encode_int8(const float* m, int64_t n, int64_t rows, int8_t* codes, float* scale) {
  int64_t R = rows > 0 ? rows : 1;
  int64_t C = n / R;
#pragma omp parallel for schedule(static)
  for (int64_t r = 0; r < R; ++r) {
    float amax = 0.0f;
    for (int64_t c = 0; c < C; ++c) amax = fmaxf(amax, fabsf(m[r * C + c]));
    amax = fmaxf(amax, 1e-12f);
    float sc = amax / 127.0f;
    scale[r] = sc;
    for (int64_t c = 0; c < C; ++c) {
      float q = rintf(m[r * C + c] / sc);
      q = fminf(fmaxf(q, -127.0f), 127.0f);
      codes[r * C + c] = (int8_t)q;
    }
  }
}

/* _momentum_codec.py:293-301 (dequant = code * row scale) */
void ko_decode_int8(const int8_t* codes, const float* scale, int64_t n, int64_t rows, float* m) {
  int64_t R = rows > 0 ? rows : 1;
  int64_t C = n / R;
#pragma omp parallel for schedule(static)
  for (int64_t r = 0; r < R; ++r)
    for (int64_t c = 0; c < C; ++c) m[r * C + c] = (float)codes[r * C + c] * scale[r];
}

/* _momentum_codec.py:100-141  flat blocks of `block` elements over the row-major flattened tensor,
 * last block zero-padded; scale = max(absmax,1e-12)/7; q = clamp(rint(m/scale), +-7); nibble = q+8;
 * even flat index in the low nibble; odd numel leaves a zero high nibble in the last byte. */
void ko_encode_4bit(const float* m, int64_t n, int64_t block, uint8_t* packed, float* scale) {
  int64_t nb = (n + block - 1) / block;
  uint8_t* nib = (uint8_t*)malloc((size_t)(n + 1));
  nib[n] = 0;
#pragma omp parallel for schedule(static)
  for (int64_t b = 0; b < nb; ++b) {
    int64_t e0 = b * block, e1 = e0 + block < n ? e0 + block : n;
    float amax = 0.0f;
    for (int64_t e = e0; e < e1; ++e) amax = fmaxf(amax, fabsf(m[e]));
    amax = fmaxf(amax, 1e-12f);
    float sc = amax / 7.0f;
    scale[b] = sc;
    for (int64_t e = e0; e < e1; ++e) {
      float q = rintf(m[e] / sc);
      q = fminf(fmaxf(q, -7.0f), 7.0f);
      nib[e] = (uint8_t)((int)q + 8);
    }
  }
  int64_t nbytes = (n + 1) / 2;
#pragma omp parallel for schedule(static)
  for (int64_t i = 0; i < nbytes; ++i) packed[i] = (uint8_t)(nib[2 * i] | (nib[2 * i + 1] << 4));
  free(nib);
}

/* _momentum_codec.py:144-155 */
void ko_decode_4bit(const uint8_t* packed, const float* scale, int64_t n, int64_t block, float* m) {
#pragma omp parallel for schedule(static)
  for (int64_t e = 0; e < n; ++e) {
    uint8_t byte = packed[e >> 1];
    int nibv = (e & 1) ? (byte >> 4) & 0xF : byte & 0xF;
    m[e] = ((float)nibv - 8.0f) * scale[e / block];
  }
}

static void decode_m(int mkind, const void* m, const float* m_scale, int64_t n, int64_t rows,
                     int64_t block, float* out) {
  if (mkind == KO_M_INT8) ko_decode_int8((const int8_t*)m, m_scale, n, rows, out);
  else if (mkind == KO_M_4BIT) ko_decode_4bit((const uint8_t*)m, m_scale, n, block, out);
  else
    for (int64_t i = 0; i < n; ++i) out[i] = ld(m, mkind == KO_M_BF16 ? KO_BF16 : KO_F32, i);
}

static void encode_m(int mkind, const float* in, int64_t n, int64_t rows, int64_t block, void* m,
                     float* m_scale) {
  if (mkind == KO_M_INT8) ko_encode_int8(in, n, rows, (int8_t*)m, m_scale);
  else if (mkind == KO_M_4BIT) ko_encode_4bit(in, n, block, (uint8_t*)m, m_scale);
  else if (mkind == KO_M_BF16)
    for (int64_t i = 0; i < n; ++i) ((uint16_t*)m)[i] = f32_to_bf16(in[i]);
  else
    memcpy(m, in, (size_t)n * 4);
}

/* ------------------------------------------------------------------ a7: cautious masking */

/* _backend.py:127-142.  mask = (delta*g > 0); delta = delta*mask / max(mean(mask), 1e-8).
 * mean(mask) equals float(count)/float(n).  Returns the kept count. */
int64_t ko_cautious(float* delta, const float* g, int64_t n) {
  int64_t cnt = 0;
#pragma omp parallel for reduction(+ : cnt) schedule(static)
  for (int64_t i = 0; i < n; ++i) cnt += (delta[i] * g[i] > 0.0f) ? 1 : 0;
  float denom = fmaxf((float)cnt / (float)n, 1e-8f);
#pragma omp parallel for schedule(static)
  for (int64_t i = 0; i < n; ++i) {
    float mask = (delta[i] * g[i] > 0.0f) ? 1.0f : 0.0f;
    delta[i] = (delta[i] * mask) / denom;
  }
  return cnt;
}

/* ------------------------------------------------------------------ a8: weight write  p += alpha*delta */

/* _backend.py:82-122 and _stochastic_rounding.py:70-103.  alpha is -1 (update) or +1 (Nekaon climb).
 * fp32 params: one fma.  bf16 "none": p - bf16(delta) rounded to nearest even (alpha=-1 only).
 * bf16 SR: res = fma(delta, alpha, fp32(p)); bits(res) + U{0..65535}; clear the low 16 bits. */
/* The Kahan write needs one more per-tensor buffer (state["shift"], bf16) than the step functions'
 * signatures carry: the caller names it here before the step and clears it afterwards. */
static uint16_t* ko_kahan_shift = NULL;
void ko_set_kahan_shift(uint16_t* shift) { ko_kahan_shift = shift; }

void ko_write(void* p, int dtype, const float* delta, int64_t n, float alpha, int method,
              uint64_t seed, uint32_t step, uint32_t tensor_id, uint32_t tag,
              const uint16_t* noise) {
  if (dtype == KO_F32) {
    float* pf = (float*)p;
#pragma omp parallel for schedule(static)
    for (int64_t i = 0; i < n; ++i) pf[i] = fmaf(delta[i], alpha, pf[i]);
    return;
  }
  uint16_t* pb = (uint16_t*)p;
  if (method == KO_W_KAHAN) {
    /* _backend.py:89-94, every line a bf16 tensor op (fp32 arithmetic, result rounded to bf16):
     *   shift -= bf16(delta); p_before = p; p += shift; shift += (p_before - p) */
    uint16_t* sh = ko_kahan_shift;
#pragma omp parallel for schedule(static)
    for (int64_t i = 0; i < n; ++i) {
      float pv = bf16_to_f32(pb[i]);
      float s1 = rbf16(bf16_to_f32(sh[i]) + alpha * rbf16(delta[i]));
      float pn = rbf16(pv + s1);
      float s2 = rbf16(s1 + rbf16(pv - pn));
      pb[i] = f32_to_bf16(pn);
      sh[i] = f32_to_bf16(s2);
    }
    return;
  }
#pragma omp parallel for schedule(static)
  for (int64_t i = 0; i < n; ++i) {
    float pv = bf16_to_f32(pb[i]);
    if (method == KO_W_NONE) {
      pb[i] = f32_to_bf16(pv + alpha * rbf16(delta[i]));
    } else {
      float res = fmaf(delta[i], alpha, pv);
      uint32_t bits;
      memcpy(&bits, &res, 4);
      uint32_t nz = (method == KO_W_SR_NOISE) ? noise[i] : ko_sr_noise(seed, step, tensor_id, tag, i);
      bits = (bits + nz) & 0xFFFF0000u;
      pb[i] = (uint16_t)(bits >> 16);
    }
  }
}

/* ------------------------------------------------------------------ a6: Lion */

/* lion.py:416-485 (one tensor).  rows = shape[0] for ndim>=2 tensors, 0 for 1-D.
 *   g  <- centralize(g) if gc and ndim>=2          (_backend.py:147-177)
 *   c   = fma(g, f32(1-b1), m*f32(b1));  d = sign(c)
 *   m   = fma(g, f32(1-b2), m*f32(b2));  store through the codec
 *   d   = fma(p, f32(wd), d) if wd;  cautious;  d *= f32(lr);  p -= d
 * kept_out (optional) receives the cautious kept count. */
int ko_lion_step(void* p, const void* g, int dtype, int64_t n, int64_t rows, int mkind, void* m,
                 float* m_scale, int64_t block, double lr, double beta1, double beta2, double wd,
                 int cautious, int gc, int method, uint64_t seed, uint32_t step,
                 uint32_t tensor_id, const uint16_t* noise, int64_t* kept_out) {
  float* G = (float*)malloc((size_t)n * 4);
  float* M = (float*)malloc((size_t)n * 4);
  float* D = (float*)malloc((size_t)n * 4);
  if (!G || !M || !D) return 1;
  if (gc && rows > 0) ko_centralize(g, dtype, rows, n / rows, G);
  else
    for (int64_t i = 0; i < n; ++i) G[i] = ld(g, dtype, i);
  decode_m(mkind, m, m_scale, n, rows, block, M);
  const float b1 = (float)beta1, w1 = (float)(1.0 - beta1);
  const float b2 = (float)beta2, w2 = (float)(1.0 - beta2);
#pragma omp parallel for schedule(static)
  for (int64_t i = 0; i < n; ++i) {
    float c = fmaf(G[i], w1, M[i] * b1);
    D[i] = (c > 0.0f) ? 1.0f : ((c < 0.0f) ? -1.0f : 0.0f);
    M[i] = fmaf(G[i], w2, M[i] * b2);
  }
  encode_m(mkind, M, n, rows, block, m, m_scale);
  if (wd != 0.0) {
    const float fwd = (float)wd;
#pragma omp parallel for schedule(static)
    for (int64_t i = 0; i < n; ++i) D[i] = fmaf(ld(p, dtype, i), fwd, D[i]);
  }
  int64_t kept = -1;
  if (cautious) kept = ko_cautious(D, G, n);
  if (kept_out) *kept_out = kept;
  const float flr = (float)lr;
#pragma omp parallel for schedule(static)
  for (int64_t i = 0; i < n; ++i) D[i] = D[i] * flr;
  ko_write(p, dtype, D, n, -1.0f, method, seed, step, tensor_id, 0u, noise);
  free(G); free(M); free(D);
  return 0;
}

/* ------------------------------------------------------------------ a2/a3: Adakaon */

/* Factored second moment + clip, _factored.py:26-83 and adakaon.py:865-888 / 984-1002.
 * In: X[R*C] (the signal whose second moment is tracked).  Updates row[R], col[C] in place and
 * writes U = ((X*r)*c) / max(rms/clip,1) * f32(scale).   scale = lr (Adakaon) or 0.2*lr (AdaMuon). */
static void factored_update(const float* X, int64_t R, int64_t C, float* row, float* col,
                            double beta2, double eps1, double clip, double scale, float* U,
                            float* rms_out) {
  const float w2 = (float)(1.0 - beta2);
  const float e1 = (float)eps1;
  double* colsum = (double*)calloc((size_t)C, 8);
  for (int64_t r = 0; r < R; ++r) {
    double s = 0.0;
    for (int64_t c = 0; c < C; ++c) {
      float sq = X[r * C + c] * X[r * C + c];
      if (eps1 > 0) sq = sq + e1;
      s += (double)sq;
      colsum[c] += (double)sq;
    }
    float mean = (float)s / (float)C;
    row[r] = ko_lerp(row[r], mean, w2);
  }
  for (int64_t c = 0; c < C; ++c) {
    float mean = (float)colsum[c] / (float)R;
    col[c] = ko_lerp(col[c], mean, w2);
  }
  free(colsum);
  double rs = 0.0;
  for (int64_t r = 0; r < R; ++r) rs += (double)row[r];
  float rowmean = (float)rs / (float)R;
  float* rf = (float*)malloc((size_t)R * 4);
  float* cf = (float*)malloc((size_t)C * 4);
  for (int64_t r = 0; r < R; ++r) rf[r] = 1.0f / sqrtf(row[r] / rowmean);
  for (int64_t c = 0; c < C; ++c) cf[c] = 1.0f / sqrtf(col[c]);
  double ss = 0.0;
#pragma omp parallel for reduction(+ : ss) schedule(static)
  for (int64_t r = 0; r < R; ++r)
    for (int64_t c = 0; c < C; ++c) {
      float u = (X[r * C + c] * rf[r]) * cf[c];
      U[r * C + c] = u;
      ss += (double)u * (double)u;
    }
  float rms = (float)sqrt(ss) / (float)sqrt((double)(R * C));
  if (rms_out) *rms_out = rms;
  float divisor = fmaxf(rms / (float)clip, 1.0f);
  const float fs = (float)scale;
#pragma omp parallel for schedule(static)
  for (int64_t i = 0; i < R * C; ++i) U[i] = (U[i] / divisor) * fs;
  free(rf); free(cf);
}

/* Non-factored (1-D) second moment, adakaon.py:908-948 / 992-1002. */
static void flat_update(const float* X, int64_t n, float* v, double beta2, double eps1, double clip,
                        double scale, float* U, float* rms_out) {
  const float w2 = (float)(1.0 - beta2);
  const float e1 = (float)eps1;
  double ss = 0.0;
  for (int64_t i = 0; i < n; ++i) {
    float sq = X[i] * X[i];
    if (eps1 > 0) sq = sq + e1;
    v[i] = ko_lerp(v[i], sq, w2);
    float u = X[i] * (1.0f / sqrtf(v[i]));
    U[i] = u;
    ss += (double)u * (double)u;
  }
  float rms = (float)sqrt(ss) / (float)sqrt((double)n);
  if (rms_out) *rms_out = rms;
  float divisor = fmaxf(rms / (float)clip, 1.0f);
  const float fs = (float)scale;
  for (int64_t i = 0; i < n; ++i) U[i] = (U[i] / divisor) * fs;
}

/* Codec EMA, _momentum_codec.py:303-340 / 357-389:  m = lerp(decode(m), u, f32(1-b1)); delta = m
 * (the fp32 value BEFORE requantisation); store encode(m). */
static void codec_ema(int mkind, void* m, float* m_scale, int64_t n, int64_t rows, int64_t block,
                      const float* U, double beta1, float* delta) {
  const float w1 = (float)(1.0 - beta1);
  decode_m(mkind, m, m_scale, n, rows, block, delta);
  if (mkind == KO_M_BF16) {
    /* _FloatCodec: the EMA runs in the stored dtype (bf16 lerp: fp32 math, bf16 rounding) */
    for (int64_t i = 0; i < n; ++i) delta[i] = rbf16(ko_lerp(delta[i], rbf16(U[i]), w1));
  } else {
#pragma omp parallel for schedule(static)
    for (int64_t i = 0; i < n; ++i) delta[i] = ko_lerp(delta[i], U[i], w1);
  }
  encode_m(mkind, delta, n, rows, block, m, m_scale);
}

/* adakaon.py:840-906 (factored), :908-966 (1-D), :968-1014 (per-param), one tensor.
 * stat_a = row[R] (factored) or v[n] (1-D);  stat_b = col[C] (factored only). */
int ko_adakaon_step(void* p, const void* g, int dtype, int64_t n, int64_t rows, int mkind, void* m,
                    float* m_scale, int64_t block, float* stat_a, float* stat_b, double lr,
                    double beta1, double beta2, double eps1, double wd, double clip, int cautious,
                    int gc, int method, uint64_t seed, uint32_t step, uint32_t tensor_id,
                    const uint16_t* noise, int64_t* kept_out, float* rms_out) {
  float* G = (float*)malloc((size_t)n * 4);
  float* U = (float*)malloc((size_t)n * 4);
  float* D = (float*)malloc((size_t)n * 4);
  if (!G || !U || !D) return 1;
  if (gc && rows > 0) ko_centralize(g, dtype, rows, n / rows, G);
  else
    for (int64_t i = 0; i < n; ++i) G[i] = ld(g, dtype, i);
  if (rows > 0) factored_update(G, rows, n / rows, stat_a, stat_b, beta2, eps1, clip, lr, U, rms_out);
  else flat_update(G, n, stat_a, beta2, eps1, clip, lr, U, rms_out);
  if (beta1 > 0) codec_ema(mkind, m, m_scale, n, rows, block, U, beta1, D);
  else memcpy(D, U, (size_t)n * 4);
  if (wd != 0.0) {
    const float a = (float)(lr * wd);
#pragma omp parallel for schedule(static)
    for (int64_t i = 0; i < n; ++i) D[i] = fmaf(ld(p, dtype, i), a, D[i]);
  }
  int64_t kept = -1;
  if (cautious) kept = ko_cautious(D, G, n);
  if (kept_out) *kept_out = kept;
  ko_write(p, dtype, D, n, -1.0f, method, seed, step, tensor_id, 0u, noise);
  free(G); free(U); free(D);
  return 0;
}

/* ------------------------------------------------------------------ a9: Nekaon climb / removal */

/* msam.py:201-235 with norm="none":  e = clamp(nan_to_num(decode(m_stored) * f32(sign*rho)), +-bound),
 * bound = f32(|rho| * clip_threshold * lr) frozen at climb time (msam.py:169-188);  p += e
 * (fp32: plain add; bf16: stochastic rounding, msam.py:231-235). */
int ko_msam_apply(void* p, int dtype, int64_t n, int64_t rows, int mkind, const void* m,
                  const float* m_scale, int64_t block, double alpha, double bound, int method,
                  uint64_t seed, uint32_t step, uint32_t tensor_id, uint32_t tag,
                  const uint16_t* noise) {
  float* E = (float*)malloc((size_t)n * 4);
  if (!E) return 1;
  decode_m(mkind, m, m_scale, n, rows, block, E);
  const float a = (float)alpha, b = (float)bound;
#pragma omp parallel for schedule(static)
  for (int64_t i = 0; i < n; ++i) {
    float e = E[i] * a;
    if (isnan(e)) e = 0.0f;
    e = fminf(fmaxf(e, -b), b);
    E[i] = e;
  }
  if (dtype == KO_F32) {
    float* pf = (float*)p;
    for (int64_t i = 0; i < n; ++i) pf[i] = pf[i] + E[i];
  } else {
    ko_write(p, dtype, E, n, 1.0f, method == KO_W_SR_NOISE ? KO_W_SR_NOISE : KO_W_SR, seed, step,
             tensor_id, tag, noise);
  }
  free(E);
  return 0;
}

/* ------------------------------------------------------------------ a10: Newton–Schulz */

/* C[MxN] = bf16( A[MxK] * B^T[NxK] ) with fp32-valued bf16 inputs, double accumulate. */
static void gemm_nt_bf16(const float* A, const float* B, int64_t M, int64_t N, int64_t K, float* C) {
#pragma omp parallel for schedule(static)
  for (int64_t i = 0; i < M; ++i)
    for (int64_t j = 0; j < N; ++j) {
      double s = 0.0;
      for (int64_t k = 0; k < K; ++k) s += (double)A[i * K + k] * (double)B[j * K + k];
      C[i * N + j] = rbf16((float)s);
    }
}

/* adamuon.py:97-118.  Every intermediate is a bf16 tensor (values held here as bf16-representable
 * floats).  in: M_in[R*C] fp32; out: O[R*C] = fp32 view of the bf16 result. */
int ko_newton_schulz(const float* M_in, int64_t R, int64_t C, int steps, float* O) {
  const float a = 3.4445f, b = -4.7750f, c = 2.0315f;
  int transposed = R > C;
  int64_t r = transposed ? C : R, k = transposed ? R : C; /* x is [r, k], r <= k */
  float* X = (float*)malloc((size_t)(r * k) * 4);
  float* Xt = (float*)malloc((size_t)(r * k) * 4);
  float* A = (float*)malloc((size_t)(r * r) * 4);
  float* A2 = (float*)malloc((size_t)(r * r) * 4);
  float* Bm = (float*)malloc((size_t)(r * r) * 4);
  float* BX = (float*)malloc((size_t)(r * k) * 4);
  if (!X || !Xt || !A || !A2 || !Bm || !BX) return 1;
  double ss = 0.0;
  for (int64_t i = 0; i < R; ++i)
    for (int64_t j = 0; j < C; ++j) {
      float v = rbf16(M_in[i * C + j]);
      if (transposed) X[j * k + i] = v; else X[i * k + j] = v;
      ss += (double)v * (double)v;
    }
  float nrm = rbf16((float)sqrt(ss));       /* x.norm() is a bf16 scalar */
  float den = rbf16(nrm + 1e-7f);           /* bf16 + python float -> bf16 */
  for (int64_t i = 0; i < r * k; ++i) X[i] = rbf16(X[i] / den);
  for (int s = 0; s < steps; ++s) {
    gemm_nt_bf16(X, X, r, r, k, A);          /* aa = x @ x.mT */
    for (int64_t i = 0; i < r; ++i)           /* aa @ aa as written (not aa @ aa.mT): feed A^T as the NT operand */
      for (int64_t j = 0; j < r; ++j) Bm[j * r + i] = A[i * r + j];
    gemm_nt_bf16(A, Bm, r, r, r, A2);
    for (int64_t i = 0; i < r * r; ++i) Bm[i] = rbf16(rbf16(b * A[i]) + rbf16(c * A2[i]));
    for (int64_t i = 0; i < r; ++i)
      for (int64_t j = 0; j < k; ++j) Xt[j * r + i] = X[i * k + j];
    gemm_nt_bf16(Bm, Xt, r, k, r, BX);       /* bb @ x */
    for (int64_t i = 0; i < r * k; ++i) X[i] = rbf16(rbf16(a * X[i]) + BX[i]);
  }
  for (int64_t i = 0; i < R; ++i)
    for (int64_t j = 0; j < C; ++j) O[i * C + j] = transposed ? X[j * k + i] : X[i * k + j];
  free(X); free(Xt); free(A); free(A2); free(Bm); free(BX);
  return 0;
}

/* ------------------------------------------------------------------ a11: AdaMuon */

/* adamuon.py:434-501 / 557-615 (one tensor).  ndim>=2: m = EMA of the raw grad (codec), O = NS(m_fp32
 * pre-requant), factored second moment of O, clip, scale 0.2*lr, wd, cautious against the raw grad.
 * 1-D: Adam-style like Adakaon's flat branch scaled by 0.2*lr, momentum of the update.
 * ns_in (optional, may be NULL): if given, receives the fp32 momentum fed to NS; ns_override
 * (optional): if given, used INSTEAD of running NS here (lets a test feed another NS result). */
int ko_adamuon_step(void* p, const void* g, int dtype, int64_t n, int64_t rows, int mkind, void* m,
                    float* m_scale, int64_t block, float* stat_a, float* stat_b, double lr,
                    double beta1, double beta2, double eps1, double wd, double clip, int ns_steps,
                    int cautious, int gc, int method, uint64_t seed, uint32_t step,
                    uint32_t tensor_id, const uint16_t* noise, float* ns_in,
                    const float* ns_override) {
  float* G = (float*)malloc((size_t)n * 4);
  float* U = (float*)malloc((size_t)n * 4);
  float* D = (float*)malloc((size_t)n * 4);
  if (!G || !U || !D) return 1;
  if (gc && rows > 0) ko_centralize(g, dtype, rows, n / rows, G);
  else
    for (int64_t i = 0; i < n; ++i) G[i] = ld(g, dtype, i);
  const double scale = 0.2 * lr;
  if (rows > 0) {
    int64_t R = rows, C = n / rows;
    if (beta1 > 0) codec_ema(mkind, m, m_scale, n, rows, block, G, beta1, D);
    else memcpy(D, G, (size_t)n * 4);
    if (ns_in) memcpy(ns_in, D, (size_t)n * 4);
    float* O = (float*)malloc((size_t)n * 4);
    if (ns_override) memcpy(O, ns_override, (size_t)n * 4);
    else ko_newton_schulz(D, R, C, ns_steps, O);
    factored_update(O, R, C, stat_a, stat_b, beta2, eps1, clip, scale, D, NULL);
    free(O);
  } else {
    flat_update(G, n, stat_a, beta2, eps1, clip, scale, U, NULL);
    if (beta1 > 0) codec_ema(mkind, m, m_scale, n, rows, block, U, beta1, D);
    else memcpy(D, U, (size_t)n * 4);
  }
  if (wd != 0.0) {
    const float a = (float)(lr * wd);
    for (int64_t i = 0; i < n; ++i) D[i] = fmaf(ld(p, dtype, i), a, D[i]);
  }
  if (cautious) ko_cautious(D, G, n);
  ko_write(p, dtype, D, n, -1.0f, method, seed, step, tensor_id, 0u, noise);
  free(G); free(U); free(D);
  return 0;
}

/* ------------------------------------------------------------------ AdaPNM (two momenta) */

/* adapnm.py:1209-1273 (per-param) = :1069-1172 (foreach), one tensor; coefficients adapnm.py:998-1017.
 * pos / neg are the two stored momenta in the roles of THIS step (adapnm.py:588-596: "m_pos" is positive
 * on odd steps).  t is the group's 1-based step.  stat_a = row[R] or v[n]; stat_b = col[C]; max_v only
 * with ams_bound on a 1-D tensor.
 *   p *= f32(1 - lr*wd)                                   (before the moments; bf16: rounded to bf16)
 *   factored: row/col EMA of g^2 (+eps);  inv = (rf*cf) * f32(sqrt(1-b2^t))
 *   1-D:      v = fma(f32(1-b2)*g, g, v*f32(b2));  den = (sqrt(max_v|v + 1e-15) + f32(eps)) / f32(bc2_sq)
 *   pos = fma(g, f32(1-b1^2), pos*f32(b1^2));  store pos through the codec
 *   pn  = fma(neg, f32(-b0), pos*f32(1+b0)) * f32(1/noise_norm)
 *   u   = pn*inv (factored) | pn/den (1-D);  u /= max(rms(u)/f32(clip), 1) if clip > 0
 *   delta = u * f32(lr/bc1);  cautious against g;  p -= delta */
int ko_adapnm_step(void* p, const void* g, int dtype, int64_t n, int64_t rows, int mkind, void* pos,
                   float* pos_scale, const void* neg, const float* neg_scale, int64_t block,
                   float* stat_a, float* stat_b, float* max_v, double lr, double beta1, double beta2,
                   double beta0, double eps, double wd, double clip, int cautious, int gc, int ams,
                   int method, uint32_t t, uint64_t seed, uint32_t step, uint32_t tensor_id,
                   const uint16_t* noise, int64_t* kept_out, float* rms_out) {
  float* G = (float*)malloc((size_t)n * 4);
  float* MP = (float*)malloc((size_t)n * 4);
  float* MN = (float*)malloc((size_t)n * 4);
  float* U = (float*)malloc((size_t)n * 4);
  if (!G || !MP || !MN || !U) return 1;
  if (gc && rows > 0) ko_centralize(g, dtype, rows, n / rows, G);
  else
    for (int64_t i = 0; i < n; ++i) G[i] = ld(g, dtype, i);
  const double b1sq = beta1 * beta1;
  const double noise_norm = sqrt((1.0 + beta0) * (1.0 + beta0) + beta0 * beta0);
  const double bc1 = 1.0 - pow(beta1, (double)t);
  const double bc2_sq = sqrt(1.0 - pow(beta2, (double)t));
  const float f_bc2 = (float)bc2_sq, f_step = (float)(lr / bc1);
  if (wd != 0.0) {
    const float sc = (float)(1.0 - lr * wd);
    if (dtype == KO_F32) {
      float* pf = (float*)p;
      for (int64_t i = 0; i < n; ++i) pf[i] = pf[i] * sc;
    } else {
      uint16_t* pb = (uint16_t*)p;
      for (int64_t i = 0; i < n; ++i) pb[i] = f32_to_bf16(bf16_to_f32(pb[i]) * sc);
    }
  }
  /* momenta: read both, EMA the positive one with the raw gradient, store it */
  decode_m(mkind, pos, pos_scale, n, rows, block, MP);
  decode_m(mkind, neg, neg_scale, n, rows, block, MN);
  {
    const float fb = (float)b1sq, fw = (float)(1.0 - b1sq);
#pragma omp parallel for schedule(static)
    for (int64_t i = 0; i < n; ++i) MP[i] = fmaf(G[i], fw, MP[i] * fb);
  }
  encode_m(mkind, MP, n, rows, block, pos, pos_scale);
  {
    const float c1 = (float)(1.0 + beta0), c2 = (float)(-beta0), c3 = (float)(1.0 / noise_norm);
#pragma omp parallel for schedule(static)
    for (int64_t i = 0; i < n; ++i) MP[i] = fmaf(MN[i], c2, MP[i] * c1) * c3;
  }
  if (rows > 0) {
    const int64_t R = rows, C = n / rows;
    const float w2 = (float)(1.0 - beta2), e1 = (float)eps;
    double* colsum = (double*)calloc((size_t)C, 8);
    for (int64_t r = 0; r < R; ++r) {
      double s = 0.0;
      for (int64_t c = 0; c < C; ++c) {
        float sq = G[r * C + c] * G[r * C + c];
        if (eps > 0) sq = sq + e1;
        s += (double)sq;
        colsum[c] += (double)sq;
      }
      stat_a[r] = ko_lerp(stat_a[r], (float)s / (float)C, w2);
    }
    for (int64_t c = 0; c < C; ++c) stat_b[c] = ko_lerp(stat_b[c], (float)colsum[c] / (float)R, w2);
    free(colsum);
    double rs = 0.0;
    for (int64_t r = 0; r < R; ++r) rs += (double)stat_a[r];
    const float rowmean = (float)rs / (float)R;
    float* rf = (float*)malloc((size_t)R * 4);
    float* cf = (float*)malloc((size_t)C * 4);
    for (int64_t r = 0; r < R; ++r) rf[r] = 1.0f / sqrtf(stat_a[r] / rowmean);
    for (int64_t c = 0; c < C; ++c) cf[c] = 1.0f / sqrtf(stat_b[c]);
#pragma omp parallel for schedule(static)
    for (int64_t r = 0; r < R; ++r)
      for (int64_t c = 0; c < C; ++c) U[r * C + c] = MP[r * C + c] * ((rf[r] * cf[c]) * f_bc2);
    free(rf); free(cf);
  } else {
    const float fb2 = (float)beta2, fw2 = (float)(1.0 - beta2), fe = (float)eps;
    for (int64_t i = 0; i < n; ++i) {
      float v = fmaf(fw2 * G[i], G[i], stat_a[i] * fb2);
      stat_a[i] = v;
      if (ams) {
        max_v[i] = fmaxf(max_v[i], v);
        v = max_v[i];
      }
      float den = sqrtf(v + 1e-15f) + fe;
      den = den / f_bc2;
      U[i] = MP[i] / den;
    }
  }
  double ss = 0.0;
#pragma omp parallel for reduction(+ : ss) schedule(static)
  for (int64_t i = 0; i < n; ++i) ss += (double)U[i] * (double)U[i];
  const float rms = (float)sqrt(ss) / (float)sqrt((double)(n > 0 ? n : 1));
  if (rms_out) *rms_out = rms;
  const float divisor = clip > 0.0 ? fmaxf(rms / (float)clip, 1.0f) : 1.0f;
#pragma omp parallel for schedule(static)
  for (int64_t i = 0; i < n; ++i) U[i] = (clip > 0.0 ? U[i] / divisor : U[i]) * f_step;
  int64_t kept = -1;
  if (cautious) kept = ko_cautious(U, G, n);
  if (kept_out) *kept_out = kept;
  ko_write(p, dtype, U, n, -1.0f, method, seed, step, tensor_id, 0u, noise);
  free(G); free(MP); free(MN); free(U);
  return 0;
}

/* ------------------------------------------------------------------ KProdigy (two passes around the distance estimate d) */

/* Pass 1 of one tensor, kprodigy.py:417-478 (= :482-703 batched): the D statistics on every slice_p-th
 * element, the d-scaled momentum EMA, the second-moment EMA.
 *   g <- centralize(g) if gc and ndim>=2;  g <- fma(p, f32(wd), g) for coupled weight decay
 *   do_d:  num = sum(g_i * (p0_i - p_i));  s_i = fma(g_i, f32(alpha_s), s_i*f32(beta3));  den = sum|s_i|
 *   momentum (kprodigy.py:762-782): int8 / fp32: fma(g, f32(d*(1-b1)), m*f32(b1)); bf16: the same two
 *     steps in bf16 (each result rounded to bf16, the gradient and the weight d*(1-b1) cast to bf16
 *     first, the decay b1 not); 4-bit: the codec's
 *     lerp(m, g*f32(d), f32(1-b1)) (g itself when d == 1)
 *   second moment: full  v = fma(f32(d*d*(1-b2))*g, g, v*f32(b2));  factored: Adakaon's row/col EMA of
 *     g^2 + eps_factored (no d in it)
 * p0 == NULL stands for the zero reference point (kprodigy.py:277-280). */
int ko_kprodigy_pass1(const void* p, const void* g, int dtype, int64_t n, int64_t rows, int mkind, void* m,
                      float* m_scale, int64_t block, float* stat_a, float* stat_b, int factored, float* s,
                      const float* p0, int64_t slice_p, int do_d, double beta1, double beta2, double beta3,
                      double d, double alpha_s, double wd_coupled, double eps_factored, int gc,
                      float* num_out, float* den_out) {
  float* G = (float*)malloc((size_t)n * 4);
  float* M = (float*)malloc((size_t)n * 4);
  if (!G || !M) return 1;
  if (gc && rows > 0) ko_centralize(g, dtype, rows, n / rows, G);
  else
    for (int64_t i = 0; i < n; ++i) G[i] = ld(g, dtype, i);
  if (wd_coupled != 0.0) {
    const float fw = (float)wd_coupled;
    for (int64_t i = 0; i < n; ++i) G[i] = fmaf(ld(p, dtype, i), fw, G[i]);
  }
  if (do_d) {
    const float fb3 = (float)beta3, fa = (float)alpha_s;
    double num = 0.0, den = 0.0;
    for (int64_t i = 0, j = 0; i < n; i += slice_p, ++j) {
      const float pr = p0 ? p0[j] : 0.0f;
      num += (double)(G[i] * (pr - ld(p, dtype, i)));
      s[j] = fmaf(G[i], fa, s[j] * fb3);
      den += (double)fabsf(s[j]);
    }
    if (num_out) *num_out = (float)num;
    if (den_out) *den_out = (float)den;
  }
  if (beta1 > 0) {
    const float fb1 = (float)beta1, ft = (float)(d * (1.0 - beta1));
    if (mkind == KO_M_4BIT) {
      const float fd = (float)d;
      if (d != 1.0)
        for (int64_t i = 0; i < n; ++i) M[i] = G[i] * fd;
      else memcpy(M, G, (size_t)n * 4);
      float* D = (float*)malloc((size_t)n * 4);
      codec_ema(mkind, m, m_scale, n, rows, block, M, beta1, D);
      free(D);
    } else if (mkind == KO_M_BF16) {
      uint16_t* mb = (uint16_t*)m;
      const float ftb = rbf16(ft);  /* add_'s alpha is cast to the tensor's dtype, mul_'s scalar is not */
      for (int64_t i = 0; i < n; ++i) {
        const float a = rbf16(bf16_to_f32(mb[i]) * fb1);
        mb[i] = f32_to_bf16(fmaf(rbf16(G[i]), ftb, a));
      }
    } else {
      decode_m(mkind, m, m_scale, n, rows, block, M);
      for (int64_t i = 0; i < n; ++i) M[i] = fmaf(G[i], ft, M[i] * fb1);
      encode_m(mkind, M, n, rows, block, m, m_scale);
    }
  }
  if (!factored || rows <= 0) {
    const float fb2 = (float)beta2, fv = (float)(d * d * (1.0 - beta2));
    for (int64_t i = 0; i < n; ++i) stat_a[i] = fmaf(fv * G[i], G[i], stat_a[i] * fb2);
  } else {
    const int64_t R = rows, C = n / rows;
    const float w2 = (float)(1.0 - beta2), e1 = (float)eps_factored;
    double* colsum = (double*)calloc((size_t)C, 8);
    for (int64_t r = 0; r < R; ++r) {
      double rs = 0.0;
      for (int64_t c = 0; c < C; ++c) {
        float sq = G[r * C + c] * G[r * C + c];
        if (eps_factored > 0) sq = sq + e1;
        rs += (double)sq;
        colsum[c] += (double)sq;
      }
      stat_a[r] = ko_lerp(stat_a[r], (float)rs / (float)C, w2);
    }
    for (int64_t c = 0; c < C; ++c) stat_b[c] = ko_lerp(stat_b[c], (float)colsum[c] / (float)R, w2);
    free(colsum);
  }
  free(G); free(M);
  return 0;
}

/* Pass 2 of one tensor, kprodigy.py:800-840 (= :889-949 batched).  dlr is the one of the top of the step; d is
 * the estimate as just updated (kprodigy.py:379-403 reassigns it before the call):
 *   numer = decode(m as stored by pass 1) (beta1 > 0) or g
 *   full:     delta = numer / max(sqrt(v), f32(d*eps))
 *   factored: delta = numer * min((rf*cf) / f32(d), f32(1/(d*eps)))
 *   delta *= f32(dlr);  delta = fma(p, f32(decay*dlr), delta) (decoupled decay);  cautious against g;  p -= delta */
int ko_kprodigy_pass2(void* p, const void* g, int dtype, int64_t n, int64_t rows, int mkind, const void* m,
                      const float* m_scale, int64_t block, const float* stat_a, const float* stat_b,
                      int factored, int has_m, double d, double dlr, double eps, double decay_dlr, int cautious,
                      int gc, int method, uint64_t seed, uint32_t step, uint32_t tensor_id,
                      const uint16_t* noise, int64_t* kept_out) {
  float* G = (float*)malloc((size_t)n * 4);
  float* D = (float*)malloc((size_t)n * 4);
  if (!G || !D) return 1;
  if (gc && rows > 0) ko_centralize(g, dtype, rows, n / rows, G);
  else
    for (int64_t i = 0; i < n; ++i) G[i] = ld(g, dtype, i);
  if (has_m) decode_m(mkind, m, m_scale, n, rows, block, D);
  else memcpy(D, G, (size_t)n * 4);
  const float fd = (float)d, fdlr = (float)dlr;
  if (!factored || rows <= 0) {
    const float floor_ = (float)(d * eps);
    for (int64_t i = 0; i < n; ++i) D[i] = (D[i] / fmaxf(sqrtf(stat_a[i]), floor_)) * fdlr;
  } else {
    const int64_t R = rows, C = n / rows;
    double rs = 0.0;
    for (int64_t r = 0; r < R; ++r) rs += (double)stat_a[r];
    const float rowmean = (float)rs / (float)R;
    const float cap = (float)(1.0 / (d * eps));
    for (int64_t r = 0; r < R; ++r) {
      const float rf = 1.0f / sqrtf(stat_a[r] / rowmean);
      for (int64_t c = 0; c < C; ++c) {
        const float inv = fminf((rf * (1.0f / sqrtf(stat_b[c]))) / fd, cap);
        D[r * C + c] = (D[r * C + c] * inv) * fdlr;
      }
    }
  }
  if (decay_dlr != 0.0) {
    const float a = (float)decay_dlr;
    for (int64_t i = 0; i < n; ++i) D[i] = fmaf(ld(p, dtype, i), a, D[i]);
  }
  int64_t kept = -1;
  if (cautious) kept = ko_cautious(D, G, n);
  if (kept_out) *kept_out = kept;
  ko_write(p, dtype, D, n, -1.0f, method, seed, step, tensor_id, 0u, noise);
  free(G); free(D);
  return 0;
}

int ko_version(void) { return 1; }
