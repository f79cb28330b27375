// Building blocks of the warp sweeps: eight consecutive elements a lane and trip, packed pairs, rows a multiple of eight
// elements, 4-bit blocks of 128 (so half a warp shares a scale).  Used by Lion, the Adakaon family, AdaMuon's EMA, AdaPNM
// and KProdigy.
#pragma once

#include <cuda_bf16.h>

#include "kaon_device.cuh"
#include "kaon_elem.cuh"
#include "kaon_ops.cuh"
#include "kaon_packed.cuh"

namespace kaon {

// The cautious mask of one element as a factor: x > 0 (x < 0) as 1.0f / 0.0f in one instruction, by comparison, so that a
// product in the subnormal range decides like any other.  A NaN gives 0.
__device__ __forceinline__ float gt0(float x) {
  float r;
  asm("set.gt.f32.f32 %0, %1, 0f00000000;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float lt0(float x) {
  float r;
  asm("set.lt.f32.f32 %0, %1, 0f00000000;" : "=f"(r) : "f"(x));
  return r;
}

// gt0, or 1.0f where `off`
__device__ __forceinline__ float gt0_or(float x, int off) {
  float r;
  asm("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %2, 0;\n\tset.gt.or.f32.f32 %0, %1, 0f00000000, p;\n\t}" : "=f"(r) : "f"(x), "r"(off));
  return r;
}

// Philox with the round keys from the host (HP: a hyper-parameter block with `step`, `rk0`, `rk1`)
template <typename HP>
__device__ __forceinline__ void philox8(const HP& hp, uint32_t tensor, uint64_t q, uint32_t tag, uint32_t out[4]) {
  uint32_t c0 = (uint32_t)q, c1 = tensor, c2 = hp.step, c3 = tag | ((uint32_t)(q >> 32) << 8);
#pragma unroll
  for (int r = 0; r < KAON_PHILOX_ROUNDS; ++r) {
    const unsigned long long p0 = (unsigned long long)0xD2511F53u * c0;
    const unsigned long long p1 = (unsigned long long)0xCD9E8D57u * c2;
    const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c1 ^ hp.rk0[r];
    const uint32_t n2 = (uint32_t)(p0 >> 32) ^ c3 ^ hp.rk1[r];
    c1 = (uint32_t)p1;
    c3 = (uint32_t)p0;
    c0 = n0;
    c2 = n2;
  }
  out[0] = c0; out[1] = c1; out[2] = c2; out[3] = c3;
}

// Eight weights on their way through a step: bf16 stays packed between the writes (four registers, not eight).
template <typename PT>
struct W8;

template <>
struct W8<__nv_bfloat16> {
  uint32_t w[4];
  __device__ __forceinline__ void load(const void* p) {
    const uint4 q = *reinterpret_cast<const uint4*>(p);
    w[0] = q.x; w[1] = q.y; w[2] = q.z; w[3] = q.w;
  }
  __device__ __forceinline__ f32x2 pair(int j) const { return pack2(bf16lo(w[j]), bf16hi(w[j])); }
  // stochastic rounding of w + D: 16 noise bits (the halves of nz[j], added by one dot-product instruction each) below
  // the kept mantissa
  __device__ __forceinline__ void add_sr(const f32x2 D[4], const uint32_t nz[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const f32x2 r = add2(pair(j), D[j]);
      w[j] = prmt(__dp2a_lo(nz[j], 0x00000001u, __float_as_uint(r.x)), __dp2a_lo(nz[j], 0x00000100u, __float_as_uint(r.y)), 0x7632u);
    }
  }
  __device__ __forceinline__ void set(int j, f32x2 v) { w[j] = prmt(__float_as_uint(v.x), __float_as_uint(v.y), 0x7632u); }
  __device__ __forceinline__ void store(void* p, const Peers* pr) const {
    const uint4 q = make_uint4(w[0], w[1], w[2], w[3]);
    *reinterpret_cast<uint4*>(p) = q;
    mirror16(pr, p, q);
  }
};

template <>
struct W8<float> {
  f32x2 v[4];
  __device__ __forceinline__ void load(const void* p) {
    const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    v[0] = pack2(a.x, a.y); v[1] = pack2(a.z, a.w); v[2] = pack2(b.x, b.y); v[3] = pack2(b.z, b.w);
  }
  __device__ __forceinline__ f32x2 pair(int j) const { return v[j]; }
  __device__ __forceinline__ void set(int j, f32x2 x) { v[j] = x; }
  __device__ __forceinline__ void store(void* p, const Peers* pr) const {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      unsigned char* a = reinterpret_cast<unsigned char*>(p) + 16 * h;
      const uint4 q = make_uint4(__float_as_uint(v[2 * h].x), __float_as_uint(v[2 * h].y),
                                 __float_as_uint(v[2 * h + 1].x), __float_as_uint(v[2 * h + 1].y));
      *reinterpret_cast<uint4*>(a) = q;
      mirror16(pr, a, q);
    }
  }
};

// x less a row mean (bits as the row table holds them; 0 without centralization), rounded to x's dtype
template <typename T>
__device__ __forceinline__ void center(const W8<T>& x, float mu, f32x2 out[4]) {
  if constexpr (Elems<T>::IS_BF16) {
    const uint32_t m2 = __float_as_uint(mu);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t w = sub_bf16x2(x.w[j], m2);
      out[j] = pack2(bf16lo(w), bf16hi(w));
    }
  } else {
    const f32x2 M = pack2(mu, mu);
#pragma unroll
    for (int j = 0; j < 4; ++j) out[j] = sub2(x.pair(j), M);
  }
}

// The stored momentum of eight elements as it lies in memory.
template <int MK> struct MRaw { };
template <> struct MRaw<KAON_M_4BIT> {
  uint32_t w;
  float sc;
  __device__ __forceinline__ void load(const void* p) { w = *reinterpret_cast<const uint32_t*>(p); }
  // nibble n as the float 2^23 + n by a byte permute, less 2^23 + 8
  __device__ __forceinline__ void decode(float scale, f32x2 M[4]) const {
    const uint32_t wl = w & 0x0F0F0F0Fu, wh = (w >> 4) & 0x0F0F0F0Fu;
    const f32x2 BIAS = pack2(-8388616.0f, -8388616.0f), SC = pack2(scale, scale);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      M[j] = mul2(add2(pack2(__uint_as_float(prmt(wl, 0x4B000000u, 0x7540u | (uint32_t)j)),
                             __uint_as_float(prmt(wh, 0x4B000000u, 0x7540u | (uint32_t)j))), BIAS), SC);
  }
};
template <> struct MRaw<KAON_M_INT8> {
  uint2 w;
  __device__ __forceinline__ void load(const void* p) { w = *reinterpret_cast<const uint2*>(p); }
  __device__ __forceinline__ void decode(float scale, f32x2 M[4]) const {
    const uint32_t x0 = w.x ^ 0x80808080u, x1 = w.y ^ 0x80808080u;  // code + 128 in every byte
    const f32x2 BIAS = pack2(-8388736.0f, -8388736.0f), SC = pack2(scale, scale);   // -(2^23 + 128)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t x = j < 2 ? x0 : x1;
      const uint32_t b = (uint32_t)(2 * (j & 1));
      M[j] = mul2(add2(pack2(__uint_as_float(prmt(x, 0x4B000000u, 0x7540u | b)),
                             __uint_as_float(prmt(x, 0x4B000000u, 0x7540u | (b + 1u)))), BIAS), SC);
    }
  }
};
template <typename T> struct MPlain {
  W8<T> w;
  __device__ __forceinline__ void load(const void* p) { w.load(p); }
  __device__ __forceinline__ void decode(float, f32x2 M[4]) const {
#pragma unroll
    for (int j = 0; j < 4; ++j) M[j] = w.pair(j);
  }
};
template <> struct MRaw<KAON_M_BF16> : MPlain<__nv_bfloat16> { };
template <> struct MRaw<KAON_M_F32> : MPlain<float> { };

// bytes of eight stored momenta
template <int MK> struct MBytes { static constexpr int V = MK == KAON_M_4BIT ? 4 : MK == KAON_M_INT8 ? 8 : MK == KAON_M_BF16 ? 16 : MK == KAON_M_F32 ? 32 : 0; };

__device__ __forceinline__ float amax8(const f32x2 M[4]) {
  float a = max3f(fabsf(M[0].x), fabsf(M[0].y), fabsf(M[1].x));
  a = max3f(a, fabsf(M[1].y), fabsf(M[2].x));
  a = max3f(a, fabsf(M[2].y), fabsf(M[3].x));
  return fmaxf(a, fabsf(M[3].y));
}

// Store eight new momenta at mp (every lane of the warp calls it; `cnt` of the lane's exist, 0..8, M is 0 beyond an odd end).  bf16 momentum is
// already rounded in M.  `amax`: int8 only, the finished maximum of the row; returns the scale (4-bit: the block's,
// to be stored by the first lane of a half warp).  Codes are rounded from m' / scale by an approximate reciprocal (within an
// ulp) and one correction with the exact residual: the correctly rounded quotient but where m' / scale lies within
// 2^-21 ulp of the middle between two floats.
// `stored`, where given: the momenta as they were stored.
template <int MK>
__device__ __forceinline__ float store_m8(void* mp, const f32x2 M[4], float amax, const int cnt, const int lane, f32x2* stored = nullptr) {
  if constexpr (MK == KAON_M_4BIT || MK == KAON_M_INT8) {
    float sc;
    if constexpr (MK == KAON_M_4BIT) sc = div7_exact(fmaxf(half_warp_max(cnt > 0 ? amax8(M) : 0.0f, lane), 1e-12f));
    else sc = div127_exact(fmaxf(amax, 1e-12f));
    float inv;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(sc));
    constexpr float MAGIC = MK == KAON_M_4BIT ? 12582920.0f : 12582912.0f;   // 1.5 * 2^23 (+ 8)
    const f32x2 INV = pack2(inv, inv), MG = pack2(MAGIC, MAGIC), NSC = pack2(-sc, -sc);
    f32x2 R[4];   // rint(m'/sc) + magic
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const f32x2 qq = mul2(M[j], INV);
      R[j] = add2(fma2(fma2(qq, NSC, M[j]), INV, qq), MG);
    }
    f32x2 T[4];   // -rint(m'/sc)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      T[j] = sub2(MG, R[j]);
      if (stored) stored[j] = mul2(T[j], NSC);
    }
    if constexpr (MK == KAON_M_4BIT) {
      // sum_k (8 - t_k) 16^k = 0x8888 - (t0 + 16 t1 + 256 t2 + 4096 t3), exact in fp32; adding 2^23 leaves it in the low
      // 16 mantissa bits
      const f32x2 K256 = pack2(256.0f, 256.0f);
      const f32x2 Xl = fma2(T[1], K256, T[0]), Yl = fma2(T[3], K256, T[2]);
      const float lo4 = __fsub_rn(8423560.0f, __fmaf_rn(Xl.y, 16.0f, Xl.x));
      const float hi4 = __fsub_rn(8423560.0f, __fmaf_rn(Yl.y, 16.0f, Yl.x));
      const uint32_t w = prmt(__float_as_uint(lo4), __float_as_uint(hi4), 0x5410u);
      if (cnt == 8) stg_u32(mp, w);
      else
        for (int b = 0; 2 * b < cnt; ++b)
          reinterpret_cast<unsigned char*>(mp)[b] = (unsigned char)((w >> (8 * b)) & (2 * b + 1 < cnt ? 0xffu : 0xfu));
    } else if (cnt > 0) {  // the low byte of every R is the code in two's complement
      const uint32_t w0 = prmt(prmt(__float_as_uint(R[0].x), __float_as_uint(R[0].y), 0x0040u),
                               prmt(__float_as_uint(R[1].x), __float_as_uint(R[1].y), 0x0040u), 0x5410u);
      const uint32_t w1 = prmt(prmt(__float_as_uint(R[2].x), __float_as_uint(R[2].y), 0x0040u),
                               prmt(__float_as_uint(R[3].x), __float_as_uint(R[3].y), 0x0040u), 0x5410u);
      *reinterpret_cast<uint2*>(mp) = make_uint2(w0, w1);   // (int8 rows are whole vectors)
    }
    return sc;
  } else {
    MRaw<MK> o;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      o.w.set(j, M[j]);
      if (stored) stored[j] = M[j];
    }
    if (cnt == 8) o.w.store(mp, nullptr);
    else
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k < cnt) {
          const float x = k & 1 ? M[k >> 1].y : M[k >> 1].x;
          if constexpr (MK == KAON_M_BF16) reinterpret_cast<uint16_t*>(mp)[k] = (uint16_t)(__float_as_uint(x) >> 16);
          else reinterpret_cast<float*>(mp)[k] = x;
        }
    return 1.0f;
  }
}

// p <- p + D: bf16 by stochastic rounding, fp32 as is
template <typename PT, typename HP>
__device__ __forceinline__ void add_noisy8(const HP& hp, const DevTensor& d, uint64_t q, uint32_t tag, W8<PT>& P, const f32x2 D[4]) {
  if constexpr (Elems<PT>::IS_BF16) {
    uint32_t nz[4];
    philox8(hp, d.tensor_id, q, tag, nz);
    P.add_sr(D, nz);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) P.v[j] = add2(P.v[j], D[j]);
  }
}

// The weight write p <- round(p + F) of vector q of a tensor: stochastic, Kahan-compensated or to nearest
template <typename PT, typename HP>
__device__ __forceinline__ void write8(const HP& hp, const DevTensor& d, uint64_t q, const bool act, W8<PT>& P, const f32x2 F[4]) {
  if constexpr (Elems<PT>::IS_BF16) {
    if (hp.sr) {
      add_noisy8(hp, d, q, KAON_TAG_UPDATE, P, F);
    } else if (hp.kahan) {
      unsigned char* she = reinterpret_cast<unsigned char*>(d.shift) + q * 16;
      W8<PT> SH;
      if (act) SH.load(she); else SH.load(d.shift);
#pragma unroll
      for (int j = 0; j < 4; ++j) {   // kahan_step in bf16 arithmetic: 5 instructions a pair for 28
        const uint32_t s1 = add_bf16x2(SH.w[j], pack_bf16_rn(F[j].x, F[j].y));
        const uint32_t pn = add_bf16x2(P.w[j], s1);
        SH.w[j] = add_bf16x2(s1, sub_bf16x2(P.w[j], pn));
        P.w[j] = pn;
      }
      if (act) SH.store(she, nullptr);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) P.w[j] = add_bf16x2(P.w[j], pack_bf16_rn(F[j].x, F[j].y));
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) P.v[j] = add2(P.v[j], F[j]);
  }
}

__device__ __forceinline__ float round_to(float x, __nv_bfloat16) { return round_bf16(x); }
__device__ __forceinline__ float round_to(float x, float) { return x; }

// A lane's part of the sum of a row of whole vectors
template <typename PT>
__device__ __forceinline__ float row_part(const unsigned char* rowp, int C, int lane) {
  f32x2 a = pack2(0.0f, 0.0f), b = pack2(0.0f, 0.0f);
#pragma unroll 4
  for (int v = lane * 8; v < C; v += 256) {
    W8<PT> w;
    w.load(rowp + v * Elems<PT>::BYTES);
    a = add2(a, add2(w.pair(0), w.pair(1)));
    b = add2(b, add2(w.pair(2), w.pair(3)));
  }
  a = add2(a, b);
  return a.x + a.y;
}

// put(i, mean of row r0 + i), i < n, means as the gradient's dtype holds them, by one warp: rows of up to 64 elements a lane
// each, longer ones the whole warp (put is then lane 0's).  g: element 0 of row 0, 16-byte aligned.
template <typename PT, typename Put>
__device__ __forceinline__ void row_means(const unsigned char* g, int C, int r0, int n, int lane, Put out) {
  using E = Elems<PT>;
  const bool vec = (C & 7) == 0;
  const float fC = (float)C, rC = __frcp_rn(fC);
  auto put = [&](int r, float s) { out(r, round_to(div_by(s, fC, rC), PT())); };
  if (C <= 64) {
    for (int r = lane; r < n; r += 32) {
      const unsigned char* rowp = g + (long long)(r0 + r) * C * E::BYTES;
      float s = 0.0f;
      if (vec) {
        f32x2 a = pack2(0.0f, 0.0f);
        for (int v = 0; v < C; v += 8) {
          W8<PT> w;
          w.load(rowp + v * E::BYTES);
          a = add2(a, add2(add2(w.pair(0), w.pair(1)), add2(w.pair(2), w.pair(3))));
        }
        s = a.x + a.y;
      } else {
        for (int i = 0; i < C; ++i) s += E::load1(rowp, i);
      }
      put(r, s);
    }
    return;
  }
  for (int r = 0; r < n; ++r) {
    const unsigned char* rowp = g + (long long)(r0 + r) * C * E::BYTES;
    float s = 0.0f;
    if (vec) {
      s = row_part<PT>(rowp, C, lane);
    } else {
      // whole vectors, and a lane each for the elements before the first and after the last
      const long long e = (long long)(r0 + r) * C, a = (e + 7) / 8 * 8, b = (e + C) / 8 * 8;
      s = row_part<PT>(g + a * E::BYTES, (int)(b - a), lane);
      const long long i = lane < 8 ? e + lane : b + lane - 8;
      if (lane < 8 ? i < a : i < e + C) s += E::load1(g, i);
    }
    s = warp_sum(s);
    if (lane == 0) put(r, s);
  }
}

}  // namespace kaon
