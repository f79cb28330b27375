// AdaPNM (positive-negative momentum over Adakaon's factored second moment) on the plan machinery of
// the Adakaon step.  Replaces reference src/kaon/adapnm.py:1039-1273 (the foreach buckets and the
// per-parameter step).
//
// One step of a plan:
//   1. STATS + FINAL of the Adakaon kernels (row / column statistics of the centralised gradient, the
//      factors r_i = rsqrt(row_i / mean(row)), c_j = rsqrt(col_j), the centralisation means) - the second
//      moment is the same recurrence as Adakaon's (reference src/kaon/_factored.py:26-83).
//   2. SUM: flat units over every factored tensor (a warp's, or items of 16 K for odd row lengths): both momenta are decoded, the positive
//      one takes the gradient, u = pn * ((r*c) * bc2); each leaves its sum of u^2 (double), its count
//      of u*g > 0 and, for int8 momentum, the row maxima of the new positive momentum.
//   3. REDUCE: one CTA per factored tensor adds the partials in order: clip divisor, cautious
//      denominator.
//   4. APPLY: the same units again: recompute, weight decay, clip, mask, weight write, store the
//      positive momentum through its codec.
//   5. FLAT: one CTA per 1-D tensor (full second moment v, optional running maximum) doing 2-4 in place.
// The two stored momenta swap roles every step (reference src/kaon/adapnm.py:588-596); `swap` selects.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include <type_traits>

#include "ada_lists.h"
#include "adakaon_dev.h"
#include "kaon_device.cuh"
#include "kaon_host.h"
#include "kaon_elem.cuh"
#include "kaon_ops.cuh"
#include "kaon_sweep.cuh"

namespace kaon {

constexpr int PNM_ITEM = 16384;
constexpr int PT_THREADS = 256;

struct PnmDev {
  float fb, fw;          // beta1^2, 1 - beta1^2
  float c1, c2, c3;      // 1 + beta0, -beta0, 1 / noise_norm
  float bc2, fstep;      // sqrt(1 - beta2^t), lr / (1 - beta1^t)
  float wdsc;            // 1 - lr * weight_decay
  float fb2, fw2, eps;   // 1-D second moment: beta2, 1 - beta2, eps on the denominator
  float clip;
  int has_wd, clip_on, cautious, gc, ams, sr, kahan, swap;
  uint32_t step, k0, k1;
  uint32_t rk0[KAON_PHILOX_ROUNDS], rk1[KAON_PHILOX_ROUNDS];
};

struct PnmBufs {
  void* m[2];       // stored "m_pos", "m_neg"
  float* sc[2];
  float* max_v;     // 1-D tensors with ams_bound, else null
};

struct PnmView {
  const Task* units;      // warp units of the factored tensors whose rows are a multiple of eight elements
  const Task* items;      // flat items of the other factored tensors
  int n_units, n_items;
  const int* item_begin;  // [n_tensors + 1] ranges of units / items (Task::slot)
  const PnmBufs* bufs;    // [n_tensors]
  double* part;           // [slot] sum of u^2
  unsigned* kpart;        // [slot] count of u*g > 0
  float* scal;            // [n_tensors][2] clip divisor, cautious denominator
  const int* fact;        // indices of the factored tensors
  int n_fact;
  const int* flat;        // indices of the 1-D tensors
  int n_flat;
};

// Weight write of one trip (reference src/kaon/adapnm.py:1090-1092, 1117-1124; _backend.py:82-142).
template <typename PT>
__device__ __forceinline__ void pnm_write(const PnmDev& hp, const DevTensor& d, const PnmTrip& tr, long long e, int cnt,
                                          float div, float denom, const SrStream& s_upd, const Peers* peers) {
  using E = Elems<PT>;
  unsigned char* pe = reinterpret_cast<unsigned char*>(d.p) + e * E::BYTES;
  float pw[8], sh[8];
  load8_guard<PT>(pe, cnt, pw);
  uint32_t nz[4] = {0u, 0u, 0u, 0u};
  if (hp.sr) s_upd.draw8(d.tensor_id, (uint64_t)(e >> 3), nz);
  const bool kahan = E::IS_BF16 && hp.kahan;
  const float rdiv = __frcp_rn(div), rdenom = __frcp_rn(denom);
  unsigned char* she = kahan ? reinterpret_cast<unsigned char*>(d.shift) + e * 2 : nullptr;
  if (kahan) load8_guard<__nv_bfloat16>(she, cnt, sh);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (k >= cnt) continue;
    float p0 = pw[k];
    if (hp.has_wd) p0 = E::IS_BF16 ? round_bf16(__fmul_rn(p0, hp.wdsc)) : __fmul_rn(p0, hp.wdsc);
    float dl = hp.clip_on ? div_by(tr.u[k], div, rdiv) : tr.u[k];
    dl = __fmul_rn(dl, hp.fstep);
    if (hp.cautious) dl = (__fmul_rn(dl, tr.y[k]) > 0.0f) ? div_by(dl, denom, rdenom) : 0.0f;
    if (kahan) kahan_step(p0, sh[k], dl);
    else p0 = write_step_pnm<PT>(p0, dl, hp.sr != 0, noise_lane_pnm(nz, k));
    pw[k] = p0;
  }
  if constexpr (E::IS_BF16) {
    // every value is a bf16 already: the high halves are the bits
    if (cnt >= 8) {
      const uint4 out = make_uint4((__float_as_uint(pw[0]) >> 16) | (__float_as_uint(pw[1]) & 0xFFFF0000u),
                                   (__float_as_uint(pw[2]) >> 16) | (__float_as_uint(pw[3]) & 0xFFFF0000u),
                                   (__float_as_uint(pw[4]) >> 16) | (__float_as_uint(pw[5]) & 0xFFFF0000u),
                                   (__float_as_uint(pw[6]) >> 16) | (__float_as_uint(pw[7]) & 0xFFFF0000u));
      *reinterpret_cast<uint4*>(pe) = out;
      mirror16(peers, pe, out);
      if (kahan)
        *reinterpret_cast<uint4*>(she) =
            make_uint4((__float_as_uint(sh[0]) >> 16) | (__float_as_uint(sh[1]) & 0xFFFF0000u),
                       (__float_as_uint(sh[2]) >> 16) | (__float_as_uint(sh[3]) & 0xFFFF0000u),
                       (__float_as_uint(sh[4]) >> 16) | (__float_as_uint(sh[5]) & 0xFFFF0000u),
                       (__float_as_uint(sh[6]) >> 16) | (__float_as_uint(sh[7]) & 0xFFFF0000u));
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) if (k < cnt) {
        reinterpret_cast<uint16_t*>(pe)[k] = (uint16_t)(__float_as_uint(pw[k]) >> 16);
        if (kahan) reinterpret_cast<uint16_t*>(she)[k] = (uint16_t)(__float_as_uint(sh[k]) >> 16);
      }
      mirror_copy(peers, pe, cnt * 2);
    }
  } else {
    float* pf = reinterpret_cast<float*>(pe);
    if (cnt >= 8) {
      reinterpret_cast<float4*>(pf)[0] = make_float4(pw[0], pw[1], pw[2], pw[3]);
      reinterpret_cast<float4*>(pf)[1] = make_float4(pw[4], pw[5], pw[6], pw[7]);
      mirror16(peers, pf, make_uint4(__float_as_uint(pw[0]), __float_as_uint(pw[1]), __float_as_uint(pw[2]), __float_as_uint(pw[3])));
      mirror16(peers, pf + 4, make_uint4(__float_as_uint(pw[4]), __float_as_uint(pw[5]), __float_as_uint(pw[6]), __float_as_uint(pw[7])));
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) if (k < cnt) pf[k] = pw[k];
      mirror_copy(peers, pf, cnt * 4);
    }
  }
}

// ----------------------------------------------------------------------------- factored tensors

// The two sweeps over tensors whose rows are a multiple of eight elements (4-bit blocks of 128): a warp per unit of up
// to 4096 elements, nothing shared between warps.  Bound by instruction issue, so on packed pairs, the mask one
// comparison an element, rows and columns advanced by an addition.  (A CTA per 16 K-element item with guarded
// elements and a scalar encode: SUM 409 us and APPLY 972 us on 269 M elements of 4-bit momentum; here 260 and 550 us.)
template <typename PT, int MK, bool APPLY>
__global__ void __launch_bounds__(PT_THREADS, 4) pnm_sweep_kernel(const __grid_constant__ PlanView pv, const __grid_constant__ PnmDev hp,
                                                                  const __grid_constant__ PnmView x) {
  using E = Elems<PT>;
  constexpr int MV = MBytes<MK>::V;
  const int lane = threadIdx.x & 31;
  const int nw = gridDim.x * (PT_THREADS / 32);
  for (int it = __shfl_sync(0xffffffffu, (int)(blockIdx.x * (PT_THREADS / 32) + (threadIdx.x >> 5)), 0); it < x.n_units; it += nw) {
    const Task t = x.units[it];
    const unsigned char* g = reinterpret_cast<const unsigned char*>(pv.grads[t.tensor]);
    if (g == nullptr) continue;
    const DevTensor& d = pv.tensors[t.tensor];
    const PnmBufs& b = x.bufs[t.tensor];
    const int nvec = t.n >> 3, nv = d.cols >> 3;
    const float* rfac = pv.aux + aux_rfac(d);
    const float* cfac = pv.aux + aux_cfac(d);
    const float* mean = pv.aux + aux_mean(d);
    unsigned* rowmax = reinterpret_cast<unsigned*>(pv.aux + aux_rowmax(d));
    const unsigned char* gp = g + (t.e0 + lane * 8) * E::BYTES;
    unsigned char* pp = reinterpret_cast<unsigned char*>(d.p) + (t.e0 + lane * 8) * E::BYTES;
    unsigned char* pos = reinterpret_cast<unsigned char*>(b.m[hp.swap]) + ((t.e0 >> 3) + lane) * MV;
    const unsigned char* neg = reinterpret_cast<const unsigned char*>(b.m[hp.swap ^ 1]) + ((t.e0 >> 3) + lane) * MV;
    // 4-bit: the block's scale; int8: the row's (the positive buffer's as they were before this step)
    const long long blk = (t.e0 >> 7) + (lane >> 4);
    float* psc = b.sc[hp.swap] + (MK == KAON_M_4BIT ? blk : 0);
    const float* nsc = b.sc[hp.swap ^ 1] + (MK == KAON_M_4BIT ? blk : 0);
    const float* old = pv.aux + aux_oldsc(d);
    uint64_t q = (uint64_t)(t.e0 >> 3) + (unsigned)lane;
    int row = t.row0, cv = (t.pad >> 3) + lane;
    if (cv >= nv) { const int k = cv / nv; row += k; cv -= k * nv; }
    const int adv_r = 32 / nv, adv_c = 32 - adv_r * nv;
    float div = 1.0f, denom = 1.0f;
    if (APPLY) { div = x.scal[2 * t.tensor]; denom = hp.cautious ? x.scal[2 * t.tensor + 1] : 1.0f; }
    const float rdiv = __frcp_rn(div), rdenom = __frcp_rn(denom);
    double ss = 0.0;
    f32x2 kept2 = pack2(0.0f, 0.0f);
    auto trip = [&](const bool act) {
      W8<PT> gq, P;
      MRaw<MK> mp, mn;
      f32x2 Y[4], MP[4], MN[4], U[4];
      gq.load(act ? gp : g);
      mp.load(act ? pos : b.m[hp.swap]);
      mn.load(act ? neg : b.m[hp.swap ^ 1]);
      if constexpr (APPLY) P.load(act ? pp : d.p);
      const int r = act ? row : 0, c = act ? cv : 0;
      float sp = 1.0f, sn = 1.0f;
      if constexpr (MK == KAON_M_4BIT) { sp = act ? *psc : 1.0f; sn = act ? *nsc : 1.0f; }
      if constexpr (MK == KAON_M_INT8) { sp = old[r]; sn = nsc[r]; }
      const float rf = rfac[r];
      const float mu = hp.gc ? mean[r] : 0.0f;
      const float4 ca = __ldg(reinterpret_cast<const float4*>(cfac) + 2 * c), cb = __ldg(reinterpret_cast<const float4*>(cfac) + 2 * c + 1);
      const f32x2 CF[4] = {pack2(ca.x, ca.y), pack2(ca.z, ca.w), pack2(cb.x, cb.y), pack2(cb.z, cb.w)};
      center<PT>(gq, E::IS_BF16 ? __uint_as_float(pack_bf16_rn(mu, mu)) : mu, Y);
      mp.decode(sp, MP);
      mn.decode(sn, MN);
      const f32x2 RF = pack2(rf, rf);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        MP[j] = fma2(Y[j], pack2(hp.fw, hp.fw), mul2(MP[j], pack2(hp.fb, hp.fb)));
        const f32x2 pn = mul2(fma2(MN[j], pack2(hp.c2, hp.c2), mul2(MP[j], pack2(hp.c1, hp.c1))), pack2(hp.c3, hp.c3));
        U[j] = mul2(pn, mul2(mul2(RF, CF[j]), pack2(hp.bc2, hp.bc2)));
      }
      if constexpr (!APPLY) {
        // the trip's eight squares in fp32, then one wide addition
        const f32x2 s2 = fma2(U[3], U[3], fma2(U[2], U[2], fma2(U[1], U[1], mul2(U[0], U[0]))));
        f32x2 K[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const f32x2 X = mul2(U[j], Y[j]);
          K[j] = pack2(gt0(X.x), gt0(X.y));
        }
        if (act) {
          ss += (double)(s2.x + s2.y);
          kept2 = add2(kept2, add2(add2(K[0], K[1]), add2(K[2], K[3])));
        }
        if constexpr (MK == KAON_M_INT8) {
          unsigned bits = act ? __float_as_uint(amax8(MP)) : 0u;
          const int row_l0 = __shfl_sync(0xffffffffu, row, 0);
          if (__all_sync(0xffffffffu, !act || row == row_l0)) {
            bits = __reduce_max_sync(0xffffffffu, bits);
            if (lane == 0) atomicMax(rowmax + row_l0, bits);
          } else if (act) {
            atomicMax(rowmax + row, bits);
          }
        }
      } else {
        // -(u / div * lr), masked by its sign against the gradient's, over the kept share
        f32x2 F[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          f32x2 u = U[j];
          if (hp.clip_on) {
            const f32x2 q0 = mul2(u, pack2(rdiv, rdiv));
            u = fma2(fma2(q0, pack2(-div, -div), u), pack2(rdiv, rdiv), q0);
          }
          u = mul2(u, pack2(-hp.fstep, -hp.fstep));
          if (hp.cautious) {
            const f32x2 X = mul2(u, Y[j]);
            const f32x2 q0 = mul2(u, pack2(rdenom, rdenom));
            u = fma2(fma2(q0, pack2(-denom, -denom), u), pack2(rdenom, rdenom), q0);
            u = mul2(u, pack2(lt0(X.x), lt0(X.y)));
          }
          F[j] = u;
        }
        if (hp.has_wd) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            f32x2 w = mul2(P.pair(j), pack2(hp.wdsc, hp.wdsc));
            if constexpr (E::IS_BF16) w = pack2(round_bf16(w.x), round_bf16(w.y));
            P.set(j, w);
          }
        }
        write8(hp, d, q, act, P, F);
        if (act) P.store(pp, &pv.peers);
        float rm = 0.0f;
        if constexpr (MK == KAON_M_INT8) rm = __uint_as_float(__ldcg(rowmax + r));
        if constexpr (MK == KAON_M_BF16) {
#pragma unroll
          for (int j = 0; j < 4; ++j) MP[j] = pack2(round_bf16(MP[j].x), round_bf16(MP[j].y));
        }
        const float sc = store_m8<MK>(pos, MP, rm, act ? 8 : 0, lane);
        if constexpr (MK == KAON_M_4BIT) { if (act && (lane & 15) == 0) stg_f32(psc, sc); }
        if constexpr (MK == KAON_M_INT8) { if (act && cv == 0) psc[row] = sc; }
      }
    };
    for (int full = nvec >> 5; full > 0; --full) {
      trip(true);
      gp += 256 * E::BYTES; pp += 256 * E::BYTES; pos += 32 * MV; neg += 32 * MV;
      if constexpr (MK == KAON_M_4BIT) { psc += 2; nsc += 2; }
      q += 32;
      row += adv_r; cv += adv_c;
      if (cv >= nv) { cv -= nv; ++row; }
    }
    if (nvec & 31) trip(lane < (nvec & 31));
    if constexpr (!APPLY) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      const unsigned kept = __reduce_add_sync(0xffffffffu, (unsigned)(kept2.x + kept2.y + 0.5f));
      if (lane == 0) { x.part[t.slot] = ss; x.kpart[t.slot] = kept; }
    }
  }
}

// The other factored tensors, eight elements a thread with every element guarded.
template <typename PT, int MK, bool APPLY>
__global__ void __launch_bounds__(PT_THREADS, 4) pnm_pass_kernel(PlanView pv, PnmDev hp, PnmView x) {
  using E = Elems<PT>;
  __shared__ double red_d[PT_THREADS / 32];
  __shared__ unsigned red_u[PT_THREADS / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const SrStream s_upd{Philox{hp.k0, hp.k1}, hp.step, KAON_TAG_UPDATE};
  for (int it = blockIdx.x; it < x.n_items; it += gridDim.x) {
    const Task t = x.items[it];
    const DevTensor d = pv.tensors[t.tensor];
    const unsigned char* g = reinterpret_cast<const unsigned char*>(pv.grads[t.tensor]);
    double ss = 0.0;
    unsigned kept = 0;
    if (g != nullptr) {
      const PnmBufs b = x.bufs[t.tensor];
      void* pos = b.m[hp.swap];
      float* psc = b.sc[hp.swap];
      const void* neg = b.m[hp.swap ^ 1];
      const float* nsc = b.sc[hp.swap ^ 1];
      const int C = d.cols;
      const float* rfac = pv.aux + aux_rfac(d);
      const float* cfac = pv.aux + aux_cfac(d);
      const float* mean = pv.aux + aux_mean(d);
      unsigned* rowmax = reinterpret_cast<unsigned*>(pv.aux + aux_rowmax(d));
      // int8: the positive buffer's row scales as they were before this step (its rows get new ones in APPLY)
      const float* psc_rd = MK == KAON_M_INT8 ? pv.aux + aux_oldsc(d) : psc;
      const int bsh = d.bshift;  // 4-bit: element -> block shift (31: one block)
      float div = 1.0f, denom = 1.0f;
      if (APPLY) { div = x.scal[2 * t.tensor]; denom = x.scal[2 * t.tensor + 1]; }
      const int nvec = (t.n + 7) >> 3;
      for (int v0 = 0; v0 < nvec; v0 += PT_THREADS) {
        const int v = v0 + tid;
        const long long e = t.e0 + (long long)v * 8;
        const int cnt_rt = v < nvec ? min(8, (int)(t.e0 + t.n - e)) : 0;
        int r0 = 0, c0 = 0;
        if (cnt_rt > 0) {
          r0 = e < 0x100000000ll ? (int)((unsigned)e / (unsigned)C) : (int)(e / C);
          c0 = (int)(e - (long long)r0 * C);
        }
        // FULL: every lane of the warp has eight elements inside one row, so the element guards and the
        // row bookkeeping fold away at compile time; anything else (a row end, a tensor's tail) takes
        // the guarded form.  The choice is per warp: the 4-bit store shuffles block maxima across lanes.
        auto trip = [&](auto full_tag) {
          constexpr bool FULL = decltype(full_tag)::value;
          const int cnt = FULL ? 8 : cnt_rt;
          PnmTrip tr;
          tr.first = 0u;
          if (cnt > 0) {
            float gx[8], mpo[8], mno[8];
            int cl[8];
            load8_guard<PT>(g + e * E::BYTES, cnt, gx);
            int r = r0, c = c0;
            // the common trip: eight elements of one row (no row bookkeeping, one row factor, one mean)
            const bool one_row = FULL || (cnt == 8 && c + 8 <= C);
            if (one_row) {
  #pragma unroll
              for (int k = 0; k < 8; ++k) { tr.rw[k] = r; cl[k] = c + k; }
              if (c == 0) tr.first = 1u;
            } else {
  #pragma unroll
              for (int k = 0; k < 8; ++k) {
                tr.rw[k] = 0; cl[k] = 0;
                if (k < cnt) {
                  while (c >= C) { c -= C; ++r; }
                  tr.rw[k] = r;
                  cl[k] = c;
                  if (c == 0) tr.first |= 1u << k;
                  ++c;
                }
              }
            }
            pnm_decode8<MK>(pos, psc_rd, e, cnt, tr.rw, bsh, mpo);
            pnm_decode8<MK>(neg, nsc, e, cnt, tr.rw, bsh, mno);
            auto chain = [&](int k, float rf, float mu, float cf) {
              const float yk = pnm_centered<PT>(gx[k], mu, hp.gc != 0);
              const float mpn = __fmaf_rn(yk, hp.fw, __fmul_rn(mpo[k], hp.fb));
              const float pn = __fmul_rn(__fmaf_rn(mno[k], hp.c2, __fmul_rn(mpn, hp.c1)), hp.c3);
              const float inv = __fmul_rn(__fmul_rn(rf, cf), hp.bc2);
              tr.y[k] = yk; tr.mp[k] = mpn; tr.u[k] = __fmul_rn(pn, inv);
            };
            if (one_row) {
              const float rf = rfac[tr.rw[0]], mu = hp.gc ? mean[tr.rw[0]] : 0.0f;
              float cf[8];
              ld8f(cfac + cl[0], 8, cf);  // the eight column factors: two vector loads where the address allows
              // the same chain on pairs (each lane of a packed instruction is the scalar IEEE operation)
              const f32x2 FW = pack2(hp.fw, hp.fw), FB = pack2(hp.fb, hp.fb), C1 = pack2(hp.c1, hp.c1);
              const f32x2 C2 = pack2(hp.c2, hp.c2), C3 = pack2(hp.c3, hp.c3), BC2 = pack2(hp.bc2, hp.bc2);
              const f32x2 RF = pack2(rf, rf), MUN = pack2(-mu, -mu);
  #pragma unroll
              for (int j = 0; j < 4; ++j) {
                f32x2 y2 = pack2(gx[2 * j], gx[2 * j + 1]);
                if (hp.gc) {
                  y2 = add2(y2, MUN);
                  if constexpr (E::IS_BF16) {
                    const uint32_t w = pack_bf16_rn(y2.x, y2.y);
                    y2 = pack2(bf16lo(w), bf16hi(w));
                  }
                }
                const f32x2 mp2 = fma2(y2, FW, mul2(pack2(mpo[2 * j], mpo[2 * j + 1]), FB));
                const f32x2 pn2 = mul2(fma2(pack2(mno[2 * j], mno[2 * j + 1]), C2, mul2(mp2, C1)), C3);
                const f32x2 inv2 = mul2(mul2(RF, pack2(cf[2 * j], cf[2 * j + 1])), BC2);
                const f32x2 u2 = mul2(pn2, inv2);
                tr.y[2 * j] = y2.x; tr.y[2 * j + 1] = y2.y;
                tr.mp[2 * j] = mp2.x; tr.mp[2 * j + 1] = mp2.y;
                tr.u[2 * j] = u2.x; tr.u[2 * j + 1] = u2.y;
              }
            } else {
  #pragma unroll
              for (int k = 0; k < 8; ++k) {
                tr.y[k] = 0.0f; tr.mp[k] = 0.0f; tr.u[k] = 0.0f;
                if (k < cnt) chain(k, rfac[tr.rw[k]], hp.gc ? mean[tr.rw[k]] : 0.0f, cfac[cl[k]]);
              }
            }
          } else {
  #pragma unroll
            for (int k = 0; k < 8; ++k) { tr.y[k] = 0.0f; tr.mp[k] = 0.0f; tr.u[k] = 0.0f; tr.rw[k] = 0; }
          }
          if constexpr (!APPLY) {
            float s8 = 0.0f;  // the trip's eight squares in fp32, then one wide addition
  #pragma unroll
            for (int k = 0; k < 8; ++k) if (k < cnt) {
              s8 = __fmaf_rn(tr.u[k], tr.u[k], s8);
              kept += (__fmul_rn(tr.u[k], tr.y[k]) > 0.0f) ? 1u : 0u;
            }
            ss += (double)s8;
            if constexpr (MK == KAON_M_INT8) {
              int cr = -1;
              float mx = 0.0f;
  #pragma unroll
              for (int k = 0; k < 8; ++k) if (k < cnt) {
                if (tr.rw[k] != cr) {
                  if (cr >= 0) atomicMax(rowmax + cr, __float_as_uint(mx));
                  cr = tr.rw[k];
                  mx = 0.0f;
                }
                mx = fmaxf(mx, fabsf(tr.mp[k]));
              }
              if (cr >= 0) atomicMax(rowmax + cr, __float_as_uint(mx));
            }
          } else {
            if (cnt > 0) pnm_write<PT>(hp, d, tr, e, cnt, div, denom, s_upd, &pv.peers);
            pnm_store_m<MK>(pos, psc, tr, e, cnt, bsh, lane,
                            [&](int r) { return __uint_as_float(__ldcg(rowmax + r)); });
          }
        };
        if (__all_sync(0xffffffffu, cnt_rt == 8 && c0 + 8 <= C)) trip(std::true_type{});
        else trip(std::false_type{});
      }
    }
    if constexpr (!APPLY) {
      // the item's partial sums, lanes then warps in order
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        ss += __shfl_xor_sync(0xffffffffu, ss, o);
        kept += __shfl_xor_sync(0xffffffffu, kept, o);
      }
      __syncthreads();
      if (lane == 0) { red_d[warp] = ss; red_u[warp] = kept; }
      __syncthreads();
      if (tid == 0) {
        double s = 0.0;
        unsigned kk = 0;
        for (int w = 0; w < PT_THREADS / 32; ++w) { s += red_d[w]; kk += red_u[w]; }
        x.part[t.slot] = s;
        x.kpart[t.slot] = kk;
      }
    }
  }
}

// int8 momentum: before SUM, zero the row maxima and set the positive buffer's row scales aside.
__global__ void __launch_bounds__(PT_THREADS) pnm_prep_kernel(PlanView pv, PnmDev hp, PnmView x) {
  const int ti = x.fact[blockIdx.x];
  if (pv.grads[ti] == nullptr) return;
  const DevTensor d = pv.tensors[ti];
  unsigned* rowmax = reinterpret_cast<unsigned*>(pv.aux + aux_rowmax(d));
  float* oldsc = pv.aux + aux_oldsc(d);
  const float* psc = x.bufs[ti].sc[hp.swap];
  for (int r = threadIdx.x; r < d.rows; r += PT_THREADS) { rowmax[r] = 0u; oldsc[r] = psc[r]; }
}

// One CTA per factored tensor: item partials in item order -> clip divisor, cautious denominator.
__global__ void __launch_bounds__(PT_THREADS) pnm_reduce_kernel(PlanView pv, PnmDev hp, PnmView x) {
  __shared__ double red_d[PT_THREADS];
  __shared__ unsigned red_u[PT_THREADS];
  const int ti = x.fact[blockIdx.x];
  if (pv.grads[ti] == nullptr) return;
  const DevTensor d = pv.tensors[ti];
  const int b0 = x.item_begin[ti], b1 = x.item_begin[ti + 1];
  // thread j takes the contiguous run of items [b0 + j*per, ...): the order of the additions is fixed
  const int per = (b1 - b0 + PT_THREADS - 1) / PT_THREADS;
  double s = 0.0;
  unsigned kk = 0;
  for (int i = b0 + threadIdx.x * per; i < min(b1, b0 + (threadIdx.x + 1) * per); ++i) { s += x.part[i]; kk += x.kpart[i]; }
  red_d[threadIdx.x] = s;
  red_u[threadIdx.x] = kk;
  __syncthreads();
  if (threadIdx.x == 0) {
    double tot = 0.0;
    unsigned kept = 0;
    for (int j = 0; j < PT_THREADS; ++j) { tot += red_d[j]; kept += red_u[j]; }
    const float rms = __fdiv_rn((float)sqrt(tot), (float)sqrt((double)d.numel));
    x.scal[2 * ti] = hp.clip_on ? fmaxf(__fdiv_rn(rms, hp.clip), 1.0f) : 1.0f;
    x.scal[2 * ti + 1] = fmaxf(__fdiv_rn((float)kept, (float)d.numel), 1e-8f);
    pv.kept[ti] = kept;
  }
}

// ----------------------------------------------------------------------------- 1-D tensors

// reference src/kaon/adapnm.py:1126-1172 / 1238-1249: full second moment v (optionally its running
// maximum), eps on the denominator.  One CTA per tensor, any length: a first sweep updates v and takes
// the tensor-wide sums, a second one recomputes the chain and writes.
template <typename PT, int MK>
__global__ void __launch_bounds__(PT_THREADS) pnm_flat_kernel(PlanView pv, PnmDev hp, PnmView x) {
  using E = Elems<PT>;
  __shared__ double red_d[PT_THREADS / 32];
  __shared__ unsigned red_u[PT_THREADS / 32];
  __shared__ float red_f[PT_THREADS / 32];
  __shared__ float bc_s[3];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ti = x.flat[blockIdx.x];
  const unsigned char* g = reinterpret_cast<const unsigned char*>(pv.grads[ti]);
  if (g == nullptr) return;
  const DevTensor d = pv.tensors[ti];
  const PnmBufs b = x.bufs[ti];
  void* pos = b.m[hp.swap];
  float* psc = b.sc[hp.swap];
  const void* neg = b.m[hp.swap ^ 1];
  const float* nsc = b.sc[hp.swap ^ 1];
  const int bsh = d.bshift;  // 4-bit: element -> block shift (31: one block)
  const long long n = d.numel;
  const long long nvec = (n + 7) >> 3;
  float* v = d.stat_a;
  float* max_v = hp.ams ? b.max_v : nullptr;
  const SrStream s_upd{Philox{hp.k0, hp.k1}, hp.step, KAON_TAG_UPDATE};
  // int8: one scalar scale; every thread keeps the old one before anything is written
  __shared__ float old_sc_s;
  const bool one_scale = MK == KAON_M_INT8 || (MK == KAON_M_4BIT && bsh >= 31);
  if (tid == 0) old_sc_s = one_scale ? psc[0] : 0.0f;
  __syncthreads();
  const float old_sc = old_sc_s;
  const float* psc_rd = one_scale ? &old_sc : psc;

  auto chain = [&](long long e, int cnt, bool first_sweep, PnmTrip& tr) {
    float gx[8], vv[8], mx[8], mpo[8], mno[8];
    load8_guard<PT>(g + e * E::BYTES, cnt, gx);
    ld8f(v + e, cnt, vv);
    if (max_v != nullptr) ld8f(max_v + e, cnt, mx);
#pragma unroll
    for (int k = 0; k < 8; ++k) tr.rw[k] = 0;
    pnm_decode8<MK>(pos, psc_rd, e, cnt, tr.rw, bsh, mpo);
    pnm_decode8<MK>(neg, nsc, e, cnt, tr.rw, bsh, mno);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      tr.y[k] = 0.0f; tr.mp[k] = 0.0f; tr.u[k] = 0.0f;
      if (k < cnt) {
        const float yk = gx[k];
        if (first_sweep) {
          vv[k] = __fmaf_rn(__fmul_rn(hp.fw2, yk), yk, __fmul_rn(vv[k], hp.fb2));
          if (max_v != nullptr) mx[k] = fmaxf(mx[k], vv[k]);
        }
        const float vd = max_v != nullptr ? mx[k] : vv[k];
        const float den = __fdiv_rn(__fadd_rn(__fsqrt_rn(__fadd_rn(vd, 1e-15f)), hp.eps), hp.bc2);
        const float mpn = __fmaf_rn(yk, hp.fw, __fmul_rn(mpo[k], hp.fb));
        const float pn = __fmul_rn(__fmaf_rn(mno[k], hp.c2, __fmul_rn(mpn, hp.c1)), hp.c3);
        tr.y[k] = yk; tr.mp[k] = mpn; tr.u[k] = __fdiv_rn(pn, den);
      }
    }
    if (first_sweep) {
      st8f(v + e, cnt, vv);
      if (max_v != nullptr) st8f(max_v + e, cnt, mx);
    }
  };

  double ss = 0.0;
  unsigned kept = 0;
  float amax = 0.0f;
  for (long long v0 = 0; v0 < nvec; v0 += PT_THREADS) {
    const long long vi = v0 + tid;
    const long long e = vi * 8;
    const int cnt = vi < nvec ? (int)min(8ll, n - e) : 0;
    if (cnt > 0) {
      PnmTrip tr;
      chain(e, cnt, true, tr);
#pragma unroll
      for (int k = 0; k < 8; ++k) if (k < cnt) {
        ss += (double)tr.u[k] * (double)tr.u[k];
        kept += (__fmul_rn(tr.u[k], tr.y[k]) > 0.0f) ? 1u : 0u;
        amax = fmaxf(amax, fabsf(tr.mp[k]));
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ss += __shfl_xor_sync(0xffffffffu, ss, o);
    kept += __shfl_xor_sync(0xffffffffu, kept, o);
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  }
  if (lane == 0) { red_d[warp] = ss; red_u[warp] = kept; red_f[warp] = amax; }
  __syncthreads();  // also: every write of v / max_v by this CTA is visible to it from here on
  if (tid == 0) {
    double tot = 0.0;
    unsigned kk = 0;
    float am = 0.0f;
    for (int w = 0; w < PT_THREADS / 32; ++w) { tot += red_d[w]; kk += red_u[w]; am = fmaxf(am, red_f[w]); }
    const float rms = __fdiv_rn((float)sqrt(tot), (float)sqrt((double)n));
    bc_s[0] = hp.clip_on ? fmaxf(__fdiv_rn(rms, hp.clip), 1.0f) : 1.0f;
    bc_s[1] = fmaxf(__fdiv_rn((float)kk, (float)n), 1e-8f);
    bc_s[2] = am;
    pv.kept[ti] = kk;
  }
  __syncthreads();
  const float div = bc_s[0], denom = bc_s[1], tmax = bc_s[2];
  for (long long v0 = 0; v0 < nvec; v0 += PT_THREADS) {
    const long long vi = v0 + tid;
    const long long e = vi * 8;
    const int cnt = vi < nvec ? (int)min(8ll, n - e) : 0;
    PnmTrip tr;
    tr.first = 0u;
    if (cnt > 0) {
      chain(e, cnt, false, tr);
      pnm_write<PT>(hp, d, tr, e, cnt, div, denom, s_upd, &pv.peers);
    }
    pnm_store_m<MK>(pos, psc, tr, e, cnt, bsh, lane, [&](int) { return tmax; },
                    (MK == KAON_M_4BIT && bsh >= 31) ? tmax : -1.0f);
  }
  if constexpr (MK == KAON_M_INT8 || MK == KAON_M_4BIT) {
    // the one scale of the tensor (int8, or a 4-bit block that covers it), once every thread has decoded with the old one
    __syncthreads();
    if (tid == 0 && (MK == KAON_M_INT8 || bsh >= 31)) psc[0] = __fdiv_rn(fmaxf(tmax, 1e-12f), MK == KAON_M_INT8 ? 127.0f : 7.0f);
  }
}

// ----------------------------------------------------------------------------- host

struct PnmHost {
  PnmView view{};
  void* block = nullptr;
  Task* d_stats = nullptr;   // STATS items the launch of its own takes
  Task* d_final = nullptr;   // the other STATS items and the FINAL items, for the persistent kernel
  Task* d_strips = nullptr;  // and their FINAL strips and row-table runs
  int n_stats = 0, n_final = 0, n_strips = 0, n_final_items = 0, order = ADA_KEPT_FIRST;
  bool attached = false;
  int64_t bytes = 0;
};

typedef void (*PnmPass)(PlanView, PnmDev, PnmView);

template <typename PT, bool APPLY>
static PnmPass pick_pass_pt(int mk) {
  switch (mk) {
    case KAON_M_F32: return pnm_pass_kernel<PT, KAON_M_F32, APPLY>;
    case KAON_M_BF16: return pnm_pass_kernel<PT, KAON_M_BF16, APPLY>;
    case KAON_M_INT8: return pnm_pass_kernel<PT, KAON_M_INT8, APPLY>;
    case KAON_M_4BIT: return pnm_pass_kernel<PT, KAON_M_4BIT, APPLY>;
    default: return nullptr;
  }
}
template <typename PT, bool APPLY>
static PnmPass pick_sweep_pt(int mk) {
  switch (mk) {
    case KAON_M_F32: return pnm_sweep_kernel<PT, KAON_M_F32, APPLY>;
    case KAON_M_BF16: return pnm_sweep_kernel<PT, KAON_M_BF16, APPLY>;
    case KAON_M_INT8: return pnm_sweep_kernel<PT, KAON_M_INT8, APPLY>;
    case KAON_M_4BIT: return pnm_sweep_kernel<PT, KAON_M_4BIT, APPLY>;
    default: return nullptr;
  }
}
template <typename PT>
static PnmPass pick_flat_pt(int mk) {
  switch (mk) {
    case KAON_M_F32: return pnm_flat_kernel<PT, KAON_M_F32>;
    case KAON_M_BF16: return pnm_flat_kernel<PT, KAON_M_BF16>;
    case KAON_M_INT8: return pnm_flat_kernel<PT, KAON_M_INT8>;
    case KAON_M_4BIT: return pnm_flat_kernel<PT, KAON_M_4BIT>;
    default: return nullptr;
  }
}

void pnm_free(kaon_plan* pl) {
  PnmHost* h = reinterpret_cast<PnmHost*>(pl->pnm);
  if (!h) return;
  cudaFree(h->block);
  delete h;
  pl->pnm = nullptr;
}

// Lists, partial-sum buffers and the table of the second momentum, built by kaon_adapnm_attach.
static int pnm_build(kaon_plan* pl, const void* const* m_neg, float* const* m_neg_scale, float* const* max_v) {
  pnm_free(pl);
  PnmHost* h = new PnmHost();
  pl->pnm = h;
  const int n = pl->n_tensors;
  std::vector<Task> units, items, stats, strips, fin;
  int slots = 0;
  std::vector<int> begin(n + 1, 0), fact, flat;
  std::vector<PnmBufs> bufs(n);
  for (int i = 0; i < n; ++i) {
    const DevTensor& t = pl->h_tensors[i];
    begin[i] = slots;
    bufs[i].m[0] = t.m; bufs[i].sc[0] = t.m_scale;
    bufs[i].m[1] = const_cast<void*>(m_neg[i]);
    bufs[i].sc[1] = m_neg_scale ? m_neg_scale[i] : nullptr;
    bufs[i].max_v = max_v ? max_v[i] : nullptr;
    if (t.numel == 0) continue;
    if (!m_neg[i]) return fail(KAON_E_INVALID, "kaon_adapnm_attach: tensor %d has no second momentum", i);
    if ((uintptr_t)m_neg[i] & 15) return fail(KAON_E_INVALID, "kaon_adapnm_attach: tensor %d: second momentum not 16-byte aligned", i);
    if ((pl->momentum_kind == KAON_M_INT8 || pl->momentum_kind == KAON_M_4BIT) && !bufs[i].sc[1])
      return fail(KAON_E_INVALID, "kaon_adapnm_attach: tensor %d: scales of the second momentum missing", i);
    if (t.rows <= 0) { flat.push_back(i); continue; }
    fact.push_back(i);
    if ((t.cols & 7) == 0 && (pl->momentum_kind != KAON_M_4BIT || t.bshift == 7)) {
      // a warp's unit: small tensors in more pieces (the tensor alone decides, so the order of its sums stays)
      long long u = 512;
      while (u < 4096 && u * 128 <= t.numel) u *= 2;
      for (long long e = 0; e < t.numel; e += u)
        units.push_back(Task{i, PH_ADA_APPLY, e, (int)std::min<long long>(u, t.numel - e), (int)(e / t.cols), slots++, (int)(e % t.cols)});
      continue;
    }
    for (long long e = 0; e < t.numel; e += PNM_ITEM)
      items.push_back(Task{i, PH_ADA_APPLY, e, (int)std::min<long long>(PNM_ITEM, t.numel - e), 0, slots++, 0});
  }
  begin[n] = slots;
  {
    std::vector<Task> hm((size_t)pl->n_tasks_main);
    KAON_CUDA(cudaMemcpy(hm.data(), pl->d_tasks_main, sizeof(Task) * hm.size(), cudaMemcpyDeviceToHost));
    // STATS items the small-CTA launch can take go there, the others stay with FINAL in the persistent
    // kernel (which stages whole rows, so it cannot take rows longer than a work item)
    // the tensors whose STATS are a launch of their own, and their FINAL, unless it had better stay
    std::vector<char> leaves = pl->param_dtype == KAON_DT_BF16 ? stats_tensors(pl, hm) : std::vector<char>(n, 0);
    int n_final = 0;
    for (const Task& t : hm) {
      if (t.phase == PH_ADA_STATS) {
        if (leaves[t.tensor]) stats.push_back(t);
        else if (pl->h_tensors[t.tensor].cols > CAP)
          return fail(KAON_E_UNSUPPORTED, "AdaPNM: tensor %d: rows longer than %d elements need bf16 weights and a row length that is a multiple of 8", t.tensor, CAP);
        else fin.push_back(t);
      } else if (t.phase == PH_ADA_FINAL) {
        if (leaves[t.tensor]) ++n_final;
        else fin.push_back(t);
      }
    }
    h->order = kept_place((int)fin.size(), false, (int)stats.size(), n_final, pl->sm_count);
    if (h->order == ADA_KEPT_WAITS) {
      for (const Task& t : hm) if (t.phase == PH_ADA_FINAL && leaves[t.tensor]) fin.push_back(t);
      leaves.assign(n, 0);
    }
    final_items(pl, leaves, strips, h->n_strips);
  }
  auto up = [](size_t b) { return (b + 255) / 256 * 256; };
  size_t o = 0;
  auto take = [&](size_t b) { size_t r = o; o += up(b); return r; };
  const size_t o_items = take(sizeof(Task) * items.size()), o_units = take(sizeof(Task) * units.size()), o_begin = take(sizeof(int) * (n + 1));
  const size_t o_bufs = take(sizeof(PnmBufs) * n), o_part = take(sizeof(double) * slots);
  const size_t o_kpart = take(sizeof(unsigned) * slots), o_scal = take(sizeof(float) * 2 * n);
  const size_t o_fact = take(sizeof(int) * fact.size()), o_flat = take(sizeof(int) * flat.size());
  const size_t o_strips = take(sizeof(Task) * strips.size()), o_stats = take(sizeof(Task) * stats.size());
  const size_t o_fin = take(sizeof(Task) * fin.size());
  KAON_CUDA(cudaMalloc(&h->block, std::max<size_t>(o, 256)));
  unsigned char* base = reinterpret_cast<unsigned char*>(h->block);
  h->bytes = (int64_t)o;
  auto put = [&](size_t off, const void* src, size_t b) -> cudaError_t {
    return b ? cudaMemcpy(base + off, src, b, cudaMemcpyHostToDevice) : cudaSuccess;
  };
  KAON_CUDA(put(o_items, items.data(), sizeof(Task) * items.size()));
  KAON_CUDA(put(o_units, units.data(), sizeof(Task) * units.size()));
  KAON_CUDA(put(o_begin, begin.data(), sizeof(int) * (n + 1)));
  KAON_CUDA(put(o_bufs, bufs.data(), sizeof(PnmBufs) * n));
  KAON_CUDA(put(o_fact, fact.data(), sizeof(int) * fact.size()));
  KAON_CUDA(put(o_flat, flat.data(), sizeof(int) * flat.size()));
  KAON_CUDA(put(o_strips, strips.data(), sizeof(Task) * strips.size()));
  KAON_CUDA(put(o_stats, stats.data(), sizeof(Task) * stats.size()));
  KAON_CUDA(put(o_fin, fin.data(), sizeof(Task) * fin.size()));
  KAON_CUDA(cudaMemset(base + o_scal, 0, sizeof(float) * 2 * n));
  PnmView& x = h->view;
  x.items = reinterpret_cast<const Task*>(base + o_items); x.n_items = (int)items.size();
  x.units = reinterpret_cast<const Task*>(base + o_units); x.n_units = (int)units.size();
  x.item_begin = reinterpret_cast<const int*>(base + o_begin);
  x.bufs = reinterpret_cast<const PnmBufs*>(base + o_bufs);
  x.part = reinterpret_cast<double*>(base + o_part);
  x.kpart = reinterpret_cast<unsigned*>(base + o_kpart);
  x.scal = reinterpret_cast<float*>(base + o_scal);
  x.fact = reinterpret_cast<const int*>(base + o_fact); x.n_fact = (int)fact.size();
  x.flat = reinterpret_cast<const int*>(base + o_flat); x.n_flat = (int)flat.size();
  h->d_stats = reinterpret_cast<Task*>(base + o_stats); h->n_stats = (int)stats.size();
  h->d_strips = reinterpret_cast<Task*>(base + o_strips); h->n_final_items = (int)strips.size();
  h->d_final = reinterpret_cast<Task*>(base + o_fin); h->n_final = (int)fin.size();
  h->attached = true;
  pl->device_bytes += h->bytes;
  return KAON_OK;
}

}  // namespace kaon

using namespace kaon;

extern "C" int kaon_adapnm_attach(kaon_plan* pl, const void* const* m_neg, float* const* m_neg_scale,
                                  float* const* max_v, int n) {
  if (!pl || !m_neg) return fail(KAON_E_INVALID, "kaon_adapnm_attach: null argument");
  if (pl->optimizer != KAON_OPT_ADAPNM) return fail(KAON_E_INVALID, "plan was not built for AdaPNM");
  if (n != pl->n_tensors) return fail(KAON_E_INVALID, "kaon_adapnm_attach: %d pointers for a plan of %d tensors", n, pl->n_tensors);
  if (int rc = check_device(pl)) return rc;
  pl->pnm_has_max_v = max_v != nullptr;
  if (max_v)
    for (int i = 0; i < n; ++i)
      if (pl->h_tensors[i].rows <= 0 && pl->h_tensors[i].numel > 0 && !max_v[i]) pl->pnm_has_max_v = false;
  return pnm_build(pl, m_neg, m_neg_scale, max_v);
}

extern "C" int kaon_adapnm_step(kaon_plan* pl, const kaon_adapnm_hparams* h, uint64_t seed, uint32_t step,
                                void* stream) {
  if (!pl || !h) return fail(KAON_E_INVALID, "kaon_adapnm_step: null argument");
  if (pl->optimizer != KAON_OPT_ADAPNM) return fail(KAON_E_INVALID, "plan was not built for AdaPNM");
  if (int rc = check_device(pl)) return rc;
  PnmHost* ph = reinterpret_cast<PnmHost*>(pl->pnm);
  if (!ph || !ph->attached) return fail(KAON_E_INVALID, "kaon_adapnm_step: call kaon_adapnm_attach first (the second momentum)");
  if (pl->momentum_kind == KAON_M_NONE) return fail(KAON_E_INVALID, "AdaPNM needs its two momenta");
  if (h->bf16_method < KAON_W_NONE || h->bf16_method > KAON_W_KAHAN) return fail(KAON_E_UNSUPPORTED, "bf16_method %d", h->bf16_method);
  if (int rc = check_kahan(pl, h->bf16_method)) return rc;
  if (h->group_step < 1) return fail(KAON_E_INVALID, "group_step is the 1-based step count of the parameter group");
  if (h->ams_bound && ph->view.n_flat > 0 && !pl->pnm_has_max_v)
    return fail(KAON_E_INVALID, "ams_bound: the 1-D tensors need their max_v buffers (kaon_adapnm_attach)");
  const double b1 = h->beta1, b2 = h->beta2, b0 = h->beta0, t = (double)h->group_step;
  const double b1sq = b1 * b1, nn = std::sqrt((1.0 + b0) * (1.0 + b0) + b0 * b0);
  const double bc1 = 1.0 - std::pow(b1, t), bc2 = std::sqrt(1.0 - std::pow(b2, t));
  PnmDev hp{};
  hp.fb = (float)b1sq; hp.fw = (float)(1.0 - b1sq);
  hp.c1 = (float)(1.0 + b0); hp.c2 = (float)(-b0); hp.c3 = (float)(1.0 / nn);
  hp.bc2 = (float)bc2; hp.fstep = (float)(h->lr / bc1);
  hp.wdsc = (float)(1.0 - h->lr * h->weight_decay); hp.has_wd = h->weight_decay != 0.0;
  hp.fb2 = (float)b2; hp.fw2 = (float)(1.0 - b2); hp.eps = (float)h->eps;
  hp.clip = (float)h->clip_threshold; hp.clip_on = h->clip_threshold > 0.0;
  hp.cautious = h->cautious != 0; hp.gc = h->gradient_centralization != 0; hp.ams = h->ams_bound != 0;
  hp.sr = h->bf16_method == KAON_W_SR && pl->param_dtype == KAON_DT_BF16;
  hp.kahan = h->bf16_method == KAON_W_KAHAN && pl->param_dtype == KAON_DT_BF16;
  hp.swap = (h->group_step & 1u) ? 0 : 1;  // odd steps: "m_pos" is positive
  hp.step = step; hp.k0 = (uint32_t)seed; hp.k1 = (uint32_t)(seed >> 32);
  philox_round_keys(hp);
  cudaStream_t s = (cudaStream_t)stream;
  const bool bf = pl->param_dtype == KAON_DT_BF16;
  const int mk = pl->momentum_kind;
  const PnmView& x = ph->view;
  // 1. second moment of the factored tensors: Adakaon's STATS and FINAL items
  if (x.n_fact > 0) {
    AdaDev ad{};
    ad.w2 = (float)(1.0 - b2); ad.w2m1 = ad.w2 - 1.0f; ad.small_w2 = ad.w2 < 0.5f;
    ad.w1 = 1.0f; ad.eps1 = (float)h->eps; ad.has_eps = h->eps > 0.0; ad.clip = 1.0f;
    ad.gc = hp.gc; ad.step = step; ad.k0 = hp.k0; ad.k1 = hp.k1; ad.stats_only = 1;
    ada_finish(ad);
    PlanView v = pl->view;
    KAON_CUDA(cudaMemsetAsync(v.task_counter, 0, pl->counters_bytes - sizeof(unsigned), s));
    const AdaStages st{ph->d_final, ph->n_final, ph->order, ph->d_stats, ph->n_stats,
                       ph->d_strips, ph->n_strips, ph->n_final_items};
    if (int rc = launch_statistics(pl, v, ad, st, s)) return rc;
    if (int rc = launch_small(pl, pl->view, ad, s)) return rc;
    // 2-4. the two sweeps over the flat items
    const int grid = std::min(x.n_items, pl->sm_count * 8);
    const int gridu = std::min((x.n_units + PT_THREADS / 32 - 1) / (PT_THREADS / 32), pl->sm_count * 4);
    if (mk == KAON_M_INT8) {
      pnm_prep_kernel<<<x.n_fact, PT_THREADS, 0, s>>>(pl->view, hp, x);
      pl->launches += 1;
    }
    PnmPass sum = bf ? pick_pass_pt<__nv_bfloat16, false>(mk) : pick_pass_pt<float, false>(mk);
    PnmPass app = bf ? pick_pass_pt<__nv_bfloat16, true>(mk) : pick_pass_pt<float, true>(mk);
    if (!sum || !app) return fail(KAON_E_INVALID, "no AdaPNM kernel for this dtype combination");
    if (gridu > 0) (bf ? pick_sweep_pt<__nv_bfloat16, false>(mk) : pick_sweep_pt<float, false>(mk))<<<gridu, PT_THREADS, 0, s>>>(pl->view, hp, x);
    if (grid > 0) sum<<<grid, PT_THREADS, 0, s>>>(pl->view, hp, x);
    pnm_reduce_kernel<<<x.n_fact, PT_THREADS, 0, s>>>(pl->view, hp, x);
    if (gridu > 0) (bf ? pick_sweep_pt<__nv_bfloat16, true>(mk) : pick_sweep_pt<float, true>(mk))<<<gridu, PT_THREADS, 0, s>>>(pl->view, hp, x);
    if (grid > 0) app<<<grid, PT_THREADS, 0, s>>>(pl->view, hp, x);
    KAON_CUDA(cudaGetLastError());
    pl->launches += 1 + 2 * (gridu > 0) + 2 * (grid > 0);
  }
  if (x.n_flat > 0) {
    PnmPass fl = bf ? pick_flat_pt<__nv_bfloat16>(mk) : pick_flat_pt<float>(mk);
    if (!fl) return fail(KAON_E_INVALID, "no AdaPNM kernel for this dtype combination");
    fl<<<x.n_flat, PT_THREADS, 0, s>>>(pl->view, hp, x);
    KAON_CUDA(cudaGetLastError());
    pl->launches += 1;
  }
  return KAON_OK;
}
