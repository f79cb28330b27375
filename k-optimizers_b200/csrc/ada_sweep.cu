// COUNT and APPLY of the Adakaon family's factored tensors as launches of their own (rows a multiple of eight
// elements; 4-bit blocks of 128).
//
// COUNT: the update chain and the momentum EMA, the kept count of the cautious mask and the row maxima int8 momentum
// is scaled by.  APPLY: the chain again, momentum encoded and stored, weights written; the Nekaon removal of the
// previous climb and the new climb ride on the same read and write of each weight (with weight decay the mask looks
// at the weights after the removal, so then COUNT takes the climb out and APPLY finds the weights without it).
//
// Bound by instruction issue, so the work is arranged for few instructions: a WARP claims a unit of 512..8192
// consecutive elements and streams it, eight elements a lane and trip, with nothing shared between warps: no staging, no
// barrier.  What is per row is one 16-byte table entry (left by FINAL), what is per column two vector loads that hit
// L1; rows and columns advance by an addition, without a division.  Arithmetic is on packed pairs in the
// reference's order of roundings; the mask is one comparison an element; codes are rounded from m' / scale
// as corrected by its exact residual (see store_m8), so no vector needs a second look.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "ada_lists.h"
#include "adakaon_dev.h"
#include "kaon_host.h"
#include "kaon_ops.cuh"
#include "kaon_sweep.cuh"

namespace kaon {

constexpr int SWT = 256;   // threads per CTA

// The vectors first, first + STRIDE, ... of a unit, 32 consecutive ones per warp (`first` includes the lane).  OWN: the
// CTA itself has just written the row table and the column factors.
// MUON (AdaMuon's factored tensors): the signal is the orthogonalised matrix (bf16, `pv.signal`), the chain carries no
// momentum, and the mask compares with the raw gradient.  MS: the build with the Nekaon climb.
// CP (COUNT): with weight decay, where the mask looks at the weights.
template <typename PT, int MKP, bool MUON, bool MS, bool APPLY, bool CP, int STRIDE, bool OWN>
__device__ __forceinline__ void sweep_unit(const PlanView& pv, const AdaDev& hp, const Task& t, const unsigned char* gbase,
                                           const int first, const int lane) {
  using E = Elems<PT>;
  using ST = typename std::conditional<MUON, __nv_bfloat16, PT>::type;
  using S = Elems<ST>;
  constexpr int MK = MUON ? KAON_M_NONE : MKP;
  constexpr bool CODED = MK == KAON_M_INT8 || MK == KAON_M_4BIT;
  constexpr int MBITS = MK == KAON_M_4BIT ? 4 : MK == KAON_M_INT8 ? 8 : MK == KAON_M_BF16 ? 16 : MK == KAON_M_F32 ? 32 : 0;
  // with weight decay the mask looks at the weights after the removal: COUNT writes them, APPLY finds them
  const bool count_p = APPLY ? hp.has_wd && hp.cautious : CP;
  const bool rem_here = MS && hp.remove && (APPLY ? !count_p : count_p);
  const bool need_p = APPLY || count_p;
  const DevTensor& d = pv.tensors[t.tensor];
  const long long e0 = t.e0;
  const int nvec = t.n >> 3;
  const int nv = d.cols >> 3;                       // vectors per row
  const unsigned char* sig = MUON ? reinterpret_cast<const unsigned char*>(pv.signal[t.tensor]) : gbase;
  const unsigned char* sp = sig + (e0 + first * 8) * S::BYTES;
  const unsigned char* rawp = gbase + (e0 + first * 8) * E::BYTES;
  unsigned char* pp = reinterpret_cast<unsigned char*>(d.p) + (e0 + first * 8) * E::BYTES;
  unsigned char* mp = MBITS ? reinterpret_cast<unsigned char*>(d.m) + (e0 + first * 8) * MBITS / 8 : nullptr;
  float* msc = d.m_scale + (MK == KAON_M_4BIT ? (e0 >> 7) + (first >> 4) : 0);
  const float4 scal = __ldcg(reinterpret_cast<const float4*>(pv.aux + aux_scal(d)));
  const float div = scal.y, rcp_div = scal.w;       // the clip divisor
  const bool clipped = div != 1.0f;
  float denom = 1.0f;                               // the kept share
  if (APPLY && hp.cautious)
    denom = fmaxf(__fdiv_rn((float)__ldcg(pv.kept + t.tensor), (float)d.numel), 1e-8f);
  const float nrcp_denom = -__fdiv_rn(1.0f, denom);
  // (plain loads, not the read-only ones: a launch that began early must not have them ahead of its wait)
  const float4* rowtab = reinterpret_cast<const float4*>(pv.aux + aux_rowtab(d));
  const float* cfac = pv.aux + aux_cfac(d);
  unsigned* rowmax = reinterpret_cast<unsigned*>(pv.aux + aux_rowmax(d));
  uint64_t q = (uint64_t)(e0 >> 3) + (unsigned)first;
  // row and vector-in-row of this lane; a trip advances by STRIDE vectors
  int row = t.row0, cv = (t.pad >> 3) + first;
  if (cv >= nv) { const int k = cv / nv; row += k; cv -= k * nv; }
  const int adv_r = STRIDE / nv, adv_c = STRIDE - adv_r * nv;
  f32x2 kept2 = pack2(0.0f, 0.0f);
  // int8 COUNT: every trip lies in one row (rows and the unit's start are whole trips); the running maximum of the row's codes
  const bool whole = !OWN && ((nv | (t.pad >> 3) | nvec) & 31) == 0;
  unsigned run = 0u;

  // int8 momentum: a trip's signal and momentum are loaded by the trip before it, as soon as that has unpacked its own (no
  // register but the words' own), its weights, which are used last, at its start.  (2.6 B list: COUNT 2110 -> 1740 us, APPLY 3921
  // -> 3510.)  Otherwise all at its start: with 4-bit and bf16 momentum the words' registers are short (COUNT 256 -> 278 us on
  // 269 M elements of bf16 momentum when loaded ahead).
  constexpr bool AHEAD = !OWN && MK == KAON_M_INT8;
  W8<ST> gq;
  W8<PT> P, rq;
  MRaw<MK> mq;
  auto load = [&](auto ahead) {
    constexpr int A = decltype(ahead)::value;   // trips ahead
    gq.load(sp + A * STRIDE * 8 * S::BYTES);
    if constexpr (MK != KAON_M_NONE) mq.load(mp + A * STRIDE * MBITS);
    if constexpr (MK == KAON_M_4BIT) mq.sc = msc[A * STRIDE / 16];
    if constexpr (MUON) rq.load(rawp + A * STRIDE * 8 * E::BYTES);
  };
  // a climb of eight elements (reference src/kaon/msam.py:222-230); `wild`: a momentum that decodes to NaN or
  // infinity (a corrupt scale) keeps the reference's nan_to_num
  auto climb8 = [&](const f32x2 M[4], float alpha, float bound, bool wild, f32x2 D[4]) {
    const f32x2 A = pack2(alpha, alpha);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      f32x2 e = mul2(M[j], A);
      if (wild) { if (e.x != e.x) e.x = 0.0f; if (e.y != e.y) e.y = 0.0f; }
      D[j] = pack2(fminf(fmaxf(e.x, -bound), bound), fminf(fmaxf(e.y, -bound), bound));
    }
  };
  auto add_noisy = [&](const f32x2 D[4], uint32_t tag) {
    add_noisy8(hp, d, q, tag, P, D);
  };
  // the vector whose words are in gq, mq; `act`: this lane has one; `more`: and one in the next trip
  auto trip = [&](const bool act, const bool more) {
    if (!AHEAD && act) load(std::integral_constant<int, 0>{});
    const float4 f = rowtab[row];   // {mean, r_i, int8: scale of the stored codes, -}
    if (need_p) P.load(act ? pp : reinterpret_cast<unsigned char*>(d.p));
    f32x2 CF[4], G[4], MO[4];
    {
      const float4* cp = reinterpret_cast<const float4*>(cfac) + 2 * cv;
      const float4 a = cp[0], b = cp[1];
      CF[0] = pack2(a.x, a.y); CF[1] = pack2(a.z, a.w); CF[2] = pack2(b.x, b.y); CF[3] = pack2(b.z, b.w);
    }
    center<ST>(gq, MUON ? 0.0f : f.x, G);
    f32x2 GM[4];   // MUON: the raw gradient, which the mask compares with
    if constexpr (MUON) center<PT>(rq, f.x, GM);
    // ---- stored momentum ----
    float sc_old = 1.0f;
    if constexpr (MK == KAON_M_4BIT) sc_old = mq.sc;
    if constexpr (MK == KAON_M_INT8) sc_old = f.z;
    if constexpr (MK != KAON_M_NONE) mq.decode(sc_old, MO);
    if (AHEAD && more) load(std::integral_constant<int, 1>{});
    if (MS && rem_here) {   // take the previous climb out (the mirrors get the step's last write only)
      f32x2 D[4];
      climb8(MO, hp.a_remove, hp.b_remove, CODED ? !(fabsf(sc_old) <= 3.0e38f) : true, D);
      add_noisy(D, KAON_TAG_REMOVE);
      if (!APPLY && act) P.store(pp, nullptr);
    }
    // ---- u = ((g r) c) / div * scale (reference src/kaon/adakaon.py:885-888), m' = lerp(m, u) ----
    // (the same roundings in COUNT and APPLY: what is counted is what APPLY keeps, also where an ulp turns a sign)
    f32x2 MN[4], F[4];
    const f32x2 RF = pack2(f.y, f.y);
#pragma unroll
    for (int j = 0; j < 4; ++j) MN[j] = mul2(mul2(G[j], RF), CF[j]);
    if (clipped) {
      const f32x2 DIVN = pack2(-div, -div), RCPD = pack2(rcp_div, rcp_div);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const f32x2 qq = mul2(MN[j], RCPD);
        MN[j] = fma2(fma2(qq, DIVN, MN[j]), RCPD, qq);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      MN[j] = mul2(MN[j], pack2(hp.upd_scale, hp.upd_scale));
      if constexpr (MK == KAON_M_BF16) {
        const uint32_t ub = pack_bf16_rn(MN[j].x, MN[j].y);
        MN[j] = pack2(bf16lo(ub), bf16hi(ub));
      }
    }
    if constexpr (MK != KAON_M_NONE) {
      if (hp.small_w1) {
#pragma unroll
        for (int j = 0; j < 4; ++j) MN[j] = fma2(pack2(hp.w1, hp.w1), sub2(MN[j], MO[j]), MO[j]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) MN[j] = fma2(pack2(hp.w1m1, hp.w1m1), sub2(MN[j], MO[j]), MN[j]);
      }
    }
    if constexpr (MK == KAON_M_BF16) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t mb = pack_bf16_rn(MN[j].x, MN[j].y);
        MN[j] = pack2(bf16lo(mb), bf16hi(mb));
      }
    }
    // ---- delta = m' + (lr wd) p; the mask; APPLY: the update, negated: -(delta if kept else 0) / (kept / numel) ----
#pragma unroll
    for (int j = 0; j < 4; ++j) F[j] = MN[j];
    if (APPLY ? hp.has_wd != 0 : CP) {
#pragma unroll
      for (int j = 0; j < 4; ++j) F[j] = fma2(P.pair(j), pack2(hp.lrwd, hp.lrwd), F[j]);
    }
    f32x2 K[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const f32x2 X = mul2(F[j], MUON ? GM[j] : G[j]);
      K[j] = pack2(gt0_or(X.x, hp.mask_off), gt0_or(X.y, hp.mask_off));
    }
    if constexpr (!APPLY) {
      if (act) kept2 = add2(kept2, add2(add2(K[0], K[1]), add2(K[2], K[3])));
      if constexpr (MK == KAON_M_INT8) {
        unsigned bits = act ? __float_as_uint(amax8(MN)) : 0u;
        if (whole) {   // to the row's atomic when it ends
          run = max(run, bits);
          if (cv + adv_c >= nv || adv_r > 0 || !more) {
            run = __reduce_max_sync(0xffffffffu, run);
            if (lane == 0) atomicMax(rowmax + row, run);
            run = 0u;
          }
          return;
        }
        const int row_l0 = __shfl_sync(0xffffffffu, row, 0);
        if (__all_sync(0xffffffffu, !act || row == row_l0)) {
          bits = __reduce_max_sync(0xffffffffu, bits);
          if (lane == 0) atomicMax(rowmax + row_l0, bits);
        } else if (act) {
          atomicMax(rowmax + row, bits);
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {   // minus the correctly rounded quotient
        const f32x2 NR = pack2(nrcp_denom, nrcp_denom), qq = mul2(F[j], NR);
        F[j] = mul2(fma2(fma2(qq, pack2(denom, denom), F[j]), NR, qq), K[j]);
      }
      // ---- store the new momentum; MO <- the momentum as stored ----
      float sc = 1.0f;
      if constexpr (MK != KAON_M_NONE) {
        float amax = 0.0f;
        if constexpr (MK == KAON_M_INT8) amax = __uint_as_float(OWN ? __ldcg(rowmax + row) : rowmax[row]);
        sc = store_m8<MK>(mp, MN, amax, act ? 8 : 0, lane, MS ? MO : nullptr);
        if constexpr (MK == KAON_M_4BIT) { if (act && (lane & 15) == 0) stg_f32(msc, sc); }
        if constexpr (MK == KAON_M_INT8) { if (act && cv == 0) msc[row] = sc; }
      }
      // ---- weights: p <- round(p - update), then the climb from the momentum as stored ----
      write8(hp, d, q, act, P, F);
      if (MS && hp.climb) {
        f32x2 D[4];
        climb8(MO, hp.a_climb, hp.b_climb, CODED ? !(sc <= 3.0e38f) : true, D);
        add_noisy(D, KAON_TAG_CLIMB);
      }
      if (act) P.store(pp, &pv.peers);
    }
  };
  auto advance = [&]() {
    sp += STRIDE * 8 * S::BYTES;
    rawp += STRIDE * 8 * E::BYTES;
    pp += STRIDE * 8 * E::BYTES;
    if constexpr (MBITS > 0) mp += STRIDE * MBITS;
    if constexpr (MK == KAON_M_4BIT) msc += STRIDE / 16;
    q += STRIDE;
    row += adv_r;
    cv += adv_c;
    if (cv >= nv) { cv -= nv; ++row; }
  };
  const int left = nvec - (first - lane);                 // vectors from the warp's first on
  int full = left >= 32 ? (left - 32) / STRIDE + 1 : 0;   // trips of the whole warp
  const int tail = left - full * STRIDE;
  const bool act = lane < tail;                           // in a tensor's last vectors
  if (AHEAD && (full > 0 || act)) load(std::integral_constant<int, 0>{});
  for (; full > 0; --full) {
    trip(true, full > 1 || act);
    advance();
  }
  if (tail > 0) {
    if (!act) { row = t.row0; cv = 0; }   // (in bounds; what such a lane computes is of no consequence)
    trip(act, false);
  }
  if constexpr (!APPLY) {
    const unsigned kept = __reduce_add_sync(0xffffffffu, (unsigned)(kept2.x + kept2.y + 0.5f));
    if (lane == 0 && kept) atomicAdd(pv.kept + t.tensor, kept);
  }
}

template <typename PT, int MKP, bool MUON, bool MS, bool APPLY, bool CP>
__global__ void __launch_bounds__(SWT, 4) ada_sweep_kernel(const __grid_constant__ PlanView pv, const __grid_constant__ AdaDev hp) {
  if (on_reserved_sm(pv.sm_reserve)) return;
  early_launch();
  after_launch_before();
  const int lane = threadIdx.x & 31;
  // The first unit is the warp's own number (with reserved multiprocessors, whose warps leave, a claimed one), the
  // others are claimed, one ahead.
  const int warps = pv.sm_reserve ? 0 : (int)gridDim.x * (SWT / 32);
  auto claim = [&]() -> int {
    int i = 0x7fffffff;
    if (lane == 0 && warps < pv.n_tasks) {
      const unsigned st = *reinterpret_cast<volatile unsigned*>(pv.status);
      if (!st) i = warps + (int)atomicAdd(pv.task_counter, 1u);
    }
    return i;   // lane 0's: broadcast where it is used, so that the atomic is in flight meanwhile
  };
  // (by a broadcast, so that the compiler knows the number, and all that follows from it, to be the warp's own)
  int cur = __shfl_sync(0xffffffffu, warps ? (int)(blockIdx.x * (SWT / 32) + (threadIdx.x >> 5)) : claim(), 0);
  while (cur < pv.n_tasks) {
    const int next = claim();
    const Task t = pv.tasks[cur];
    const unsigned char* gbase = reinterpret_cast<const unsigned char*>(pv.grads[t.tensor]);
    if (gbase != nullptr) sweep_unit<PT, MKP, MUON, MS, APPLY, CP, 32, false>(pv, hp, t, gbase, lane, lane);
    cur = __shfl_sync(0xffffffffu, next, 0);
  }
}

// ----------------------------------------------------------------------------- small tensors

// A factored tensor of at most ADA_SMALL_MAX elements in ONE CTA: row statistics, column statistics, clip divisor,
// COUNT and APPLY with barriers in between.  A list of adapter matrices has hundreds of them, each far too small to
// share out; as items of the stages above they spent the step waiting for one another (720 matrices of 10 240
// elements: 700 us).  The gradient is kept in shared memory for the statistics.  Sums in a fixed order.
// Bound by the latency of a matrix's phases, so by the rounds of blocks a list takes: BLOCKS of them an SM (small_takes_five).
__device__ __forceinline__ double small_sum(double v, double* red, int tid) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((tid & 31) == 0) red[tid >> 5] = v;
  __syncthreads();
  double t = 0.0;
#pragma unroll
  for (int w = 0; w < SWT / 32; ++w) t += red[w];
  return t;
}

template <typename PT, int MKP, bool MUON, bool MS, int BLOCKS>
__global__ void __launch_bounds__(SWT, BLOCKS) ada_small_kernel(const __grid_constant__ PlanView pv, const __grid_constant__ AdaDev hp) {
  using ST = typename std::conditional<MUON, __nv_bfloat16, PT>::type;
  using S = Elems<ST>;
  extern __shared__ __align__(128) unsigned char g_s[];
  __shared__ double red[SWT / 32];
  __shared__ float xs[2][SWT];
  const int tid = threadIdx.x, lane = tid & 31;
  const int ti = pv.tasks[blockIdx.x].tensor;
  const unsigned char* g = reinterpret_cast<const unsigned char*>(pv.grads[ti]);
  if (g == nullptr) return;
  const DevTensor d = pv.tensors[ti];
  const unsigned char* sig = MUON ? reinterpret_cast<const unsigned char*>(pv.signal[ti]) : g;
  const int n = (int)d.numel, R = d.rows, C = d.cols;
  const bool gc = hp.gc != 0 && !MUON;   // AdaMuon's statistics are of a matrix that is not centralised
#pragma unroll 4
  for (int k = tid; k < n * S::BYTES / 16; k += SWT)
    reinterpret_cast<uint4*>(g_s)[k] = reinterpret_cast<const uint4*>(sig)[k];
  __syncthreads();
  // ---- rows: T consecutive threads each, T a power of two of at least one vector a thread; the centralised gradient
  //      goes back to shared memory, 1 / row statistic to the scratch ----
  const int nv = C >> 3;
  int T = 1;
  while (T < 32 && T < nv) T *= 2;
  const int per = SWT / T, sub = tid & (T - 1), rr = tid / T;
  float4* rowtab = reinterpret_cast<float4*>(pv.aux + aux_rowtab(d));
  auto row_sum = [&](float part) -> float {
    double v = (double)part;
    for (int o = T >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return (float)v;
  };
  const f32x2 EPS = pack2(hp.eps1, hp.eps1);
  double rowsum = 0.0;
  for (int r0 = 0; r0 < R; r0 += per) {
    const int r = r0 + rr;
    const bool act = r < R;
    const int vecs = act ? nv : 0;   // (a thread without a row reads none: its owner writes it back meanwhile)
    unsigned char* rowp = g_s + (size_t)(act ? r : 0) * C * S::BYTES;
    float mu = 0.0f;
    if (gc) {
      float s = 0.0f;
      for (int v = sub; v < vecs; v += T) {
        W8<ST> x;
        x.load(rowp + (size_t)v * 8 * S::BYTES);
        const f32x2 a = add2(add2(x.pair(0), x.pair(1)), add2(x.pair(2), x.pair(3)));
        s += a.x + a.y;
      }
      mu = __fdiv_rn(row_sum(s), (float)C);
      if (S::IS_BF16) mu = round_bf16(mu);
    }
    const float mb = S::IS_BF16 ? __uint_as_float(pack_bf16_rn(mu, mu)) : mu;
    float s2 = 0.0f;
    for (int v = sub; v < vecs; v += T) {
      W8<ST> x;
      f32x2 y[4];
      x.load(rowp + (size_t)v * 8 * S::BYTES);
      center<ST>(x, mb, y);
      f32x2 a = pack2(0.0f, 0.0f);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        a = add2(a, add2(mul2(y[j], y[j]), EPS));
        x.set(j, y[j]);
      }
      s2 += a.x + a.y;
      x.store(rowp + (size_t)v * 8 * S::BYTES, nullptr);
    }
    s2 = row_sum(s2);
    if (act && sub == 0) {
      const float rn = lerp_torch(d.stat_a[r], __fdiv_rn(s2, (float)C), hp.w2, hp.w2m1, hp.small_w2 != 0);
      d.stat_a[r] = rn;
      if (gc) pv.aux[aux_mean(d) + r] = mu;
      const float raw_mu = (MUON && hp.gc) ? pv.aux[aux_mean(d) + r] : mu;
      if (hp.int8) reinterpret_cast<unsigned*>(pv.aux + aux_rowmax(d))[r] = 0u;
      rowtab[r] = make_float4(Elems<PT>::IS_BF16 ? __uint_as_float(pack_bf16_rn(raw_mu, raw_mu)) : raw_mu, __fdiv_rn(1.0f, rn),
                              hp.int8 ? d.m_scale[r] : 1.0f, 0.0f);
      rowsum += (double)rn;
    }
  }
  const double rs = small_sum(rowsum, red, tid);
  const float rowmean = __fdiv_rn((float)rs, (float)R);
  __syncthreads();
  // ---- columns: with fewer than SWT of them, SWT / C threads to a column (every Q-th row), added in order ----
  float* cfac = pv.aux + aux_cfac(d);
  double tl = 0.0;
  const int Q = C >= SWT ? 1 : SWT / C, q = C >= SWT ? 0 : tid / C;
  for (int c0 = 0; c0 < C; c0 += SWT) {
    const int c = c0 + (C >= SWT ? tid : tid - q * C);
    const bool act = c < C && q < Q;
    float a1 = 0.0f, a2 = 0.0f;
    if (act) {
#pragma unroll 4
      for (int r = q; r < R; r += Q) {
        const float x = S::load1(g_s, r * C + c);
        const float sq = __fmul_rn(x, x);
        a1 += __fadd_rn(sq, hp.eps1);
        a2 = __fmaf_rn(sq, rowtab[r].y, a2);
      }
    }
    if (Q > 1) {
      // power-of-two rows of at most a warp: the groups of a warp first, by shuffles
      int G = Q, stride = C;
      if (C < 32 && (C & (C - 1)) == 0) {
        for (int o = C; o < 32; o <<= 1) {
          a1 += __shfl_xor_sync(0xffffffffu, a1, o);
          a2 += __shfl_xor_sync(0xffffffffu, a2, o);
        }
        G = SWT / 32; stride = 32;
      }
      xs[0][tid] = a1; xs[1][tid] = a2;
      __syncthreads();
      if (tid < C) {
        a1 = a2 = 0.0f;
        for (int k = 0; k < G; ++k) { a1 += xs[0][k * stride + tid]; a2 += xs[1][k * stride + tid]; }
      }
    }
    if (act && q == 0) {
      const float cn = lerp_torch(d.stat_b[c], __fdiv_rn(a1, (float)R), hp.w2, hp.w2m1, hp.small_w2 != 0);
      d.stat_b[c] = cn;
      cfac[c] = rsqrt_torch(cn);
      tl += (double)a2 / (double)cn;
    }
  }
  const double T2 = small_sum(tl, red, tid);
  // ---- the whole tensor: mean(row), rms, clip divisor; r_i of every row ----
  const double ss = (double)rowmean * T2;
  const float rms = __fdiv_rn((float)sqrt(ss), (float)sqrt((double)R * (double)C));
  const float div = fmaxf(__fdiv_rn(rms, hp.clip), 1.0f);
  if (tid == 0) *reinterpret_cast<float4*>(pv.aux + aux_scal(d)) = make_float4(rowmean, div, rms, __fdiv_rn(1.0f, div));
  for (int r = tid; r < R; r += SWT) {
    const float rf = rsqrt_torch(__fdiv_rn(d.stat_a[r], rowmean));
    rowtab[r].y = rf;
    pv.aux[aux_rfac(d) + r] = rf;
  }
  if (hp.stats_only) return;
  __syncthreads();
  const Task t{ti, 0, 0, n, 0, 0, 0};
  if (hp.cautious || hp.int8) {
    if (hp.has_wd && hp.cautious) sweep_unit<PT, MKP, MUON, MS, false, true, SWT, true>(pv, hp, t, g, tid, lane);
    else sweep_unit<PT, MKP, MUON, MS, false, false, SWT, true>(pv, hp, t, g, tid, lane);
    __threadfence_block();
    __syncthreads();
  }
  sweep_unit<PT, MKP, MUON, MS, true, false, SWT, true>(pv, hp, t, g, tid, lane);
}

// ----------------------------------------------------------------------------- host

typedef void (*SweepKernel)(PlanView, AdaDev);

template <typename PT, bool MS, bool APPLY, bool CP>
static SweepKernel pick_sweep_pt(int mk) {
  switch (mk) {
    case KAON_M_F32: return ada_sweep_kernel<PT, KAON_M_F32, false, MS, APPLY, CP>;
    case KAON_M_BF16: return ada_sweep_kernel<PT, KAON_M_BF16, false, MS, APPLY, CP>;
    case KAON_M_INT8: return ada_sweep_kernel<PT, KAON_M_INT8, false, MS, APPLY, CP>;
    case KAON_M_4BIT: return ada_sweep_kernel<PT, KAON_M_4BIT, false, MS, APPLY, CP>;
    case KAON_M_NONE: return ada_sweep_kernel<PT, KAON_M_NONE, false, false, APPLY, CP>;
    default: return nullptr;
  }
}
template <bool APPLY, bool CP>
static SweepKernel pick_sweep(int pdt, int mk, bool muon, bool ms) {
  const bool bf = pdt == KAON_DT_BF16;
  if (muon) return bf ? ada_sweep_kernel<__nv_bfloat16, KAON_M_NONE, true, false, APPLY, CP> : ada_sweep_kernel<float, KAON_M_NONE, true, false, APPLY, CP>;
  if (ms) return bf ? pick_sweep_pt<__nv_bfloat16, true, APPLY, CP>(mk) : pick_sweep_pt<float, true, APPLY, CP>(mk);
  return bf ? pick_sweep_pt<__nv_bfloat16, false, APPLY, CP>(mk) : pick_sweep_pt<float, false, APPLY, CP>(mk);
}

typedef void (*SmallKernel)(PlanView, AdaDev);
template <typename PT, bool MS, int BLOCKS>
static SmallKernel pick_small_pt(int mk) {
  switch (mk) {
    case KAON_M_F32: return ada_small_kernel<PT, KAON_M_F32, false, MS, BLOCKS>;
    case KAON_M_BF16: return ada_small_kernel<PT, KAON_M_BF16, false, MS, BLOCKS>;
    case KAON_M_INT8: return ada_small_kernel<PT, KAON_M_INT8, false, MS, BLOCKS>;
    case KAON_M_4BIT: return ada_small_kernel<PT, KAON_M_4BIT, false, MS, BLOCKS>;
    case KAON_M_NONE: return ada_small_kernel<PT, KAON_M_NONE, false, false, BLOCKS>;
    default: return nullptr;
  }
}
template <int BLOCKS>
static SmallKernel pick_small(int pdt, int mk, bool muon, bool ms) {
  const bool bf = pdt == KAON_DT_BF16;
  if (muon) return bf ? ada_small_kernel<__nv_bfloat16, KAON_M_NONE, true, false, BLOCKS> : ada_small_kernel<float, KAON_M_NONE, true, false, BLOCKS>;
  if (ms) return bf ? pick_small_pt<__nv_bfloat16, true, BLOCKS>(mk) : pick_small_pt<float, true, BLOCKS>(mk);
  return bf ? pick_small_pt<__nv_bfloat16, false, BLOCKS>(mk) : pick_small_pt<float, false, BLOCKS>(mk);
}

// The plan's small tensors (their statistics only, for AdaPNM and KProdigy).
int launch_small(kaon_plan* pl, const PlanView& base, const AdaDev& hp, cudaStream_t s) {
  if (pl->n_tasks_small == 0) return KAON_OK;
  const bool muon = pl->optimizer == KAON_OPT_ADAMUON;
  const bool ms = hp.remove || hp.climb;
  const int mk = hp.stats_only ? KAON_M_NONE : pl->momentum_kind;
  SmallKernel k = pick_small<4>(pl->param_dtype, mk, muon, ms);
  if (!k) return fail(KAON_E_INVALID, "no Adakaon kernel for this dtype combination");
  const size_t smem = (size_t)pl->small_max * (muon || pl->param_dtype == KAON_DT_BF16 ? 2 : 4);
  const SmallKernel five = pick_small<5>(pl->param_dtype, mk, muon, ms);
  int* blocks = pl->small_blocks[ms];
  if (blocks[0] == 0) {
    KAON_CUDA(cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, ADA_SMALL_MAX * 4));
    KAON_CUDA(cudaFuncSetAttribute((const void*)five, cudaFuncAttributeMaxDynamicSharedMemorySize, ADA_SMALL_MAX * 4));
    KAON_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks[1], (const void*)five, SWT, smem));
    KAON_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks[0], (const void*)k, SWT, smem));
  }
  if (small_takes_five(pl->n_tasks_small, blocks[0], blocks[1], pl->sm_count)) k = five;
  PlanView v = base;
  v.tasks = pl->d_tasks_small;
  v.n_tasks = pl->n_tasks_small;
  k<<<pl->n_tasks_small, SWT, smem, s>>>(v, hp);
  KAON_CUDA(cudaGetLastError());
  pl->launches += 1;
  return KAON_OK;
}

// The units of the tensors marked in `elig`: as large as leaves each warp of the machine a dozen (a warp's time per
// unit is then small beside the launch's), at most 8192 elements, where the fetches at a unit's head cost little.  AdaMuon's
// chain is short (no momentum), so that a unit's head and its claim cost more beside it: three to a warp, at most 32 768 elements
// (COUNT of four width-3072 blocks 617 -> 313 us, 334 since it rounds as APPLY does; Nekaon's APPLY, on 269 M elements,
// 568 -> 625 with such units).
void sweep_units(const kaon_plan* pl, const std::vector<char>& elig, std::vector<Task>& out) {
  const bool muon = pl->optimizer == KAON_OPT_ADAMUON;
  long long total = 0;
  for (int i = 0; i < pl->n_tensors; ++i) if (elig[i]) total += pl->h_tensors[i].numel;
  long long u = muon ? 32768 : 8192;
  while (u > 512 && total / u < (muon ? 3ll : 12ll) * pl->sm_count * 32) u /= 2;
  for (int i = 0; i < pl->n_tensors; ++i) {
    if (!elig[i]) continue;
    const DevTensor& t = pl->h_tensors[i];
    for (long long e = 0; e < t.numel; e += u)
      out.push_back(Task{i, PH_ADA_APPLY, e, (int)std::min<long long>(u, t.numel - e), (int)(e / t.cols), 0, (int)(e % t.cols)});
  }
}

// The COUNT (where something is counted) and APPLY launches over the plan's units; `base` carries the plan's
// pointers (and AdaMuon's signal column).
int launch_count_apply(kaon_plan* pl, const PlanView& base, const AdaDev& hp, cudaStream_t s) {
  const bool muon = pl->optimizer == KAON_OPT_ADAMUON;
  const bool ms = hp.remove || hp.climb;
  PlanView va = base;
  va.tasks = pl->d_tasks_apply2;
  va.n_tasks = pl->n_tasks_apply2;
  if (va.n_tasks == 0) return KAON_OK;
  const int want = (pl->n_tasks_apply2 + SWT / 32 - 1) / (SWT / 32), most = pl->sm_count * 4;
  const int grid = base.sm_reserve ? most : std::max(1, std::min(want, most));
  if (hp.cautious || hp.int8) {
    va.task_counter = base.counters2 + 1;
    SweepKernel k = hp.has_wd && hp.cautious ? pick_sweep<false, true>(pl->param_dtype, pl->momentum_kind, muon, ms)
                                             : pick_sweep<false, false>(pl->param_dtype, pl->momentum_kind, muon, false);
    KAON_CUDA(launch_early(!base.sm_reserve, k, grid, SWT, 0, s, va, hp));
    pl->launches += 1;
  }
  va.task_counter = base.counters2 + 2;
  KAON_CUDA(launch_early(!base.sm_reserve, pick_sweep<true, false>(pl->param_dtype, pl->momentum_kind, muon, ms), grid, SWT, 0, s, va, hp));
  pl->launches += 1;
  return KAON_OK;
}

}  // namespace kaon
