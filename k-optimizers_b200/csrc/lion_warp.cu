// The cautious Lion step, a warp per unit of 512 to 16384 consecutive elements, nothing shared between warps.
//
// MAIN unit: the means of the rows it touches, then per eight elements of a lane the direction sign(b1*m + (1-b1)*g), the
// new momentum, its codes, and two bits an element for APPLY (element e, o of a pair: nibble kept_e | kept_o << 1 |
// neg_e << 2 | neg_o << 3; with weight decay (w_e + 1) + 4 (w_o + 1), w the update's sign or 2 where masked out).  APPLY unit: once every MAIN
// unit of the tensor has finished, the weights with the tensor-wide rescale 1/max(kept/numel, 1e-8).  Units are claimed in
// list order, all of MAIN first; small lists are one launch, large ones a launch each (see lion_warp_units).
//
// Bound by instruction issue (4-bit momentum: MAIN 69 % of the slots, 224 warp instructions per 256 elements) or HBM (wider
// states; APPLY 5.3 TB/s), so: packed pairs; the mask from the sign bytes of the products; momentum codes packed as small
// integers by FMAs; rows advanced by an addition; the next trip's words loaded ahead; no staging and no barrier.  (Rows staged in shared memory by a CTA per 16 K-element item: 5.30 ms on the
// 2.6 B-parameter list with 4-bit momentum, 267 us on ragged fp32 lists.)
#include <algorithm>
#include <type_traits>
#include <vector>

#include "kaon_host.h"
#include "kaon_ops.cuh"
#include "kaon_sweep.cuh"
#include "lion_dev.h"

namespace kaon {

constexpr int LWT = 256;            // threads per CTA
constexpr int LW_ROWS = 64;         // rows a unit may touch
constexpr int LW_MAX_COLS = 16384;  // longer rows: the staged kernel, whose row means come from a launch of their own

// Eight consecutive elements of which `cnt` exist (the end of a tensor whose length is no multiple of eight)
template <typename T>
__device__ __forceinline__ void load_some(W8<T>& w, const void* p, int cnt) {
  float x[8];
  load8_guard<T>(p, cnt, x);
#pragma unroll
  for (int j = 0; j < 4; ++j) w.set(j, pack2(x[2 * j], x[2 * j + 1]));
}
__device__ __forceinline__ void load_some(MRaw<KAON_M_4BIT>& w, const void* p, int cnt) {
  w.w = 0x88888888u;
#pragma unroll
  for (int b = 0; b < 4; ++b)
    if (2 * b < cnt) w.w = (w.w & ~(0xffu << (8 * b))) | ((uint32_t) reinterpret_cast<const unsigned char*>(p)[b] << (8 * b));
  if (cnt & 1) w.w = (w.w & ~(0xfu << (4 * cnt))) | (8u << (4 * cnt));
}
template <typename T>
__device__ __forceinline__ void load_some(MPlain<T>& w, const void* p, int cnt) { load_some(w.w, p, cnt); }

// SIGNAL: APPLY units of the same launch wait for this one.
template <typename PT, int MK, bool WD, bool SIGNAL>
__device__ __forceinline__ void lion_main_unit(const PlanView& pv, const LionDev& hp, const Task& t, const unsigned char* gbase,
                                               float* mean_s, const int lane) {
  using E = Elems<PT>;
  constexpr int MV = MBytes<MK>::V;
  const DevTensor& d = pv.tensors[t.tensor];
  const bool gc = hp.gc && d.rows > 0;
  const int C = d.cols;
  // rows that start on vector and block boundaries go one by one (mean and sweep of a row back to back: the second
  // reading hits L1); others with the whole unit's means first
  const bool by_row = gc && (C & 127) == 0 && C >= 512;
  const int seg = by_row ? C : t.n;
  const float fC = (float)C, rC = __frcp_rn(fC);
  unsigned kept = 0;
  for (int s0 = 0; s0 < t.n; s0 += seg) {
    const int n = min(seg, t.n - s0);
    const long long e0 = t.e0 + s0;
    const unsigned char* gp = gbase + e0 * E::BYTES;
    const unsigned char* pp = reinterpret_cast<const unsigned char*>(d.p) + e0 * E::BYTES;
    unsigned char* mp = reinterpret_cast<unsigned char*>(d.m) + (e0 >> 3) * MV;
    float* scp = MK == KAON_M_4BIT ? d.m_scale + (e0 >> 7) : nullptr;
    uint16_t* cp = reinterpret_cast<uint16_t*>(pv.codes + d.code_off + (e0 >> 2));
    const int nvec = n >> 3;

    W8<PT> gq;
    MRaw<MK> mq;
    W8<PT> P;
    auto load = [&](unsigned v) {
      gq.load(gp + v * (8u * E::BYTES));
      mq.load(mp + v * (unsigned)MV);
      if constexpr (MK == KAON_M_4BIT) mq.sc = scp[v >> 4];
      if constexpr (WD) P.load(pp + v * (8u * E::BYTES));
    };
    if (lane < nvec) load((unsigned)lane);   // in flight over the means
    float mean = 0.0f;   // by_row: the segment's
    if (by_row) {
      mean = round_to(div_by(warp_sum(row_part<PT>(gp, C, lane)), fC, rC), PT());
    } else if (gc) {
      __syncwarp();
      row_means<PT>(gbase, C, t.row0, (t.pad + n + C - 1) / C, lane, [&](int r, float mean) { mean_s[r] = mean; });
      __syncwarp();
    }
    const float mean_bits = E::IS_BF16 ? __uint_as_float(pack_bf16_rn(mean, mean)) : mean;
    // row (of the unit's) and column of the lane's next vector; a trip advances by 256 elements
    int lr = 0, col = t.pad + lane * 8;
    if (gc && !by_row && col >= C) { const int k = col / C; lr = k; col -= k * C; }
    const int adv_r = gc ? 256 / C : 0, adv_c = 256 - adv_r * C;

    // the vector in g, m, p; `cnt` of its elements exist (8 but at the end of a tensor)
    auto trip = [&](const W8<PT>& g, const MRaw<MK>& m, const W8<PT>& p, const unsigned v, const int cnt, auto rows_tag) {
      constexpr int ROWS = decltype(rows_tag)::value;   // 0: one mean, 1: a row per vector, 2: rows end inside vectors
      f32x2 G[4], MO[4], CD[4], N[4];
      if constexpr (ROWS == 0) {
        center<PT>(g, mean_bits, G);
      } else if constexpr (ROWS == 1) {
        const float mu = mean_s[lr];
        center<PT>(g, E::IS_BF16 ? __uint_as_float(pack_bf16_rn(mu, mu)) : mu, G);
      } else {
        float mu[8];
        if (C >= 8) {
          const float a = mean_s[lr], b = mean_s[min(lr + 1, LW_ROWS - 1)];
#pragma unroll
          for (int k = 0; k < 8; ++k) mu[k] = k < C - col ? a : b;
        } else {
          int r = lr, c = col;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            mu[k] = mean_s[min(r, LW_ROWS - 1)];
            if (++c >= C) { c = 0; ++r; }
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          G[j] = sub2(g.pair(j), pack2(mu[2 * j], mu[2 * j + 1]));
          if constexpr (E::IS_BF16) {
            const uint32_t w = pack_bf16_rn(G[j].x, G[j].y);
            G[j] = pack2(bf16lo(w), bf16hi(w));
          }
        }
      }
      float sc_old = 1.0f;
      if constexpr (MK == KAON_M_4BIT) sc_old = m.sc;
      m.decode(sc_old, MO);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        CD[j] = fma2(G[j], pack2(hp.w1, hp.w1), mul2(MO[j], pack2(hp.b1, hp.b1)));
        N[j] = fma2(G[j], pack2(hp.w2, hp.w2), mul2(MO[j], pack2(hp.b2, hp.b2)));
      }
      uint32_t code;
      if constexpr (!WD) {
        // kept: direction and gradient have the same sign; the update's sign is then the gradient's
        float x[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) unpack2(mul2(CD[j], G[j]), x[2 * j], x[2 * j + 1]);
        float low = min3f(fabsf(x[0]), fabsf(x[1]), fabsf(x[2]));
        low = min3f(low, fabsf(x[3]), fabsf(x[4]));
        low = min3f(low, fabsf(x[5]), fabsf(x[6]));
        low = fminf(low, fabsf(x[7]));
        // bytes 0xFF where the product is negative (masked out), where the gradient is negative
        auto signs = [](float a, float b, float c, float d) {
          return prmt(prmt(__float_as_uint(a), __float_as_uint(b), 0x00FBu), prmt(__float_as_uint(c), __float_as_uint(d), 0x00FBu), 0x5410u);
        };
        const uint32_t a_lo = signs(x[0], x[1], x[2], x[3]), a_hi = signs(x[4], x[5], x[6], x[7]);
        const uint32_t g_lo = signs(G[0].x, G[0].y, G[1].x, G[1].y), g_hi = signs(G[2].x, G[2].y, G[3].x, G[3].y);
        // element b of each four lives in byte b: kept bits 0,1,4,5 and neg bits 2,3,6,7 of the code byte, all disjoint, so
        // that the sum of the bytes (top byte of t * 0x01010101) is their OR
        const uint32_t t_lo = ~a_lo & ((g_lo & 0x80400804u) | 0x20100201u);
        const uint32_t t_hi = ~a_hi & ((g_hi & 0x80400804u) | 0x20100201u);
        code = prmt(t_lo * 0x01010101u, t_hi * 0x01010101u, 0x0073u) & 0xffffu;
        if (!(low > 0.0f)) {   // a zero, or a product that underflows: by comparisons
          code = 0u;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const float c = k & 1 ? CD[k >> 1].y : CD[k >> 1].x, gr = k & 1 ? G[k >> 1].y : G[k >> 1].x;
            const uint32_t bit = 1u << (4 * (k >> 1) + (k & 1));
            if (c > 0.0f && gr > 0.0f) code |= bit;
            if (c < 0.0f && gr < 0.0f) code |= 5u * bit;
          }
        }
        if (cnt < 8) {
#pragma unroll
          for (int k = 0; k < 8; ++k) if (k >= cnt) code &= ~(5u << (4 * (k >> 1) + (k & 1)));
        }
        kept += __popc(code & 0x3333u);
      } else {
        f32x2 W[4];
        auto one = [&](float c, float gr, float w) {
          const float s = c > 0.0f ? 1.0f : (c < 0.0f ? -1.0f : 0.0f);
          return __fmul_rn(__fmaf_rn(w, hp.wd, s), gr) > 0.0f ? s : 2.0f;
        };
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const f32x2 w = p.pair(j);
          W[j] = pack2(one(CD[j].x, G[j].x, w.x), one(CD[j].y, G[j].y, w.y));
        }
        // sum of (w_k + 1) 4^k, exact in fp32, in the low 16 mantissa bits
        const f32x2 K16 = pack2(16.0f, 16.0f);
        const f32x2 D = fma2(fma2(W[3], K16, W[2]), pack2(256.0f, 256.0f), fma2(W[1], K16, W[0]));
        code = __float_as_uint(__fadd_rn(__fmaf_rn(D.y, 4.0f, D.x), 8388608.0f + 21845.0f)) & 0xffffu;
        if (cnt < 8) code |= 0xffffu & ~((1u << (2 * cnt)) - 1u);
        kept += 8u - __popc(code & (code >> 1) & 0x5555u);
      }
      if (cnt < 8) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (k >= cnt) { if (k & 1) N[k >> 1].y = 0.0f; else N[k >> 1].x = 0.0f; }
      }
      if constexpr (MK == KAON_M_BF16) {
#pragma unroll
        for (int j = 0; j < 4; ++j) N[j] = pack2(round_bf16(N[j].x), round_bf16(N[j].y));
      }
      const float sc = store_m8<MK>(mp + v * (unsigned)MV, N, 0.0f, cnt, lane);
      if constexpr (MK == KAON_M_4BIT) { if (cnt > 0 && (lane & 15) == 0) stg_f32(scp + (v >> 4), sc); }
      if (cnt > 0) stg_u16(cp + v, code);
    };
    auto sweep = [&](auto rows_tag) {
      int v0 = 0;
      for (; v0 + 32 <= nvec; v0 += 32) {
        const W8<PT> g = gq;
        const MRaw<MK> m = mq;
        const W8<PT> p = P;
        const unsigned v = (unsigned)(v0 + lane);
        if (v + 32u < (unsigned)nvec) load(v + 32u);
        trip(g, m, p, v, 8, rows_tag);
        if constexpr (decltype(rows_tag)::value != 0) {
          lr += adv_r;
          col += adv_c;
          if (col >= C) { col -= C; ++lr; }
        }
      }
      if (v0 * 8 < n) {   // the last trip of the unit
        const unsigned v = (unsigned)(v0 + lane);
        const int cnt = max(0, min(8, n - (int)v * 8));
        if (cnt > 0 && cnt < 8) {
          load_some(gq, gp + v * (8u * E::BYTES), cnt);
          load_some(mq, mp + v * (unsigned)MV, cnt);
          if constexpr (MK == KAON_M_4BIT) mq.sc = scp[v >> 4];
          if constexpr (WD) load_some(P, pp + v * (8u * E::BYTES), cnt);
        } else if (cnt == 0) {
#pragma unroll
          for (int j = 0; j < 4; ++j) { gq.set(j, pack2(0.0f, 0.0f)); if constexpr (WD) P.set(j, pack2(0.0f, 0.0f)); }
          load_some(mq, nullptr, 0);
          if constexpr (MK == KAON_M_4BIT) mq.sc = 1.0f;
          lr = 0;
        }
        trip(gq, mq, P, v, cnt, rows_tag);
      }
    };
    if (!gc || by_row) sweep(std::integral_constant<int, 0>{});
    else if (C & 7) sweep(std::integral_constant<int, 2>{});
    else sweep(std::integral_constant<int, 1>{});
  }
  kept = __reduce_add_sync(0xffffffffu, kept);
  if (lane == 0 && kept) atomicAdd(pv.kept + t.tensor, kept);
  if constexpr (SIGNAL) {
    __syncwarp();   // orders the other lanes' stores before the release
    if (lane == 0) signal_counter(pv.done + t.tensor, 1u);
  }
}

template <typename PT, bool WD, bool WAIT>
__device__ __forceinline__ void lion_apply_unit(const PlanView& pv, const LionDev& hp, const Task& t, float2* lut_s, const int lane) {
  using E = Elems<PT>;
  const DevTensor& d = pv.tensors[t.tensor];
  bool ok = true;
  if (WAIT && lane == 0) ok = wait_counter(pv.done + t.tensor, (unsigned)d.n_main, pv.status, 2001u, pv.spin_limit ? pv.spin_limit : KAON_SPIN_LIMIT);
  if (WAIT && !__all_sync(0xffffffffu, ok)) return;
  // cautious rescale (reference src/kaon/_backend.py:127-134): mean(mask) = count / numel in fp32
  const float denom = fmaxf(__fdiv_rn((float)__ldcg(pv.kept + t.tensor), (float)d.numel), 1e-8f);
  const float rdenom = __frcp_rn(denom);
  const float vpos = __fmul_rn(__fdiv_rn(1.0f, denom), hp.lr);  // |update| of a kept element, no weight decay
  // the pair a nibble of the codes stands for: minus the updates, or (weight decay) the signs, 2 where masked out
  if (lane < 16) {
    if (WD) lut_s[lane] = make_float2((float)(lane & 3) - 1.0f, (float)(lane >> 2) - 1.0f);
    else lut_s[lane] = make_float2((lane & 1) ? ((lane & 4) ? vpos : -vpos) : 0.0f, (lane & 2) ? ((lane & 8) ? vpos : -vpos) : 0.0f);
  }
  __syncwarp();
  unsigned char* pp = reinterpret_cast<unsigned char*>(d.p) + t.e0 * E::BYTES;
  const uint16_t* cp = reinterpret_cast<const uint16_t*>(pv.codes + d.code_off + (t.e0 >> 2));
  const uint64_t q0 = (uint64_t)(t.e0 >> 3);
  auto update = [&](const W8<PT>& P, uint32_t code, f32x2 F[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 u = lut_s[(code >> (4 * j)) & 15u];
      F[j] = pack2(u.x, u.y);
      if constexpr (WD) {
        const f32x2 dv = fma2(P.pair(j), pack2(hp.wd, hp.wd), F[j]);
        const f32x2 q = mul2(dv, pack2(rdenom, rdenom));
        const f32x2 x = mul2(fma2(fma2(q, pack2(-denom, -denom), dv), pack2(rdenom, rdenom), q), pack2(-hp.lr, -hp.lr));
        F[j] = pack2(u.x < 1.5f ? x.x : 0.0f, u.y < 1.5f ? x.y : 0.0f);
      }
    }
  };
  auto one = [&](W8<PT>& P, uint32_t code, unsigned v) {
    f32x2 F[4];
    update(P, code, F);
    write8(hp, d, q0 + v, true, P, F);
    P.store(pp + v * (8u * E::BYTES), &pv.peers);
  };
  const unsigned nvec = (unsigned)t.n >> 3;
  unsigned v = (unsigned)lane;
  for (; v + 32u < nvec; v += 64u) {
    W8<PT> A, B;
    A.load(pp + v * (8u * E::BYTES));
    const uint32_t ca = __ldcg(cp + v);
    B.load(pp + (v + 32u) * (8u * E::BYTES));
    const uint32_t cb = __ldcg(cp + v + 32u);
    one(A, ca, v);
    one(B, cb, v + 32u);
  }
  if (v < nvec) {
    W8<PT> A;
    A.load(pp + v * (8u * E::BYTES));
    one(A, __ldcg(cp + v), v);
  }
  if ((t.n & 7) && lane == 0) {   // the elements after the last whole vector of the tensor
    const int cnt = t.n & 7;
    W8<PT> A;
    load_some(A, pp + nvec * (8u * E::BYTES), cnt);
    f32x2 F[4];
    update(A, __ldcg(cp + nvec), F);
    const float dlt[8] = {F[0].x, F[0].y, F[1].x, F[1].y, F[2].x, F[2].y, F[3].x, F[3].y};
    float neg[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) neg[k] = -dlt[k];
    const SrStream st{Philox{hp.k0, hp.k1}, hp.step, KAON_TAG_UPDATE};
    update8<PT>(pp + nvec * (8u * E::BYTES), cnt, neg, -1.0f, hp.sr != 0, st, d.tensor_id, q0 + nvec, &pv.peers,
                hp.kahan ? reinterpret_cast<unsigned char*>(d.shift) + (q0 + nvec) * 16 : nullptr);
  }
  __syncwarp();
}

// Units in list order, each claimed while the one before it is worked on.
template <typename Unit>
__device__ __forceinline__ void claimed_units(const PlanView& pv, const int lane, Unit unit) {
  if (on_reserved_sm(pv.sm_reserve)) return;
  auto claim = [&]() -> int {
    int i = 0x7fffffff;
    if (lane == 0) {
      const unsigned st = *reinterpret_cast<volatile unsigned*>(pv.status);
      if (!st) i = (int)atomicAdd(pv.task_counter, 1u);
    }
    return i;   // lane 0's: broadcast where it is used, so that the atomic is in flight meanwhile
  };
  int cur = __shfl_sync(0xffffffffu, claim(), 0);
  while (cur < pv.n_tasks) {
    const int next = claim();
    const Task t = pv.tasks[cur];
    const unsigned char* g = reinterpret_cast<const unsigned char*>(pv.grads[t.tensor]);
    if (g != nullptr) unit(t, g);
    cur = __shfl_sync(0xffffffffu, next, 0);
  }
}

template <typename PT, int MK, bool WD>
__global__ void __launch_bounds__(LWT, 4) lion_warp_kernel(const __grid_constant__ PlanView pv, const __grid_constant__ LionDev hp) {
  __shared__ float mean_s[LWT / 32][LW_ROWS];
  __shared__ float2 lut_s[LWT / 32][16];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  claimed_units(pv, lane, [&](const Task& t, const unsigned char* g) {
    if (t.phase == PH_LION_MAIN) lion_main_unit<PT, MK, WD, true>(pv, hp, t, g, mean_s[warp], lane);
    else lion_apply_unit<PT, WD, true>(pv, hp, t, lut_s[warp], lane);
  });
}

template <typename PT, int MK, bool WD>
__global__ void __launch_bounds__(LWT, 4) lion_main_kernel(const __grid_constant__ PlanView pv, const __grid_constant__ LionDev hp) {
  __shared__ float mean_s[LWT / 32][LW_ROWS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  claimed_units(pv, lane, [&](const Task& t, const unsigned char* g) { lion_main_unit<PT, MK, WD, false>(pv, hp, t, g, mean_s[warp], lane); });
}

template <typename PT, bool WD>
__global__ void __launch_bounds__(LWT, 4) lion_apply_kernel(const __grid_constant__ PlanView pv, const __grid_constant__ LionDev hp) {
  __shared__ float2 lut_s[LWT / 32][16];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  claimed_units(pv, lane, [&](const Task& t, const unsigned char*) { lion_apply_unit<PT, WD, false>(pv, hp, t, lut_s[warp], lane); });
}

// ----------------------------------------------------------------------------- host

bool lion_warp_tensor(const DevTensor& t, int momentum_kind) {
  if (momentum_kind != KAON_M_4BIT && momentum_kind != KAON_M_BF16 && momentum_kind != KAON_M_F32) return false;
  // a block of its own for a tensor of up to 128 elements is block 0 of a blocked one
  if (momentum_kind == KAON_M_4BIT && t.bshift != 7 && !(t.bshift >= 31 && t.numel <= 128)) return false;
  return t.numel > 0 && (t.rows <= 0 || (t.cols >= 3 && t.cols <= LW_MAX_COLS));
}

// Units: about 4096 elements (small tensors in more pieces, large lists in fewer), starting on 128-element boundaries.  Whole rows where rows are a
// multiple of 128; otherwise at least two rows' worth, since the rows at both ends are averaged by two units, and at most
// LW_ROWS rows.
// Order: all MAIN units, then all APPLY units (APPLY units between them would empty the first level caches by their acquiring
// reads, where the second reading of a row's gradient hits).  Up to 64 M elements one launch; larger lists two (returns
// the number of MAIN units; 0: one launch), without the counters, whose fences then cost more than a launch (2.6 B list in
// units of 4096: 4.59 ms, in one launch 4.98; in units of 8192 4.40).
int lion_warp_units(const std::vector<DevTensor>& tensors, const std::vector<char>& elig, std::vector<Task>& out, std::vector<int>& n_main) {
  long long total = 0;
  for (size_t i = 0; i < tensors.size(); ++i) if (elig[i]) total += tensors[i].numel;
  const bool split = total > (64ll << 20);
  const int n = (int)tensors.size();
  n_main.assign(n, 0);
  out.reserve((size_t)(total / 2048) + 64 * (size_t)n);
  const long long most = split ? 8192 : 4096;   // (large lists: a shorter list of units to build and to claim)
  auto apply = [&](int i) {
    const DevTensor& t = tensors[i];
    long long u = 512;
    while (u < (split ? 2 : 1) * most && u * 128 <= t.numel) u *= 2;
    for (long long e = 0; e < t.numel; e += u)
      out.push_back(Task{i, PH_LION_APPLY, e, (int)std::min<long long>(u, t.numel - e), 0, 0, 0});
  };
  for (int i = 0; i < n; ++i) {
    if (!elig[i]) continue;
    const DevTensor& t = tensors[i];
    const long long C = t.cols;
    long long u = 512;
    while (u < most && u * 128 <= t.numel) u *= 2;
    if (t.rows > 0) {
      if (C % 128 == 0) u = std::min<long long>(std::max<long long>(1, u / C), LW_ROWS) * C;
      else u = std::min(std::max(u, (2 * C + 127) / 128 * 128), (LW_ROWS - 2) * C / 128 * 128);
    }
    for (long long e = 0; e < t.numel; e += u) {
      out.push_back(Task{i, PH_LION_MAIN, e, (int)std::min<long long>(u, t.numel - e), t.rows > 0 ? (int)(e / C) : 0, 0,
                         t.rows > 0 ? (int)(e % C) : 0});
      ++n_main[i];
    }
  }
  const int mains = split ? (int)out.size() : 0;
  for (int i = 0; i < n; ++i)
    if (elig[i]) apply(i);
  return mains;
}

typedef void (*LionWarp)(PlanView, LionDev);

template <typename PT, bool WD>
static LionWarp pick(int mk, bool split) {
  switch (mk) {
    case KAON_M_4BIT: return split ? lion_main_kernel<PT, KAON_M_4BIT, WD> : lion_warp_kernel<PT, KAON_M_4BIT, WD>;
    case KAON_M_BF16: return split ? lion_main_kernel<PT, KAON_M_BF16, WD> : lion_warp_kernel<PT, KAON_M_BF16, WD>;
    case KAON_M_F32: return split ? lion_main_kernel<PT, KAON_M_F32, WD> : lion_warp_kernel<PT, KAON_M_F32, WD>;
    default: return nullptr;
  }
}

int launch_lion_warp(kaon_plan* pl, const PlanView& base, const LionDev& hp, cudaStream_t s) {
  const bool bf = pl->param_dtype == KAON_DT_BF16, split = pl->n_tasks_warp_main > 0;
  const int mk = pl->momentum_kind;
  LionWarp k = hp.has_wd ? (bf ? pick<__nv_bfloat16, true>(mk, split) : pick<float, true>(mk, split))
                         : (bf ? pick<__nv_bfloat16, false>(mk, split) : pick<float, false>(mk, split));
  LionWarp ka = hp.has_wd ? (bf ? lion_apply_kernel<__nv_bfloat16, true> : lion_apply_kernel<float, true>)
                          : (bf ? lion_apply_kernel<__nv_bfloat16, false> : lion_apply_kernel<float, false>);
  if (!k) return fail(KAON_E_INVALID, "no Lion kernel for this dtype combination");
  auto run = [&](LionWarp kernel, const Task* tasks, int n, unsigned* counter) {
    PlanView v = base;
    v.tasks = tasks;
    v.n_tasks = n;
    v.task_counter = counter;
    const int most = pl->sm_count * 4;
    const int grid = base.sm_reserve ? most : std::max(1, std::min((n + LWT / 32 - 1) / (LWT / 32), most));
    kernel<<<grid, LWT, 0, s>>>(v, hp);
    pl->launches += 1;
  };
  const int first = split ? pl->n_tasks_warp_main : pl->n_tasks_warp;
  run(k, pl->d_tasks_warp, first, base.task_counter);
  if (split) run(ka, pl->d_tasks_warp + first, pl->n_tasks_warp - first, base.counters2 + 1);
  KAON_CUDA(cudaGetLastError());
  return KAON_OK;
}

}  // namespace kaon
