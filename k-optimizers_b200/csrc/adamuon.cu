// AdaMuon step for sm_100a (reference src/kaon/adamuon.py:327-352, 434-615).
//
// Per >=2-D tensor:  (1) EMA pre-pass: m <- lerp(decode(m), g, 1-b1) with g optionally centralised (each
// row less its mean, adamuon.py:334-335), re-encode and store m, write the fp32 pre-requant momentum as
// bf16 into the workspace;  (2) Newton-Schulz of that matrix on the tensor
// cores (ns.cu);  (3) the Adakaon STATS/FINAL/COUNT/APPLY work items with the orthogonalised matrix O as
// the signal, no further momentum, scale 0.2*lr, and the cautious mask taken against the raw gradient.
// 1-D tensors run the FLAT work item (Adam-style, momentum of the update) inside step (3)'s kernel.
#include <algorithm>
#include <cstring>
#include <vector>

#include "adakaon_dev.h"
#include "kaon_host.h"
#include "kaon_ops.cuh"
#include "kaon_sweep.cuh"
#include "ns_batch.h"

namespace kaon {

constexpr int ET = 256;

struct EmaOut { __nv_bfloat16* x; long long ld; };   // a tensor's matrix for Newton-Schulz and its row stride

// The general form, a CTA per item (a run of whole rows): any row length, block size, centralization.  Gradient and
// momentum straight from global memory; the item's sum of squares of what Newton-Schulz will read goes along.
template <typename PT, int MK>
__global__ void __launch_bounds__(ET) muon_ema_kernel(PlanView pv, const Task* tasks, int n_tasks,
                                                      float w1, float w1m1, int small_w1, int gc,
                                                      const EmaOut* outs, double* part) {
  using E = Elems<PT>;
  __shared__ unsigned rowmax_s[MAX_TASK_ROWS];
  __shared__ float scale_s[MAX_TASK_ROWS];
  __shared__ float mean_s[MAX_TASK_ROWS];  // centralization mean of each row of the item
  __shared__ double red_s[ET / 32];
  const int tid = threadIdx.x;
  for (int ti = blockIdx.x; ti < n_tasks; ti += gridDim.x) {
    const Task t = tasks[ti];
    if (pv.grads[t.tensor] == nullptr) continue;
    const EmaOut xo_t = outs[t.tensor];
    double ss = 0.0;
    const DevTensor d = pv.tensors[t.tensor];
    const unsigned char* g = reinterpret_cast<const unsigned char*>(pv.grads[t.tensor]) + t.e0 * E::BYTES;
    const int n = t.n, C = d.cols;
    const int nrows = n / C;
    const int nvec = (n + 7) >> 3, nvec_pad = (nvec + 31) & ~31;
    const bool row_uniform = (C & 7) == 0;
    const unsigned char* mbase = reinterpret_cast<const unsigned char*>(d.m);
    if (gc) {
      // one warp per row; the mean also goes to the scratch, where the cautious mask of the weight stage
      // finds it (the mask compares with the centralised gradient)
      for (int r = tid >> 5; r < nrows; r += ET / 32) {
        const unsigned char* rowp = g + (size_t)r * C * E::BYTES;
        float sum = 0.0f;
        if (row_uniform) {
          for (int v = tid & 31; v < (C >> 3); v += 32) {
            float x[8];
            E::load8(rowp + (size_t)v * 8 * E::BYTES, x);
            sum += ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
          }
        } else {
          for (int i = tid & 31; i < C; i += 32) sum += E::load1(rowp, i);
        }
        sum = warp_sum(sum);
        const float mean = __fdiv_rn(sum, (float)C);
        const float mu = E::IS_BF16 ? round_bf16(mean) : mean;
        if ((tid & 31) == 0) { mean_s[r] = mu; pv.aux[aux_mean(d) + t.row0 + r] = mu; }
      }
      __syncthreads();
    }
    auto m_new8 = [&](int v, int cnt, float mn[8]) {
      float gv[8], mo[8];
      load8_guard<PT>(g + (size_t)v * 8 * E::BYTES, cnt, gv);
      if (gc) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float x = __fsub_rn(gv[k], mean_s[row_uniform ? row_of((unsigned)v * 8u, d) : row_of((unsigned)(v * 8 + min(k, max(cnt - 1, 0))), d)]);
          gv[k] = E::IS_BF16 ? round_bf16(x) : x;
        }
      }
      if constexpr (MK == KAON_M_4BIT) {
        const long long blk = blk_of(d, t.e0 + (long long)v * 8);
        decode8<MK>(mbase + (t.e0 >> 1), v, cnt, d.m_scale[blk], mo);
      } else if constexpr (MK == KAON_M_INT8) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
          mo[k] = (k < cnt) ? __fmul_rn((float)(signed char)mbase[t.e0 + v * 8 + k],
                                        scale_s[row_uniform ? row_of((unsigned)v * 8u, d) : row_of((unsigned)(v * 8 + k), d)])
                            : 0.0f;
      } else if constexpr (MK == KAON_M_BF16) {
        decode8<MK>(mbase + t.e0 * 2, v, cnt, 1.0f, mo);
      } else if constexpr (MK == KAON_M_F32) {
        decode8<MK>(mbase + t.e0 * 4, v, cnt, 1.0f, mo);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        float r;
        if constexpr (MK == KAON_M_NONE) r = gv[k];
        else if constexpr (MK == KAON_M_BF16) r = round_bf16(lerp_torch(mo[k], round_bf16(gv[k]), w1, w1m1, small_w1 != 0));
        else r = lerp_torch(mo[k], gv[k], w1, w1m1, small_w1 != 0);
        mn[k] = (k < cnt) ? r : 0.0f;
      }
    };
    if constexpr (MK == KAON_M_INT8) {
      for (int r = tid; r < nrows; r += ET) { rowmax_s[r] = 0u; scale_s[r] = d.m_scale[t.row0 + r]; }
      __syncthreads();
      for (int v = tid; v < nvec; v += ET) {
        const int cnt = min(8, n - v * 8);
        float mn[8];
        m_new8(v, cnt, mn);
        if (row_uniform) {
          float a = 0.0f;
#pragma unroll
          for (int k = 0; k < 8; ++k) a = fmaxf(a, fabsf(mn[k]));
          atomicMax(rowmax_s + row_of((unsigned)v * 8u, d), __float_as_uint(a));
        } else {
          for (int k = 0; k < cnt; ++k) atomicMax(rowmax_s + row_of((unsigned)(v * 8 + k), d), __float_as_uint(fabsf(mn[k])));
        }
      }
      __syncthreads();
    }
    for (int v = tid; v < nvec_pad; v += ET) {
      const int cnt = max(0, min(8, n - v * 8));
      float mn[8];
      if (cnt > 0) m_new8(v, cnt, mn);
      else {
#pragma unroll
        for (int k = 0; k < 8; ++k) mn[k] = 0.0f;
      }
      if constexpr (MK == KAON_M_4BIT) {
        float a = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) a = fmaxf(a, fabsf(mn[k]));
        a = fmaxf(group_max(a, blk_lanes(d)), 1e-12f);
        const float sc = __fdiv_rn(a, 7.0f);
        const float inv = __fdividef(1.0f, sc);
        uint32_t word = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int qi = min(max((int)quant_round(mn[k], sc, inv, 1e-4f), -7), 7);
          if (k < cnt) word |= (uint32_t)(qi + 8) << (4 * k);
        }
        if (cnt > 0) {
          unsigned char* mdst = (unsigned char*)d.m + (t.e0 >> 1) + (size_t)v * 4;
          if (cnt == 8) *reinterpret_cast<uint32_t*>(mdst) = word;
          else
            for (int b = 0; b < (cnt + 1) / 2; ++b) mdst[b] = (unsigned char)(word >> (8 * b));
          if ((v & (blk_lanes(d) - 1)) == 0) d.m_scale[blk_of(d, t.e0 + (long long)v * 8)] = sc;
        }
      } else if constexpr (MK == KAON_M_INT8) {
        if (cnt > 0) {
          unsigned char* mdst = (unsigned char*)d.m + t.e0 + (size_t)v * 8;
          float sc = 0.0f, inv = 0.0f;
          int rprev = -1;
          for (int k = 0; k < cnt; ++k) {
            const int r = row_uniform ? row_of((unsigned)v * 8u, d) : row_of((unsigned)(v * 8 + k), d);
            if (r != rprev) {
              sc = __fdiv_rn(fmaxf(__uint_as_float(rowmax_s[r]), 1e-12f), 127.0f);
              inv = __fdividef(1.0f, sc);
              rprev = r;
              if ((unsigned)(v * 8 + k) == (unsigned)r * (unsigned)C) d.m_scale[t.row0 + r] = sc;
            }
            mdst[k] = (unsigned char)(min(max((int)quant_round(mn[k], sc, inv, 1e-3f), -127), 127) & 0xFF);
          }
        }
      } else if constexpr (MK == KAON_M_BF16) {
        if (cnt > 0)
          for (int k = 0; k < cnt; ++k)
            reinterpret_cast<uint16_t*>((unsigned char*)d.m + t.e0 * 2)[v * 8 + k] = (uint16_t)(__float_as_uint(mn[k]) >> 16);
      } else if constexpr (MK == KAON_M_F32) {
        if (cnt > 0)
          for (int k = 0; k < cnt; ++k) reinterpret_cast<float*>((unsigned char*)d.m + t.e0 * 4)[v * 8 + k] = mn[k];
      }
      // the matrix Newton-Schulz reads: bf16 of the fp32 pre-requant momentum
      if (cnt > 0) {
        if (cnt == 8 && row_uniform) {   // (its rows are then not padded)
          *reinterpret_cast<uint4*>(xo_t.x + t.e0 + (size_t)v * 8) =
              make_uint4(pack_bf16_rn(mn[0], mn[1]), pack_bf16_rn(mn[2], mn[3]), pack_bf16_rn(mn[4], mn[5]), pack_bf16_rn(mn[6], mn[7]));
        } else {
          for (int k = 0; k < cnt; ++k) {
            const int r = row_of((unsigned)(v * 8 + k), d);
            xo_t.x[(t.row0 + r) * xo_t.ld + (v * 8 + k - r * C)] = __float2bfloat16_rn(mn[k]);
          }
        }
        for (int k = 0; k < cnt; ++k) {
          const float x = round_bf16(mn[k]);
          ss += (double)x * (double)x;
        }
      }
    }
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((tid & 31) == 0) red_s[tid >> 5] = ss;
    __syncthreads();
    if (tid == 0) {
      double tot = 0.0;
      for (int w = 0; w < ET / 32; ++w) tot += red_s[w];
      part[t.slot] = tot;
    }
    __syncthreads();
  }
}

// The common case (rows a multiple of eight elements, 4-bit blocks of 128, no centralization), a warp per unit: runs of
// whole rows with int8 momentum (a row's maximum comes before its codes: two passes over the row, the second from
// L1), flat runs otherwise.  No barriers; packed pairs; the unit's sum of squares of what Newton-Schulz will read goes
// along.  (A CTA per 16 K-element item with scalar arithmetic and a separate norm pass: 2.4 + 1.2 ms on 453 M elements.)
template <typename PT, int MK>
__global__ void __launch_bounds__(ET, 4) muon_ema_fast_kernel(const __grid_constant__ PlanView pv, const Task* tasks, int n_tasks,
                                                              float w1, float w1m1, int small_w1, const EmaOut* outs, double* part) {
  using E = Elems<PT>;
  constexpr int MV = MBytes<MK>::V;
  const int lane = threadIdx.x & 31;
  const int nw = gridDim.x * (ET / 32);
  for (int i = __shfl_sync(0xffffffffu, (int)(blockIdx.x * (ET / 32) + (threadIdx.x >> 5)), 0); i < n_tasks; i += nw) {
    const Task t = tasks[i];
    const unsigned char* g = reinterpret_cast<const unsigned char*>(pv.grads[t.tensor]);
    if (g == nullptr) continue;
    const DevTensor& d = pv.tensors[t.tensor];
    __nv_bfloat16* x_out = outs[t.tensor].x;
    unsigned char* m = reinterpret_cast<unsigned char*>(d.m);
    const int nv = MK == KAON_M_INT8 ? d.cols >> 3 : t.n >> 3;   // vectors of a row (or of the flat run)
    const int rows = MK == KAON_M_INT8 ? t.n / d.cols : 1;
    double ss = 0.0;
    for (int r = 0; r < rows; ++r) {
      const long long e0 = t.e0 + (long long)r * (MK == KAON_M_INT8 ? d.cols : 0);
      const float row_sc = MK == KAON_M_INT8 ? d.m_scale[t.row0 + r] : 1.0f;
      // the new momentum of vector v
      auto fresh = [&](int v, f32x2 MN[4]) {
        const long long e = e0 + v * 8ll;
        W8<PT> gq;
        MRaw<MK> mq;
        f32x2 MO[4];
        gq.load(g + e * E::BYTES);
        if constexpr (MK != KAON_M_NONE) {
          mq.load(m + (e >> 3) * MV);
          mq.decode(MK == KAON_M_4BIT ? d.m_scale[e >> 7] : row_sc, MO);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          f32x2 G = gq.pair(j);
          if constexpr (MK == KAON_M_NONE) {
            MN[j] = G;
          } else {
            if constexpr (MK == KAON_M_BF16) G = pack2(round_bf16(G.x), round_bf16(G.y));
            MN[j] = small_w1 ? fma2(pack2(w1, w1), sub2(G, MO[j]), MO[j]) : fma2(pack2(w1m1, w1m1), sub2(G, MO[j]), G);
            if constexpr (MK == KAON_M_BF16) MN[j] = pack2(round_bf16(MN[j].x), round_bf16(MN[j].y));
          }
        }
      };
      float amax = 0.0f;
      if constexpr (MK == KAON_M_INT8) {
#pragma unroll 2
        for (int v = lane; v < nv; v += 32) {
          f32x2 MN[4];
          fresh(v, MN);
          amax = fmaxf(amax, amax8(MN));
        }
        __syncwarp();
        amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(amax)));
      }
      for (int v0 = 0; v0 < nv; v0 += 32) {
        const int v = v0 + lane;
        const bool act = v < nv;
        f32x2 MN[4];
        fresh(act ? v : 0, MN);
        const long long e = e0 + v * 8ll;
        if constexpr (MK != KAON_M_NONE) {
          const float sc = store_m8<MK>(m + (e >> 3) * MV, MN, amax, act ? 8 : 0, lane);
          if constexpr (MK == KAON_M_4BIT) { if (act && (lane & 15) == 0) d.m_scale[e >> 7] = sc; }
          if constexpr (MK == KAON_M_INT8) { if (v == 0) d.m_scale[t.row0 + r] = sc; }
        }
        if (!act) continue;
        const uint4 x = make_uint4(pack_bf16_rn(MN[0].x, MN[0].y), pack_bf16_rn(MN[1].x, MN[1].y),
                                   pack_bf16_rn(MN[2].x, MN[2].y), pack_bf16_rn(MN[3].x, MN[3].y));
        *reinterpret_cast<uint4*>(x_out + e) = x;   // bf16 of the momentum before requantisation
        const uint32_t xw[4] = {x.x, x.y, x.z, x.w};
        f32x2 q = pack2(0.0f, 0.0f);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const f32x2 y = pack2(bf16lo(xw[j]), bf16hi(xw[j]));
          q = fma2(y, y, q);
        }
        ss += (double)(q.x + q.y);
      }
      __syncwarp();
    }
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) part[t.slot] = ss;
  }
}

typedef void (*EmaKernel)(PlanView, const Task*, int, float, float, int, int, const EmaOut*, double*);
typedef void (*EmaFastKernel)(PlanView, const Task*, int, float, float, int, const EmaOut*, double*);

template <typename PT>
static EmaKernel pick_ema_pt(int mk) {
  switch (mk) {
    case KAON_M_F32: return muon_ema_kernel<PT, KAON_M_F32>;
    case KAON_M_BF16: return muon_ema_kernel<PT, KAON_M_BF16>;
    case KAON_M_INT8: return muon_ema_kernel<PT, KAON_M_INT8>;
    case KAON_M_4BIT: return muon_ema_kernel<PT, KAON_M_4BIT>;
    case KAON_M_NONE: return muon_ema_kernel<PT, KAON_M_NONE>;
    default: return nullptr;
  }
}
template <typename PT>
static EmaFastKernel pick_ema_fast_pt(int mk) {
  switch (mk) {
    case KAON_M_F32: return muon_ema_fast_kernel<PT, KAON_M_F32>;
    case KAON_M_BF16: return muon_ema_fast_kernel<PT, KAON_M_BF16>;
    case KAON_M_INT8: return muon_ema_fast_kernel<PT, KAON_M_INT8>;
    case KAON_M_4BIT: return muon_ema_fast_kernel<PT, KAON_M_4BIT>;
    case KAON_M_NONE: return muon_ema_fast_kernel<PT, KAON_M_NONE>;
    default: return nullptr;
  }
}

static size_t up256(size_t x) { return (x + 255) / 256 * 256; }

// Matrices are independent of each other until the second-moment stage: they run in batches, every matrix of a batch
// at the same stage of its chain in one launch (EMA, norms, three products per iteration).  A batch holds what NS_BATCH
// bytes of scratch allow (a list of small matrices is one batch; a width-3072 DiT block is one).  Batches alternate
// between NS_LANES internal streams with a scratch each, so that one's last tiles and pre-pass share the machine with
// the other's products.
constexpr int NS_LANES = 2;
constexpr size_t NS_BATCH = (size_t)768 << 20;

struct MuonLayout {
  std::vector<size_t> o_off;     // per tensor: byte offset of O in the workspace (factored tensors)
  std::vector<int> batch;        // per tensor: its batch, or -1
  std::vector<size_t> s_off;     // per tensor: offset of its scratch inside its lane's
  int n_batches = 0;
  size_t scratch_off = 0, lane_stride = 0, total = 0;
};

static MuonLayout muon_layout(const kaon_plan* pl) {
  MuonLayout L;
  L.o_off.assign(pl->n_tensors, 0);
  L.s_off.assign(pl->n_tensors, 0);
  L.batch.assign(pl->n_tensors, -1);
  size_t cur = 0, used = 0;
  for (int i = 0; i < pl->n_tensors; ++i) {
    const DevTensor& t = pl->h_tensors[i];
    if (t.rows <= 0 || t.numel == 0) continue;
    L.o_off[i] = cur;
    cur += up256((size_t)t.numel * 2);
    const size_t need = up256(ns_scratch_bytes(t.rows, t.cols));
    if (L.n_batches == 0 || used + need > NS_BATCH) { ++L.n_batches; used = 0; }
    L.batch[i] = L.n_batches - 1;
    L.s_off[i] = used;
    used += need;
    L.lane_stride = std::max(L.lane_stride, used);
  }
  L.scratch_off = cur;
  L.total = cur + (size_t)std::min(NS_LANES, std::max(L.n_batches, 1)) * L.lane_stride + 256;
  return L;
}

// What a plan keeps between steps: the batches' launch tables, rebuilt when the workspace or the number of iterations
// changes.  They cover every matrix; one without a gradient is passed over by the kernels.
struct MuonHost {
  MuonLayout layout;
  struct Batch {
    NsBatch ns;
    size_t ns_off = 0;                    // its tables in `block`
    int fast0 = 0, n_fast = 0;            // EMA units, general items of the tensors without units, items of all
    int rest0 = 0, n_rest = 0;
    int all0 = 0, n_all = 0;
    int scale_f0 = 0, scale_a0 = 0;
    std::vector<int> tensors;
  };
  std::vector<Batch> batches;
  const void* base = nullptr;
  int steps = 0;
  unsigned char* block = nullptr;
  size_t block_bytes = 0, off_fast = 0, off_rest = 0, off_all = 0, off_outs = 0, off_scale = 0, off_part = 0;
};

void muon_free(kaon_plan* pl) {
  MuonHost* h = reinterpret_cast<MuonHost*>(pl->muon);
  if (!h) return;
  cudaFree(h->block);
  delete h;
  pl->muon = nullptr;
}

static int muon_build(kaon_plan* pl, MuonHost& h, unsigned char* ws, int steps, cudaStream_t s) {
  const int n = pl->n_tensors;
  const MuonLayout& L = h.layout;
  std::vector<Task> fast, rest, all;
  std::vector<EmaOut> outs(n, EmaOut{nullptr, 0});
  std::vector<NsScale> scales;
  NsShares shares;
  h.batches.assign(L.n_batches, MuonHost::Batch());
  int slots = 0;
  size_t tab = 0;
  for (int b = 0; b < L.n_batches; ++b) {
    MuonHost::Batch& B = h.batches[b];
    B.fast0 = (int)fast.size(); B.rest0 = (int)rest.size(); B.all0 = (int)all.size();
    std::vector<NsMat> mats;
    std::vector<NsScale> sf, sa;
    for (int i = 0; i < n; ++i) {
      if (L.batch[i] != b) continue;
      const DevTensor& t = pl->h_tensors[i];
      NsMat m{};
      m.R = t.rows; m.C = t.cols;
      ns_scratch_layout(m, ws + L.scratch_off + (size_t)(b % NS_LANES) * L.lane_stride + L.s_off[i]);
      m.out = reinterpret_cast<__nv_bfloat16*>(ws + L.o_off[i]);
      m.tensor = i;
      mats.push_back(m);
      B.tensors.push_back(i);
      outs[i] = EmaOut{m.x0, m.ld};
      // general items: runs of whole rows
      const int a0 = slots;
      const size_t first = all.size();
      for (long long r = 0; r < t.rows; r += t.chunk_rows) {
        const long long nr = std::min<long long>(t.chunk_rows, t.rows - r);
        all.push_back(Task{i, 0, r * t.cols, (int)(nr * t.cols), (int)r, slots++, 0});
      }
      sa.push_back(NsScale{a0, slots, m.scal});
      const bool units = (t.cols & 7) == 0 && (pl->momentum_kind != KAON_M_4BIT || t.bshift == 7);
      if (!units) {
        rest.insert(rest.end(), all.begin() + (long)first, all.end());
        sf.push_back(sa.back());
        continue;
      }
      // a warp's units: about 4096 elements, of whole rows with int8 momentum
      const int f0 = slots;
      const long long len = pl->momentum_kind == KAON_M_INT8 ? std::max<long long>(1, 4096 / t.cols) * t.cols : 4096;
      for (long long e = 0; e < t.numel; e += len)
        fast.push_back(Task{i, 0, e, (int)std::min<long long>(len, t.numel - e), (int)(e / t.cols), slots++, 0});
      sf.push_back(NsScale{f0, slots, m.scal});
    }
    B.n_fast = (int)fast.size() - B.fast0; B.n_rest = (int)rest.size() - B.rest0; B.n_all = (int)all.size() - B.all0;
    B.scale_f0 = (int)scales.size(); scales.insert(scales.end(), sf.begin(), sf.end());
    B.scale_a0 = (int)scales.size(); scales.insert(scales.end(), sa.begin(), sa.end());
    if (int rc = ns_batch_build(mats, steps, shares, B.ns)) return rc;
    B.ns_off = tab;
    tab += up256(B.ns.bytes);
  }
  size_t o = tab;
  auto take = [&](size_t bytes) { const size_t at = o; o += up256(std::max<size_t>(bytes, 1)); return at; };
  h.off_fast = take(sizeof(Task) * fast.size());
  h.off_rest = take(sizeof(Task) * rest.size());
  h.off_all = take(sizeof(Task) * all.size());
  h.off_outs = take(sizeof(EmaOut) * outs.size());
  h.off_scale = take(sizeof(NsScale) * scales.size());
  const size_t uploaded = o;
  h.off_part = take(sizeof(double) * (size_t)slots);
  if (o > h.block_bytes) {
    if (h.block) { KAON_CUDA(cudaStreamSynchronize(s)); cudaFree(h.block); h.block = nullptr; }
    KAON_CUDA(cudaMalloc((void**)&h.block, o));
    pl->device_bytes += (int64_t)(o - h.block_bytes);
    h.block_bytes = o;
  }
  std::vector<unsigned char> img(uploaded, 0);
  for (const MuonHost::Batch& B : h.batches)
    if (B.ns.bytes) std::memcpy(img.data() + B.ns_off, B.ns.host.data(), B.ns.bytes);
  auto put = [&](size_t at, const void* src, size_t bytes) { if (bytes) std::memcpy(img.data() + at, src, bytes); };
  put(h.off_fast, fast.data(), sizeof(Task) * fast.size());
  put(h.off_rest, rest.data(), sizeof(Task) * rest.size());
  put(h.off_all, all.data(), sizeof(Task) * all.size());
  put(h.off_outs, outs.data(), sizeof(EmaOut) * outs.size());
  put(h.off_scale, scales.data(), sizeof(NsScale) * scales.size());
  // pageable source: staged before the call returns, ordered on the step's stream after the steps before it
  KAON_CUDA(cudaMemcpyAsync(h.block, img.data(), uploaded, cudaMemcpyHostToDevice, s));
  for (MuonHost::Batch& B : h.batches) { B.ns.host.clear(); B.ns.host.shrink_to_fit(); }
  h.base = ws;
  h.steps = steps;
  return KAON_OK;
}

}  // namespace kaon

using namespace kaon;

extern "C" int64_t kaon_adamuon_workspace_bytes(const kaon_plan* pl) {
  if (!pl || pl->optimizer != KAON_OPT_ADAMUON) return 0;
  return (int64_t)muon_layout(pl).total;
}

extern "C" int64_t kaon_adamuon_signal_offset(const kaon_plan* pl, int tensor) {
  if (!pl || pl->optimizer != KAON_OPT_ADAMUON || tensor < 0 || tensor >= pl->n_tensors) return -1;
  if (pl->h_tensors[tensor].rows <= 0) return -1;
  return (int64_t)muon_layout(pl).o_off[tensor];
}

extern "C" int kaon_adamuon_step(kaon_plan* pl, const kaon_adamuon_hparams* h, void* workspace,
                                 int64_t workspace_bytes, uint64_t seed, uint32_t step, void* stream) {
  if (!pl || !h) return fail(KAON_E_INVALID, "kaon_adamuon_step: null argument");
  if (pl->optimizer != KAON_OPT_ADAMUON) return fail(KAON_E_INVALID, "plan was not built for AdaMuon");
  if (int rc = check_device(pl)) return rc;
  if (h->bf16_method < KAON_W_NONE || h->bf16_method > KAON_W_KAHAN) return fail(KAON_E_UNSUPPORTED, "bf16_method %d", h->bf16_method);
  if (int rc = check_kahan(pl, h->bf16_method)) return rc;
  if (!(h->clip_threshold > 0.0)) return fail(KAON_E_INVALID, "clip_threshold must be > 0");
  if (h->ns_steps < 1) return fail(KAON_E_INVALID, "ns_steps must be >= 1");
  const bool has_m = pl->momentum_kind != KAON_M_NONE;
  if (has_m != (h->beta1 > 0.0)) return fail(KAON_E_INVALID, "beta1 %g does not match the plan's momentum kind", h->beta1);
  if (!pl->muon) {
    MuonHost* fresh = new MuonHost();
    fresh->layout = muon_layout(pl);
    pl->muon = fresh;
  }
  MuonHost& H = *reinterpret_cast<MuonHost*>(pl->muon);
  const MuonLayout& L = H.layout;
  if (!workspace || ((uintptr_t)workspace & 255) || workspace_bytes < (int64_t)L.total)
    return fail(KAON_E_INVALID, "kaon_adamuon_step: workspace missing, misaligned or smaller than %zu bytes", L.total);
  cudaStream_t s = (cudaStream_t)stream;
  unsigned char* ws = reinterpret_cast<unsigned char*>(workspace);
  const int n = pl->n_tensors;

  // one-time: the O column; per workspace and iteration count: the batches' tables
  if (!pl->d_signal) {
    KAON_CUDA(cudaMalloc((void**)&pl->d_signal, sizeof(void*) * (size_t)n));
    pl->device_bytes += (int64_t)(sizeof(void*) * n);
  }
  if (H.base != workspace || H.steps != h->ns_steps)
    if (int rc = muon_build(pl, H, ws, h->ns_steps, s)) { H.base = nullptr; return rc; }
  if (pl->signal_base != workspace) {
    std::vector<const void*> sig(n, nullptr);
    for (int i = 0; i < n; ++i)
      if (pl->h_tensors[i].rows > 0 && pl->h_tensors[i].numel) sig[i] = ws + L.o_off[i];
    KAON_CUDA(cudaMemcpyAsync((void*)pl->d_signal, sig.data(), sizeof(void*) * (size_t)n, cudaMemcpyHostToDevice, s));
    pl->signal_base = workspace;
  }

  const float w1 = (float)(1.0 - h->beta1);
  const bool bf = pl->param_dtype == KAON_DT_BF16;
  EmaKernel ek = bf ? pick_ema_pt<__nv_bfloat16>(pl->momentum_kind) : pick_ema_pt<float>(pl->momentum_kind);
  EmaFastKernel ef = bf ? pick_ema_fast_pt<__nv_bfloat16>(pl->momentum_kind) : pick_ema_fast_pt<float>(pl->momentum_kind);
  if (!ek || !ef) return fail(KAON_E_INVALID, "no AdaMuon EMA kernel for this dtype combination");
  PlanView v = pl->view;
  v.signal = pl->d_signal;
  KAON_CUDA(cudaMemsetAsync(v.task_counter, 0, pl->counters_bytes - sizeof(unsigned), s));

  // (1) + (2): batch by batch, EMA pre-pass and Newton-Schulz into the O slots, on the caller's stream or (more than
  // one batch) alternating over the lanes, forked from it and joined before stage 3
  const bool lanes = H.batches.size() > 1;
  if (lanes && !pl->muon_lanes_ready) {
    for (int l = 0; l < NS_LANES; ++l) {
      KAON_CUDA(cudaStreamCreateWithFlags(&pl->muon_stream[l], cudaStreamNonBlocking));
      KAON_CUDA(cudaEventCreateWithFlags(&pl->muon_join[l], cudaEventDisableTiming));
    }
    KAON_CUDA(cudaEventCreateWithFlags(&pl->muon_fork, cudaEventDisableTiming));
    pl->muon_lanes_ready = true;
  }
  if (lanes) {
    KAON_CUDA(cudaEventRecord(pl->muon_fork, s));
    for (int l = 0; l < NS_LANES; ++l) KAON_CUDA(cudaStreamWaitEvent(pl->muon_stream[l], pl->muon_fork, 0));
  }
  const bool gc = h->gradient_centralization != 0;
  const EmaOut* outs = reinterpret_cast<const EmaOut*>(H.block + H.off_outs);
  double* part = reinterpret_cast<double*>(H.block + H.off_part);
  for (size_t b = 0; b < H.batches.size(); ++b) {
    const MuonHost::Batch& B = H.batches[b];
    const int n_mats = (int)B.tensors.size();
    const int live = (int)std::count_if(B.tensors.begin(), B.tensors.end(), [&](int i) { return pl->h_grads[i] != nullptr; });
    if (live == 0) continue;
    cudaStream_t sl = lanes ? pl->muon_stream[b % NS_LANES] : s;
    const int n_gen = gc ? B.n_all : B.n_rest;   // centralization takes the general form throughout
    if (!gc && B.n_fast) {
      const int grid = std::min((B.n_fast + ET / 32 - 1) / (ET / 32), pl->sm_count * 4);
      ef<<<grid, ET, 0, sl>>>(v, reinterpret_cast<const Task*>(H.block + H.off_fast) + B.fast0, B.n_fast, w1, w1 - 1.0f, w1 < 0.5f, outs, part);
      pl->launches += 1;
    }
    if (n_gen) {
      const Task* list = gc ? reinterpret_cast<const Task*>(H.block + H.off_all) + B.all0 : reinterpret_cast<const Task*>(H.block + H.off_rest) + B.rest0;
      ek<<<std::min(n_gen, pl->sm_count * 8), ET, 0, sl>>>(v, list, n_gen, w1, w1 - 1.0f, w1 < 0.5f, gc, outs, part);
      pl->launches += 1;
    }
    ns_batch_scale(reinterpret_cast<const NsScale*>(H.block + H.off_scale) + (gc ? B.scale_a0 : B.scale_f0), n_mats, part, sl);
    KAON_CUDA(cudaGetLastError());
    long long nl = 1;
    if (int rc = ns_batch_run(B.ns, H.block + B.ns_off, live < n_mats ? v.grads : nullptr, v.status, sl, &nl)) return rc;
    pl->launches += nl;
  }
  if (lanes) {
    for (int l = 0; l < NS_LANES; ++l) {
      KAON_CUDA(cudaEventRecord(pl->muon_join[l], pl->muon_stream[l]));
      KAON_CUDA(cudaStreamWaitEvent(s, pl->muon_join[l], 0));
    }
  }

  // (3) second moment of O, clip, scale, cautious, weight write (and the whole 1-D branch)
  AdaDev hp{};
  hp.w1 = w1; hp.w1m1 = w1 - 1.0f; hp.small_w1 = w1 < 0.5f;
  hp.w2 = (float)(1.0 - h->beta2); hp.w2m1 = hp.w2 - 1.0f; hp.small_w2 = hp.w2 < 0.5f;
  hp.eps1 = (float)h->eps1; hp.has_eps = h->eps1 > 0.0;
  hp.clip = (float)h->clip_threshold;
  hp.lrwd = (float)(h->lr * h->weight_decay); hp.has_wd = h->weight_decay != 0.0;
  hp.upd_scale = (float)(0.2 * h->lr);  // _UPDATE_RMS * lr, product taken in double (adamuon.py:88, 489)
  hp.cautious = h->cautious != 0;
  hp.gc = h->gradient_centralization != 0;  // the statistics of O ignore it; the mask centres the raw gradient
  hp.sr = h->bf16_method == KAON_W_SR && pl->param_dtype == KAON_DT_BF16;
  hp.kahan = h->bf16_method == KAON_W_KAHAN && pl->param_dtype == KAON_DT_BF16;
  hp.has_m = has_m;
  hp.step = step; hp.k0 = (uint32_t)seed; hp.k1 = (uint32_t)(seed >> 32);
  ada_finish(hp);
  if (int rc = ensure_apply2(pl)) return rc;
  const bool three = pl->apply2 == 1;  // STATS/FINAL/FLAT here, COUNT and APPLY as launches of their own
  if (three) {
    if (int rc = launch_statistics(pl, v, hp, ada_stages(pl, hp.cautious), s)) return rc;
  } else {
    PlanView w = v;
    w.tasks = hp.cautious ? pl->d_tasks_full : pl->d_tasks_main;
    w.n_tasks = hp.cautious ? pl->n_tasks_full : pl->n_tasks_main;
    if (int rc = launch_persistent(pl, w, hp, false, s)) return rc;
  }
  if (int rc = launch_small(pl, v, hp, s)) return rc;
  if (three) {
    if (int rc = launch_count_apply(pl, v, hp, s)) return rc;
  }
  return KAON_OK;
}
