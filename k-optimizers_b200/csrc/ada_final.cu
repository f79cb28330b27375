// FINAL of the Adakaon family as launches of their own, for the tensors whose STATS, COUNT and APPLY are: column statistics, the
// clip divisor, and the row table the sweeps read.
#include <algorithm>
#include <vector>

#include "adakaon_dev.h"
#include "kaon_host.h"
#include "kaon_ops.cuh"

namespace kaon {

// Column statistics of a strip of FS_COLS columns from the STATS runs' partial sums, and by the tensor's last strip to arrive
// the row mean and the clip divisor.  A warp takes every FS_WARPS-th run, four columns a lane: a tall tensor
// has a hundred runs, which one thread a column (ada_final in adakaon.cu, for tensors that stay in the persistent kernel)
// went through in a chain of a dozen loads.  Sums in a fixed order, in double; with a Kahan compensation in fp32 and
// in the order of the runs (the rule at warp_sum_d in adakaon.cu).
constexpr int FS_COLS = 128, FS_THREADS = 256, FS_WARPS = FS_THREADS / 32;

__device__ __forceinline__ void final_strip(const PlanView& pv, const AdaDev& hp, const Task& t) {
  __shared__ double sum_s[FS_WARPS][2][FS_COLS];
  __shared__ double red[FS_WARPS];
  if (pv.grads[t.tensor] == nullptr) return;
  const DevTensor& d = pv.tensors[t.tensor];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int C = d.cols, S = d.n_stats, c0 = t.row0;
  const float* part = pv.aux + d.aux_off;
  const bool plain = d.shift != nullptr;
  const int c = c0 + tid;   // the column of a thread below FS_COLS
  const bool own = tid < FS_COLS && c < C;
  const float old = own ? d.stat_b[c] : 0.0f;
  double s1 = 0.0, s2 = 0.0;
  if (plain) {
    if (own) {
      float a = 0.0f, b = 0.0f;
#pragma unroll 8
      for (int s = 0; s < S; ++s) {
        a += __ldcg(part + 2ll * s * C + c);
        b += __ldcg(part + 2ll * s * C + C + c);
      }
      s1 = (double)a; s2 = (double)b;
    }
  } else {
    const int cl = c0 + lane * 4;
    double a[4] = {0.0, 0.0, 0.0, 0.0}, b[4] = {0.0, 0.0, 0.0, 0.0};
    if (cl < C) {
#pragma unroll 4
      for (int s = warp; s < S; s += FS_WARPS) {
        const float4 x = __ldcg(reinterpret_cast<const float4*>(part + 2ll * s * C + cl));
        const float4 y = __ldcg(reinterpret_cast<const float4*>(part + 2ll * s * C + C + cl));
        a[0] += (double)x.x; a[1] += (double)x.y; a[2] += (double)x.z; a[3] += (double)x.w;
        b[0] += (double)y.x; b[1] += (double)y.y; b[2] += (double)y.z; b[3] += (double)y.w;
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      sum_s[warp][0][lane * 4 + k] = a[k];
      sum_s[warp][1][lane * 4 + k] = b[k];
    }
    __syncthreads();
    if (own)
      for (int w = 0; w < FS_WARPS; ++w) { s1 += sum_s[w][0][tid]; s2 += sum_s[w][1][tid]; }
  }
  auto block_sum = [&](double v) -> double {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double r = 0.0;
    for (int w = 0; w < FS_WARPS; ++w) r += red[w];
    return r;
  };
  double tl = 0.0;
  if (own) {
    const float cn = lerp_torch(old, __fdiv_rn((float)s1, (float)d.rows), hp.w2, hp.w2m1, hp.small_w2 != 0);
    d.stat_b[c] = cn;
    pv.aux[aux_cfac(d) + c] = rsqrt_torch(cn);
    tl = s2 / (double)cn;
  }
  tl = block_sum(tl);
  double* tpart = reinterpret_cast<double*>(pv.aux + aux_tpart(d));
  const int strips = (C + FS_COLS - 1) / FS_COLS;
  int last = 0;
  if (tid == 0) {
    tpart[t.slot] = tl;
    __threadfence();
    unsigned before;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(pv.done + 1 * pv.n_tensors + t.tensor) : "memory");
    last = before == (unsigned)strips - 1u;
    if (last) __threadfence();
  }
  if (!__syncthreads_or(last)) return;
  // the last strip of the tensor
  const double* rowpart = reinterpret_cast<const double*>(pv.aux + aux_rowpart(d));
  double rs = 0.0, T = 0.0;
  for (int s = tid; s < S; s += FS_THREADS) rs += __ldcg(rowpart + s);
  for (int s = tid; s < strips; s += FS_THREADS) T += __ldcg(tpart + s);
  rs = block_sum(rs);
  T = block_sum(T);
  if (tid == 0) {
    const float rowmean = __fdiv_rn((float)rs, (float)d.rows);
    const double ss = (double)rowmean * T;
    const float rms = __fdiv_rn((float)sqrt(ss), (float)sqrt((double)d.rows * (double)C));
    const float div = fmaxf(__fdiv_rn(rms, hp.clip), 1.0f);
    *reinterpret_cast<float4*>(pv.aux + aux_scal(d)) = make_float4(rowmean, div, rms, __fdiv_rn(1.0f, div));
  }
}

// The row table of FINAL's tensors, FS_THREADS rows a CTA.  (By the tensor's last strip alone it was the step's longest chain
// of loads: 68 us of FINAL on the 269 M list, whose tallest tensors have 10 240 rows.)
__device__ __forceinline__ void rowtab_run(const PlanView& pv, const AdaDev& hp, const Task& t) {
  if (pv.grads[t.tensor] == nullptr) return;
  const DevTensor& d = pv.tensors[t.tensor];
  const int r = t.row0 + threadIdx.x;
  if ((int)threadIdx.x >= t.n) return;
  const float rn = __ldcg(d.stat_a + r), mu = hp.gc ? __ldcg(pv.aux + aux_mean(d) + r) : 0.0f, sc = hp.int8 ? __ldcg(d.m_scale + r) : 1.0f;
  const float rf = rsqrt_torch(__fdiv_rn(rn, __ldcg(pv.aux + aux_scal(d))));
  pv.aux[aux_rfac(d) + r] = rf;
  reinterpret_cast<float4*>(pv.aux + aux_rowtab(d))[r] =
      make_float4(pv.param_bf16 ? __uint_as_float(pack_bf16_rn(mu, mu)) : mu, rf, sc, 0.0f);
  if (hp.int8) {   // COUNT starts from zeroed row maxima; APPLY decodes with the old scales
    reinterpret_cast<unsigned*>(pv.aux + aux_rowmax(d))[r] = 0u;
    pv.aux[aux_oldsc(d) + r] = sc;
  }
}

// A block an item; with reserved multiprocessors, whose blocks leave, the others claim the items.  Nothing where a wait of this
// plan has run out: STATS then left no sums to go by (the status stays).
template <typename Item>
__device__ __forceinline__ void each_item(const PlanView& pv, const Item& item) {
  __shared__ int next_s;
  if (on_reserved_sm(pv.sm_reserve)) return;
  auto failed = [&]() { return __syncthreads_or(*reinterpret_cast<volatile unsigned*>(pv.status) != 0u) != 0; };   // (the block's)
  if (pv.sm_reserve == 0u) {
    const Task t = pv.tasks[blockIdx.x];
    early_launch();
    after_launch_before();
    if (failed()) return;
    item(t);
    return;
  }
  if (failed()) return;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) next_s = (int)atomicAdd(pv.task_counter, 1u);
    __syncthreads();
    if (next_s >= pv.n_tasks) return;
    item(pv.tasks[next_s]);
  }
}

__global__ void __launch_bounds__(FS_THREADS) ada_final_kernel(const __grid_constant__ PlanView pv, const __grid_constant__ AdaDev hp) {
  each_item(pv, [&](const Task& t) { final_strip(pv, hp, t); });
}
__global__ void __launch_bounds__(FS_THREADS) ada_rowtab_kernel(const __grid_constant__ PlanView pv, const __grid_constant__ AdaDev hp) {
  each_item(pv, [&](const Task& t) { rowtab_run(pv, hp, t); });
}

// ----------------------------------------------------------------------------- host

// The strips of the FINAL launch for the tensors marked in `elig`, then the runs of rows of the row-table launch.
void final_items(const kaon_plan* pl, const std::vector<char>& elig, std::vector<Task>& out, int& n_strips) {
  for (int i = 0; i < pl->n_tensors; ++i) {
    if (!elig[i]) continue;
    const int C = pl->h_tensors[i].cols;
    for (int c = 0; c < C; c += FS_COLS) out.push_back(Task{i, PH_ADA_FINAL, 0, std::min(FS_COLS, C - c), c, c / FS_COLS, 0});
  }
  n_strips = (int)out.size();
  for (int i = 0; i < pl->n_tensors; ++i)
    if (elig[i])
      for (int r = 0; r < pl->h_tensors[i].rows; r += FS_THREADS)
        out.push_back(Task{i, PH_ADA_FINAL, 0, std::min(FS_THREADS, pl->h_tensors[i].rows - r), r, 0, 0});
}

int launch_final(kaon_plan* pl, const PlanView& base, const AdaDev& hp, const Task* items, int n_strips, int n, cudaStream_t s) {
  if (n == 0) return KAON_OK;
  const int most = pl->sm_count * 4;
  PlanView v = base;
  v.tasks = items; v.n_tasks = n_strips; v.task_counter = base.counters2 + 3;
  KAON_CUDA(launch_early(!v.sm_reserve, ada_final_kernel, v.sm_reserve ? most : v.n_tasks, FS_THREADS, 0, s, v, hp));
  v.tasks = items + n_strips; v.n_tasks = n - n_strips; v.task_counter = base.counters2 + 4;
  KAON_CUDA(launch_early(!v.sm_reserve, ada_rowtab_kernel, v.sm_reserve ? most : v.n_tasks, FS_THREADS, 0, s, v, hp));
  pl->launches += 2;
  return KAON_OK;
}

}  // namespace kaon
