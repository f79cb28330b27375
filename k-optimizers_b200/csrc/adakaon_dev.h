// Device-side hyper-parameter block of the Adakaon / AdaMuon kernels and the launch helpers other
// translation units use.
#pragma once

#include <stddef.h>
#include <stdint.h>

#include <vector>

#include "kaon_device.cuh"
#include "kaon_plan.h"

namespace kaon {

struct AdaDev {
  float w1, w1m1, w2, w2m1, eps1, clip, lrwd, upd_scale;
  int small_w1, small_w2, has_eps, has_wd, cautious, gc, sr, has_m;
  int remove, climb, kahan, int8;
  float a_remove, b_remove, a_climb, b_climb;
  uint32_t step, k0, k1;
  uint32_t rk0[KAON_PHILOX_ROUNDS], rk1[KAON_PHILOX_ROUNDS];  // Philox round keys (k + r * Weyl), from the host
  int mask_off;          // !cautious
  int stats_only;        // second moment only (AdaPNM, KProdigy)
};

// Philox round keys of a hyper-parameter block from its k0, k1
template <typename HP>
inline void philox_round_keys(HP& hp) {
  for (int r = 0; r < KAON_PHILOX_ROUNDS; ++r) { hp.rk0[r] = hp.k0 + 0x9E3779B9u * (uint32_t)r; hp.rk1[r] = hp.k1 + 0xBB67AE85u * (uint32_t)r; }
}

// round keys from k0, k1; no eps is an eps of 0
inline void ada_finish(AdaDev& hp) {
  philox_round_keys(hp);
  if (!hp.has_eps) hp.eps1 = 0.0f;
  hp.mask_off = !hp.cautious;
}

int launch_persistent(kaon_plan* pl, const PlanView& v, const AdaDev& hp, bool early, cudaStream_t s);
// COUNT and APPLY as launches of their own (ada_sweep.cu), for the factored tensors whose rows stream
void sweep_units(const kaon_plan* pl, const std::vector<char>& elig, std::vector<Task>& out);
int ensure_apply2(kaon_plan* pl);
int launch_small(kaon_plan* pl, const PlanView& base, const AdaDev& hp, cudaStream_t s);
int launch_count_apply(kaon_plan* pl, const PlanView& base, const AdaDev& hp, cudaStream_t s);
// the STATS launch over a caller's list of STATS items (all of which pass stats_item_ok, ada_lists.h); `beside`: the launch
// before it on the stream is the persistent kernel's, and the two may run at the same time
int launch_stats(kaon_plan* pl, const PlanView& base, const AdaDev& hp, const Task* tasks, int n, bool beside, cudaStream_t s);
// FINAL as launches of its own (ada_final.cu)
void final_items(const kaon_plan* pl, const std::vector<char>& elig, std::vector<Task>& out, int& n_strips);
int launch_final(kaon_plan* pl, const PlanView& base, const AdaDev& hp, const Task* items, int n_strips, int n, cudaStream_t s);

// All of that over a plan's lists: the persistent kernel's and its place (ada_lists.h); the STATS launch's; the FINAL launch's
// strips and the row-table launch's runs
struct AdaStages {
  const Task* keep; int n_keep;
  int order;
  const Task* stats; int n_stats;
  const Task* final; int n_strips, n_final;
};
int launch_statistics(kaon_plan* pl, const PlanView& base, const AdaDev& hp, const AdaStages& st, cudaStream_t s);
inline AdaStages ada_stages(const kaon_plan* pl, bool cautious) {   // (of a plan with apply2 == 1)
  const int i = cautious ? 1 : 0;
  return AdaStages{pl->d_tasks_na[i], pl->n_tasks_na[i], pl->ada_order[i], pl->d_tasks_stats, pl->n_tasks_stats,
                   pl->d_tasks_final, pl->n_tasks_strips, pl->n_tasks_final};
}

}  // namespace kaon
