// Which of a plan's work items the persistent kernel of the Adakaon family keeps and which the launches beside it take
// (host code; looked over by tests/test_ada_lists.py).
#pragma once

#include <algorithm>
#include <vector>

#include "kaon_plan.h"

namespace kaon {

constexpr int ST_MAXROWS = 1024;   // rows of one item of the STATS launch at most

// A STATS item (of bf16 rows) the STATS launch can take
inline bool stats_item_ok(const kaon_plan* pl, const Task& t) {
  const DevTensor& dt = pl->h_tensors[t.tensor];
  return dt.cols >= 256 && (dt.cols & 7) == 0 && t.n / dt.cols <= ST_MAXROWS && (dt.aux_off & 3) == 0;
}

// Whether a list of n small tensors runs the build of ada_small_kernel for five blocks an SM (48 registers, which spill) or the one
// for four: `four`, `five`: the blocks that registers and shared memory let in of either.  Only where that saves a round of blocks.
inline bool small_takes_five(int n, int four, int five, int sms) {
  auto rounds = [&](int blocks) { return (n - 1) / (blocks * sms) + 1; };
  return five > four && four > 0 && rounds(five) < rounds(four);
}

// The tensors (of bf16 rows) whose STATS items in `list` the STATS launch can take, all of them
inline std::vector<char> stats_tensors(const kaon_plan* pl, const std::vector<Task>& list) {
  std::vector<char> ok((size_t)pl->n_tensors, 0);
  for (const Task& t : list) if (t.phase == PH_ADA_STATS) ok[t.tensor] = 1;
  for (const Task& t : list) if (t.phase == PH_ADA_STATS && !stats_item_ok(pl, t)) ok[t.tensor] = 0;
  return ok;
}

// Whether the persistent kernel's list of n items runs beside a STATS launch of n_stats: a few 1-D tensors, or any list where both
// launches find room.  (Its blocks fill a multiprocessor each: beside a STATS that needs the whole machine, a list with
// stages that wait for one another cost 40 us more than the two in turn, and the 540 1-D tensors of the 2.6 B list gained nothing.)
inline bool runs_beside(int n, bool flat_only, int n_stats, int sms) {
  return n > 0 && ((flat_only && n <= sms / 2) || n + n_stats / 4 <= sms);
}

struct AdaLists {
  bool any = false;               // some tensor's COUNT and APPLY are launches of their own; nothing below where none's are
  std::vector<char> elig;         // those tensors
  std::vector<char> leaves;       // and those of them whose FINAL is a launch, too
  std::vector<Task> stats;        // the STATS launch's items
  std::vector<Task> keep[2];      // the persistent kernel's: from the list without COUNT items, from the full list
  bool stats_first = false;       // its FINAL items wait for items of the STATS launch, which then has to come before it
  bool beside[2] = {false, false};  // the list may run beside the STATS launch
  bool long_rows_ok = true;       // no tensor whose rows exceed a work item is left to it
};

// Per factored tensor: COUNT and APPLY leave the persistent kernel when its rows stream (a multiple of 8 elements; 4-bit
// block 128), its STATS items when they qualify (stats_item_ok, bf16 gradients or AdaMuon's bf16 signal), and FINAL with both: a COUNT
// that stays waits for its FINAL.  Everything else - the 1-D tensors, the stages of tensors that do not qualify - stays.
// `src`: the plan's list without COUNT items and its full one; `small`: the tensors one CTA steps on its own.
inline AdaLists ada_lists(const kaon_plan* pl, const std::vector<Task>& small, const std::vector<Task> src[2]) {
  AdaLists a;
  const bool muon = pl->optimizer == KAON_OPT_ADAMUON;
  const int mk = muon ? KAON_M_NONE : pl->momentum_kind;
  const bool stats_dtype = muon || pl->param_dtype == KAON_DT_BF16;
  a.elig.assign((size_t)pl->n_tensors, 0);
  a.leaves.assign((size_t)pl->n_tensors, 0);
  for (int i = 0; i < pl->n_tensors; ++i) {
    const DevTensor& t = pl->h_tensors[i];
    if (t.rows <= 0 || t.numel == 0 || (t.cols & 7) != 0) continue;
    if (mk == KAON_M_4BIT && t.block != 128u) continue;
    a.elig[i] = 1;
  }
  for (const Task& t : small) a.elig[t.tensor] = 0;
  a.any = std::find(a.elig.begin(), a.elig.end(), 1) != a.elig.end();
  if (!a.any) return a;
  // the tensors whose STATS leave
  const std::vector<char> gone = stats_dtype ? stats_tensors(pl, src[0]) : std::vector<char>((size_t)pl->n_tensors, 0);
  for (const Task& t : src[0])
    if (t.phase == PH_ADA_STATS && gone[t.tensor]) a.stats.push_back(t);
  for (int i = 0; i < pl->n_tensors; ++i) a.leaves[i] = gone[i] && a.elig[i];
  for (int variant = 0; variant < 2; ++variant) {
    bool flat_only = true;
    for (const Task& t : src[variant]) {
      if (t.phase == PH_ADA_FINAL && a.leaves[t.tensor]) continue;
      if ((t.phase == PH_ADA_APPLY || t.phase == PH_ADA_COUNT) && a.elig[t.tensor]) continue;
      if (t.phase == PH_ADA_STATS && gone[t.tensor]) continue;
      // what stays here is staged row by row: a tensor whose rows exceed a work item cannot stay
      if (t.phase != PH_ADA_FINAL && t.phase != PH_ADA_FLAT && pl->h_tensors[t.tensor].cols > CAP) a.long_rows_ok = false;
      if (t.phase == PH_ADA_FINAL && gone[t.tensor]) a.stats_first = true;
      flat_only = flat_only && t.phase == PH_ADA_FLAT;
      a.keep[variant].push_back(t);
    }
    a.beside[variant] = runs_beside((int)a.keep[variant].size(), flat_only, (int)a.stats.size(), pl->sm_count);
  }
  if (a.stats_first) a.beside[0] = a.beside[1] = false;
  return a;
}

}  // namespace kaon
