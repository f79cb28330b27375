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

// The place of the persistent kernel's list among the STATS and FINAL launches of the tensors whose FINAL may leave: first, and beside
// STATS; first; last, beginning while FINAL and the row table drain; or between STATS and FINAL, because its own FINAL items
// wait for STATS items that left.
enum : int { ADA_KEPT_BESIDE = 0, ADA_KEPT_FIRST = 1, ADA_KEPT_LAST = 2, ADA_KEPT_WAITS = 3 };

// The place of a list of n items that waits for nothing of the others', beside n_stats STATS items and n_final FINAL items (strips of
// FINAL_STRIP columns) of theirs; ADA_KEPT_WAITS: their FINAL had better stay in the list.  A block of the persistent kernel
// fills a multiprocessor.  Us a step:
// - beside STATS where both find room, or where 1-D tensors alone leave half the machine (AdaPNM, width-448 UNet: 252, as separate launches
//   300; beside a STATS that needs the whole machine, 40 more than the two in turn);
// - 1-D tensors alone, many: first (the 540 of the 2.6 B list gained nothing elsewhere);
// - stages that wait for one another, with little else in STATS: last (Adakaon int8, ragged list: 76, first 95, FINAL kept 90);
// - with STATS enough to fill half the machine, but few strips: FINAL kept, which such a list finds blocks for while it waits
//   (Nekaon, forty pairs of rank 32 and width 1280: 173, last 226); with many strips last (120 pairs of rank 64 and width 1536: 455,
//   FINAL kept 491).
inline int kept_place(int n, bool flat_only, int n_stats, int n_final, int sms) {
  if (n == 0) return ADA_KEPT_FIRST;
  if ((flat_only && n <= sms / 2) || n + n_stats / 4 <= sms) return ADA_KEPT_BESIDE;
  if (flat_only) return ADA_KEPT_FIRST;
  return n_stats <= sms / 2 || n_final > 2 * sms ? ADA_KEPT_LAST : ADA_KEPT_WAITS;
}

struct AdaLists {
  bool any = false;               // some tensor's COUNT and APPLY are launches of their own; nothing below where none's are
  std::vector<char> elig;         // those tensors
  std::vector<char> leaves;       // and those of them whose FINAL is a launch, too
  std::vector<Task> stats;        // the STATS launch's items
  std::vector<Task> keep[2];      // the persistent kernel's: from the list without COUNT items, from the full list
  int order[2] = {ADA_KEPT_FIRST, ADA_KEPT_FIRST};   // and their place
  bool long_rows_ok = true;       // no tensor whose rows exceed a work item is left to it
};

// Per factored tensor: COUNT and APPLY leave the persistent kernel when its rows stream (a multiple of 8 elements; 4-bit
// block 128), its STATS items when they qualify (stats_item_ok, bf16 gradients or AdaMuon's bf16 signal), and FINAL with both (a COUNT
// that stays waits for its FINAL), unless it had better stay (kept_place).  Everything else - the 1-D tensors, the stages of tensors that do not qualify - stays.
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
  // the list a tensor's FINAL may leave, without what leaves in any case
  auto stays = [&](const Task& t) {
    return !((t.phase == PH_ADA_APPLY || t.phase == PH_ADA_COUNT) && a.elig[t.tensor]) && !(t.phase == PH_ADA_STATS && gone[t.tensor]);
  };
  {
    int n = 0, n_final = 0;
    bool flat_only = true, waits = false;
    for (const Task& t : src[1]) {
      if (!stays(t)) continue;
      if (t.phase == PH_ADA_FINAL && a.leaves[t.tensor]) { ++n_final; continue; }
      ++n;
      flat_only = flat_only && t.phase == PH_ADA_FLAT;
      waits = waits || (t.phase == PH_ADA_FINAL && gone[t.tensor]);
    }
    int place = kept_place(n, flat_only, (int)a.stats.size(), n_final, pl->sm_count);
    if (place == ADA_KEPT_WAITS) a.leaves.assign((size_t)pl->n_tensors, 0);
    if (waits) place = ADA_KEPT_WAITS;
    a.order[0] = a.order[1] = place;
  }
  for (int variant = 0; variant < 2; ++variant)
    for (const Task& t : src[variant]) {
      if (!stays(t) || (t.phase == PH_ADA_FINAL && a.leaves[t.tensor])) continue;
      // what stays here is staged row by row: a tensor whose rows exceed a work item cannot stay
      if (t.phase != PH_ADA_FINAL && t.phase != PH_ADA_FLAT && pl->h_tensors[t.tensor].cols > CAP) a.long_rows_ok = false;
      a.keep[variant].push_back(t);
    }
  return a;
}

}  // namespace kaon
