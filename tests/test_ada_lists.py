"""The share-out of the Adakaon family's work items (csrc/ada_lists.h, host code): every item has one place, and no item waits
for a launch that comes after its own.  On the GPU, a list whose tensors part ways: 4-bit blocks of 256 beside a matrix of 128
elements, which is one block of 128; and lists long enough to run five blocks an SM."""
import os
import subprocess

import numpy as np
import pytest
import torch

import kaon_oracle as ko

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "k-optimizers_b200", "csrc")
CUDA = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <set>
#include <tuple>
#include "ada_lists.h"
using namespace kaon;
// arguments: optimizer, weight dtype, momentum kind, then rows cols block (rows 0: one dimension); prints how many tensors stay,
// leave with STATS and FINAL, and leave but for STATS and FINAL, and whether STATS comes first; exit code 0 where the lists are sound
int main(int argc, char** argv) {
  kaon_plan pl;
  pl.optimizer = atoi(argv[1]); pl.param_dtype = atoi(argv[2]); pl.momentum_kind = atoi(argv[3]);
  pl.sm_count = 148;
  std::vector<Task> src[2], small;
  for (int i = 4; i + 2 < argc; i += 3) {
    const int ti = pl.n_tensors++;
    DevTensor t{};
    t.rows = atoi(argv[i]); t.cols = atoi(argv[i + 1]); t.block = (unsigned)atoi(argv[i + 2]);
    t.numel = (long long)(t.rows ? t.rows : 1) * t.cols;
    pl.h_tensors.push_back(t);
    if (!t.rows) {
      for (auto& l : src) l.push_back(Task{ti, PH_ADA_FLAT, 0, (int)t.numel, 0, 0, 0});
      continue;
    }
    for (int ph : {PH_ADA_STATS, PH_ADA_FINAL, PH_ADA_COUNT, PH_ADA_APPLY})
      for (int r = 0; r < (ph == PH_ADA_FINAL ? 1 : t.rows); r += 32) {
        const Task k{ti, ph, (long long)r * t.cols, (t.rows - r < 32 ? t.rows - r : 32) * t.cols, r, r / 32, 0};
        src[1].push_back(k);
        if (ph != PH_ADA_COUNT) src[0].push_back(k);
      }
  }
  const AdaLists a = ada_lists(&pl, small, src);
  if (!a.any) return 10;
  typedef std::tuple<int, int, long long> Id;
  auto id = [](const Task& t) { return Id(t.tensor, t.phase, t.e0); };
  for (int v = 0; v < 2; ++v) {
    std::set<Id> kept, stats;
    for (const Task& t : a.keep[v]) if (!kept.insert(id(t)).second) return 1;
    for (const Task& t : a.stats) if (!stats.insert(id(t)).second) return 2;
    bool flat_only = true;
    for (const Task& t : src[v]) {
      const bool here = kept.count(id(t)) != 0, there = stats.count(id(t)) != 0;
      const bool sweep = (t.phase == PH_ADA_COUNT || t.phase == PH_ADA_APPLY) && a.elig[t.tensor];
      const bool final_launch = t.phase == PH_ADA_FINAL && a.leaves[t.tensor];
      if ((int)here + there + sweep + final_launch != 1) return 3;
      if (final_launch)   // (that launch may run ahead of the persistent kernel)
        for (const Task& k : src[v])
          if (k.tensor == t.tensor && k.phase == PH_ADA_STATS && !stats.count(id(k))) return 8;
      if (!here) continue;
      flat_only = flat_only && t.phase == PH_ADA_FLAT;
      // a kept COUNT or APPLY waits for its FINAL, which has to be kept; a kept FINAL for its STATS, kept or launched before
      if ((t.phase == PH_ADA_COUNT || t.phase == PH_ADA_APPLY) && !kept.count(Id(t.tensor, PH_ADA_FINAL, 0))) return 4;
      if (t.phase == PH_ADA_FINAL)
        for (const Task& k : src[v])
          if (k.tensor == t.tensor && k.phase == PH_ADA_STATS && !kept.count(id(k)) && a.order[v] != ADA_KEPT_WAITS) return 5;
    }
    if ((int)kept.size() != (int)a.keep[v].size()) return 7;
  }
  int stay = 0, out = 0, part = 0;
  for (int i = 0; i < pl.n_tensors; ++i) {
    if (a.leaves[i]) ++out;
    else if (a.elig[i]) ++part;
    else ++stay;
  }
  std::printf("%d %d %d %d\n", stay, out, part, (int)(a.order[1] == ADA_KEPT_WAITS));
  return 0;
}
"""

ADAKAON, ADAMUON, F32, BF16, INT8, BITS4 = 1, 2, 0, 1, 2, 3


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("ada_lists")
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", f"-I{CSRC}", f"-I{CUDA}", str(d / "main.cpp"), "-o", str(d / "main")])
    return str(d / "main")


@pytest.mark.parametrize("head,tensors,want", [
    # 4-bit blocks of 256, and one of 128 in the same list: FINAL of the former stays, so their STATS are launched first
    ((ADAKAON, BF16, BITS4), [(8, 16, 128), (1024, 1024, 256), (1024, 1024, 256)], "2 0 1 1"),
    ((ADAKAON, F32, BITS4), [(8, 16, 128), (1024, 1024, 256)], "1 0 1 0"),
    ((ADAKAON, BF16, BITS4), [(1024, 1024, 128), (512, 264, 64), (300, 77, 128), (0, 1280, 128)], "3 1 0 1"),
    ((ADAKAON, BF16, INT8), [(1024, 1024, 0), (64, 128, 0), (0, 1280, 0), (333, 77, 0)], "2 1 1 0"),
    ((ADAMUON, F32, BITS4), [(1024, 1024, 256), (1024, 520, 256), (0, 640, 128)], "1 2 0 0"),
])
def test_no_item_waits_for_a_later_launch(program, head, tensors, want):
    out = subprocess.run([program, *map(str, head), *(str(x) for t in tensors for x in t)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.returncode
    assert out.stdout.strip() == want


@pytest.mark.gpu
@pytest.mark.parametrize("name,kw", [("Adakaon", dict()), ("Nekaon", dict(weight_decay=0.1))])
def test_blocks_of_256_beside_a_block_of_128_vs_oracle(name, kw):
    import kaon_b200
    from _gpu import state_np, to_bits
    shapes = [(8, 16), (1024, 1024), (1024, 1024), (640, 264)]
    kw = dict(kw, lr=1e-3, momentum_dtype="4bit", momentum_4bit_block=256)
    gen = torch.Generator().manual_seed(3)
    host = [(torch.randn(s, generator=gen) * 0.02).bfloat16() for s in shapes]
    params = [torch.nn.Parameter(h.clone().cuda()) for h in host]
    opt = getattr(kaon_b200, name)(params, **kw)
    opt.sr_seed = 5
    inner = getattr(opt, "base_optimizer", opt)
    orc = getattr(ko, "Oracle" + name)([to_bits(h) for h in host], shapes, seed=5, **kw)
    for step in range(2):
        grads = [(torch.randn(s, generator=gen) * 1e-3).bfloat16() for s in shapes]
        for p, g in zip(params, grads):
            p.grad = g.cuda()
        opt.step()
        torch.cuda.synchronize()
        opt.check_device_status()
        orc.step([to_bits(g) for g in grads])
        for i, p in enumerate(params):
            # statistics summed in another order: an ulp or two (2e-6); a code or a weight at a rounding boundary one step off
            for key, want in orc.tensors[i].state.items():
                got = state_np(inner.state[p], key)
                if not isinstance(want, np.ndarray) or got is None or want.size == 0:
                    continue
                got, want = got.reshape(-1), want.reshape(-1)
                if got.dtype.kind == "f":
                    assert np.abs(got - want).max() <= 2e-6 * np.abs(want).max(), (step, shapes[i], key)
                else:
                    assert (got != want).sum() <= 2 + 2e-4 * got.size, (step, shapes[i], key)
            diff = np.abs(to_bits(p).astype(np.int32) - orc.tensors[i].p.reshape(-1).astype(np.int32))
            assert diff.max() <= (2 if name == "Nekaon" else 1) and (diff != 0).sum() <= 1 + 1e-3 * diff.size, (step, shapes[i])


RULE = r"""
#include <cstdlib>
#include "ada_lists.h"
int main(int argc, char** argv) { return kaon::small_takes_five(atoi(argv[1]), atoi(argv[2]), atoi(argv[3]), 148); }
"""


def test_five_blocks_only_where_they_save_a_round(tmp_path):
    (tmp_path / "main.cpp").write_text(RULE)
    subprocess.check_call(["g++", "-std=c++17", "-O1", f"-I{CSRC}", f"-I{CUDA}", str(tmp_path / "main.cpp"), "-o", str(tmp_path / "main")])
    takes = lambda n, four=4, five=5: subprocess.run([str(tmp_path / "main"), str(n), str(four), str(five)]).returncode == 1  # noqa: E731
    assert [n for n in (1, 16, 592, 593, 740, 741, 1184, 1185, 1480, 1481, 1776, 1777, 2220, 2221) if takes(n)] == [593, 740, 1185, 1480, 1777, 2220]
    assert not takes(700, 3, 3) and not takes(700, 4, 4)   # (shared memory lets no fifth in)


@pytest.mark.gpu
@pytest.mark.parametrize("name,kw", [("Adakaon", dict()), ("Adakaon", dict(momentum_dtype="int8", weight_decay=0.1)), ("Nekaon", dict())])
def test_a_long_list_steps_as_two_short_ones(name, kw):
    """700 matrices in one list (five blocks an SM) and in two of 350 (four): the same arithmetic, the same bits."""
    import kaon_b200
    gen = torch.Generator(device="cuda").manual_seed(3)
    shapes = [(8, 128), (64, 8), (16, 264), (128, 32), (5, 1600)] * 140
    values = [(torch.randn(s, device="cuda", generator=gen) * 0.02, torch.randn(s, device="cuda", generator=gen) * 1e-3) for s in shapes]
    runs = []
    for parts in (1, 2):
        params = [torch.nn.Parameter(v.clone()) for v, _ in values]
        for p, (_, g) in zip(params, values):
            p.grad = g.clone()
        n = len(params) // parts
        opts = [getattr(kaon_b200, name)(params[i * n:(i + 1) * n], lr=1e-3, **kw) for i in range(parts)]
        for _ in range(2):
            for o in opts:
                o.step()
        torch.cuda.synchronize()
        for o in opts:
            o.check_device_status()
        runs.append([p.detach() for p in params])
    for a, b in zip(*runs):
        assert torch.equal(a, b), a.shape
