"""Products by pairs of CTAs (csrc/ns_share.h, csrc/ns_gemm.cuh): their tiles are handed out once each with the coordinates they
have; on the GPU, the iteration against fp64 over batches small and large, and over batches all of whose products are pairs'
(the share-out says so), at extents that end inside a tile, inside either CTA's half of it and inside a k-block."""
import os
import subprocess

import pytest
import torch

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "k-optimizers_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "ns_share.h"
using namespace kaon;
// arguments: pairs, then M N K sym of each product; exit code 0 where the share-out is sound
int main(int argc, char** argv) {
  std::vector<NsShape> ps;
  for (int i = 2; i + 3 < argc; i += 4) ps.push_back(NsShape{atoi(argv[i]), atoi(argv[i + 1]), atoi(argv[i + 2]), atoi(argv[i + 3]) != 0});
  const int pairs = atoi(argv[1]);
  const NsShare s = ns_share_out(ps, pairs, true);
  const int grid = (int)s.begin.size() - 1;
  if (!s.pair || grid < 1 || grid > pairs || s.begin[0] != 0 || s.begin[grid] != (int)s.tiles.size()) return 1;
  for (size_t i = 0; i < ps.size(); ++i) {
    const int w = ns_tile_cols(s.bn, ps[i].N, true), tn = ns_tiles(ps[i].N, w), tm = ns_tiles(ps[i].M, 2 * NS_TILE_M);
    if (w != 128 && w != 256) return 2;
    std::vector<char> seen((size_t)tm * tn, 0);
    for (const NsTile& t : s.tiles)
      if (t.prob == (int)i) {
        if (t.mi < 0 || t.mi >= tm || t.ni < 0 || t.ni >= tn || seen[(size_t)t.mi * tn + t.ni]++) return 3;
      }
    for (int mi = 0; mi < tm; ++mi)
      for (int ni = 0; ni < tn; ++ni)   // below the diagonal: from its mirror image
        if (seen[(size_t)mi * tn + ni] != (ps[i].sym && (ni + 1) * w - 1 < mi * 2 * NS_TILE_M ? 0 : 1)) return 4;
  }
  // no share-out where none stays below the bound given
  if (ns_share_out(ps, pairs, true, s.most).bn != 0) return 5;
  return 0;
}
"""


@pytest.mark.parametrize("products", [
    [(1, 1, 1, 0)],
    [(257, 129, 65, 0), (256, 256, 64, 1), (300, 300, 1000, 1)],
    [(3072, 3072, 9216, 1), (3072, 12288, 3072, 0), (9216, 3072, 3072, 0)],
])
def test_share_out_of_pairs(products, tmp_path):
    (tmp_path / "main.cpp").write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O2", f"-I{CSRC}", str(tmp_path / "main.cpp"), "-o", str(tmp_path / "main")])
    subprocess.check_call([str(tmp_path / "main"), "74", *[str(x) for p in products for x in p]])


@pytest.mark.gpu
@pytest.mark.parametrize("shapes", [
    [(640, 640)] * 4 + [(5120, 640), (640, 2560)],
    [(1100, 520), (520, 1100), (1000, 1000), (1400, 1288), (264, 4104)],
    [(3072, 3072), (3072, 12288)],
])
def test_iteration_vs_fp64(shapes):
    import kaon_b200
    gen = torch.Generator(device="cuda").manual_seed(5)
    runs = []
    for _ in range(2):
        gen.manual_seed(5)
        params = [torch.nn.Parameter((torch.randn(s, device="cuda", generator=gen) * 0.02).bfloat16()) for s in shapes]
        for p in params:
            p.grad = (torch.randn(p.shape, device="cuda", generator=gen) * 1e-3).bfloat16()
        opt = kaon_b200.AdaMuon(params, lr=1e-3, betas=(0.0, 0.999), bf16_method="none")   # no momentum: X is the gradient
        opt.step()
        torch.cuda.synchronize()
        opt.check_device_status()
        runs.append([opt.orthogonalised(p).clone() for p in params])
    for p, got, again in zip(params, *runs):
        assert torch.equal(got.view(torch.int16), again.view(torch.int16)), p.shape
        x = p.grad.double()
        x /= x.norm() + 1e-7
        for _ in range(opt.param_groups[0]["ns_steps"]):
            a = x @ x.T
            x = 3.4445 * x + (-4.7750 * a + 2.0315 * a @ a) @ x
        # a chain of bf16 products: a few 2^-8 of an entry's size
        assert ((got.double() - x).norm() / x.norm()).item() < 2e-2, p.shape


PAIRS = r"""
#include <cstdio>
#include <cstdlib>
#include "ns_share.h"
using namespace kaon;
// arguments: multiprocessors, then R C of each matrix of a batch; exit code 0 where every product of an iteration takes pairs
int main(int argc, char** argv) {
  NsShares::Key key;
  for (int i = 2; i + 1 < argc; i += 2) key.push_back({atoll(argv[i]), atoll(argv[i + 1])});
  NsShares shares;
  for (const NsShare& s : shares.get(key, atoi(argv[1]))) if (!s.pair) return 1;
  return 0;
}
"""

# 3080 = 12 x 256 + 8: the last tile's second CTA has no row; 2952 = 11 x 256 + 136: it has eight; 100, 104: tiles of 128 columns;
# 264 and 3336 end inside a k-block of 64; 2001: rows of the last product off the 16-byte grid
RAGGED = [
    [(2952, 4104), (4104, 2952), (3096, 3096), (100, 3000), (3000, 104)],
    [(3080, 3400), (3400, 3080), (264, 3336), (3001, 264), (264, 2001)],
]


@pytest.mark.parametrize("shapes", RAGGED)
def test_ragged_batches_take_pairs(shapes, tmp_path):
    (tmp_path / "main.cpp").write_text(PAIRS)
    subprocess.check_call(["g++", "-std=c++17", "-O2", f"-I{CSRC}", str(tmp_path / "main.cpp"), "-o", str(tmp_path / "main")])
    subprocess.check_call([str(tmp_path / "main"), "148", *[str(x) for s in shapes for x in s]])


@pytest.mark.gpu
@pytest.mark.parametrize("shapes", RAGGED)
def test_ragged_pairs_vs_fp64(shapes):
    assert torch.cuda.get_device_properties(0).multi_processor_count == 148   # (of the share-out above)
    test_iteration_vs_fp64(shapes)
