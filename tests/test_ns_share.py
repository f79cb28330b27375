"""The tiles of grouped matrix products (csrc/ns_share.h, host code): every tile that has to be computed is handed out once,
with the coordinates it has, up to the tallest matrices a plan takes."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "k-optimizers_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "ns_share.h"
using namespace kaon;
// arguments: CTAs, then M N K sym of each product; exit code 0 where the share-out is sound
int main(int argc, char** argv) {
  std::vector<NsShape> ps;
  for (int i = 2; i + 3 < argc; i += 4) ps.push_back(NsShape{atoi(argv[i]), atoi(argv[i + 1]), atoi(argv[i + 2]), atoi(argv[i + 3]) != 0});
  const int ctas = atoi(argv[1]);
  const NsShare s = ns_share_out(ps, ctas);
  const int grid = (int)s.begin.size() - 1;
  if (grid < 1 || grid > ctas || s.begin[0] != 0 || s.begin[grid] != (int)s.tiles.size()) return 1;
  for (int c = 0; c < grid; ++c) if (s.begin[c] >= s.begin[c + 1]) return 2;   // (a CTA without a tile)
  std::vector<std::vector<char>> seen(ps.size());
  std::vector<int> tn(ps.size());
  for (size_t i = 0; i < ps.size(); ++i) {
    tn[i] = ns_tiles(ps[i].N, ns_tile_cols(s.bn, ps[i].N));
    seen[i].assign((size_t)ns_tiles(ps[i].M, NS_TILE_M) * tn[i], 0);
  }
  for (const NsTile& t : s.tiles) {
    if (t.prob < 0 || t.prob >= (int)ps.size() || t.mi < 0 || t.ni < 0 || t.ni >= tn[t.prob]) return 3;
    const size_t at = (size_t)t.mi * tn[t.prob] + t.ni;
    if (at >= seen[t.prob].size() || seen[t.prob][at]++) return 4;
  }
  for (size_t i = 0; i < ps.size(); ++i) {
    const long long w = ns_tile_cols(s.bn, ps[i].N);
    for (size_t at = 0; at < seen[i].size(); ++at) {
      // a symmetric product's tile that lies wholly below the diagonal comes from its mirror image
      const long long last_col = ((long long)(at % tn[i]) + 1) * w - 1, first_row = (long long)(at / tn[i]) * NS_TILE_M;
      if (seen[i][at] != (ps[i].sym && last_col < first_row ? 0 : 1)) return 5;
    }
  }
  std::printf("%d %zu\n", s.bn, s.tiles.size());
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("ns_share")
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O2", f"-I{CSRC}", str(d / "main.cpp"), "-o", str(d / "main")])
    return str(d / "main")


@pytest.mark.parametrize("shapes", [
    [(1, 1, 1, 0)],
    [(320, 320, 1280, 1), (320, 320, 320, 1), (36, 36, 320, 1), (4, 4, 2880, 1)],
    [(333, 77, 77, 0), (129, 65, 64, 0), (128, 64, 65, 0)],
    [(3072, 3072, 3072, 1)] * 2 + [(3072, 3072, 9216, 1), (3072, 3072, 12288, 1)],
    [(4194560, 8, 8, 0), (64, 64, 64, 1)],              # more row tiles than 15 bits hold
    [(2147483647, 1, 1, 0)],                            # the tallest matrix of a plan
])
@pytest.mark.parametrize("ctas", [1, 148])
def test_every_tile_once(program, shapes, ctas):
    out = subprocess.run([program, str(ctas), *(str(x) for s in shapes for x in s)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, (out.returncode, out.stderr)


def test_stages_of_a_batch_are_shared_out_once(tmp_path):
    """Batches of the same shapes get the same share-out, and its shapes are those of the iteration's products."""
    (tmp_path / "m.cpp").write_text(r"""
#include "ns_share.h"
using namespace kaon;
int main() {
  NsShares s;
  const NsShares::Key wide{{320, 1280}, {64, 64}}, tall{{1280, 320}, {64, 64}};
  const auto* a = &s.get(wide, 148);
  const auto* b = &s.get(tall, 148);
  if (a != &s.get(wide, 148) || b == a || s.known.size() != 2) return 1;
  const NsShape x = ns_stage_shape(2, 320, 1280), y = ns_stage_shape(2, 1280, 320), z = ns_stage_shape(0, 1280, 320);
  return x.M == 320 && x.N == 1280 && x.K == 320 && y.M == 1280 && y.N == 320 && y.K == 320 && z.M == 320 && z.K == 1280 && z.sym ? 0 : 2;
}
""")
    subprocess.check_call(["g++", "-std=c++17", f"-I{CSRC}", str(tmp_path / "m.cpp"), "-o", str(tmp_path / "m")])
    assert subprocess.run([str(tmp_path / "m")]).returncode == 0
