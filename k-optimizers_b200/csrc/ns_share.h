// The tiles of a batch's grouped products and how they are shared out over the CTAs of a launch (ns.cu).  Host code,
// compiled without CUDA too.
#pragma once

#include <algorithm>
#include <array>
#include <functional>
#include <map>
#include <queue>
#include <utility>
#include <vector>

#ifdef __CUDACC__
#define NS_HD __host__ __device__
#else
#define NS_HD
#endif

namespace kaon {

constexpr int NS_TILE_M = 128, NS_TILE_K = 64;   // rows of an output tile, K elements of a pipeline stage

// (tile coordinates are int: a matrix of 2^31 - 1 rows, the most a plan takes, has 2^24 row tiles)
constexpr long long NS_PAIR_MIN = 20000;         // the least work of a pair (see ns_share_out's cost: 80 k-blocks of a widest tile)
struct NsTile { int prob, mi, ni; };

// one product: out[M, N], K deep; sym: only the tiles that reach the diagonal are computed
struct NsShape { int M, N, K; bool sym; };

// A stage's tiles: CTA (pair of CTAs) b takes tiles[begin[b]] .. tiles[begin[b + 1]].
struct NsShare {
  bool pair = false;         // tiles of 2 x NS_TILE_M rows, a pair of CTAs each
  int bn = 0;                // width of the stage's tiles (a narrower matrix: its own, see ns_tile_cols)
  long long most = 0;        // the longest CTA's work
  std::vector<NsTile> tiles;
  std::vector<int> begin;
};

NS_HD inline int ns_tiles(int extent, int tile) { return (extent - 1) / tile + 1; }   // (extent >= 1; no sum that overflows)
inline int ns_tile_cols(int bn, int N, bool pair = false) {   // (a pair's CTAs hold half the columns each, in boxes of 64)
  const int g = pair ? 128 : 64;
  return std::min(bn, ns_tiles(N, g) * g);
}
inline int ns_tile_rows(bool pair) { return pair ? 2 * NS_TILE_M : NS_TILE_M; }
inline int ns_first_col(const NsShape& p, int bn, int mi, bool pair = false) {
  return p.sym ? std::min(ns_tiles(p.N, bn), (int)((long long)mi * ns_tile_rows(pair) / bn)) : 0;
}

// Tiles of one stage shared out over at most `ctas` CTAs (`pair`: pairs of CTAs), the longest first to the one with the least
// work.  The cost of a tile is a CTA's bytes into shared memory per k-block (128 + BN rows of 128 bytes, a pair's CTA
// 128 + BN / 2: what a tile of up to 256 columns waits for, not the tensor cores) times its k-blocks, plus its epilogue.  Tile widths: the one of 256 / 192 / 128 / 64 columns (the
// same for a stage) whose longest CTA has the least work: wide tiles need fewer bytes, narrow ones fill the machine.
// A width whose mean work is no less than the longest CTA's so far cannot win and is not shared out: of a large batch
// only the widest is.  `under`: nor is one that does not stay below this; nothing (bn 0) where none does.
inline NsShare ns_share_out(const std::vector<NsShape>& ps, int ctas, bool pair = false, long long under = 0) {
  NsShare best;
  best.most = under;
  for (int bn : {256, 192, 128, 64}) {
    if (pair && bn % 128) continue;
    struct P { long long cost; int prob; };
    std::vector<P> order;
    long long count = 0, work = 0;
    for (int i = 0; i < (int)ps.size(); ++i) {
      const int w = ns_tile_cols(bn, ps[i].N, pair), tm = ns_tiles(ps[i].M, ns_tile_rows(pair)), tn = ns_tiles(ps[i].N, w);
      const long long cost = (long long)ns_tiles(ps[i].K, NS_TILE_K) * (128 + (pair ? w / 2 : w)) + 400 + w;
      long long c = (long long)tm * tn;
      for (int mi = 0; ps[i].sym && mi < tm; ++mi) c -= ns_first_col(ps[i], w, mi, pair);
      order.push_back(P{cost, i});
      count += c;
      work += c * cost;
    }
    const int grid = (int)std::min<long long>(ctas, count);
    if (best.most && work >= best.most * grid) continue;
    std::stable_sort(order.begin(), order.end(), [](const P& a, const P& b) { return a.cost > b.cost; });
    typedef std::pair<long long, int> Load;
    std::priority_queue<Load, std::vector<Load>, std::greater<Load>> q;
    for (int c = 0; c < grid; ++c) q.push(Load(0, c));
    std::vector<std::vector<NsTile>> mine(grid);
    long long most = 0;
    for (const P& o : order) {
      const NsShape& p = ps[o.prob];
      const int w = ns_tile_cols(bn, p.N, pair), tm = ns_tiles(p.M, ns_tile_rows(pair)), tn = ns_tiles(p.N, w);
      for (int mi = 0; mi < tm; ++mi)
        for (int ni = ns_first_col(p, w, mi, pair); ni < tn; ++ni) {
          Load l = q.top();
          q.pop();
          l.first += o.cost;
          most = std::max(most, l.first);
          mine[l.second].push_back(NsTile{o.prob, mi, ni});
          q.push(l);
        }
    }
    if (best.most && most >= best.most) continue;
    best = NsShare();
    best.pair = pair;
    best.bn = bn;
    best.most = most;
    for (int c = 0; c < grid; ++c) {
      best.begin.push_back((int)best.tiles.size());
      best.tiles.insert(best.tiles.end(), mine[c].begin(), mine[c].end());
    }
    best.begin.push_back((int)best.tiles.size());
  }
  return best;
}

// The three products of an iteration on a matrix stored [R, C] (r, k: its smaller and larger side):
// A = X X^T [r, r], B = b A + c A A [r, r], X <- a X + B X as stored.
inline NsShape ns_stage_shape(int stage, long long R, long long C) {
  const int r = (int)std::min(R, C), k = (int)std::max(R, C);
  if (stage == 0) return NsShape{r, r, k, true};
  if (stage == 1) return NsShape{r, r, r, true};
  return R > C ? NsShape{k, r, r, false} : NsShape{r, k, r, false};
}

// Share-outs by the shapes of a batch: all iterations of a batch have the same, and most batches of a list too.
struct NsShares {
  typedef std::vector<std::pair<long long, long long>> Key;   // the matrices' [R, C]
  std::map<Key, std::array<NsShare, 3>> known;
  const std::array<NsShare, 3>& get(const Key& key, int ctas) {
    const auto it = known.find(key);
    if (it != known.end()) return it->second;
    std::array<NsShare, 3> a;
    for (int stage = 0; stage < 3; ++stage) {
      std::vector<NsShape> shapes;
      for (const auto& m : key) shapes.push_back(ns_stage_shape(stage, m.first, m.second));
      // Pairs, unless single CTAs are done earlier (a small batch fills the machine with those only) or the work is short.  What
      // pairs save is energy, on a machine that runs long products at its power limit: four width-3072 blocks 11.4 -> 10.9 ms a
      // step; the products of a width-320 list, a few k-blocks a CTA, 343 us with single CTAs and 361 with pairs.
      a[stage] = ctas > 1 ? ns_share_out(shapes, ctas / 2, true) : NsShare();
      if (a[stage].most < NS_PAIR_MIN) a[stage] = NsShare();
      NsShare one = ns_share_out(shapes, ctas, false, a[stage].most);
      if (one.bn) a[stage] = std::move(one);
    }
    return known.emplace(key, std::move(a)).first->second;
  }
};

}  // namespace kaon
