// Host rules that choose between launches: plain functions of sizes and counts, so
// that they can be tested without a GPU.
#pragma once
#include <algorithm>

namespace nddo {

// Size buckets of a molecule list: each has launches of its own, with its own
// shared-memory footprint.  The first edge keeps bases below the cluster Jacobi's
// minimum apart from the ones it serves, 194 those below the cluster
// tridiagonalisation's, so a molecule's kernel follows its own size.
constexpr int kSizeBuckets = 9;
constexpr int kSizeBucketEdges[kSizeBuckets] = {31, 64, 96, 128, 160, 194, 256, 338, 1 << 30};
inline int size_bucket(int n) { return (int)(std::lower_bound(kSizeBucketEdges, kSizeBucketEdges + kSizeBuckets, n) - kSizeBucketEdges); }

// Tridiagonalisation by a cluster of eight CTAs per molecule (tridiag.cu) instead
// of one CTA, for `count` molecules of up to n basis functions tridiagonalised at
// about the same time: those of the launch's list and of the other groups' lists
// beside it.  A cluster has an SM for each CTA, so 15 or so (`clusters`) run at a
// time; a wave of them has to cost less than its share of the one-CTA kernel, whose
// time grows as N^3 while its SMs hold up to 152 molecules: two waves at N = 234
// 2.9 ms against 3.5, three at 300 6.8 against 7.3, three at 396 11.7 against 16; two
// at 180 2.0 against 1.8.  Counted by group, 152 molecules of N = 300 in four groups
// took three waves each, at once: eight iterations 281 ms, 172 with one CTA a molecule.
constexpr int kHhClusterMinN = 195;   // its smallest basis, one more than an edge of the size buckets
constexpr int kHhClusterWaveN = 100;  // basis functions that pay for a wave of clusters
inline bool hh_cluster_pays(int count, int n, int clusters) {
  return n >= kHhClusterMinN && (count + clusters - 1) / clusters * kHhClusterWaveN <= n;
}

// The effort of each SCF iteration of a batch whose density comes from the
// purification.  Effort 0: few purification steps (18 to 24 are the rule), 1: as many
// as it has, 2: the eigensolver as well.  A molecule that the purification did not
// treat waits without advancing until the host has read the counts of its block and
// enqueues an iteration of more effort.  The first `early` iterations, whose gaps are
// small, have effort 1 from the start.  A wait after few steps asks for all of them in
// the next blocks, and for good at the second time; a wait although a block had all of
// them asks for the eigensolver in the first iteration of the next blocks, and in
// every iteration from the second time on.  tiled: some molecule is on the tile kernel;
// the one-CTA kernel takes the steps it needs at any effort.
// Raised only for a block's first iteration, effort 1 could not settle a molecule that
// keeps needing more than the few steps: it was counted as waiting again at the
// block's end and the whole batch went over to the eigensolver.
// gapless: some molecule is known to have no gap (a lone atom), so the eigensolver is
// there from the start: an oxygen atom's two iterations take 0.5 ms with it and took
// 2.8 waiting for it.
class EffortPlan {
 public:
  EffortPlan(bool tiled, int early, bool gapless) : tiled_(tiled), early_(tiled ? early : 0) {
    if (gapless) first_ = rest_ = 2;
  }
  // effort of the b-th iteration of block `block`, the it-th of all
  int next(int block, int b, int it) {
    const int e = std::max(b == 0 ? first_ : rest_, it < early_ ? 1 : 0);
    int& low = low_[block & 1];
    low = b == 0 ? e : std::min(low, e);
    return e;
  }
  // whether a molecule was waiting at the end of block `block`; `upcoming` is the
  // next one to be enqueued
  void seen(int block, bool waiting, int upcoming) {
    if (rest_ == 2 || block < since_) return;   // nothing more to raise, or enqueued before the last raise
    if (!waiting) {
      first_ = rest_ = step_waits_ > 1 ? 1 : 0;
      return;
    }
    if (tiled_ && low_[block & 1] == 0) {
      ++step_waits_;
      first_ = rest_ = 1;
    } else {
      ++eigen_waits_;
      first_ = 2;
      rest_ = eigen_waits_ > 1 ? 2 : tiled_ ? 1 : 0;
    }
    since_ = upcoming;
  }

 private:
  bool tiled_;
  int early_;
  int first_ = 0, rest_ = 0;                // effort of a block's first iteration and of its others
  int step_waits_ = 0, eigen_waits_ = 0;
  int since_ = 0;                           // first block enqueued with the efforts of the last raise
  int low_[2] = {0, 0};                     // lowest effort of the last two blocks
};

// molecules still active after a block, and those of them that wait
struct BlockCounts { int active, waiting; };

// The SCF loop: blocks of iterations, enqueued one ahead of the counts that are read.
// iterate(effort) enqueues an iteration, count(slot) the counts after a block, read(slot)
// waits for them (slot 0 or 1, alternately).  Past max_iter only molecules that waited
// are still active.
template <typename Iterate, typename Count, typename Read>
void run_blocks(int block, int max_iter, bool purified, EffortPlan plan, Iterate iterate, Count count, Read read) {
  int it = 0, nblock = 0;
  for (;;) {
    for (int b = 0; b < block && (b == 0 || it < max_iter); ++b, ++it) iterate(plan.next(nblock, b, it));
    const bool last = it >= max_iter;
    count(nblock & 1);
    ++nblock;
    if (last && !purified) break;
    if (nblock < 2 && !last) continue;
    const int seen = last ? nblock - 1 : nblock - 2;
    const BlockCounts c = read(seen & 1);
    if (c.active == 0) break;
    if (purified) plan.seen(seen, c.waiting > 0, nblock);
  }
}

}  // namespace nddo
