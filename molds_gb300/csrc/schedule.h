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

}  // namespace nddo
