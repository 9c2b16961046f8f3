// Which walk answers a kNN or normal batch, and how its lists start.  Plain
// functions of sizes and settings, compiled for the host by a test.
#pragma once

#include <stdint.h>

namespace pptkg {

constexpr int KNN_MAX_K = 64;     // largest k of the packets' register lists
constexpr int WARP_MAX_K = 256;   // largest k of the warp lists

// What puts a batch's queries in tree order, which packets need: nothing (all
// points of a tree, of a forest), a counting sort of their row numbers' tree
// positions, or that after a descent per point.
enum class BatchOrder { tree, rows, points };

// What a batch answers.  Lists that leave the query's own point out (knn,
// both) cost packets more: their own first chunk is never full.
enum class Answer { knn, both, normals };

// Largest batch in tree order, over trees of p points each, that runs one warp
// per query.  Trees of a few leaf ranges need no walk, which packets then
// answer from the warm start.  us, packets / warps, on a surface (c x p: c
// clouds of p points):
//   normals, float:   k = 4: 50x200 78 / 81, 100x200 72 / 92, 1x40k 81 / 142; k = 16: 1x20k 114 / 116,
//                     12x5k 134 / 191; k = 32: 1x20k 178 / 144, 60x1k 219 / 229, 1x1M 2625 / 2954
//                     k = 64: 300x200 430 / 368, 1x1M 8054 / 6454, 1300x50 164 / 263
//   kNN, float:       k = 8: 50x200 80 / 79, 6x5k 90 / 98; k = 16: 100x200 92 / 81, 60x1k 126 / 153,
//                     1x60k 196 / 169, 5x60k 465 / 636; k = 32: 300x200 153 / 154, 60x5k 784 / 712,
//                     1x1M 2760 / 2739; k = 64: 1x1M 7862 / 4566
//   both, float:      k = 10: 1x57k 124 / 190; k = 16: 50x200 101 / 87, 300x200 129 / 166, 1x60k 219 / 220
//                     k = 24: 11x8k 339 / 379, 1x4.8M (k = 20) 0.89 x; k = 32: 300x200 176 / 204,
//                     1x60k 511 / 276, 200x5k 2974 / 2617; k = 64: 1x1M 8703 / 6647
//   double:           normals k = 8: 100x200 99 / 102; k = 16: 6x5k 186 / 179, 1x60k 210 / 299; k = 30:
//                     175x94 238 / 145, 1300x50 195 / 269; k = 32: 1x1M 6598 / 4737
//                     kNN k = 16: 300x1k 728 / 800; k = 64: 1x1M 25593 / 8337
inline int64_t tree_line(int64_t p, int k, bool f64, Answer a) {
  const int64_t all = INT64_MAX;
  const bool knn = a == Answer::knn, both = a == Answer::both;
  if (p < 128) {
    if (p >= 64 && k > (f64 ? 16 : 32)) return 65536;
    return f64 && k > 8 ? 16384 : 4096;
  }
  if (k <= 4) return !knn ? 10240 : f64 ? 20480 : 12288;
  if (k <= 8) return !knn ? (f64 ? 16384 : 12288) : f64 ? 28672 : p >= 1000 ? 24576 : 10240;
  if (k <= 16) {
    if (f64) return knn ? 200000 : 40960;
    // (k = 16 fills its list, which costs packets more than 9 to 15 do)
    const bool full = k == 16 && p >= 5000;
    return knn ? (full ? 98304 : 32768) : both ? (full ? 65536 : 16384) : 20480;
  }
  if (f64 || (knn && k > 32)) return all;
  if (k > 32) return 131072;  // (above, 0.82 to 1.35 x, by the cloud)
  if (p < 1000) return knn ? 65536 : 20480;
  if (k < 32) return knn ? 131072 : 45056;
  return knn ? 524288 : both ? 131072 : 40960;
}

// Whether m queries run one warp per query in place of 32-query packets:
// beyond the packets' lists (k > 64) always, otherwise a batch too small to
// fill the GPU with packets, or too scattered to share their walks.  nv: the
// points asked, in tree order those of one tree on average.  Where queries
// have to be sorted first, packets have a floor (that, and a few hundred slow
// warps) that grows with the tree, so the line lies at m * m = c * nv.  `span`
// is the lane_span setting: 1024 is the line as measured, which moves with its
// inverse; -1: packets wherever they can, 0: warps.  us, packets / warps:
//   rows of 2M points:   k = 8: 40k 1.14 x, 70k 219 / 232; k = 16: 70k 286 / 260, 100k 292 / 374
//                        k = 32: 200k 860 / 828, 300k 1126 / 1000
//   rows of 20M points:  k = 8: 140k 572 / 448, 200k 554 / 740; k = 32: 500k 2796 / 1994
//   points of 2M:        k = 1: 100k 187 / 187, 200k 226 / 317; k = 16: 140k 348 / 351
//                        k = 32: 500k 1544 / 1341; double k = 8: 200k 707 / 584, 300k 809 / 844
//   points of 20M:       k = 1: 200k 427 / 375, 300k 494 / 535; k = 16: 300k 900 / 824, 500k 1163 / 1324
//   points of 65k:       k = 4: 65k 150 / 151; k = 16: 65k 213 / 178
inline bool by_warp(int64_t nv, int64_t m, int k, bool f64, Answer a, BatchOrder order, int span) {
  if (k > WARP_MAX_K) return false;
  if (k > KNN_MAX_K) return true;
  if (span < 0) return false;
  if (span == 0) return true;
  const double s = span / 1024.0;
  if (order == BatchOrder::tree) return m * s <= (double)tree_line(nv, k, f64, a);
  int64_t small = 65536;
  double c;
  if (k > (f64 ? 16 : 32)) {
    c = 1e9;  // (at every measured size)
  } else if (order == BatchOrder::rows) {
    if (k <= 8) small = 40960;
    c = k <= 8 ? 1500 : k <= 16 ? (f64 ? 20000 : 2500) : 40000;
  } else {
    c = k <= 8 ? (f64 ? 15000 : 3600) : k <= 16 ? (f64 ? 500000 : 8000) : 200000;
  }
  return m * s <= (double)small || (double)m * m * s * s <= c * (double)nv;
}

// Queries that a warp batch takes in the order they come.  Sorted ones share
// cached nodes, which pays for the sort only in large batches.  us, as they
// come / sorted, 20M points: rows, k = 8, 200k 740 / 736, 500k 1408 / 1328;
// points, k = 32, 500k 1669 / 1792, 1M 3254 / 3389, k = 64, 1M 5383 / 5281.
inline int warp_unsorted(BatchOrder order) { return order == BatchOrder::points ? 1 << 20 : 1 << 18; }

// Window of a packet's warm lists, in multiples of k: one more than the
// warm_mult setting where packets span over 256 tree positions and lists are
// short.  Their queries' walks share less, so candidates found before them
// save more (1M scattered queries, k = 16: 2.35 -> 2.10 ms; queries in tree
// order: 31.8 -> 32.7).  A setting of 1 is the k-position start everywhere.
inline int warm_window(int mult, int64_t nv, int64_t m, int kmax) {
  return mult + (mult > 1 && kmax <= 16 && 32 * nv > 256 * m ? 1 : 0);
}

}  // namespace pptkg
