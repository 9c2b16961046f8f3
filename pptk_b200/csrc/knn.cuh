// k-d tree traversals for kNN and r-near queries.
//
// kNN: a warp carries a packet of 32 queries that are close in tree order
// (queries are sorted by the tree position of the point or of the bucket they
// fall in), or answers one query with all its lanes; both walk the wide
// hierarchy, a node's children one per lane.  r-near packets walk the binary
// hierarchy: each node is one broadcast load, the two children are tested per
// lane, and leaf buckets are staged in shared memory with one coalesced 16 B
// load per lane and read back as broadcasts.
//
// Distances follow the reference exactly (kdtree-impl.h:331-339): per-axis
// (point - query) in the distance type, squared, summed in axis order, each
// operation rounded separately.  Box distances use the same operations, so a
// box's nearest distance never exceeds the distance of a point inside it and
// pruning can never drop an answer.
#pragma once

#include "tree.cuh"

namespace pptkg {

// ------------------------------------------------------------- distances --
template <typename T, typename DistT, int D>
__device__ __forceinline__ DistT point_dist2(const T* p, const DistT* q) {
  DistT s = xmul(xsub((DistT)p[0], q[0]), xsub((DistT)p[0], q[0]));
#pragma unroll
  for (int d = 1; d < D; d++) {
    DistT t = xsub((DistT)p[d], q[d]);
    s = xadd(s, xmul(t, t));
  }
  return s;
}

template <typename T, typename DistT, int D>
__device__ __forceinline__ DistT box_min_dist2(const T* lo, const T* hi, const DistT* q) {
  DistT s = (DistT)0;
#pragma unroll
  for (int d = 0; d < D; d++) {
    DistT a = xsub((DistT)lo[d], q[d]);
    DistT c = xsub((DistT)hi[d], q[d]);
    DistT v = a > (DistT)0 ? xmul(a, a) : (c < (DistT)0 ? xmul(c, c) : (DistT)0);
    s = xadd(s, v);
  }
  return s;
}

template <typename T, typename DistT, int D>
__device__ __forceinline__ DistT box_max_dist2(const T* lo, const T* hi, const DistT* q) {
  DistT s = (DistT)0;
#pragma unroll
  for (int d = 0; d < D; d++) {
    DistT a = xsub((DistT)lo[d], q[d]);
    DistT c = xsub((DistT)hi[d], q[d]);
    a = xmul(a, a);
    c = xmul(c, c);
    s = xadd(s, a > c ? a : c);
  }
  return s;
}

// ---------------------------------------------------------------- top-k ---
// The k best (dist2, point id) pairs, held in registers in descending order
// so that the current k-th best is always slot 0.  The id is the point's
// original index, so among equal distances the smaller index wins -- both
// for the order of a result and for which point takes the k-th slot.  (The
// reference keeps whichever equal-distance candidate its std::priority_queue
// happens to retain, kdtree-impl.h:360-373, 894-899; an index order makes the
// answer a function of the input alone.)  KMAX is the compile time capacity;
// for a run-time k < KMAX the slots [k, KMAX) hold entries that compare below
// every candidate and never move.
template <int KMAX, typename DistT>
struct TopK;

// Sort of N 64-bit keys held in registers (fully unrolled), into descending
// (desc = true) or ascending order: Batcher's odd-even merge exchange (Knuth,
// The Art of Computer Programming, vol. 3, algorithm 5.2.2M), 63 exchanges
// for 16 keys and 191 for 32, against 80 and 240 of a bitonic network (kNN k = 32 of 20M points:
// 56.5 -> 54.4 ms; k = 16 within the noise).
template <int N, int P = 1, int K = P>
__device__ __forceinline__ void network_sort(unsigned long long (&a)[N], bool desc) {
#pragma unroll
  for (int c = 0; c < N - K; c++) {
    // c = i + j of the algorithm: blocks of K out of every 2K, from K mod P on
    const int from = K % P;
    if (c < from || ((c - from) / K) % 2 || c / (2 * P) != (c + K) / (2 * P)) continue;
    const unsigned long long x = a[c], y = a[c + K];
    const bool sw = desc ? x < y : y < x;
    a[c] = sw ? y : x;
    a[c + K] = sw ? x : y;
  }
  if constexpr (K > 1)
    network_sort<N, P, K / 2>(a, desc);
  else if constexpr (2 * P < N)
    network_sort<N, 2 * P, 2 * P>(a, desc);
}

// float distances: (dist2 bits << 32 | id) packed into one 64-bit key;
// non-negative floats order like their bit patterns.
template <int KMAX>
struct TopK<KMAX, float> {
  static constexpr int CAP = KMAX;
  unsigned long long s[KMAX];
  unsigned long long lim;
  __device__ __forceinline__ void reset(int k, float r2) {
    lim = (unsigned long long)__float_as_uint(r2) << 32;
#pragma unroll
    for (int j = 0; j < KMAX; j++) s[j] = j < k ? lim : 0ull;
  }
  __device__ __forceinline__ float worst() const { return __uint_as_float((unsigned)(s[0] >> 32)); }
  __device__ __forceinline__ void offer(float d2, int id) {
    unsigned long long c = ((unsigned long long)__float_as_uint(d2) << 32) | (unsigned)id;
    if (c < s[0]) insert(c);
  }
  __device__ __forceinline__ void insert(unsigned long long c) {
#pragma unroll
    for (int j = 0; j < KMAX - 1; j++) {
      unsigned long long nx = s[j + 1];
      s[j] = nx > c ? nx : (s[j] > c ? c : s[j]);
    }
    s[KMAX - 1] = s[KMAX - 1] > c ? c : s[KMAX - 1];
  }
  // Lowers the bound of the k live slots to b, inclusively (distances equal
  // to b still enter): live keys above the seed key become the seed key,
  // which sorts after every real key of distance b, so the list stays
  // sorted.  Only valid when at least k real candidates with distance <= b
  // are in the list or will be offered, so that every seed key is pushed out
  // by the end of the search.
  __device__ __forceinline__ void seed(int k, float b, float) {
    const unsigned long long key = ((unsigned long long)__float_as_uint(b) << 32) | 0xffffffffull;
    if (!(b >= 0.f) || key >= lim) return;
#pragma unroll
    for (int j = 0; j < KMAX; j++)
      if (j < k && s[j] > key) s[j] = key;
  }
  __device__ __forceinline__ bool valid(int j) const { return s[j] < lim && (unsigned)s[j] != 0xffffffffu; }
  __device__ __forceinline__ int id(int j) const { return (int)(unsigned)(s[j] & 0xffffffffull); }
  // Slot j sorts before the key (0, id0) of a point at distance 0.
  __device__ __forceinline__ bool below_zero(int j, int id0) const {
    return s[j] < (unsigned long long)(unsigned)id0;
  }
  __device__ __forceinline__ float dist(int j) const { return __uint_as_float((unsigned)(s[j] >> 32)); }
  // Warm start (see warm_topk): slot j holds a real candidate, an empty
  // live slot (no candidate yet) or a dead slot (beyond k); sort_desc()
  // then restores the list order.
  __device__ __forceinline__ void set_real(int j, float d2, int id) {
    s[j] = ((unsigned long long)__float_as_uint(d2) << 32) | (unsigned)id;
  }
  __device__ __forceinline__ void set_empty(int j) { s[j] = lim; }
  __device__ __forceinline__ void set_dead(int j) { s[j] = 0ull; }
  __device__ __forceinline__ void sort_desc() { network_sort<KMAX>(s, true); }
  // The KMAX smallest of this list (sorted descending) and t (Q <= KMAX
  // keys sorted ascending, read as padded with keys above every list key),
  // sorted descending: the element-wise minimum of the two is a bitonic
  // sequence holding them, and a bitonic merge sorts it.
  template <int Q>
  __device__ __forceinline__ void merge_smallest(const unsigned long long (&t)[Q]) {
    static_assert(Q <= KMAX, "merge of at most KMAX keys");
#pragma unroll
    for (int j = 0; j < Q; j++) s[j] = t[j] < s[j] ? t[j] : s[j];
#pragma unroll
    for (int stride = KMAX / 2; stride > 0; stride >>= 1)
#pragma unroll
      for (int i = 0; i < KMAX; i++) {
        const int j = i ^ stride;
        if (j > i) {
          const unsigned long long x = s[i], y = s[j];
          const bool sw = x < y;
          s[i] = sw ? y : x;
          s[j] = sw ? x : y;
        }
      }
  }
  __device__ __forceinline__ unsigned long long key_real(float d2, int id) const {
    return ((unsigned long long)__float_as_uint(d2) << 32) | (unsigned)id;
  }
  __device__ __forceinline__ unsigned long long key_empty() const { return lim; }
};

// double distances: parallel (dist2, id) arrays compared lexicographically.
template <int KMAX>
struct TopK<KMAX, double> {
  static constexpr int CAP = KMAX;
  double d[KMAX];
  int p[KMAX];
  double lim_d;
  __device__ __forceinline__ void reset(int k, double r2) {
    lim_d = r2;
#pragma unroll
    for (int j = 0; j < KMAX; j++) {
      d[j] = j < k ? r2 : -1.0;
      p[j] = -1;
    }
  }
  __device__ __forceinline__ double worst() const { return d[0]; }
  __device__ __forceinline__ static bool gt(double da, int pa, double db, int pb) {
    return da > db || (da == db && pa > pb);
  }
  __device__ __forceinline__ void offer(double d2, int id) {
    if (gt(d[0], p[0], d2, id)) insert(d2, id);
  }
  __device__ __forceinline__ void insert(double cd, int cp) {
#pragma unroll
    for (int j = 0; j < KMAX - 1; j++) {
      const bool nx = gt(d[j + 1], p[j + 1], cd, cp);
      const bool cur = gt(d[j], p[j], cd, cp);
      d[j] = nx ? d[j + 1] : (cur ? cd : d[j]);
      p[j] = nx ? p[j + 1] : (cur ? cp : p[j]);
    }
    if (gt(d[KMAX - 1], p[KMAX - 1], cd, cp)) {
      d[KMAX - 1] = cd;
      p[KMAX - 1] = cp;
    }
  }
  // As TopK<KMAX, float>::seed; r2 is the bound the slots were reset to.
  __device__ __forceinline__ void seed(int k, double b, double r2) {
    if (!(b >= 0.0) || !(b < r2)) return;
#pragma unroll
    for (int j = 0; j < KMAX; j++)
      if (j < k && gt(d[j], p[j], b, 0x7fffffff)) {
        d[j] = b;
        p[j] = 0x7fffffff;
      }
  }
  __device__ __forceinline__ bool valid(int j) const { return p[j] >= 0 && p[j] != 0x7fffffff && d[j] >= 0.0; }
  __device__ __forceinline__ int id(int j) const { return p[j]; }
  __device__ __forceinline__ bool below_zero(int j, int id0) const { return d[j] == 0.0 && p[j] < id0; }
  __device__ __forceinline__ double dist(int j) const { return d[j]; }
  __device__ __forceinline__ void set_real(int j, double d2, int id) {
    d[j] = d2;
    p[j] = id;
  }
  __device__ __forceinline__ void set_empty(int j) {
    d[j] = lim_d;
    p[j] = -1;
  }
  __device__ __forceinline__ void set_dead(int j) {
    d[j] = -1.0;
    p[j] = -1;
  }
  __device__ __forceinline__ void sort_desc() {
#pragma unroll
    for (int size = 2; size <= KMAX; size <<= 1)
#pragma unroll
      for (int stride = size / 2; stride > 0; stride >>= 1)
#pragma unroll
        for (int i = 0; i < KMAX; i++) {
          const int j = i ^ stride;
          if (j > i) {
            const double da = d[i], db = d[j];
            const int pa = p[i], pb = p[j];
            const bool up = (i & size) != 0;
            const bool sw = up ? gt(da, pa, db, pb) : gt(db, pb, da, pa);
            d[i] = sw ? db : da;
            d[j] = sw ? da : db;
            p[i] = sw ? pb : pa;
            p[j] = sw ? pa : pb;
          }
        }
  }
};

// ----------------------------------------------------- packet traversal --
// Per-warp shared memory: the traversal stack and one leaf staging buffer.
template <typename T, int D>
struct WarpScratch {
  int* stack;
  PointRec<T, D>* buf;                   // 32 entries (r-near staging)
  int* log;                              // per-lane neighbour lists, lane-strided; null when unused
  WNode<T, D>* nodes;                    // the 32 nodes of a step (kNN)
  typename DistOf<T>::type* box;         // the packet's two boxes: [2][lo, hi][D] (kNN)
};

// A lane's query as the rest of its warp reads it during a bucket scan:
// the coordinates and the entry bound (a candidate enters the list iff its
// dist2 <= thr).
template <typename DistT, int D>
struct alignas(16) QStage {
  DistT q[D];
  DistT thr;
};

// The largest value below r2 (r2 > 0), -1 for r2 <= 0, so that for every
// distance d2 >= 0: d2 < r2  <=>  d2 <= below(r2).
__device__ __forceinline__ float below(float r2) {
  if (!(r2 > 0.f)) return -1.f;
  return __uint_as_float(__float_as_uint(r2) - 1u);  // +inf -> FLT_MAX
}
__device__ __forceinline__ double below(double r2) {
  if (!(r2 > 0.0)) return -1.0;
  return __longlong_as_double(__double_as_longlong(r2) - 1ll);  // +inf -> DBL_MAX
}

// Entry bound of a list whose k-th distance is `worst` (worst <= r2 always):
// d2 <= entry_bound  <=>  d2 <= worst && d2 < r2.
template <typename DistT>
__device__ __forceinline__ DistT entry_bound(DistT worst, DistT r2_below) {
  return worst < r2_below ? worst : r2_below;
}

template <typename T, int D>
__device__ __forceinline__ TNode<T, D> load_node(const TNode<T, D>* nodes, int i) {
  static_assert(sizeof(TNode<T, D>) % 16 == 0, "TNode must be a multiple of 16 bytes");
  TNode<T, D> n;
  const float4* src = reinterpret_cast<const float4*>(nodes + i);
  float4* dst = reinterpret_cast<float4*>(&n);
#pragma unroll
  for (int j = 0; j < (int)(sizeof(TNode<T, D>) / 16); j++) dst[j] = __ldg(src + j);
  return n;
}

// Bits [a, a + n) of a 32-bit chunk mask (clipped to the chunk; 0 if empty).
__device__ __forceinline__ unsigned window_bits(int a, int n) {
  const int lo = max(a, 0), hi = min(a + n, 32);
  if (hi <= lo) return 0u;
  const unsigned top = hi >= 32 ? 0xffffffffu : ((1u << hi) - 1u);
  return top & ~((1u << lo) - 1u);
}

// Lower bound, in float, of the squared distance between a box and any query
// of the packet whose coordinates lie in [plo, phi]: per axis the rounded
// operations of box_min_dist2 at the nearest packet coordinate, which are
// monotone, so no query of the packet is nearer to the box.
template <typename T, typename DistT, int D>
__device__ __forceinline__ float packet_min_dist2(const T* lo, const T* hi, const DistT* plo, const DistT* phi) {
  DistT s = (DistT)0;
#pragma unroll
  for (int d = 0; d < D; d++) {
    const DistT a = xsub((DistT)lo[d], phi[d]);
    const DistT c = xsub((DistT)hi[d], plo[d]);
    const DistT v = a > (DistT)0 ? xmul(a, a) : (c < (DistT)0 ? xmul(c, c) : (DistT)0);
    s = xadd(s, v);
  }
  if constexpr (std::is_same<DistT, float>::value)
    return s;
  else
    return __double2float_rd(s);
}

__device__ __forceinline__ float float_above(float x) { return x; }
__device__ __forceinline__ float float_above(double x) { return __double2float_ru(x); }

template <typename V>
__device__ __forceinline__ V lanes_min(V v) {
  if constexpr (std::is_same<V, float>::value) {
    return from_ord(__reduce_min_sync(0xffffffffu, ord_of(v)));
  } else {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
  }
}
template <typename V>
__device__ __forceinline__ V lanes_max(V v) {
  if constexpr (std::is_same<V, float>::value) {
    return from_ord(__reduce_max_sync(0xffffffffu, ord_of(v)));
  } else {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
  }
}

// Lanes with a candidate to insert that make an insertion of the whole warp
// worth while (wide_knn).  All-point normals / kNN k = 32 of the 20M-point
// scene: 38.5 / 60.8 ms at 6 lanes, 37.1 / 56.5 at 12, 36.5 / 56.5 at 18,
// against 40.5 / 68.0 when every chunk's marks are inserted at once.
constexpr int DRAIN_LANES = 16;

// Exact kNN of the lane's query over the points below node `root` of the
// wide hierarchy (-1: none), ties in dist2 broken by point id, with the top-k
// list in the lane's registers.  `own` (tree position or -1) is skipped,
// which is how self queries exclude the query point itself; so are the tree
// positions [wlo, wlo + wn), the warm-start window whose candidates the list
// holds.
//
// The leaf ranges around the queries' anchors come first, so the bounds are
// close to final before the walk starts at the top.  A step of it takes one
// node: the children arrive one per lane, and each is tested against the
// boxes of the packet's queries and the packet's largest bound.  Children
// that pass are put off (inner nodes) or, nearest first, tested by every lane
// against its own query and scanned if one needs them (leaf ranges).
//
// Every leaf range that holds a candidate within a query's final bound is
// scanned: the packet test bounds every lane's own test from below.  False
// on a full stack (the host sizes it from the level count) or more steps
// than nodes (a corrupt hierarchy).
template <typename T, int D, typename Top, typename DistT>
__device__ bool wide_knn(const TreeView<T, D>& tv, int root, const DistT* q, int anchor, int own, bool active,
                         DistT r2, Top& top, WarpScratch<T, D> ws, int wlo = 0, int wn = 0) {
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  const unsigned lt = (1u << lane) - 1u;
  // (a query with a NaN coordinate has no neighbours)
#pragma unroll
  for (int d = 0; d < D; d++) active = active && q[d] == q[d];
  if (root < 0 || !__any_sync(FULL, active)) return true;
  auto need = [&](DistT md) { return active && md < r2 && md <= top.worst(); };
  // Leaf range scan, transposed: lane j holds candidate j of the chunk (one
  // coalesced load), and the warp loops only over the lanes whose query needs
  // this range.  For such a query i every lane computes its candidate's
  // distance to q_i, and the ballot of candidates that can enter list i
  // becomes lane i's mark mask.  The queries sit in the warp's staging buffer
  // so that lane i's coordinates and bound arrive as one shared broadcast.
  //
  // Marked candidates do not enter the lists at once: a third of the lanes
  // need a chunk, each has a few marks, and a list insertion costs the warp as
  // much for one lane as for 32.  A lane keeps the marks of up to two chunks,
  // and an insertion runs once DRAIN_LANES lanes have one to make (or one
  // lane's third chunk needs room).  Bounds that lag by a few candidates only
  // cost some marks that the insertion then rejects.
  QStage<DistT, D>* qst = reinterpret_cast<QStage<DistT, D>*>(ws.buf);
  const DistT r2_below = below(r2);
#pragma unroll
  for (int d = 0; d < D; d++) qst[lane].q[d] = q[d];
  unsigned mark0 = 0, mark1 = 0;  // marks held back, and the chunks they belong to
  int base0 = 0, base1 = 0;
  // one held-back candidate of every lane that has one enters its list
  auto take = [&]() {
    if (mark0) {
      const int t = __ffs(mark0) - 1;
      mark0 &= mark0 - 1;
      const PointRec<T, D> r = tv.pt(base0 + t);
      top.offer(point_dist2<T, DistT, D>(r.c, q), r.id);
      if (!mark0) {
        mark0 = mark1;
        base0 = base1;
        mark1 = 0;
      }
    }
  };
  auto scan = [&](int begin, int count, bool mine) {
    const unsigned needm = __ballot_sync(FULL, mine);
    for (int base = begin; base < begin + count; base += 32) {
      const int nb = min(32, begin + count - base);
      T c[D];
      if (lane < nb) {
        const PointRec<T, D> pr = tv.pt(base + lane);
#pragma unroll
        for (int d = 0; d < D; d++) c[d] = pr.c[d];
      } else {
#pragma unroll
        for (int d = 0; d < D; d++) c[d] = (T)0;
      }
      // each needing lane publishes its entry bound for this chunk; the
      // loop below reads a query and its bound as one broadcast
      __syncwarp();
      qst[lane].thr = entry_bound(top.worst(), r2_below);
      __syncwarp();
      unsigned mark = 0;
      unsigned rem = needm;
      while (rem) {
        const int i = __ffs(rem) - 1;
        rem &= rem - 1;
        const QStage<DistT, D> qi = qst[i];
        const unsigned m = __ballot_sync(FULL, point_dist2<T, DistT, D>(c, qi.q) <= qi.thr);
        if (lane == i) mark = m;
      }
      if (nb < 32) mark &= (1u << nb) - 1u;
      // the query's own point never enters its list, and the positions of
      // its warm-start window are in it already
      if (own >= base && own < base + nb) mark &= ~(1u << (own - base));
      mark &= ~window_bits(wlo - base, wn);
      // (the loop ends: every pass takes a mark of each lane that has one)
      while (__any_sync(FULL, mark && mark1) || __popc(__ballot_sync(FULL, mark0 != 0)) >= DRAIN_LANES) take();
      if (mark0) {
        if (mark) {
          mark1 = mark;
          base1 = base;
        }
      } else {
        mark0 = mark;
        base0 = base;
      }
    }
  };
  // The packet's queries in two boxes, cut where the distance from one lane's
  // query to the next is largest.  Queries next to each other in tree order
  // straddle at most one boundary of a node much larger than the packet, and
  // one box over both of its sides would reach most of that node.
  float jump = 0.f;
  {
    DistT s = (DistT)0;
    bool both = lane > 0 && active;
#pragma unroll
    for (int d = 0; d < D; d++) {
      const DistT e = q[d] - __shfl_up_sync(FULL, q[d], 1);
      s += e * e;
    }
    both = __shfl_up_sync(FULL, (int)active, 1) && both;
    if (both) jump = (float)s;
  }
  const unsigned far = __reduce_max_sync(FULL, jump > 0.f ? __float_as_uint(jump) : 0u);
  const int cut = far ? __ffs(__ballot_sync(FULL, jump > 0.f && __float_as_uint(jump) == far)) - 1 : 32;
  // (in shared memory: a step reads them as broadcasts, and the lists need
  // the registers)
#pragma unroll
  for (int b = 0; b < 2; b++) {
    const bool in = active && (lane >= cut) == (b == 1);
#pragma unroll
    for (int d = 0; d < D; d++) {
      const DistT lo = lanes_min(in ? q[d] : (DistT)INFINITY), hi = lanes_max(in ? q[d] : (DistT)-INFINITY);
      if (lane == 0) {
        ws.box[2 * D * b + d] = lo;
        ws.box[2 * D * b + D + d] = hi;
      }
    }
  }
  __syncwarp();
  auto reach = [&]() {
    const DistT w = top.worst() < r2 ? top.worst() : r2;
    return __reduce_max_sync(FULL, active && w >= (DistT)0 ? __float_as_uint(float_above(w)) : 0u);
  };
  unsigned rmax = reach();
  // the leaf ranges around the queries come first
  const int home = active && anchor >= 0 ? tv.wide_of(0, min(anchor, tv.pts_cap - 1)) : -1;
  int h0 = (int)__reduce_min_sync(FULL, home >= 0 ? (unsigned)home : 0x7fffffffu);
  int h1 = min(__reduce_max_sync(FULL, home) + 1, tv.n_wide);
  if (h1 - h0 > 32 || h1 < h0) h0 = h1 = 0;
  int2* stk = reinterpret_cast<int2*>(ws.stack);
  int sp = 0, steps = 0;
  bool started = false;
  int at = h0, cnt = h1 - h0;  // nodes of this step, one per lane
  WNode<T, D> w;
  if (lane < cnt) w = tv.wnode(at + lane);
  while (true) {
    if (++steps > tv.n_wide + 1) return false;
    bool hit = lane < cnt && w.cnt != 0;
    unsigned md = 0;
    if (hit && started) {
      md = __float_as_uint(fminf(packet_min_dist2<T, DistT, D>(w.lo, w.hi, ws.box, ws.box + D),
                                 packet_min_dist2<T, DistT, D>(w.lo, w.hi, ws.box + 2 * D, ws.box + 3 * D)));
      hit = md <= rmax && !(at + lane >= h0 && at + lane < h1);
    }
    unsigned hm = __ballot_sync(FULL, hit);
    if (hm) {
      if (__any_sync(FULL, hit && w.cnt > 0)) {
        // leaf ranges, nearest first, until none is within reach
        __syncwarp();
        if (hit) ws.nodes[lane] = w;
        __syncwarp();
        do {
          const unsigned near = __reduce_min_sync(FULL, hit ? md : 0xffffffffu);
          if (near > rmax) break;
          const int s = __ffs(__ballot_sync(FULL, hit && md == near)) - 1;
          if (lane == s) hit = false;
          hm &= ~(1u << s);
          const WNode<T, D> leaf = ws.nodes[s];
          const bool mine = need(box_min_dist2<T, DistT, D>(leaf.lo, leaf.hi, q));
          if (__any_sync(FULL, mine)) {
            scan(leaf.begin, leaf.cnt, mine);
            rmax = reach();
          }
        } while (hm);
      } else {
        // inner nodes are put off, the nearest on top
        const int n = __popc(hm);
        if (sp + n > tv.wstack) return false;
        const unsigned near = __reduce_min_sync(FULL, hit ? md : 0xffffffffu);
        const int s = __ffs(__ballot_sync(FULL, hit && md == near)) - 1;
        const int r = lane == s ? n - 1 : __popc(hm & lt) - (s < lane ? 1 : 0);
        if (hit) stk[sp + r] = make_int2(at + lane, (int)md);
        sp += n;
        __syncwarp();
      }
    }
    // the next step: the root's children first, then those of a node put
    // off that a query still needs, or the rest of a node's children
    int node = root, from = 0;
    bool found = !started;
    while (!found && sp > 0) {
      const int2 e = stk[--sp];
      node = e.x;
      if (node < 0) {
        node = ~node;
        from = e.y;
      } else if ((unsigned)e.y > rmax) {
        continue;
      }
      found = true;
      const WNode<T, D> up = tv.wnode(node);
      // (its first children are on their way while its own box is tested)
      at = up.begin + from;
      cnt = -up.cnt - from;
      if (lane < cnt) w = tv.wnode(at + lane);
      if (from == 0 && !__any_sync(FULL, need(box_min_dist2<T, DistT, D>(up.lo, up.hi, q)))) found = false;
    }
    __syncwarp();
    if (!found) break;
    if (!started) {
      started = true;
      const WNode<T, D> up = tv.wnode(root);
      if (up.cnt >= 0) {  // the tree is one leaf range
        at = root;
        cnt = 1;
      } else {
        at = up.begin;
        cnt = -up.cnt;
      }
      if (lane < cnt) w = tv.wnode(at + lane);
    }
    if (cnt > 32) {
      if (sp >= tv.wstack) return false;
      if (lane == 0) stk[sp] = make_int2(~node, from + 32);
      sp++;
      __syncwarp();
      cnt = 32;
    }
  }
  while (__any_sync(FULL, mark0 != 0)) take();
  return true;
}

// ------------------------------------------------- one warp per query ----
// A (distance, point id) pair as one sortable value, ordered like the lists
// above, and the warp operations on it.
template <typename DistT>
struct WarpKey;

template <>
struct WarpKey<float> {
  unsigned long long v;  // dist2 bits << 32 | id
  static __device__ __forceinline__ WarpKey make(float d2, int id) {
    return {((unsigned long long)__float_as_uint(d2) << 32) | (unsigned)id};
  }
  static __device__ __forceinline__ WarpKey none(float r2) { return {(unsigned long long)__float_as_uint(r2) << 32}; }
  __device__ __forceinline__ bool operator<(const WarpKey& o) const { return v < o.v; }
  __device__ __forceinline__ float dist() const { return __uint_as_float((unsigned)(v >> 32)); }
  __device__ __forceinline__ int id() const { return (int)(unsigned)v; }
  __device__ __forceinline__ WarpKey from(int lane) const { return {__shfl_sync(0xffffffffu, v, lane)}; }
  __device__ __forceinline__ WarpKey below() const { return {__shfl_up_sync(0xffffffffu, v, 1)}; }
  __device__ __forceinline__ WarpKey across(int mask) const { return {__shfl_xor_sync(0xffffffffu, v, mask)}; }
};

template <>
struct WarpKey<double> {
  double d;
  int i;
  static __device__ __forceinline__ WarpKey make(double d2, int id) { return {d2, id}; }
  static __device__ __forceinline__ WarpKey none(double r2) { return {r2, -1}; }
  __device__ __forceinline__ bool operator<(const WarpKey& o) const { return d < o.d || (d == o.d && i < o.i); }
  __device__ __forceinline__ double dist() const { return d; }
  __device__ __forceinline__ int id() const { return i; }
  __device__ __forceinline__ WarpKey from(int lane) const {
    return {__shfl_sync(0xffffffffu, d, lane), __shfl_sync(0xffffffffu, i, lane)};
  }
  __device__ __forceinline__ WarpKey below() const {
    return {__shfl_up_sync(0xffffffffu, d, 1), __shfl_up_sync(0xffffffffu, i, 1)};
  }
  __device__ __forceinline__ WarpKey across(int mask) const {
    return {__shfl_xor_sync(0xffffffffu, d, mask), __shfl_xor_sync(0xffffffffu, i, mask)};
  }
};

// The k <= 32 S smallest keys of one query, spread over the warp: element
// 32 s + lane, ascending, in the lane's slot s.
template <int S, typename DistT>
struct WarpList {
  typedef WarpKey<DistT> Key;
  Key a[S];
  Key limit;  // element k - 1: what a candidate has to beat
  int k;
  __device__ __forceinline__ void reset(int k_, DistT r2) {
    k = k_;
    limit = Key::none(r2);
#pragma unroll
    for (int s = 0; s < S; s++) a[s] = limit;
  }
  __device__ __forceinline__ void tighten() {
#pragma unroll
    for (int s = 0; s < S; s++)
      if (s == (k - 1) >> 5) limit = a[s].from((k - 1) & 31);
  }
  // c (the same in every lane) takes its place; larger elements move up.
  __device__ __forceinline__ void insert(Key c) {
    const int lane = threadIdx.x & 31;
    int r = 0;
#pragma unroll
    for (int s = 0; s < S; s++) r += __popc(__ballot_sync(0xffffffffu, a[s] < c));
#pragma unroll
    for (int s = S - 1; s >= 0; s--) {
      Key up = a[s].below();
      if (s > 0) {
        const Key last = a[s > 0 ? s - 1 : 0].from(31);
        if (lane == 0) up = last;
      }
      const int e = 32 * s + lane;
      if (e == r)
        a[s] = c;
      else if (e > r)
        a[s] = up;
    }
    tighten();
  }
  static __device__ __forceinline__ void exchange(Key& x, int mask, bool low) {
    const Key y = x.across(mask);
    if ((y < x) == low) x = y;
  }
  // A key per lane, as many of them as not real: sorted across the warp
  // (bitonic, 15 exchanges), then merged through the slots.
  __device__ __forceinline__ void merge(Key c) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
      for (int m = size >> 1; m > 0; m >>= 1) exchange(c, m, ((lane & size) == 0 || size == 32) == ((lane & m) == 0));
#pragma unroll
    for (int s = 0; s < S; s++) {
      // a[s] ascending against c descending: the smaller of each pair are the
      // 32 smallest of both, in a bitonic order that five exchanges sort
      const Key d = c.across(31);
      const bool sw = d < a[s];
      c = sw ? a[s] : d;
      a[s] = sw ? d : a[s];
#pragma unroll
      for (int m = 16; m > 0; m >>= 1) {
        exchange(a[s], m, (lane & m) == 0);
        if (s + 1 < S) exchange(c, m, (lane & m) == 0);
      }
    }
    tighten();
  }
};

// Exact kNN of one query (q, the same in every lane) by a whole warp, over
// the points below node `root` of the wide hierarchy: the children of a node
// are tested one per lane against the query itself, the nearest first, and a
// leaf range's points one per lane.  `home` (a leaf range, or -1) is scanned
// first; `own` is skipped.  For batches whose packets would be too few to
// fill the GPU or whose queries lie too far apart to share a walk.
template <int S, typename T, int D, typename DistT>
__device__ __forceinline__ bool warp_knn(const TreeView<T, D>& tv, int root, const DistT* q, int home, int own,
                                         DistT r2, WarpList<S, DistT>& top, int2* stk) {
  typedef WarpKey<DistT> Key;
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  const unsigned lt = (1u << lane) - 1u;
  auto reach = [&]() { return __float_as_uint(float_above(top.limit.dist())); };
  unsigned rmax = r2 > (DistT)0 ? reach() : 0u;
  int sp = 0, steps = 0;
  bool started = home < 0;
  int at = started ? root : home, cnt = 1;
  WNode<T, D> w;
  if (lane < cnt) w = tv.wnode(at + lane);
  while (true) {
    if (++steps > tv.n_wide + 1) return false;
    bool hit = lane < cnt && w.cnt != 0 && !(started && at + lane == home);
    unsigned md = 0;
    if (hit) {
      const DistT b = box_min_dist2<T, DistT, D>(w.lo, w.hi, q);
      if constexpr (std::is_same<DistT, float>::value)
        md = __float_as_uint(b);
      else
        md = __float_as_uint(__double2float_rd(b));
      hit = md <= rmax;
    }
    unsigned hm = __ballot_sync(FULL, hit);
    if (hm) {
      if (__any_sync(FULL, hit && w.cnt > 0)) {
        do {
          const unsigned near = __reduce_min_sync(FULL, hit ? md : 0xffffffffu);
          if (near > rmax) break;
          const int s = __ffs(__ballot_sync(FULL, hit && md == near)) - 1;
          if (lane == s) hit = false;
          hm &= ~(1u << s);
          const int begin = __shfl_sync(FULL, w.begin, s), end = begin + __shfl_sync(FULL, w.cnt, s);
          for (int base = begin; base < end; base += 32) {
            const int p = base + lane;
            Key c = Key::none(r2);
            bool in = false;
            if (p < end) {
              const PointRec<T, D> pr = tv.pt(p);
              const DistT d2 = point_dist2<T, DistT, D>(pr.c, q);
              in = d2 < r2 && p != own;
              if (in) c = Key::make(d2, pr.id);
              in = in && c < top.limit;
            }
            unsigned mark = __ballot_sync(FULL, in);
            // a merge costs as much as a dozen insertions
            if (__popc(mark) > 12) {
              top.merge(in ? c : Key::none(r2));
            } else {
              while (mark) {
                const Key x = c.from(__ffs(mark) - 1);
                mark &= mark - 1;
                if (x < top.limit) top.insert(x);
              }
            }
          }
          rmax = reach();
        } while (hm);
      } else {
        const int n = __popc(hm);
        if (sp + n > tv.wstack) return false;
        const unsigned near = __reduce_min_sync(FULL, hit ? md : 0xffffffffu);
        const int s = __ffs(__ballot_sync(FULL, hit && md == near)) - 1;
        const int r = lane == s ? n - 1 : __popc(hm & lt) - (s < lane ? 1 : 0);
        if (hit) stk[sp + r] = make_int2(at + lane, (int)md);
        sp += n;
        __syncwarp();
      }
    }
    if (!started) {
      started = true;
      at = root;
      cnt = 1;
      if (lane == 0) w = tv.wnode(root);
      continue;
    }
    // the topmost entry still within reach (32 are looked at together)
    int node = -1, from = 0;
    while (sp > 0) {
      const int2 e = lane < sp ? stk[sp - 1 - lane] : make_int2(0, -1);
      const unsigned ok = __ballot_sync(FULL, lane < sp && (e.x < 0 || (unsigned)e.y <= rmax));
      if (!ok) {
        sp -= min(sp, 32);
        continue;
      }
      const int s = __ffs(ok) - 1;
      sp -= s + 1;
      node = __shfl_sync(FULL, e.x, s);
      if (node < 0) {
        node = ~node;
        from = __shfl_sync(FULL, e.y, s);
      }
      break;
    }
    __syncwarp();
    if (node < 0) break;
    at = tv.wnode(node).begin + from;
    cnt = -tv.wnode(node).cnt - from;
    if (cnt > 32) {
      if (sp >= tv.wstack) return false;
      if (lane == 0) stk[sp] = make_int2(~node, from + 32);
      sp++;
      __syncwarp();
      cnt = 32;
    }
    if (lane < cnt) w = tv.wnode(at + lane);
  }
  return true;
}

// Per-lane traversal for lists in device memory (k > 256).  Each lane walks
// its own near-first depth-first path of the binary hierarchy with a private
// stack of deferred children (reference, size and box distance, re-tested on
// pop), so the 32 walks advance side by side and their node loads overlap.
// Every point whose distance is within the query's final bound is offered.
// Requires tv.depth <= LSTACK (the caller checks); false on a corrupt tree.
template <int LSTACK, typename T, int D, typename DistT, typename Top>
__device__ bool lane_knn(const TreeView<T, D>& tv, const DistT* q, int own, bool active, DistT r2, Top& top) {
  if (!active) return true;
  int sref[LSTACK], scnt[LSTACK];
  DistT smd[LSTACK];
  int sp = 0;
  auto need = [&](DistT md) { return md < r2 && md <= top.worst(); };
  // a bucket is read four points at a time so that the loads overlap; the
  // offers then go in position order against the current bound, as one by one
  auto scan = [&](int begin, int count) {
    const int end = begin + count;
    int p = begin;
    for (; p + 4 <= end; p += 4) {
      PointRec<T, D> r[4];
      DistT d2[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        r[j] = tv.pt(p + j);
        d2[j] = point_dist2<T, DistT, D>(r[j].c, q);
      }
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (d2[j] <= top.worst() && d2[j] < r2 && p + j != own)
          top.offer(d2[j], r[j].id);
    }
    for (; p < end; p++) {
      const PointRec<T, D> r = tv.pt(p);
      const DistT d2 = point_dist2<T, DistT, D>(r.c, q);
      if (d2 <= top.worst() && d2 < r2 && p != own) top.offer(d2, r.id);
    }
  };
  int cur = tv.root, visits = 0;
  while (true) {
    if (++visits > tv.n_nodes) return false;  // a tree is acyclic: more visits mean a corrupt node array
    const TNode<T, D> nd = load_node(tv.nodes, tv.node_index(cur));
    const DistT md0 = nd.cnt[0] > 0 ? box_min_dist2<T, DistT, D>(nd.lo[0], nd.hi[0], q) : (DistT)INFINITY;
    const DistT md1 = nd.cnt[1] > 0 ? box_min_dist2<T, DistT, D>(nd.lo[1], nd.hi[1], q) : (DistT)INFINITY;
    const bool sw = md1 < md0;
    const DistT mdn = sw ? md1 : md0, mdf = sw ? md0 : md1;
    const int refn = sw ? nd.ref[1] : nd.ref[0], reff = sw ? nd.ref[0] : nd.ref[1];
    const int cntn = sw ? nd.cnt[1] : nd.cnt[0], cntf = sw ? nd.cnt[0] : nd.cnt[1];
    int next = -1;
    // the far child is never nearer than the near one, so it is needed only
    // when the near one is
    if (need(mdn)) {
      if (refn >= 0) {
        next = refn;
        if (need(mdf)) {
          if (sp >= LSTACK) return false;
          sref[sp] = reff;
          scnt[sp] = cntf;
          smd[sp] = mdf;
          sp++;
        }
      } else {
        scan(-refn - 1, cntn);
        if (need(mdf)) {
          if (reff >= 0)
            next = reff;
          else
            scan(-reff - 1, cntf);
        }
      }
    }
    while (next < 0 && sp > 0) {
      --sp;
      if (!need(smd[sp])) continue;
      if (sref[sp] < 0)
        scan(-sref[sp] - 1, scnt[sp]);
      else
        next = sref[sp];
    }
    if (next < 0) return true;
    cur = next;
  }
}

// Top-k of any size k for the per-lane walk: a binary max-heap of
// (dist2, id) pairs in device memory, ordered like the register lists
// ((dist2, id) lexicographic), so the k kept are the same k smallest.
// Slot 0 holds the current k-th once the heap is full.
template <typename DistT>
struct HeapTop {
  DistT* d;
  int* p;
  int k, size;
  DistT r2;
  __device__ __forceinline__ static bool gt(DistT da, int pa, DistT db, int pb) {
    return da > db || (da == db && pa > pb);
  }
  __device__ __forceinline__ DistT worst() const { return size < k ? r2 : d[0]; }
  __device__ void sift_down(int i, int n) {
    const DistT di = d[i];
    const int pi = p[i];
    while (true) {
      int c = 2 * i + 1;
      if (c >= n) break;
      if (c + 1 < n && gt(d[c + 1], p[c + 1], d[c], p[c])) c++;
      if (!gt(d[c], p[c], di, pi)) break;
      d[i] = d[c];
      p[i] = p[c];
      i = c;
    }
    d[i] = di;
    p[i] = pi;
  }
  __device__ void offer(DistT d2, int id) {
    if (size < k) {
      int i = size++;
      while (i > 0) {
        const int par = (i - 1) / 2;
        if (!gt(d2, id, d[par], p[par])) break;
        d[i] = d[par];
        p[i] = p[par];
        i = par;
      }
      d[i] = d2;
      p[i] = id;
    } else if (gt(d[0], p[0], d2, id)) {
      d[0] = d2;
      p[0] = id;
      sift_down(0, size);
    }
  }
  // Sorts the kept pairs ascending in place (heap sort).
  __device__ void sort() {
    for (int e = size - 1; e > 0; e--) {
      const DistT td = d[0];
      const int tp = p[0];
      d[0] = d[e];
      p[0] = p[e];
      d[e] = td;
      p[e] = tp;
      sift_down(0, e);
    }
  }
};

// r-near over the whole tree in ascending tree position (the reference's
// left-then-right order, kdtree-impl.h:519-558).  In COUNT mode a lane whose
// ball contains a whole child box adds the child's size without distance
// tests (every point of the box is provably inside, see box_max_dist2);
// otherwise every point with dist2 < r2 is passed to emit(pos) in ascending
// position.  The own position is not excluded here: for self queries the
// caller subtracts it (it is always a hit when r2 > 0).
template <typename T, int D, typename DistT, bool COUNT, typename Emit>
__device__ bool packet_rnear(const TreeView<T, D>& tv, const DistT* q, bool active, DistT r2, WarpScratch<T, D> ws,
                             long long& count, Emit emit) {
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  int sp = 0;
  int cur = tv.root;
  bool ok = true;
  auto scan = [&](int begin, int cnt, bool mine) {
    for (int base = begin; base < begin + cnt; base += 32) {
      const int nb = min(32, begin + cnt - base);
      __syncwarp();
      if (lane < nb) ws.buf[lane] = tv.pt(base + lane);
      __syncwarp();
      if (mine) {
        for (int t = 0; t < nb; t++) {
          const PointRec<T, D> pr = ws.buf[t];
          const DistT d2 = point_dist2<T, DistT, D>(pr.c, q);
          if (d2 < r2) {
            if (COUNT)
              count++;
            else
              emit(base + t, pr);
          }
        }
      }
    }
  };
  // A lane that counted a whole inner child is muted while the warp walks
  // that child's subtree for other lanes: `mute` is the stack depth at which
  // the subtree was entered, and the lane rejoins once a pop goes below it.
  int mute = -1;
  auto live = [&]() { return active && mute < 0; };
  // Handles child c of nd; returns the node to descend into, or -1.
  auto process = [&](const TNode<T, D>& nd, int c, bool& took) -> int {
    took = false;
    if (nd.cnt[c] == 0) return -1;
    bool mine = live() && box_min_dist2<T, DistT, D>(nd.lo[c], nd.hi[c], q) < r2;
    if (COUNT && mine && box_max_dist2<T, DistT, D>(nd.lo[c], nd.hi[c], q) < r2) {
      count += nd.cnt[c];
      mine = false;
      took = true;
    }
    if (!__any_sync(FULL, mine)) return -1;
    const int ref = nd.ref[c];
    if (ref < 0) {
      scan(-ref - 1, nd.cnt[c], mine);
      return -1;
    }
    return ref;
  };
  int visits = 0;
  while (true) {
    if (++visits > tv.n_nodes) {
      ok = false;
      break;
    }
    const TNode<T, D>& nd = tv.nodes[cur];
    const bool w0 = live() && nd.cnt[0] > 0 && box_min_dist2<T, DistT, D>(nd.lo[0], nd.hi[0], q) < r2;
    const bool w1 = live() && nd.cnt[1] > 0 && box_min_dist2<T, DistT, D>(nd.lo[1], nd.hi[1], q) < r2;
    const bool a0 = __any_sync(FULL, w0), a1 = __any_sync(FULL, w1);
    int next = -1;
    bool took = false;
    if (a0) {
      next = process(nd, 0, took);
      if (next >= 0 && a1) {
        if (sp >= tv.depth) {
          ok = false;
        } else {
          __syncwarp();
          if (lane == 0) ws.stack[sp] = (cur << 1) | 1;
          sp++;
        }
      }
    }
    if (next < 0 && a1) next = process(nd, 1, took);
    if (next >= 0) {
      if (took) mute = sp;
      cur = next;
      continue;
    }
    __syncwarp();
    bool found = false;
    while (sp > 0) {
      const int e = ws.stack[--sp];
      __syncwarp();
      if (mute >= 0 && sp < mute) mute = -1;
      const int r = process(tv.nodes[e >> 1], e & 1, took);
      if (r >= 0) {
        if (took) mute = sp;
        cur = r;
        found = true;
        break;
      }
    }
    if (!found) break;
  }
  return ok;
}

}  // namespace pptkg
