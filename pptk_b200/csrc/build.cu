// Level-synchronous device builder that reproduces the reference k-d tree
// exactly (pptk/kdtree/src/kdtree-impl.h:248-329 MakeNode /
// RecursiveBuildHelper, :773-818 BuildTree).
//
// The reference builds depth first; every node only permutes the indices of
// its own range, so building all nodes of a level at once gives the same
// permutation.  Nodes with more than mid_capacity() points are processed by
// grid-wide kernels over tiles of points; those of up to that many are split
// by one block each, in shared memory, until small_capacity() points are left,
// and subtrees of those are finished by one warp each.
//
// The reference partition (PartitionIndices, kdtree-impl.h:192-246) is two
// Hoare passes with converging cursors.  Each pass pairs the j-th misplaced
// element of the left zone (ascending) with the j-th misplaced element of the
// right zone (descending), so it is reproduced by ranking the two kinds of
// misplaced elements with scans and swapping rank-matched pairs.
#include <algorithm>
#include <cstddef>
#include <vector>

#include "build.cuh"
#include "build_nodes.cuh"
#include "profile.cuh"
#include "util.cuh"

namespace pptkg {

constexpr int BT = 256;     // threads per tile block
constexpr int SWAP_U = 4;   // pairs a k_swap thread has in flight
constexpr int SPLIT_U = 4;  // points a k_split thread has in flight
// Points per tile of a level: 4,096, or 1,024 in builds of less than 4M
// points, whose levels would otherwise leave SMs without a tile (200k points:
// 49 tiles, a level's pass over them 15 us against 7).  A multiple of
// SPLIT_U x BT, at most 16 x BT.
inline int tile_points(int64_t n) { return n < ((int64_t)1 << 22) ? 1024 : 4096; }
static_assert(1024 % (SPLIT_U * BT) == 0 && 4096 <= 16 * BT, "tiles are whole steps of a block, 16 points a thread");

template <typename T, int D>
struct Seg {
  int b, e;
  int parent, side;  // parent record and side; a cloud's root has parent = -1 - cloud
  int lvl;
  int rec;
  long long n_orig;  // input rows of the segment's cloud (the reference's num_points)
  T lo[D], hi[D];  // loose extent (the reference's node_box), trimmed in place
  typename OrdOf<T>::type tlo[D], thi[D];
  // tight boxes of the points below the split value and of the others,
  // which are the children's unless ties moved the split
  typename OrdOf<T>::type clo[2][D], chi[2][D];
  int act;
  int sd;
  T sv;
  int L1, L2;
  int G;
  int tile0, ntiles;
  int boxed;  // tlo / thi are known (from the parent)
};

// Ties of segments of at most this many points are moved by one block.
constexpr int TIE_BLOCK = 8192;

constexpr int MAX_LEVELS = 4096;  // grid-wide levels

struct BuildCtl {
  int status;
  int nsmall;
  int small_next;
  int nmid;
  int mid_next;
  int rec_count;
  int depth;
  int ties;     // 1 + the last level with points at a split value
  int big;      // 1 + the last level with such points in a segment too large for one block
  int stalled;  // 1 + the level that waits for a tie pass that the host has not launched
  int unboxed;  // 1 + the last level with segments whose box is not known
  int tile;     // points per tile
  int level_cnt[MAX_LEVELS + 1];    // large segments per level
  int level_tiles[MAX_LEVELS + 1];  // their tiles
};

// ----------------------------------------------------------------- helpers
template <typename T>
__device__ __forceinline__ T midpoint_ref(T a, T b) {
  if constexpr (std::is_unsigned<T>::value) {
    // kdtree-impl.h:161-164 (unsigned form), in C++ integer promotion
    if (a < b) {
      const T t = a;
      a = b;
      b = t;
    }
    return (T)((a - b) / 2 + b);
  } else if constexpr (std::is_integral<T>::value) {
    // kdtree-impl.h:167-173 (signed form), in C++ integer promotion
    if ((a >= 0 && b >= 0) || (a < 0 && b < 0)) return (T)((b - a) / (T)2 + a);
    return (T)((a + b) / (T)2);
  } else {
    // the same signed form in floating point, one rounding per operation
    if ((a >= (T)0 && b >= (T)0) || (a < (T)0 && b < (T)0)) return xadd(xdiv(xsub(b, a), (T)2), a);
    return xdiv(xadd(a, b), (T)2);
  }
}

// `T width = max - min` of ComputeSplit (kdtree-impl.h:179): integer types
// wrap as the reference's conversion back to T does.
template <typename T>
__device__ __forceinline__ T width_ref(T lo, T hi) {
  if constexpr (std::is_integral<T>::value)
    return (T)(hi - lo);
  else
    return xsub(hi, lo);
}

__device__ __forceinline__ double max0(double x) { return (0.0 < x) ? x : 0.0; }

// MakeNode's per-node decisions (kdtree-impl.h:248-297): empty-space trims of
// the loose extent against the tight box (TrimEmptyGaps, :114-158, in double),
// then the leaf test and the widest-axis midpoint split (ComputeSplit,
// :175-190, in T).  Writes the record except split_index and children.
template <typename T, int D>
__device__ void node_logic(int size, long long n_orig, bool is_top, T lo[D], T hi[D], const T tlo[D], const T thi[D],
                           int max_leaf, double thr, Rec<T, D>& rec, int& act, int& sd, T& sv) {
  for (int i = 0; i < D; i++) {
    rec.lo[i] = tlo[i];
    rec.hi[i] = thi[i];
  }
  if (is_top)
    for (int i = 0; i < D; i++) {
      lo[i] = tlo[i];
      hi[i] = thi[i];
    }
  rec.ntrim = 0;
  rec.split_dim = -1;
  rec.split_val = (T)0;
  rec.split_index = -1;
  rec.left = rec.right = -1;
  if ((long long)size != n_orig) {
    for (int guard = 0; guard <= 2 * D; guard++) {
      int gdim = -1, gside = -1;
      double gsize = 0.0;
      for (int i = 0; i < D; i++) {
        double g = max0(__dsub_rn((double)hi[i], (double)thi[i]));
        if (g >= gsize) gdim = i, gside = 1, gsize = g;
        g = max0(__dsub_rn((double)tlo[i], (double)lo[i]));
        if (g >= gsize) gdim = i, gside = 0, gsize = g;
      }
      if (gsize == 0.0) break;
      double width = __dsub_rn((double)hi[gdim], (double)lo[gdim]);
      if (__ddiv_rn(gsize, width) <= thr) break;
      if (rec.ntrim < 2 * D) rec.trim[rec.ntrim] = (uint8_t)(gdim * 2 + gside);
      rec.ntrim++;
      if (gside == 0)
        lo[gdim] = tlo[gdim];
      else
        hi[gdim] = thi[gdim];
    }
  }
  bool point = true;
  for (int i = 0; i < D; i++)
    if (tlo[i] != thi[i]) point = false;
  act = 0;
  if (!point && size > max_leaf) {
    T maxw = (T)0;
    sd = 0;
    sv = (T)0;
    for (int i = 0; i < D; i++) {
      T w = width_ref(tlo[i], thi[i]);
      if (w >= maxw) {
        maxw = w;
        sd = i;
        sv = (tlo[i] == thi[i]) ? tlo[i] : midpoint_ref(tlo[i], thi[i]);
      }
    }
    act = 1;
    rec.split_dim = (int8_t)sd;
    rec.split_val = sv;
  }
}

// num_left rule of PartitionIndices (kdtree-impl.h:234-244).
__device__ __forceinline__ int num_left_rule(int lim1, int lim2, int count) {
  int nl;
  if (lim1 > count / 2)
    nl = lim1;
  else if (lim2 < count / 2)
    nl = lim2;
  else
    nl = count / 2;
  if (lim1 == count && lim2 == 0) nl = count / 2;
  return nl;
}

template <typename T, int D>
__device__ __forceinline__ Small<T, D> small_of(const Seg<T, D>& g) {
  Small<T, D> s;
  s.b = g.b;
  s.e = g.e;
  s.parent = g.parent;
  s.lvl = (int16_t)g.lvl;
  s.side = (int16_t)g.side;
  s.n_orig = g.n_orig;
  for (int d = 0; d < D; d++) {
    s.lo[d] = g.lo[d];
    s.hi[d] = g.hi[d];
  }
  return s;
}

// Segments that the grid-wide levels leave: to k_block (`mid`, above small_cap
// points) and k_subtree (`small`).
template <typename T, int D>
struct Lists {
  Small<T, D>*mid, *small;
  int mid_capn, small_capn, mid_cap, small_cap;
};

template <typename T, int D>
__device__ __forceinline__ void hand_on(const Small<T, D>& s, const Lists<T, D>& to, BuildCtl* ctl) {
  const bool mid = s.e - s.b > to.small_cap;
  const int slot = atomicAdd(mid ? &ctl->nmid : &ctl->nsmall, 1);
  if (slot < (mid ? to.mid_capn : to.small_capn))
    (mid ? to.mid : to.small)[slot] = s;
  else
    atomicExch(&ctl->status, 7);
}

template <typename T, int D>
__device__ __forceinline__ void seg_clear(Seg<T, D>& g) {
  for (int d = 0; d < D; d++) {
    g.tlo[d] = ord_t<T>(Limits<T>::max());
    g.thi[d] = ord_t<T>(Limits<T>::lowest());
    for (int c = 0; c < 2; c++) {
      g.clo[c][d] = ord_t<T>(Limits<T>::max());
      g.chi[c][d] = ord_t<T>(Limits<T>::lowest());
    }
  }
  g.L1 = g.L2 = 0;
  g.act = 0;
  g.G = 0;
  g.boxed = 0;
}

// A large segment takes its tiles and its record.
template <typename T, int D>
__device__ __forceinline__ void take_place(Seg<T, D>& g, int lvl, int tile, BuildCtl* ctl) {
  g.ntiles = div_up_dev(g.e - g.b, tile);
  g.tile0 = atomicAdd(&ctl->level_tiles[lvl], g.ntiles);
  g.rec = atomicAdd(&ctl->rec_count, 1);
}

// ------------------------------------------------------- input staging ----
template <typename T, int D>
__global__ void k_valid(const T* __restrict__ in, int64_t n, int* __restrict__ flag) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  bool ok = true;
#pragma unroll
  for (int d = 0; d < D; d++) ok = ok && valid_coord(in[i * D + d]);
  flag[i] = ok ? 1 : 0;
}

template <typename T, int D>
__global__ void k_compact(const T* __restrict__ in, int64_t n, const int* __restrict__ flag,
                          const int* __restrict__ off, SoA<T, D> soa) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || !flag[i]) return;
  int j = off[i];
#pragma unroll
  for (int d = 0; d < D; d++) soa.x[d][j] = in[i * D + d];
  soa.id[j] = (int)i;
}

// valid_off[c] = number of valid rows before cloud c (the stable compaction
// keeps every cloud's valid rows together, in order).
static __global__ void k_cloud_off(const int* off, const int64_t* orig_off, int ncloud, int64_t* valid_off) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c <= ncloud) valid_off[c] = off[orig_off[c]];
}

// ------------------------------------------------------ grid-wide levels --
// Level `lvl` works on list segs (ctl->level_cnt[lvl] entries).  Kernels are
// launched with upper-bound grids and read the live counts from the device,
// so the host never waits between levels.
template <typename T, int D>
__global__ void k_roots(const int64_t* valid_off, const int64_t* orig_off, int ncloud, int tile, Seg<T, D>* lvl0,
                        Lists<T, D> to, BuildCtl* ctl) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c == 0) ctl->tile = tile;
  if (c >= ncloud) return;
  const int b = (int)valid_off[c], e = (int)valid_off[c + 1];
  if (e <= b) return;
  Seg<T, D> g;
  g.b = b;
  g.e = e;
  g.parent = -1 - c;
  g.side = 0;
  g.lvl = 0;
  g.rec = -1;
  g.n_orig = orig_off[c + 1] - orig_off[c];
  for (int d = 0; d < D; d++) {
    g.lo[d] = Limits<T>::max();  // replaced by the tight box at a root
    g.hi[d] = Limits<T>::lowest();
  }
  seg_clear(g);
  if (e - b > to.mid_cap) {
    ctl->unboxed = 1;
    take_place(g, 0, tile, ctl);
    lvl0[atomicAdd(&ctl->level_cnt[0], 1)] = g;
  } else {
    hand_on(small_of(g), to, ctl);
  }
}

// The segment of every tile, a warp per segment.
template <typename T, int D>
__global__ void k_tiles(const Seg<T, D>* segs, int lvl, int* tile_seg, const BuildCtl* ctl) {
  const int nseg = ctl->level_cnt[lvl], lane = threadIdx.x & 31;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nseg; i += (gridDim.x * blockDim.x) >> 5) {
    const int t0 = segs[i].tile0, nt = segs[i].ntiles;
    for (int t = lane; t < nt; t += 32) tile_seg[t0 + t] = i;
  }
}

// The tiles of a level are walked grid-stride by a grid of a few blocks per
// SM, so a level with few tiles (or none: the trailing levels of a
// capture-mode rebuild) costs a few hundred idle blocks, not one per tile of
// the largest level.
template <typename T, int D>
__device__ __forceinline__ void tile_at(const Seg<T, D>* segs, const int* tile_seg, int t, int tile, int& s, int& start,
                                        int& end) {
  s = tile_seg[t];
  start = segs[s].b + (t - segs[s].tile0) * tile;
  end = min(start + tile, segs[s].e);
}

template <typename T>
__device__ __forceinline__ T warp_min(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <typename T>
__device__ __forceinline__ T warp_max(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// The same of ordered images, in one instruction for 32-bit ones.
template <typename U>
__device__ __forceinline__ U warp_min_ord(U v) {
  if constexpr (sizeof(U) == 4)
    return __reduce_min_sync(0xffffffffu, v);
  else
    return warp_min(v);
}
template <typename U>
__device__ __forceinline__ U warp_max_ord(U v) {
  if constexpr (sizeof(U) == 4)
    return __reduce_max_sync(0xffffffffu, v);
  else
    return warp_max(v);
}

template <typename T, int D>
__global__ void __launch_bounds__(BT) k_bbox(Seg<T, D>* segs, int lvl, const int* tile_seg, const BuildCtl* ctl,
                                             SoA<T, D> soa) {
  __shared__ T shmn[D][BT / 32], shmx[D][BT / 32];
  if (ctl->unboxed != lvl + 1) return;
  const int ntiles = ctl->level_tiles[lvl], tile = ctl->tile;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    int s, start, end;
    tile_at(segs, tile_seg, t, tile, s, start, end);
    if (segs[s].boxed) continue;  // (uniform over the block)
    T mn[D], mx[D];
#pragma unroll
    for (int d = 0; d < D; d++) {
      mn[d] = Limits<T>::max();
      mx[d] = Limits<T>::lowest();
    }
    for (int i = start + threadIdx.x; i < end; i += BT) {
#pragma unroll
      for (int d = 0; d < D; d++) {
        T v = soa.x[d][i];
        mn[d] = min(mn[d], v);
        mx[d] = max(mx[d], v);
      }
    }
#pragma unroll
    for (int d = 0; d < D; d++) {
      mn[d] = warp_min(mn[d]);
      mx[d] = warp_max(mx[d]);
      if (lane == 0) {
        shmn[d][wid] = mn[d];
        shmx[d][wid] = mx[d];
      }
    }
    __syncthreads();
    if (threadIdx.x < D) {
      int d = threadIdx.x;
      T a = shmn[d][0], b = shmx[d][0];
      for (int w = 1; w < BT / 32; w++) {
        a = min(a, shmn[d][w]);
        b = max(b, shmx[d][w]);
      }
      atomicMin(&segs[s].tlo[d], ord_t<T>(a));
      atomicMax(&segs[s].thi[d], ord_t<T>(b));
    }
    __syncthreads();
  }
}

// A record takes its place and its parent learns of it.
template <typename T, int D>
__device__ __forceinline__ bool link_record(const Rec<T, D>& rec, int id, int parent, int side, Rec<T, D>* recs,
                                            int rec_cap, int* root_rec, BuildCtl* ctl) {
  if (id >= rec_cap) {
    atomicExch(&ctl->status, 6);
    return false;
  }
  recs[id] = rec;
  if (parent < 0)
    root_rec[-parent - 1] = id;
  else if (side)
    recs[parent].right = id;
  else
    recs[parent].left = id;
  return true;
}

// Split decision and record of a segment whose box is known.
template <typename T, int D>
__device__ __forceinline__ void decide(Seg<T, D>& g, BuildCtl* ctl, Rec<T, D>* recs, int rec_cap, int* root_rec,
                                       int max_leaf, double thr) {
  T tlo[D], thi[D];
  for (int d = 0; d < D; d++) {
    tlo[d] = from_ord_t<T>(g.tlo[d]);
    thi[d] = from_ord_t<T>(g.thi[d]);
  }
  Rec<T, D> rec;
  g.sd = 0;
  g.sv = (T)0;
  node_logic<T, D>(g.e - g.b, g.n_orig, g.parent < 0, g.lo, g.hi, tlo, thi, max_leaf, thr, rec, g.act, g.sd, g.sv);
  rec.begin = g.b;
  rec.end = g.e;
  if (!link_record<T, D>(rec, g.rec, g.parent, g.side, recs, rec_cap, root_rec, ctl)) g.act = 0;
  g.boxed = 1;
}

// The decisions that waited for k_bbox.
template <typename T, int D>
__global__ void k_node(Seg<T, D>* segs, int lvl, BuildCtl* ctl, Rec<T, D>* recs, int rec_cap, int* root_rec,
                       int max_leaf, double thr) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (ctl->unboxed != lvl + 1 || i >= ctl->level_cnt[lvl] || segs[i].boxed) return;
  Seg<T, D> g = segs[i];
  decide(g, ctl, recs, rec_cap, root_rec, max_leaf, thr);
  segs[i] = g;
}

// One pass over a level's points: how many lie below (L1) and at or below
// (L2) the split value, per tile how many below, which (a bit per point, for
// the ranks), and the tight boxes of both sides, so that neither the ranks nor
// the next level's boxes read the points again: 12 B a point in place of 24.
// Bound by its instructions (two-sided boxes), then by loads in flight: 20M
// points 107 us with selects for both sides, 65 with a branch.
template <typename T, int D>
__global__ void __launch_bounds__(BT) k_split(Seg<T, D>* segs, int lvl, const int* tile_seg, const BuildCtl* ctl,
                                              SoA<T, D> soa, int* tile_lt, uint32_t* tile_bits) {
  typedef typename OrdOf<T>::type U;
  __shared__ U shb[BT / 32][4 * D];
  __shared__ int shc[BT / 32][2];
  const int ntiles = ctl->level_tiles[lvl], tile = ctl->tile;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    int s, start, end;
    tile_at(segs, tile_seg, t, tile, s, start, end);
    if (!segs[s].act) continue;  // (uniform over the block)
    const T sv = segs[s].sv;
    const int sd = segs[s].sd;
    T lo[2][D], hi[2][D];
#pragma unroll
    for (int c = 0; c < 2; c++)
#pragma unroll
      for (int d = 0; d < D; d++) {
        lo[c][d] = Limits<T>::max();
        hi[c][d] = Limits<T>::lowest();
      }
    int c1 = 0, c2 = 0;
    // a full tile needs no test of its end; the loads of SPLIT_U points are
    // issued together
    auto points = [&](auto full) {
      for (int j0 = 0; j0 < tile / BT; j0 += SPLIT_U) {
        T x[SPLIT_U][D];
        bool in[SPLIT_U];
#pragma unroll
        for (int u = 0; u < SPLIT_U; u++) {
          const int i = start + (j0 + u) * BT + threadIdx.x;
          in[u] = decltype(full)::value || i < end;
#pragma unroll
          for (int d = 0; d < D; d++) x[u][d] = in[u] ? soa.x[d][i] : (T)0;
        }
#pragma unroll
        for (int u = 0; u < SPLIT_U; u++) {
          T v = x[u][0];
#pragma unroll
          for (int d = 1; d < D; d++) v = d == sd ? x[u][d] : v;
          const bool below = in[u] && v < sv;
          c2 += in[u] && v == sv;
          if (below) {
#pragma unroll
            for (int d = 0; d < D; d++) {
              lo[0][d] = min(lo[0][d], x[u][d]);
              hi[0][d] = max(hi[0][d], x[u][d]);
            }
          } else if (in[u]) {
#pragma unroll
            for (int d = 0; d < D; d++) {
              lo[1][d] = min(lo[1][d], x[u][d]);
              hi[1][d] = max(hi[1][d], x[u][d]);
            }
          }
          const unsigned m = __ballot_sync(0xffffffffu, below);
          c1 += __popc(m);
          if (lane == 0) tile_bits[(size_t)t * (tile / 32) + (j0 + u) * (BT / 32) + wid] = m;
        }
      }
    };
    if (start + tile <= end)
      points(std::true_type());
    else
      points(std::false_type());
    c2 = warp_sum(c2) + c1;  // (c1: the warp's already)
#pragma unroll
    for (int c = 0; c < 2; c++)
#pragma unroll
      for (int d = 0; d < D; d++) {
        const U a = warp_min_ord(ord_t<T>(lo[c][d])), b = warp_max_ord(ord_t<T>(hi[c][d]));
        if (lane == 0) {
          shb[wid][c * 2 * D + d] = a;
          shb[wid][c * 2 * D + D + d] = b;
        }
      }
    if (lane == 0) {
      shc[wid][0] = c1;
      shc[wid][1] = c2;
    }
    __syncthreads();
    if (threadIdx.x < 4 * D) {
      const int c = threadIdx.x / (2 * D), r = threadIdx.x % (2 * D);
      U v = shb[0][threadIdx.x];
      for (int w = 1; w < BT / 32; w++) v = r < D ? min(v, shb[w][threadIdx.x]) : max(v, shb[w][threadIdx.x]);
      if (r < D)
        atomicMin(&segs[s].clo[c][r], v);
      else
        atomicMax(&segs[s].chi[c][r - D], v);
    } else if (threadIdx.x == 4 * D) {
      int n = 0;
      for (int w = 0; w < BT / 32; w++) n += shc[w][0];
      tile_lt[t] = n;
      atomicAdd(&segs[s].L1, n);
    } else if (threadIdx.x == 4 * D + 1) {
      int n = 0;
      for (int w = 0; w < BT / 32; w++) n += shc[w][1];
      atomicAdd(&segs[s].L2, n);
    }
    __syncthreads();
  }
}

// Ranks of pass 1 from the tiles' counts: left of Z = b + L1 the points not
// below the split value are misplaced, right of it those below.  A tile on
// one side of Z needs no second look; the one that holds Z counts its bits.
template <typename T, int D>
__global__ void k_ranks(Seg<T, D>* segs, int lvl, const int* tile_lt, const uint32_t* tile_bits, long long* tile_off,
                        BuildCtl* ctl) {
  __shared__ long long sh[33];
  const int nseg = ctl->level_cnt[lvl], tile = ctl->tile;
  for (int si = blockIdx.x; si < nseg; si += gridDim.x) {
    Seg<T, D>& g = segs[si];
    if (!g.act) continue;  // (uniform over the block)
    const int b = g.b, Z = b + g.L1;
    // points below the split value among the first Z - start of the tile that
    // holds Z (one word per thread)
    const int mid = g.L1 / tile, n = g.L1 - mid * tile;
    int in = 0;
    if (mid < g.ntiles && threadIdx.x <= n >> 5 && threadIdx.x < tile / 32) {
      const uint32_t w = tile_bits[(size_t)(g.tile0 + mid) * (tile / 32) + threadIdx.x];
      in = __popc(threadIdx.x < n >> 5 ? w : w & ((1u << (n & 31)) - 1u));
    }
    const int left = (int)block_sum((long long)in, sh);
    long long carry = 0;
    for (int c0 = 0; c0 < g.ntiles; c0 += blockDim.x) {
      const int t = c0 + threadIdx.x;
      long long v = 0;
      if (t < g.ntiles) {
        const int start = b + t * tile, end = min(start + tile, g.e), lt = tile_lt[g.tile0 + t];
        if (end <= Z) {
          v = end - start - lt;
        } else if (start >= Z) {
          v = (long long)lt << 32;
        } else {
          v = (n - left) + ((long long)(lt - left) << 32);
        }
      }
      long long tot;
      const long long ex = block_excl_scan(v, sh, tot);
      if (t < g.ntiles) tile_off[g.tile0 + t] = carry + ex;
      carry += tot;
    }
    if (threadIdx.x == 0) {
      const int nbl = (int)(carry & 0xffffffffll), ngr = (int)(carry >> 32);
      g.G = nbl;
      if (nbl != ngr) atomicExch(&ctl->status, 1);
      if (g.L1 != g.L2) {
        ctl->ties = lvl + 1;
        if (g.e - g.b > TIE_BLOCK) ctl->big = lvl + 1;
      }
    }
  }
}

// The positions of pass 1's misplaced points at their ranks, from the bits.
template <typename T, int D>
__global__ void __launch_bounds__(BT) k_place_ranks(Seg<T, D>* segs, int lvl, const int* tile_seg,
                                                    const BuildCtl* ctl, const uint32_t* tile_bits, const long long* tile_off, int* blpos,
                                                    int* grpos) {
  __shared__ long long sh[33];
  const int ntiles = ctl->level_tiles[lvl], tile = ctl->tile;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    int s, start, end;
    tile_at(segs, tile_seg, t, tile, s, start, end);
    if (!segs[s].act) continue;  // (uniform over the block)
    const int b = segs[s].b, Z = b + segs[s].L1, G = segs[s].G, size = segs[s].e - b;
    // tile / BT positions per thread (4 or 16): a part of a word
    const int items = tile / BT, bit0 = threadIdx.x * items;
    const int i0 = start + bit0;
    const unsigned all = (1u << items) - 1u;
    const unsigned below = tile_bits[(size_t)t * (tile / 32) + (bit0 >> 5)] >> (bit0 & 31) & all;
    const unsigned in = i0 >= end ? 0u : end - i0 >= items ? all : (1u << (end - i0)) - 1u;
    const unsigned left = i0 >= Z ? 0u : Z - i0 >= items ? all : (1u << (Z - i0)) - 1u;
    unsigned mbl = in & left & ~below, mgr = in & ~left & below;
    const long long mine = (long long)__popc(mbl) + ((long long)__popc(mgr) << 32);
    long long tot;
    const long long ex = block_excl_scan(mine, sh, tot) + tile_off[t];
    int rb = (int)(ex & 0xffffffffll), rg = (int)(ex >> 32);
    while (mbl) {
      const int j = __ffs(mbl) - 1;
      mbl &= mbl - 1;
      if (rb < size) blpos[b + rb] = i0 + j;
      rb++;
    }
    while (mgr) {
      const int j = __ffs(mgr) - 1;
      mgr &= mgr - 1;
      const int slot = G - 1 - rg;
      if (slot >= 0 && slot < size) grpos[b + slot] = i0 + j;
      rg++;
    }
  }
}

// ---- the tie pass (PartitionIndices' second): points equal to the split
// value move to [b + L1, b + L2).  Segments of up to TIE_BLOCK points have it
// from one block each (k_ties), larger ones from the whole grid (k_flags,
// k_tscan, k_scatter, k_swap), which the host launches only once a level has
// asked for it.
template <typename T, int D>
__device__ __forceinline__ bool big_tie(const Seg<T, D>& g) {
  return g.L1 != g.L2 && g.e - g.b > TIE_BLOCK;
}

template <typename T, int D>
__global__ void __launch_bounds__(BT) k_ties(Seg<T, D>* segs, int lvl, BuildCtl* ctl, SoA<T, D> soa, int* blpos,
                                             int* grpos) {
  typedef typename OrdOf<T>::type U;
  __shared__ long long sh[33];
  __shared__ U box[4 * D];
  if (ctl->ties != lvl + 1) return;
  const int nseg = ctl->level_cnt[lvl];
  for (int si = blockIdx.x; si < nseg; si += gridDim.x) {
    Seg<T, D>& g = segs[si];
    if (!g.act || g.L1 == g.L2 || g.e - g.b > TIE_BLOCK) continue;  // (uniform over the block)
    const int b = g.b, e = g.e, L1 = g.L1, Z = b + g.L2;
    const T sv = g.sv;
    const T* v = soa.x[g.sd];
    long long carry = 0;
    for (int i0 = b + L1; i0 < e; i0 += BT) {
      const int i = i0 + threadIdx.x;
      bool bl = false, gr = false;
      if (i < e) {
        const T x = v[i];
        bl = i < Z && x > sv;
        gr = i >= Z && x <= sv;
      }
      long long tot;
      const long long ex = carry + block_excl_scan((long long)bl + ((long long)gr << 32), sh, tot);
      if (bl) blpos[b + (int)(ex & 0xffffffffll)] = i;
      if (gr) grpos[b + (int)(ex >> 32)] = i;  // (from the left: read from its end below)
      carry += tot;
    }
    const int G = (int)(carry & 0xffffffffll);
    if (G != (int)(carry >> 32)) {
      if (threadIdx.x == 0) atomicExch(&ctl->status, 1);
      continue;
    }
    __threadfence_block();
    __syncthreads();
    for (int j = threadIdx.x; j < G; j += BT) {
      const int x = blpos[b + j], y = grpos[b + G - 1 - j];
#pragma unroll
      for (int d = 0; d < D; d++) {
        const T t = soa.x[d][x];
        soa.x[d][x] = soa.x[d][y];
        soa.x[d][y] = t;
      }
      const int t = soa.id[x];
      soa.id[x] = soa.id[y];
      soa.id[y] = t;
    }
    // the children's boxes, where the ties moved the split off b + L1
    const int at = b + num_left_rule(L1, g.L2, e - b);
    if (at == b + L1) continue;  // (uniform over the block)
    if (threadIdx.x < 4 * D)
      box[threadIdx.x] = ord_t<T>((threadIdx.x / D) & 1 ? Limits<T>::lowest() : Limits<T>::max());
    __threadfence_block();
    __syncthreads();
    U lo[2][D], hi[2][D];
#pragma unroll
    for (int c = 0; c < 2; c++)
#pragma unroll
      for (int d = 0; d < D; d++) {
        lo[c][d] = ord_t<T>(Limits<T>::max());
        hi[c][d] = ord_t<T>(Limits<T>::lowest());
      }
    for (int i = b + threadIdx.x; i < e; i += BT)
#pragma unroll
      for (int d = 0; d < D; d++) {
        const U x = ord_t<T>(soa.x[d][i]);
#pragma unroll
        for (int c = 0; c < 2; c++)
          if ((i >= at) == (c == 1)) {
            lo[c][d] = min(lo[c][d], x);
            hi[c][d] = max(hi[c][d], x);
          }
      }
#pragma unroll
    for (int c = 0; c < 2; c++)
#pragma unroll
      for (int d = 0; d < D; d++) {
        atomicMin(&box[(2 * c) * D + d], lo[c][d]);
        atomicMax(&box[(2 * c + 1) * D + d], hi[c][d]);
      }
    __syncthreads();
    if (threadIdx.x < D) {
      const int d = threadIdx.x;
      for (int c = 0; c < 2; c++) {
        g.clo[c][d] = box[(2 * c) * D + d];
        g.chi[c][d] = box[(2 * c + 1) * D + d];
      }
    }
    __syncthreads();
  }
}

template <typename T>
__device__ __forceinline__ void tie_flags(int i, T x, T sv, int b, int L1, int L2, bool& bl, bool& gr) {
  const int Z = b + L2;
  bl = (i >= b + L1) && (i < Z) && (x > sv);
  gr = (i >= Z) && (x <= sv);
}

template <typename T, int D>
__global__ void __launch_bounds__(BT) k_flags(Seg<T, D>* segs, int lvl, const int* tile_seg, const BuildCtl* ctl,
                                              SoA<T, D> soa, long long* tile_cnt) {
  __shared__ long long sh[33];
  if (ctl->big != lvl + 1) return;
  const int ntiles = ctl->level_tiles[lvl], tile = ctl->tile;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    int s, start, end;
    tile_at(segs, tile_seg, t, tile, s, start, end);
    long long c = 0;
    if (segs[s].act && big_tie(segs[s])) {
      const T sv = segs[s].sv;
      const T* v = soa.x[segs[s].sd];
      const int b = segs[s].b, L1 = segs[s].L1, L2 = segs[s].L2;
      for (int i = start + threadIdx.x; i < end; i += BT) {
        bool bl, gr;
        tie_flags(i, v[i], sv, b, L1, L2, bl, gr);
        c += (long long)bl + ((long long)gr << 32);
      }
    }
    long long tot = block_sum(c, sh);
    if (threadIdx.x == 0) tile_cnt[t] = tot;
  }
}

template <typename T, int D>
__global__ void k_tscan(Seg<T, D>* segs, int lvl, const long long* tile_cnt, long long* tile_off, BuildCtl* ctl) {
  __shared__ long long sh[33];
  if (ctl->big != lvl + 1) return;
  const int nseg = ctl->level_cnt[lvl];
  for (int si = blockIdx.x; si < nseg; si += gridDim.x) {
    Seg<T, D>& g = segs[si];
    if (!g.act || !big_tie(g)) continue;  // (uniform over the block)
    long long carry = 0;
    for (int c0 = 0; c0 < g.ntiles; c0 += blockDim.x) {
      int t = c0 + threadIdx.x;
      long long v = t < g.ntiles ? tile_cnt[g.tile0 + t] : 0;
      long long tot;
      long long ex = block_excl_scan(v, sh, tot);
      if (t < g.ntiles) tile_off[g.tile0 + t] = carry + ex;
      carry += tot;
    }
    if (threadIdx.x == 0) {
      int nbl = (int)(carry & 0xffffffffll), ngr = (int)(carry >> 32);
      g.G = nbl;
      if (nbl != ngr) atomicExch(&ctl->status, 1);
    }
  }
}

template <typename T, int D>
__global__ void __launch_bounds__(BT) k_scatter(Seg<T, D>* segs, int lvl, const int* tile_seg, const BuildCtl* ctl,
                                                SoA<T, D> soa, const long long* tile_off, int* blpos, int* grpos) {
  __shared__ long long sh[33];
  if (ctl->big != lvl + 1) return;
  const int ntiles = ctl->level_tiles[lvl], tile = ctl->tile;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    int s, start, end;
    tile_at(segs, tile_seg, t, tile, s, start, end);
    if (!segs[s].act || !big_tie(segs[s])) continue;  // (uniform over the block)
    const T sv = segs[s].sv;
    const T* v = soa.x[segs[s].sd];
    const int b = segs[s].b, L1 = segs[s].L1, L2 = segs[s].L2, G = segs[s].G;
    const int items = tile / BT, i0 = start + threadIdx.x * items;
    unsigned mbl = 0, mgr = 0;
    for (int j = 0; j < items; j++) {
      int i = i0 + j;
      if (i < end) {
        bool bl, gr;
        tie_flags(i, v[i], sv, b, L1, L2, bl, gr);
        mbl |= (unsigned)bl << j;
        mgr |= (unsigned)gr << j;
      }
    }
    long long mine = (long long)__popc(mbl) + ((long long)__popc(mgr) << 32);
    long long tot;
    long long ex = block_excl_scan(mine, sh, tot) + tile_off[t];
    int rb = (int)(ex & 0xffffffffll), rg = (int)(ex >> 32);
    const int size = segs[s].e - b;
    for (int j = 0; j < items; j++) {
      if (mbl >> j & 1) {
        if (rb < size) blpos[b + rb] = i0 + j;
        rb++;
      }
      if (mgr >> j & 1) {
        const int slot = G - 1 - rg;
        if (slot >= 0 && slot < size) grpos[b + slot] = i0 + j;
        rg++;
      }
    }
  }
}

// Swaps rank-matched pairs (tie: those of the tie pass, if the level has one).
template <typename T, int D>
__global__ void __launch_bounds__(BT) k_swap(Seg<T, D>* segs, int lvl, bool tie, const int* tile_seg, BuildCtl* ctl,
                                             SoA<T, D> soa, const int* blpos, const int* grpos) {
  if (tie && ctl->big != lvl + 1) return;
  const int ntiles = ctl->level_tiles[lvl], tile = ctl->tile;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    int s, start, end;
    tile_at(segs, tile_seg, t, tile, s, start, end);
    if (!segs[s].act) continue;
    if (tie && !big_tie(segs[s])) continue;
    const int b = segs[s].b, e = segs[s].e, G = segs[s].G;
    // pair j of this tile: j = start - b + threadIdx.x + u * BT.  Every
    // position belongs to one pair only, so the loads of SWAP_U pairs are
    // issued before their stores: the swap is bound by memory latency, and
    // one pair in flight per thread left most of it exposed
    const int jend = min(end - b, G);
    for (int j0 = start - b + threadIdx.x; j0 < jend; j0 += SWAP_U * BT) {
      int x[SWAP_U], y[SWAP_U];
      bool ok[SWAP_U];
#pragma unroll
      for (int u = 0; u < SWAP_U; u++) {
        const int j = j0 + u * BT;
        ok[u] = j < jend;
        x[u] = ok[u] ? blpos[b + j] : b;
        y[u] = ok[u] ? grpos[b + j] : b;
        if (ok[u] && (x[u] < b || x[u] >= e || y[u] < b || y[u] >= e)) {
          atomicExch(&ctl->status, 4);
          ok[u] = false;
        }
      }
      T vx[SWAP_U][D], vy[SWAP_U][D];
      int ix[SWAP_U], iy[SWAP_U];
#pragma unroll
      for (int u = 0; u < SWAP_U; u++) {
        if (!ok[u]) continue;
#pragma unroll
        for (int d = 0; d < D; d++) {
          vx[u][d] = soa.x[d][x[u]];
          vy[u][d] = soa.x[d][y[u]];
        }
        ix[u] = soa.id[x[u]];
        iy[u] = soa.id[y[u]];
      }
#pragma unroll
      for (int u = 0; u < SWAP_U; u++) {
        if (!ok[u]) continue;
#pragma unroll
        for (int d = 0; d < D; d++) {
          soa.x[d][x[u]] = vy[u][d];
          soa.x[d][y[u]] = vx[u][d];
        }
        soa.id[x[u]] = iy[u];
        soa.id[y[u]] = ix[u];
      }
    }
  }
}

// The children of a level's segments: a lane per child makes it and decides
// it if it stays large, and the warp writes the map of the tiles.  (Bound by
// the decisions' serial arithmetic: both children on one lane took 24 us for
// the 400 segments of a 200k-point build's last level.)
template <typename T, int D>
__global__ void k_children(Seg<T, D>* segs, int lvl, int tied, Rec<T, D>* recs, int rec_cap, Seg<T, D>* next,
                           Lists<T, D> to, int max_leaf, double thr, int* tile_seg, BuildCtl* ctl) {
  const int c0 = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  const int i = c0 >> 1, side = c0 & 1;
  // a level whose ties had no pass (tied 0: none was launched, 1: that of
  // small segments) waits for it
  if ((tied < 1 && ctl->ties == lvl + 1) || (tied < 2 && ctl->big == lvl + 1)) {
    if (c0 == 0) ctl->stalled = lvl + 1;
    return;
  }
  const int nseg = ctl->level_cnt[lvl];
  if ((c0 & ~31) >> 1 >= nseg) return;
  int t0 = 0, nt = 0, at = 0;
  if (i < nseg && segs[i].act) {
    const Seg<T, D>& g = segs[i];
    const int si = g.b + num_left_rule(g.L1, g.L2, g.e - g.b);
    if (side == 0) recs[g.rec].split_index = si;
    const int cb = side ? si : g.b, ce = side ? g.e : si;
    if (cb < ce) {
      Seg<T, D> c;
      c.b = cb;
      c.e = ce;
      c.parent = g.rec;
      c.side = side;
      c.lvl = g.lvl + 1;
      c.rec = -1;
      c.n_orig = g.n_orig;
      for (int d = 0; d < D; d++) {
        c.lo[d] = side == 1 && d == g.sd ? g.sv : g.lo[d];
        c.hi[d] = side == 0 && d == g.sd ? g.sv : g.hi[d];
      }
      if (ce - cb > to.mid_cap) {
        seg_clear(c);
        take_place(c, lvl + 1, ctl->tile, ctl);
        if (si == g.b + g.L1 || !big_tie(g)) {
          for (int d = 0; d < D; d++) {
            c.tlo[d] = g.clo[side][d];
            c.thi[d] = g.chi[side][d];
          }
          decide(c, ctl, recs, rec_cap, (int*)nullptr, max_leaf, thr);
        } else {
          // decided by k_node once k_bbox knows its box; until then, and for
          // good below the last level of a rebuild, its record is a leaf that
          // no other record refers to (the passes over all records read it)
          Rec<T, D> rec;
          rec.begin = cb;
          rec.end = ce;
          rec.split_dim = -1;
          rec.split_index = rec.left = rec.right = -1;
          rec.ntrim = 0;
          for (int d = 0; d < D; d++) rec.lo[d] = rec.hi[d] = (T)0;
          rec.split_val = (T)0;
          if (c.rec < rec_cap) recs[c.rec] = rec;
          ctl->unboxed = lvl + 2;
        }
        t0 = c.tile0;
        nt = c.ntiles;
        at = atomicAdd(&ctl->level_cnt[lvl + 1], 1);
        next[at] = c;
      } else {
        hand_on(small_of(c), to, ctl);
      }
    }
  }
  for (unsigned rest = __ballot_sync(0xffffffffu, nt > 0); rest; rest &= rest - 1) {
    const int s = __ffs(rest) - 1;
    const int a = __shfl_sync(0xffffffffu, t0, s), n = __shfl_sync(0xffffffffu, nt, s),
              k = __shfl_sync(0xffffffffu, at, s);
    for (int t = lane; t < n; t += 32) tile_seg[a + t] = k;
  }
}

// --------------------------------------------- per-block segments ----
// Points of a warp's word whose bits are set, counted before every word: the
// words of a segment of up to 2,048 points, two per lane.
struct WordScan {
  int a0, a1, total;
  __device__ __forceinline__ WordScan(const uint32_t* bits, int words) {
    const int lane = threadIdx.x & 31;
    const int c0 = lane < words ? __popc(bits[lane]) : 0, c1 = lane + 32 < words ? __popc(bits[lane + 32]) : 0;
    const int i0 = warp_incl_scan(c0), t0 = __shfl_sync(0xffffffffu, i0, 31);
    const int i1 = warp_incl_scan(c1) + t0;
    a0 = i0 - c0;
    a1 = i1 - c1;
    total = __shfl_sync(0xffffffffu, i1, 31);
  }
  // bits set before word w (the same in every lane)
  __device__ __forceinline__ int before(int w) const { return __shfl_sync(0xffffffffu, w < 32 ? a0 : a1, w & 31); }
};

// Splits segments of small_cap to mid_cap points, one block each in shared
// memory, down to small_cap points, which go to the list of k_subtree.  A
// node's partition takes its ranks from a bit per point: a misplaced point's
// rank is the number of set (or clear) bits before it.  Persistent: a block
// takes segments from the list until it is exhausted.
//
// As grid-wide levels these segments cost a chain of launches per level for a
// few thousand points, and a cloud of long chains (a few points split off at a
// time) one chain of launches per split.  us a build with k_subtree taking
// 2,048 points / with levels down to 512 / so: 600 points 261 / 305 / 241,
// 1,000 277 / 336 / 267, 3,000 in chains 3540 / 4618 / 2016, 200k with ties
// 938 / 1023 / 895, 5M 3300 / 2971 / 2668.  A few blocks' serial splits bound
// the small ones, the levels above the large ones.
template <typename T, int D>
__global__ void __launch_bounds__(BT, 4) k_block(SoA<T, D> soa, Rec<T, D>* recs, int rec_cap, int* root_rec,
                                              Lists<T, D> to, int max_leaf, double thr, BuildCtl* ctl) {
  typedef typename OrdOf<T>::type U;
  constexpr int WARPS = BT / 32, TODO = 4;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ Small<T, D> todo[TODO];  // (disjoint, above small_cap points each: at most three)
  __shared__ U box[WARPS][2 * D];
  __shared__ uint32_t bits[64];
  __shared__ int le[WARPS];
  // (the box as values in shared memory: ptxas 12.9 does not come back from the
  // int16, 3-d kernel where the deciding lane converts it itself)
  __shared__ T s_sv, tight[2 * D];
  __shared__ int s_item, s_todo, s_act, s_sd, s_rec;
  T* X[D];
  unsigned char* p = smem;
#pragma unroll
  for (int d = 0; d < D; d++) {
    X[d] = (T*)p;
    p += sizeof(T) * to.mid_cap;
  }
  int* ID = (int*)p;
  p += sizeof(int) * to.mid_cap;
  uint16_t* S = (uint16_t*)p;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const unsigned FULL = 0xffffffffu, lt = (1u << lane) - 1u;
  const int nmid = min(ctl->nmid, to.mid_capn);
  // swaps the first G pairs of S[at ..] and, from its end, S[at + half ..]
  auto swap = [&](int at, int half, int G) {
    __syncthreads();
    for (int j = tid; j < G; j += BT) {
      const int x = S[at + j], y = S[at + half + G - 1 - j];
#pragma unroll
      for (int d = 0; d < D; d++) {
        const T t = X[d][x];
        X[d][x] = X[d][y];
        X[d][y] = t;
      }
      const int t = ID[x];
      ID[x] = ID[y];
      ID[y] = t;
    }
    __syncthreads();
  };

  while (true) {
    if (tid == 0) s_item = atomicAdd(&ctl->mid_next, 1);
    __syncthreads();
    if (s_item >= nmid) break;
    const int base = to.mid[s_item].b, n = to.mid[s_item].e - base;
    for (int i = tid; i < n; i += BT) {
#pragma unroll
      for (int d = 0; d < D; d++) X[d][i] = soa.x[d][base + i];
      ID[i] = soa.id[base + i];
    }
    if (tid == 0) {
      todo[0] = to.mid[s_item];
      s_todo = 1;
    }
    __syncthreads();
    for (int nodes = 0; s_todo > 0; nodes++) {
      const int cur = s_todo - 1;
      const int b = todo[cur].b - base, e = todo[cur].e - base, words = (e - b + 31) >> 5;
      // tight box
      T mn[D], mx[D];
#pragma unroll
      for (int d = 0; d < D; d++) {
        mn[d] = Limits<T>::max();
        mx[d] = Limits<T>::lowest();
      }
      for (int i = b + tid; i < e; i += BT)
#pragma unroll
        for (int d = 0; d < D; d++) {
          const T v = X[d][i];
          mn[d] = min(mn[d], v);
          mx[d] = max(mx[d], v);
        }
#pragma unroll
      for (int d = 0; d < D; d++) {
        const U lo = warp_min_ord(ord_t<T>(mn[d])), hi = warp_max_ord(ord_t<T>(mx[d]));
        if (lane == 0) {
          box[wid][d] = lo;
          box[wid][D + d] = hi;
        }
      }
      __syncthreads();
      if (wid == 0) {
        if (lane < 2 * D) {
          U v = box[0][lane];
          for (int w = 1; w < WARPS; w++) v = lane < D ? min(v, box[w][lane]) : max(v, box[w][lane]);
          tight[lane] = from_ord_t<T>(v);
        }
        __syncwarp();
        if (lane == 0) {
          Small<T, D> g = todo[cur];
          Rec<T, D> rec;
          int act = 0, sd = 0;
          T sv = (T)0;
          node_logic<T, D>(e - b, g.n_orig, g.parent < 0, g.lo, g.hi, tight, tight + D, max_leaf, thr, rec, act, sd, sv);
          rec.begin = g.b;
          rec.end = g.e;
          const int id = atomicAdd(&ctl->rec_count, 1);
          if (!link_record<T, D>(rec, id, g.parent, g.side, recs, rec_cap, root_rec, ctl)) act = 0;
          if (nodes >= n) {  // every split leaves fewer points
            atomicExch(&ctl->status, 5);
            act = 0;
          }
          atomicMax(&ctl->depth, g.lvl + 1);
          todo[cur] = g;  // (its extent is trimmed)
          s_act = act;
          s_sd = sd;
          s_sv = sv;
          s_rec = id;
          if (!act) s_todo = cur;
        }
      }
      __syncthreads();
      if (!s_act) continue;
      const T sv = s_sv;
      const T* v = X[0];
#pragma unroll
      for (int d = 1; d < D; d++)
        if (d == s_sd) v = X[d];
      // a bit per point: below the split value
      int c2 = 0;
      for (int w = wid; w < words; w += WARPS) {
        const int q = b + 32 * w + lane;
        const bool in = q < e;
        const T x = in ? v[q] : sv;
        const unsigned m = __ballot_sync(FULL, in && x < sv);
        c2 += __popc(__ballot_sync(FULL, in && x <= sv));
        if (lane == 0) bits[w] = m;
      }
      if (lane == 0) le[wid] = c2;
      __syncthreads();
      const int half = (e - b) / 2;
      int L1, L2 = 0;
      {
        const WordScan scan(bits, words);
        L1 = scan.total;
        for (int w = 0; w < WARPS; w++) L2 += le[w];
        const int zw = L1 >> 5;  // points below the split value among the first L1
        const int first = zw < words ? scan.before(zw) + __popc(bits[zw] & ((1u << (L1 & 31)) - 1u)) : L1;
        for (int w = wid; w < words; w += WARPS) {
          const unsigned m = bits[w];
          const int q = 32 * w + lane, r = scan.before(w) + __popc(m & lt);
          if (m >> lane & 1u) {
            if (q >= L1) S[b + half + r - first] = (uint16_t)(b + q);
          } else if (q < L1) {
            S[b + q - r] = (uint16_t)(b + q);
          }
        }
        swap(b, half, L1 - first);
      }
      if (L1 != L2) {
        // the tie pass: points equal to the split value to [b + L1, b + L2)
        for (int w = wid; w < words; w += WARPS) {
          const int q = 32 * w + lane;
          const T x = b + q < e ? v[b + q] : sv;
          const unsigned m = __ballot_sync(FULL, b + q < e && q >= L1 && (q < L2 ? x > sv : x <= sv));
          if (lane == 0) bits[w] = m;
        }
        __syncthreads();
        const WordScan scan(bits, words);
        const int zw = L2 >> 5;
        const int G = zw < words ? scan.before(zw) + __popc(bits[zw] & ((1u << (L2 & 31)) - 1u)) : scan.total;
        for (int w = wid; w < words; w += WARPS) {
          const unsigned m = bits[w];
          const int q = 32 * w + lane, r = scan.before(w) + __popc(m & lt);
          if (m >> lane & 1u) S[q < L2 ? b + r : b + half + r - G] = (uint16_t)(b + q);
        }
        swap(b, half, G);
      }
      if (tid == 0) {
        const Small<T, D> g = todo[cur];
        const int at = g.b + num_left_rule(L1, L2, e - b);
        recs[s_rec].split_index = at;
        int left = cur;
        for (int side = 0; side < 2; side++) {
          Small<T, D> c = g;
          c.b = side ? at : g.b;
          c.e = side ? g.e : at;
          if (c.b >= c.e) continue;
          c.parent = s_rec;
          c.side = (int16_t)side;
          c.lvl = (int16_t)(g.lvl + 1);
#pragma unroll
          for (int d = 0; d < D; d++)
            if (d == s_sd) (side ? c.lo[d] : c.hi[d]) = sv;
          if (c.e - c.b <= to.small_cap)
            hand_on(c, to, ctl);
          else if (left < TODO)
            todo[left++] = c;
          else
            atomicExch(&ctl->status, 3);
        }
        s_todo = left;
      }
      __syncthreads();
    }
    for (int i = tid; i < n; i += BT) {
#pragma unroll
      for (int d = 0; d < D; d++) soa.x[d][base + i] = X[d][i];
      soa.id[base + i] = ID[i];
    }
  }
}

// ------------------------------------------------- per-warp subtrees ----
// k_subtree nodes of at most this many points are split by one lane each.
constexpr int LANE_NODE = 32;

// Finishes the subtrees of small segments in shared memory, one warp per
// segment, level by level: every node above LANE_NODE points by the whole
// warp (boxes and ranks by warp reductions and ballots, the split decisions of
// all of them side by side), the others by one lane each.  A warp waits for no
// other, so the few nodes of a segment's first levels and the uneven ones of
// its last cost only their own warp.  Persistent: a warp takes segments from
// the list until it is exhausted.
template <typename T, int D>
__global__ void __launch_bounds__(32) k_subtree(const Small<T, D>* small, SoA<T, D> soa, Rec<T, D>* recs, int* root_rec,
                                                int cap_pts, int cap_list, int max_leaf, double thr, int rec_cap,
                                                int small_capn, BuildCtl* ctl) {
  extern __shared__ __align__(16) unsigned char smem[];
  T* X[D];
  unsigned char* p = smem;
#pragma unroll
  for (int d = 0; d < D; d++) {
    X[d] = (T*)p;
    p += sizeof(T) * cap_pts;
  }
  int* ID = (int*)p;
  p += sizeof(int) * cap_pts;
  Entry<T, D>* LA = (Entry<T, D>*)p;
  p += sizeof(Entry<T, D>) * cap_list;
  Entry<T, D>* LB = (Entry<T, D>*)p;
  p += sizeof(Entry<T, D>) * cap_list;
  uint16_t* S = (uint16_t*)p;
  const int lane = threadIdx.x;
  const unsigned FULL = 0xffffffffu;
  const unsigned lt = (1u << lane) - 1u;
  const int nsmall = min(ctl->nsmall, small_capn);

  while (true) {
    int item = 0;
    if (lane == 0) item = atomicAdd(&ctl->small_next, 1);
    item = __shfl_sync(FULL, item, 0);
    if (item >= nsmall) break;
    const Small<T, D> seg = small[item];
    const int n = seg.e - seg.b;
    for (int i = lane; i < n; i += 32) {
#pragma unroll
      for (int d = 0; d < D; d++) X[d][i] = soa.x[d][seg.b + i];
      ID[i] = soa.id[seg.b + i];
    }
    if (lane == 0) {
      Entry<T, D> r;
      r.b = 0;
      r.e = (uint16_t)n;
      r.parent = seg.parent;
      r.side = (uint16_t)seg.side;
#pragma unroll
      for (int d = 0; d < D; d++) {
        r.lo[d] = seg.lo[d];
        r.hi[d] = seg.hi[d];
      }
      LA[0] = r;
    }
    __syncwarp();
    int nA = 1, levels = 0;
    while (nA > 0) {
      if (levels > n + 1) {  // every level splits ranges into strictly smaller ones
        if (lane == 0) atomicExch(&ctl->status, 5);
        break;
      }
      int base = 0;
      if (lane == 0) base = atomicAdd(&ctl->rec_count, nA);
      base = __shfl_sync(FULL, base, 0);
      levels++;
      int nB = 0;
      for (int e0 = 0; e0 < nA; e0 += 32) {
        const int ei = e0 + lane;
        Entry<T, D> en;
        en.b = en.e = 0;
        if (ei < nA) en = LA[ei];
        const int b = en.b, e = en.e, size = e - b;
        const unsigned large = __ballot_sync(FULL, size > LANE_NODE);
        T mn[D], mx[D];
#pragma unroll
        for (int d = 0; d < D; d++) {
          mn[d] = Limits<T>::max();
          mx[d] = Limits<T>::lowest();
        }
        // tight boxes: of a large node by the warp, of a small one by its lane
        for (unsigned rest = large; rest; rest &= rest - 1) {
          const int s = __ffs(rest) - 1;
          const int nb = __shfl_sync(FULL, b, s), ne = __shfl_sync(FULL, e, s);
          T lo[D], hi[D];
#pragma unroll
          for (int d = 0; d < D; d++) {
            lo[d] = Limits<T>::max();
            hi[d] = Limits<T>::lowest();
          }
          for (int q = nb + lane; q < ne; q += 32)
#pragma unroll
            for (int d = 0; d < D; d++) {
              const T v = X[d][q];
              lo[d] = min(lo[d], v);
              hi[d] = max(hi[d], v);
            }
#pragma unroll
          for (int d = 0; d < D; d++) {
            lo[d] = warp_min(lo[d]);
            hi[d] = warp_max(hi[d]);
            if (lane == s) {
              mn[d] = lo[d];
              mx[d] = hi[d];
            }
          }
        }
        const bool tiny = size > 0 && size <= LANE_NODE;
        if (tiny)
          for (int q = b; q < e; q++)
#pragma unroll
            for (int d = 0; d < D; d++) {
              const T v = X[d][q];
              mn[d] = min(mn[d], v);
              mx[d] = max(mx[d], v);
            }
        int act = 0, sd = 0;
        T sv = (T)0;
        const int id = base + ei;
        if (size > 0) {
          Rec<T, D> rec;
          node_logic<T, D>(size, seg.n_orig, en.parent < 0, en.lo, en.hi, mn, mx, max_leaf, thr, rec, act, sd, sv);
          rec.begin = seg.b + b;
          rec.end = seg.b + e;
          if (!link_record<T, D>(rec, id, en.parent, en.side, recs, rec_cap, root_rec, ctl)) act = 0;
        }
        int L1 = 0, L2 = 0;
        // partition of the large nodes, by the warp
        for (unsigned rest = __ballot_sync(FULL, size > LANE_NODE && act); rest; rest &= rest - 1) {
          const int s = __ffs(rest) - 1;
          const int nb = __shfl_sync(FULL, b, s), ne = __shfl_sync(FULL, e, s), nd = __shfl_sync(FULL, sd, s);
          const T nv = __shfl_sync(FULL, sv, s);
          const T* v = X[0];
#pragma unroll
          for (int d = 1; d < D; d++)
            if (d == nd) v = X[d];
          // bits of the points below the split value: word w is lane w's
          // (cap_pts <= 1024)
          unsigned word = 0;
          int c1 = 0, c2 = 0;
          for (int q0 = nb, w = 0; q0 < ne; q0 += 32, w++) {
            const int q = q0 + lane;
            const bool in = q < ne;
            const T x = in ? v[q] : nv;
            const unsigned m = __ballot_sync(FULL, in && x < nv);
            c1 += __popc(m);
            c2 += __popc(__ballot_sync(FULL, in && x <= nv));
            if (lane == w) word = m;
          }
          // pass 1: misplaced points ranked from the bits, then swapped
          const int half = (ne - nb) / 2;
          {
            const int Z = nb + c1;
            int G = 0, a = 0;
            for (int q0 = nb, w = 0; q0 < ne; q0 += 32, w++) {
              const int q = q0 + lane;
              const bool below = __shfl_sync(FULL, word, w) >> lane & 1u;
              const unsigned bl = __ballot_sync(FULL, q < Z && !below), gr = __ballot_sync(FULL, q >= Z && below);
              if (bl >> lane & 1u) {
                const int r = G + __popc(bl & lt);
                if (r < half) S[nb + r] = (uint16_t)q;
              }
              if (gr >> lane & 1u) {
                const int r = a + __popc(gr & lt);
                if (r < half) S[nb + half + r] = (uint16_t)q;
              }
              G += __popc(bl);
              a += __popc(gr);
            }
            if ((a != G || G > half) && lane == 0) atomicExch(&ctl->status, 2);
            __syncwarp();
            if (a == G && G <= half)
              for (int j = lane; j < G; j += 32) {
                const int x = S[nb + j], y = S[nb + half + G - 1 - j];
#pragma unroll
                for (int d = 0; d < D; d++) {
                  const T t = X[d][x];
                  X[d][x] = X[d][y];
                  X[d][y] = t;
                }
                const int t = ID[x];
                ID[x] = ID[y];
                ID[y] = t;
              }
            __syncwarp();
          }
          if (c1 != c2) {
            // pass 2: points equal to the split value to [c1, c2)
            const int Z = nb + c2;
            int G = 0, a = 0;
            for (int q0 = nb + c1; q0 < ne; q0 += 32) {
              const int q = q0 + lane;
              const T x = q < ne ? v[q] : nv;
              const unsigned bl = __ballot_sync(FULL, q < Z && x > nv);
              const unsigned gr = __ballot_sync(FULL, q < ne && q >= Z && x <= nv);
              if (bl >> lane & 1u) {
                const int r = G + __popc(bl & lt);
                if (r < half) S[nb + r] = (uint16_t)q;
              }
              if (gr >> lane & 1u) {
                const int r = a + __popc(gr & lt);
                if (r < half) S[nb + half + r] = (uint16_t)q;
              }
              G += __popc(bl);
              a += __popc(gr);
            }
            if ((a != G || G > half) && lane == 0) atomicExch(&ctl->status, 2);
            __syncwarp();
            if (a == G && G <= half)
              for (int j = lane; j < G; j += 32) {
                const int x = S[nb + j], y = S[nb + half + G - 1 - j];
#pragma unroll
                for (int d = 0; d < D; d++) {
                  const T t = X[d][x];
                  X[d][x] = X[d][y];
                  X[d][y] = t;
                }
                const int t = ID[x];
                ID[x] = ID[y];
                ID[y] = t;
              }
            __syncwarp();
          }
          if (lane == s) {
            L1 = c1;
            L2 = c2;
          }
        }
        // partition of a small node by its lane, with the reference's two
        // converging cursors (the pairs a warp forms by ranks)
        if (tiny && act) {
          const T* v = X[0];
#pragma unroll
          for (int d = 1; d < D; d++)
            if (d == sd) v = X[d];
          for (int q = b; q < e; q++) {
            const T x = v[q];
            L1 += x < sv;
            L2 += x <= sv;
          }
          for (int pass = 1; pass <= (L1 == L2 ? 1 : 2); pass++) {
            const int Z = pass == 1 ? b + L1 : b + L2;
            int i = pass == 1 ? b : b + L1, j = e - 1;
            while (true) {
              while (i < Z && !(pass == 1 ? !(v[i] < sv) : (v[i] > sv))) i++;
              while (j >= Z && !(pass == 1 ? (v[j] < sv) : (v[j] <= sv))) j--;
              if (i >= Z || j < Z) break;
#pragma unroll
              for (int d = 0; d < D; d++) {
                const T t = X[d][i];
                X[d][i] = X[d][j];
                X[d][j] = t;
              }
              const int t = ID[i];
              ID[i] = ID[j];
              ID[j] = t;
              i++;
              j--;
            }
          }
        }
        // children, in the order of their parents
        const int si = b + (act ? num_left_rule(L1, L2, size) : 0);
        const bool left = act && si > b, right = act && si < e;
        if (act) recs[id].split_index = seg.b + si;
        const unsigned ml = __ballot_sync(FULL, left), mr = __ballot_sync(FULL, right);
        const int more = __popc(ml) + __popc(mr);
        if (nB + more > cap_list) {
          if (lane == 0) atomicExch(&ctl->status, 3);
          nB = 0;
          e0 = nA;  // (reported; the segment ends here)
          continue;
        }
        int slot = nB + __popc(ml & lt) + __popc(mr & lt);
        Entry<T, D> c;
        c.b = (uint16_t)b;
        c.e = (uint16_t)si;
        c.parent = id;
        c.side = 0;
        if (left) {
#pragma unroll
          for (int d = 0; d < D; d++) {
            c.lo[d] = en.lo[d];
            c.hi[d] = d == sd ? sv : en.hi[d];
          }
          LB[slot++] = c;
        }
        if (right) {
          c.b = (uint16_t)si;
          c.e = (uint16_t)e;
          c.side = 1;
#pragma unroll
          for (int d = 0; d < D; d++) {
            c.lo[d] = d == sd ? sv : en.lo[d];
            c.hi[d] = en.hi[d];
          }
          LB[slot] = c;
        }
        nB += more;
      }
      __syncwarp();
      nA = nB;
      Entry<T, D>* tmp = LA;
      LA = LB;
      LB = tmp;
    }
    __syncwarp();
    for (int i = lane; i < n; i += 32) {
#pragma unroll
      for (int d = 0; d < D; d++) soa.x[d][seg.b + i] = X[d][i];
      soa.id[seg.b + i] = ID[i];
    }
    if (lane == 0) atomicMax(&ctl->depth, seg.lvl + levels);
    __syncwarp();
  }
}

// ------------------------------------------------------- finishing ----
template <typename T, int D>
__global__ void k_finish(SoA<T, D> soa, int nv, PointRec<T, D>* pts, int* fwd, int* ids,
                         const int64_t* nv_dev = nullptr) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (nv_dev) nv = (int)*nv_dev;  // capture mode: the valid count is on the device
  if (i >= nv) return;
  PointRec<T, D> r;
#pragma unroll
  for (int d = 0; d < D; d++) r.c[d] = soa.x[d][i];
  r.id = soa.id[i];
  pts[i] = r;
  ids[i] = r.id;
  fwd[r.id] = i;
}

template <typename T, int D>
__global__ void k_tflag(const Rec<T, D>* recs, int n_recs, int bucket, int* flag, const int* n_dev = nullptr) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_recs) return;
  if (n_dev && i >= *n_dev) {  // capture mode: records beyond the live count
    flag[i] = 0;
    return;
  }
  const Rec<T, D>& r = recs[i];
  flag[i] = (r.split_dim >= 0 && r.end - r.begin > bucket && r.left >= 0 && r.right >= 0) ? 1 : 0;
}

template <typename T, int D>
__global__ void k_tfill(const Rec<T, D>* recs, int n_recs, const int* flag, const int* tid, TNode<T, D>* nodes,
                        const int* n_dev = nullptr, int node_lim = INT_MAX, int* status = nullptr) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_recs || (n_dev && i >= *n_dev) || !flag[i]) return;
  // capture mode: nodes beyond the capacity are left out (their parents
  // see them as buckets: the walks stay exact) and reported
  if (tid[i] >= node_lim) {
    atomicExch(status, 21);
    return;
  }
  const Rec<T, D>& r = recs[i];
  TNode<T, D> t;
  for (int c = 0; c < 2; c++) {
    int ch = c ? r.right : r.left;
    const Rec<T, D>& cr = recs[ch];
    for (int d = 0; d < D; d++) {
      t.lo[c][d] = cr.lo[d];
      t.hi[c][d] = cr.hi[d];
    }
    t.cnt[c] = cr.end - cr.begin;
    t.ref[c] = (flag[ch] && tid[ch] < node_lim) ? tid[ch] : -cr.begin - 1;
  }
  nodes[tid[i]] = t;
}

// Per-cloud traversal roots: the root record's node when it is an inner
// node, otherwise a dedicated node (index nt + c) whose first child is the
// whole cloud as one bucket (or nothing, for a cloud without valid points).
template <typename T, int D>
__global__ void k_troots(const Rec<T, D>* recs, const int* root_rec, const int64_t* valid_off, int ncloud,
                         const int* flag, const int* tid, int nt, TNode<T, D>* nodes, int* root_tnode,
                         double* box = nullptr) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncloud) return;
  const int r = root_rec[c];
  if (box && c == 0)  // the first cloud's box
    for (int d = 0; d < D; d++) {
      box[d] = r >= 0 ? (double)recs[r].lo[d] : 0.0;
      box[4 + d] = r >= 0 ? (double)recs[r].hi[d] : 0.0;
    }
  TNode<T, D> t;
  for (int k = 0; k < 2; k++)
    for (int d = 0; d < D; d++) {
      t.lo[k][d] = Limits<T>::max();
      t.hi[k][d] = Limits<T>::lowest();
    }
  t.ref[0] = t.ref[1] = -1;
  t.cnt[0] = t.cnt[1] = 0;
  if (r >= 0 && flag[r] && tid[r] < nt) {
    // the root record has its own node; the reserved slot stays an empty
    // node (nothing refers to it, but every slot holds a well-formed node)
    nodes[nt + c] = t;
    root_tnode[c] = tid[r];
    return;
  }
  if (r >= 0) {
    for (int d = 0; d < D; d++) {
      t.lo[0][d] = recs[r].lo[d];
      t.hi[0][d] = recs[r].hi[d];
    }
    t.ref[0] = -(int)valid_off[c] - 1;
    t.cnt[0] = (int)(valid_off[c + 1] - valid_off[c]);
  }
  nodes[nt + c] = t;
  root_tnode[c] = nt + c;
}

// --------------------------------------------------- wide hierarchy ----
// Type of the traversal data of a tree of point type T (integer trees walk
// in float).
template <typename T>
struct WalkOf {
  typedef typename std::conditional<std::is_integral<T>::value, float, T>::type type;
};

// A record that a level of nodes of at most `cap` points divides.
template <typename T, int D>
__device__ __forceinline__ bool wide_inner(const Rec<T, D>& r, long long cap) {
  return r.split_dim >= 0 && r.end - r.begin > cap && r.left >= 0 && r.right >= 0;
}

// The record that decides record r's range: r itself, or, below a record
// with one child over the same points, that child (the bound only stops a
// damaged file's cycle).
template <typename T, int D>
__device__ __forceinline__ int wide_resolve(const Rec<T, D>* recs, int r, long long cap) {
  for (int guard = 0; guard < 4096; guard++) {
    const Rec<T, D>& x = recs[r];
    if (x.split_dim < 0 || x.end - x.begin <= cap || (x.left >= 0) == (x.right >= 0)) break;
    r = x.left >= 0 ? x.left : x.right;
  }
  return r;
}

// Where the nodes of every level begin: at a cloud's first point and at the
// right child of a record that the level divides.
template <typename T, int D>
__global__ void k_wide_mark(const Rec<T, D>* recs, int n_recs, int bucket, int levels, int words,
                            const int64_t* valid_off, int ncloud, uint32_t* bits, const int* n_dev = nullptr) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < ncloud && valid_off[i + 1] > valid_off[i]) {
    const int b = (int)valid_off[i];
    for (int j = 0; j < levels; j++) atomicOr(&bits[j * words + (b >> 5)], 1u << (b & 31));
  }
  if (i >= n_recs || (n_dev && i >= *n_dev)) return;
  const Rec<T, D>& r = recs[i];
  for (int j = 0; j < levels && wide_inner(r, wide_cap(bucket, j)); j++) {
    const int b = recs[r.right].begin;
    atomicOr(&bits[j * words + (b >> 5)], 1u << (b & 31));
  }
}

// A word of the node map as its number of nodes, for the scan.
struct NodeWord {
  uint32_t bits;
  __device__ explicit operator int64_t() const { return __popc(bits); }
};

struct WideMap {
  const uint32_t* bits;
  const int* rank;
  int words, levels, cap;
  __device__ __forceinline__ int of(int j, int p) const {
    const int w = j * words + (p >> 5);
    return rank[w] + __popc(bits[w] & (0xffffffffu >> (31 - (p & 31)))) - 1;
  }
  __device__ __forceinline__ bool starts(int j, int p) const { return bits[j * words + (p >> 5)] >> (p & 31) & 1u; }
};

// Record r as a node of level j.  A record that no node begins at (a damaged
// file's) is left out; one beyond the capacity (a rebuild that needs more) is
// reported, and children beyond it are cut off.
template <typename T, int D>
__device__ __forceinline__ void wide_write(const Rec<T, D>& r, int j, const WideMap& m,
                                           WNode<typename WalkOf<T>::type, D>* nodes, int2* span, int* status) {
  typedef typename WalkOf<T>::type V;
  if (r.end <= r.begin || !m.starts(j, r.begin)) return;
  const int i = m.of(j, r.begin);
  if (i >= m.cap) {
    if (status) atomicExch(status, 21);
    return;
  }
  WNode<V, D> w;
#pragma unroll
  for (int d = 0; d < D; d++) {
    w.lo[d] = (V)r.lo[d];
    w.hi[d] = (V)r.hi[d];
  }
  w.begin = r.begin;
  w.cnt = r.end - r.begin;
  if (j > 0) {
    w.begin = m.of(j - 1, r.begin);
    w.cnt = -max(min(m.of(j - 1, r.end - 1) + 1, i) - w.begin, 0);
  }
  nodes[i] = w;
  span[i] = make_int2(r.begin, r.end - r.begin);
}

template <typename T, int D>
__global__ void k_wide_fill(const Rec<T, D>* recs, int n_recs, int bucket, const int* root_rec, int ncloud, WideMap m,
                            WNode<typename WalkOf<T>::type, D>* nodes, int2* span, const int* n_dev = nullptr,
                            int* status = nullptr) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < ncloud && root_rec[i] >= 0)
    for (int j = m.levels - 1; j >= 0; j--) {
      const int r = wide_resolve(recs, root_rec[i], wide_cap(bucket, j));
      if (wide_inner(recs[r], wide_cap(bucket, j))) break;
      wide_write<T, D>(recs[r], j, m, nodes, span, status);
    }
  if (i >= n_recs || (n_dev && i >= *n_dev)) return;
  for (int j = 0; j < m.levels && wide_inner(recs[i], wide_cap(bucket, j)); j++)
    for (int c = 0; c < 2; c++) {
      const int r = wide_resolve(recs, c ? recs[i].right : recs[i].left, wide_cap(bucket, j));
      if (!wide_inner(recs[r], wide_cap(bucket, j))) wide_write<T, D>(recs[r], j, m, nodes, span, status);
    }
}

// Marks and ranks the nodes (on a capture-ready forest over the live
// records, n_dev); wrank's last entry receives their number.
template <typename T, int D>
void wide_begin(TreeBase* t, int n_recs, cudaStream_t st, const int* n_dev = nullptr) {
  int64_t most = 1;  // points of the largest cloud
  for (int c = 0; c < t->ncloud; c++)
    most = std::max(most, t->capture ? t->orig_off_h[c + 1] - t->orig_off_h[c] : t->valid_off_h[c + 1] - t->valid_off_h[c]);
  const int levels = wide_levels(t->bucket, most);
  const int64_t words = wide_words(t->capture ? t->n : t->nv);
  if (!t->wbits || !t->wrank || t->wlevels != levels || t->wwords != (int)words) {
    if (t->wbits) dev_free(t->wbits, st);
    if (t->wrank) dev_free(t->wrank, st);
    t->wbits = nullptr;
    t->wrank = nullptr;
    t->wlevels = levels;
    t->wwords = (int)words;
    PPTKG_CUDA(dev_malloc((void**)&t->wbits, sizeof(uint32_t) * levels * words, st));
    PPTKG_CUDA(dev_malloc((void**)&t->wrank, sizeof(int) * (levels * words + 1), st));
  }
  PPTKG_CUDA(cudaMemsetAsync(t->wbits, 0, sizeof(uint32_t) * levels * words, st));
  k_wide_mark<T, D><<<div_up(std::max(n_recs, t->ncloud), 256), 256, 0, st>>>(
      (const Rec<T, D>*)t->recs, n_recs, t->bucket, levels, (int)words, t->valid_off, t->ncloud, t->wbits, n_dev);
  PPTKG_CHECK_LAUNCH();
  exclusive_scan<NodeWord, int>((const NodeWord*)t->wbits, t->wrank, levels * words, t->wrank + levels * words, st);
}

// Wide nodes that a rebuild within the capacities of records and traversal
// nodes can have: on every level one per cloud and one more per record that
// the level divides.  Those have two children, as half of all records have at
// most; above the first level they are of more than `bucket` points and so are
// traversal nodes.
static int wide_capacity(const TreeBase* t) {
  return (int)std::min<int64_t>(INT32_MAX / 2, t->cap_recs / 2 + t->ncloud + (t->wlevels - 1) * t->cap_tnodes);
}

template <typename T, int D>
void wide_alloc(TreeBase* t, int n_wide, cudaStream_t st) {
  if (t->wide) dev_free(t->wide, st);
  if (t->wspan) dev_free(t->wspan, st);
  t->wide = nullptr;
  t->wspan = nullptr;
  t->n_wide = n_wide;
  PPTKG_CUDA(dev_malloc(&t->wide, (size_t)std::max(n_wide, 1) * sizeof(WNode<typename WalkOf<T>::type, D>), st));
  PPTKG_CUDA(dev_malloc((void**)&t->wspan, (size_t)std::max(n_wide, 1) * sizeof(int2), st));
}

// Fills the nodes; `clear`: entries that no record fills hold nothing.
template <typename T, int D>
void wide_fill(TreeBase* t, int n_recs, bool clear, cudaStream_t st, const int* n_dev = nullptr,
               int* status = nullptr) {
  typedef WNode<typename WalkOf<T>::type, D> Node;
  if (t->n_wide <= 0) return;
  if (clear) {
    PPTKG_CUDA(cudaMemsetAsync(t->wide, 0, sizeof(Node) * (size_t)t->n_wide, st));
    PPTKG_CUDA(cudaMemsetAsync(t->wspan, 0, sizeof(int2) * (size_t)t->n_wide, st));
  }
  const WideMap m{t->wbits, t->wrank, t->wwords, t->wlevels, t->n_wide};
  k_wide_fill<T, D><<<div_up(std::max(n_recs, t->ncloud), 256), 256, 0, st>>>(
      (const Rec<T, D>*)t->recs, n_recs, t->bucket, t->root_rec, t->ncloud, m, (Node*)t->wide, t->wspan,
      n_dev, status);
  PPTKG_CHECK_LAUNCH();
}

template <typename V, int D>
__global__ void k_ids(const PointRec<V, D>* pts, int64_t nv, int* ids) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nv) ids[i] = pts[i].id;
}

template <typename T, int D>
void make_wide(TreeBase* t, cudaStream_t st) {
  int n = 0;
  if (!t->ids) {
    typedef typename WalkOf<T>::type V;
    PPTKG_CUDA(dev_malloc((void**)&t->ids, std::max<int64_t>(t->nv, 1) * sizeof(int), st));
    if (t->nv > 0) {
      k_ids<V, D><<<div_up(t->nv, 256), 256, 0, st>>>((const PointRec<V, D>*)t->pts, t->nv, t->ids);
      PPTKG_CHECK_LAUNCH();
    }
  }
  wide_begin<T, D>(t, t->n_recs, st);
  PPTKG_CUDA(cudaMemcpyAsync(&n, t->wrank + (int64_t)t->wlevels * t->wwords, sizeof(int), cudaMemcpyDeviceToHost, st));
  PPTKG_CUDA(cudaStreamSynchronize(st));
  wide_alloc<T, D>(t, n, st);
  wide_fill<T, D>(t, t->n_recs, true, st);
  PPTKG_CUDA(cudaStreamSynchronize(st));
  t->walkable = true;
}

// ------------------------------------------------------------ host side ----
// Points of the largest segment that k_block takes; larger ones go through
// grid-wide levels.  The levels planned for rebuilds count those: this size
// decides which trees a capture-ready forest takes, so it does not follow
// k_block's needs (2,048 float points are 37 KB of shared memory, six blocks
// per SM).  Fewer where leaves of one to three points make more records.
template <typename T, int D>
int mid_capacity(int max_leaf) {
  int cap = sizeof(T) == 4 ? 2048 : 1024;
  while (cap > 64 && (sizeof(T) * D + 8) * (size_t)cap + 4 * (8 + sizeof(T) * D) * (size_t)(2 * (cap / (max_leaf + 1)) + 2) > 72 * 1024 - 48)
    cap /= 2;
  return cap;
}

template <typename T, int D>
constexpr size_t block_smem(int cap) {
  return (sizeof(T) * D + sizeof(int) + sizeof(uint16_t)) * (size_t)cap;
}

// k_block's grid: the blocks that the shared memory of a device's SMs holds.
static int block_grid(size_t smem, int device) {
  int per_sm = 228 * 1024;
  PPTKG_CUDA(cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device));
  return sm_count(device) * std::max(1, std::min(8, (int)(per_sm / (smem + 3 * 1024))));
}

// Grid of the grid-stride level kernels: eight 256-thread blocks per SM.
static int level_grid(int device) { return sm_count(device) * 8; }

// Points of the largest segment that k_subtree takes, its list capacity and
// its shared memory: 512 float points and their lists take 15 KB, so 14 warps
// share an SM.  (1,024 points: one level less, but 128 us in place of 80 for
// the six segments of a 3,001-point cloud.)
template <typename T, int D>
int small_capacity(int max_leaf, int& cap_list, size_t& smem) {
  int cap = sizeof(T) <= 4 ? 512 : 256;
  while (true) {
    cap_list = 2 * (cap / (max_leaf + 1)) + 2;
    smem = (sizeof(T) * D + sizeof(int) + sizeof(uint16_t)) * (size_t)cap + 2 * sizeof(Entry<T, D>) * (size_t)cap_list;
    if ((smem <= 24 * 1024 && cap <= mid_capacity<T, D>(max_leaf)) || cap <= 64) break;
    cap /= 2;
  }
  return cap;
}

// ------------------------------------------------ integer point types ----
// The reference computes every distance of an integer tree in float
// (Accumulator, accumulator.h:16-19): each coordinate and box bound is
// converted to float where it is read (kdtree-impl.h:331-339, box.h:157-198).
// After the build (done exactly in T), the tree-ordered points and the
// traversal boxes are stored as those float values, so the float query
// kernels answer integer trees; the records stay in T.
template <typename T, int D>
__global__ void k_lower_points(const PointRec<T, D>* in, int64_t nv, PointRec<float, D>* out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv) return;
  PointRec<float, D> r;
#pragma unroll
  for (int d = 0; d < D; d++) r.c[d] = (float)in[i].c[d];
  r.id = in[i].id;
  out[i] = r;
}

template <typename T, int D>
__global__ void k_lower_tnodes(const TNode<T, D>* in, int n, TNode<float, D>* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  TNode<float, D> t;
#pragma unroll
  for (int k = 0; k < 2; k++) {
#pragma unroll
    for (int d = 0; d < D; d++) {
      t.lo[k][d] = (float)in[i].lo[k][d];
      t.hi[k][d] = (float)in[i].hi[k][d];
    }
    t.ref[k] = in[i].ref[k];
    t.cnt[k] = in[i].cnt[k];
  }
  out[i] = t;
}

template <typename T, int D>
void lower_points(TreeBase* tree, cudaStream_t st) {
  PointRec<float, D>* out = nullptr;
  PPTKG_CUDA(dev_malloc((void**)&out, std::max<int64_t>(tree->nv, 1) * sizeof(PointRec<float, D>), st));
  if (tree->nv > 0) {
    k_lower_points<T, D><<<(unsigned)((tree->nv + 255) / 256), 256, 0, st>>>((const PointRec<T, D>*)tree->pts,
                                                                             tree->nv, out);
    PPTKG_CHECK_LAUNCH();
  }
  dev_free(tree->pts, st);
  tree->pts = out;
  tree->dtype = F32;
}

template <typename T, int D>
void lower_tnodes(TreeBase* tree, cudaStream_t st) {
  TNode<float, D>* out = nullptr;
  const int n = tree->n_tnodes;
  PPTKG_CUDA(dev_malloc((void**)&out, std::max(n, 1) * sizeof(TNode<float, D>), st));
  if (n > 0) {
    k_lower_tnodes<T, D><<<(unsigned)((n + 255) / 256), 256, 0, st>>>((const TNode<T, D>*)tree->tnodes, n, out);
    PPTKG_CHECK_LAUNCH();
  }
  dev_free(tree->tnodes, st);
  tree->tnodes = out;
}

// k_subtree's grid: the warps that the shared memory of a device's SMs holds
// (its dynamic part stays below the 48 KB that need no opt-in).
static int subtree_grid(size_t smem, int device) {
  int per_sm = 228 * 1024;
  PPTKG_CUDA(cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device));
  return sm_count(device) * std::max(1, std::min(32, (int)(per_sm / (smem + 1024))));
}

// Segments above small_capacity() points that n points can have at a time.
template <typename T, int D>
int mid_segments(int64_t n, int max_leaf) {
  int cap_list;
  size_t smem;
  return (int)(n / (small_capacity<T, D>(max_leaf, cap_list, smem) + 1) + 2);
}

// A stretch of a scratch block, handed out piece by piece (base null: only
// measured).
struct Carve {
  char* base;
  size_t at = 0;
  template <typename V>
  V* take(size_t n) {
    V* p = base ? reinterpret_cast<V*>(base + at) : nullptr;
    at += (n * sizeof(V) + 255) & ~(size_t)255;
    return p;
  }
};

// Scratch of a build's levels, one block of device memory (an allocation of
// its own for each of the eleven arrays took 30 us of a small build), and the
// launches of one level.
template <typename T, int D>
struct Levels {
  BuildBuf<char> block;
  Seg<T, D>* seg[2];
  Lists<T, D> lists;
  int cap_list;  // of k_subtree's node lists
  size_t smem;   // its shared memory
  int *blpos, *grpos, *tile_seg, *tile_lt;
  uint32_t* bits;
  long long *tile_cnt, *tile_off;
  unsigned gt, gq, gs;
  int tile, device;
  BuildCtl* ctl;
  SoA<T, D> soa;
  Rec<T, D>* recs;
  int rec_cap;
  int* root_rec;
  int max_leaf;
  double thr;
  cudaStream_t st;

  void carve(Carve c, int64_t n, int max_tiles, int seg_cap, size_t* bytes) {
    ctl = c.take<BuildCtl>(1);
    for (auto& x : seg) x = c.take<Seg<T, D>>(seg_cap);
    lists.mid = c.take<Small<T, D>>(lists.mid_capn);
    lists.small = c.take<Small<T, D>>(lists.small_capn);
    blpos = c.take<int>(n + 1);
    grpos = c.take<int>(n + 1);
    tile_seg = c.take<int>(max_tiles);
    tile_lt = c.take<int>(max_tiles);
    bits = c.take<uint32_t>((size_t)max_tiles * (tile / 32));
    tile_cnt = c.take<long long>(max_tiles);
    tile_off = c.take<long long>(max_tiles);
    if (bytes) *bytes = c.at;
  }
  // Of a build of at most n points of tree `t` (of n_in input rows).
  Levels(const TreeBase* t, int64_t n, int64_t n_in, int small_capn, SoA<T, D> soa_, Rec<T, D>* recs_, int rec_cap_,
         cudaStream_t st_)
      : tile(tile_points(n_in)), device(t->device), soa(soa_), recs(recs_), rec_cap(rec_cap_), root_rec(t->root_rec),
        max_leaf(t->max_leaf), thr(t->empty_split), st(st_) {
    lists.mid_cap = mid_capacity<T, D>(max_leaf);
    lists.small_cap = small_capacity<T, D>(max_leaf, cap_list, smem);
    // segments of a list or level are disjoint
    lists.mid_capn = mid_segments<T, D>(n, max_leaf);
    lists.small_capn = small_capn;
    const int seg_cap = (int)(n / (lists.mid_cap + 1) + 2);
    const int max_tiles = (int)(n / tile) + seg_cap + 2;
    gt = (unsigned)std::min(max_tiles, level_grid(device));
    gq = (unsigned)std::min(seg_cap, level_grid(device));
    gs = (unsigned)div_up(seg_cap, 128);
    size_t bytes = 0;
    carve(Carve{nullptr}, n, max_tiles, seg_cap, &bytes);
    block.alloc(bytes, st);
    carve(Carve{block.get()}, n, max_tiles, seg_cap, nullptr);
    PPTKG_CUDA(cudaMemsetAsync(ctl, 0, sizeof(BuildCtl), st));
  }
  void roots(const int64_t* valid_off, const int64_t* orig_off, int ncloud) {
    k_roots<T, D><<<div_up(ncloud, 128), 128, 0, st>>>(valid_off, orig_off, ncloud, tile, seg[0], lists, ctl);
    PPTKG_CHECK_LAUNCH();
  }
  // What the grid-wide levels leave, in a cloud of up to `most` points.
  void finish(int64_t most) {
    if (most > lists.small_cap) {
      const size_t bytes = block_smem<T, D>(lists.mid_cap);
      k_block<T, D><<<std::min(lists.mid_capn, block_grid(bytes, device)), BT, bytes, st>>>(
          soa, recs, rec_cap, root_rec, lists, max_leaf, thr, ctl);
      PPTKG_CHECK_LAUNCH();
    }
    k_subtree<T, D><<<std::max(1, std::min(lists.small_capn, subtree_grid(smem, device))), 32, smem, st>>>(
        lists.small, soa, recs, root_rec, lists.small_cap, cap_list, max_leaf, thr, rec_cap, lists.small_capn, ctl);
    PPTKG_CHECK_LAUNCH();
  }

  // Boxes (where its segments' may be unknown: the roots', and those below a
  // large segment's split that ties moved), split values and pass 1 of level
  // lvl.
  void split(Seg<T, D>* A, int lvl, bool boxes) {
    if (lvl == 0) {
      k_tiles<T, D><<<gq, 128, 0, st>>>(A, lvl, tile_seg, ctl);
      PPTKG_CHECK_LAUNCH();
    }
    if (boxes) {
      k_bbox<T, D><<<gt, BT, 0, st>>>(A, lvl, tile_seg, ctl, soa);
      PPTKG_CHECK_LAUNCH();
      k_node<T, D><<<gs, 128, 0, st>>>(A, lvl, ctl, recs, rec_cap, root_rec, max_leaf, thr);
      PPTKG_CHECK_LAUNCH();
    }
    k_split<T, D><<<gt, BT, 0, st>>>(A, lvl, tile_seg, ctl, soa, tile_lt, bits);
    PPTKG_CHECK_LAUNCH();
    k_ranks<T, D><<<gq, 256, 0, st>>>(A, lvl, tile_lt, bits, tile_off, ctl);
    PPTKG_CHECK_LAUNCH();
    k_place_ranks<T, D><<<gt, BT, 0, st>>>(A, lvl, tile_seg, ctl, bits, tile_off, blpos,
                                           grpos);
    PPTKG_CHECK_LAUNCH();
    k_swap<T, D><<<gt, BT, 0, st>>>(A, lvl, false, tile_seg, ctl, soa, blpos, grpos);
    PPTKG_CHECK_LAUNCH();
  }
  // The tie pass: of small segments (tied 1), of all (2).
  void tie_pass(Seg<T, D>* A, int lvl, int tied) {
    if (tied < 1) return;
    k_ties<T, D><<<gq, BT, 0, st>>>(A, lvl, ctl, soa, blpos, grpos);
    PPTKG_CHECK_LAUNCH();
    if (tied < 2) return;
    k_flags<T, D><<<gt, BT, 0, st>>>(A, lvl, tile_seg, ctl, soa, tile_cnt);
    PPTKG_CHECK_LAUNCH();
    k_tscan<T, D><<<gq, 256, 0, st>>>(A, lvl, tile_cnt, tile_off, ctl);
    PPTKG_CHECK_LAUNCH();
    k_scatter<T, D><<<gt, BT, 0, st>>>(A, lvl, tile_seg, ctl, soa, tile_off, blpos, grpos);
    PPTKG_CHECK_LAUNCH();
    k_swap<T, D><<<gt, BT, 0, st>>>(A, lvl, true, tile_seg, ctl, soa, blpos, grpos);
    PPTKG_CHECK_LAUNCH();
  }
  void children(Seg<T, D>* A, int lvl, int tied, Seg<T, D>* B) {
    k_children<T, D><<<2 * gs, 128, 0, st>>>(A, lvl, tied, recs, rec_cap, B, lists, max_leaf, thr, tile_seg, ctl);
    PPTKG_CHECK_LAUNCH();
  }
};

template <typename T, int D>
TreeBase* build_forest(const T* d_in, int64_t n, const int64_t* orig_off_h, int ncloud, int max_leaf, double thr,
                       int bucket, cudaStream_t st) {
  if (n > (int64_t)INT32_MAX / 2 - 64) throw Error(E_INVALID, "k-d tree supports at most 2^30 points");
  if (ncloud < 1) throw Error(E_INVALID, "at least one cloud");
  if (max_leaf < 1) max_leaf = 1;
  Stage stage("build", st);
  keep_pool_cached(st);
  std::unique_ptr<TreeBase> tree(new TreeBase());
  tree->stream = st;
  tree->dtype = std::is_same<T, double>::value ? F64 : F32;
  tree->rec_dtype = dtype_code<T>();
  tree->dim = D;
  tree->n = n;
  tree->max_leaf = max_leaf;
  tree->empty_split = thr;
  tree->bucket = bucket;
  tree->ncloud = ncloud;
  PPTKG_CUDA(cudaGetDevice(&tree->device));
  tree->orig_off_h.assign(orig_off_h, orig_off_h + ncloud + 1);
  if (tree->orig_off_h[0] != 0 || tree->orig_off_h[ncloud] != n)
    throw Error(E_INVALID, "cloud offsets must start at 0 and end at n");
  for (int c = 0; c < ncloud; c++)
    if (tree->orig_off_h[c + 1] < tree->orig_off_h[c]) throw Error(E_INVALID, "cloud offsets must not decrease");
  PPTKG_CUDA(dev_malloc((void**)&tree->orig_off, sizeof(int64_t) * (ncloud + 1), st));
  PPTKG_CUDA(dev_malloc((void**)&tree->valid_off, sizeof(int64_t) * (ncloud + 1), st));
  PPTKG_CUDA(dev_malloc((void**)&tree->root_rec, sizeof(int) * ncloud, st));
  PPTKG_CUDA(dev_malloc((void**)&tree->root_tnode, sizeof(int) * ncloud, st));
  PPTKG_CUDA(cudaMemcpyAsync(tree->orig_off, orig_off_h, sizeof(int64_t) * (ncloud + 1), cudaMemcpyHostToDevice, st));
  PPTKG_CUDA(cudaMemsetAsync(tree->root_rec, 0xff, sizeof(int) * ncloud, st));

  // valid-point compaction (ValidPointIndices, kdtree-impl.h:53-75), per cloud
  std::unique_ptr<Stage> st_prep(new Stage("build.prep", st));
  BuildBuf<int> flag, off;
  auto find_valid = [&]() {
    flag.alloc(n + 1, st);
    off.alloc(n + 1, st);
    if (n > 0) {
      k_valid<T, D><<<div_up(n, 256), 256, 0, st>>>(d_in, n, flag.get());
      PPTKG_CHECK_LAUNCH();
    }
    exclusive_scan<int, int>(flag.get(), off.get(), n, off.get() + n, st);
  };
  find_valid();
  k_cloud_off<<<div_up(ncloud + 1, 256), 256, 0, st>>>(off.get(), tree->orig_off, ncloud, tree->valid_off);
  PPTKG_CHECK_LAUNCH();
  tree->valid_off_h.resize(ncloud + 1);
  PPTKG_CUDA(cudaMemcpyAsync(tree->valid_off_h.data(), tree->valid_off, sizeof(int64_t) * (ncloud + 1),
                             cudaMemcpyDeviceToHost, st));
  PPTKG_CUDA(cudaStreamSynchronize(st));
  const int nv = (int)tree->valid_off_h[ncloud];
  tree->nv = nv;

  BuildBuf<T> xs((size_t)D * nv + 1, st);
  BuildBuf<int> ids(nv + 1, st);
  SoA<T, D> soa;
  for (int d = 0; d < D; d++) soa.x[d] = xs.get() + (size_t)d * nv;
  soa.id = ids.get();
  auto take_points = [&]() {
    if (n > 0) {
      k_compact<T, D><<<div_up(n, 256), 256, 0, st>>>(d_in, n, flag.get(), off.get(), soa);
      PPTKG_CHECK_LAUNCH();
    }
    flag.release();
    off.release();
  };
  take_points();
  st_prep.reset();

  // a binary tree over nv points has at most 2 nv - 1 records
  const size_t rec_cap = 2 * (size_t)nv + 64;
  std::unique_ptr<Stage> st_scr(new Stage("build.scratch", st));
  BuildBuf<Rec<T, D>> recbuf(rec_cap, st);
  Rec<T, D>* recs = recbuf.get();
  st_scr.reset();

  const int mid_cap = mid_capacity<T, D>(max_leaf);
  // (small segments are disjoint: at most one per point)
  int64_t small_capn = std::min<int64_t>(nv, ncloud + 2 * 64 * ((int64_t)mid_segments<T, D>(nv, max_leaf) + 1));
  int64_t most = 0;  // points of the largest cloud
  for (int c = 0; c < ncloud; c++) most = std::max(most, tree->valid_off_h[c + 1] - tree->valid_off_h[c]);
  int depth = 0;
  for (int attempt = 0; attempt < 4; attempt++, small_capn = attempt < 3 ? std::min<int64_t>(nv, 4 * small_capn) : nv) {
    Stage st_att("build.attempt", st);
    if (attempt > 0) {
      find_valid();
      take_points();
    }
    Levels<T, D> lv(tree.get(), nv, n, (int)small_capn, soa, recs, (int)rec_cap, st);
    BuildCtl* ctl = lv.ctl;
    if (nv > 0) lv.roots(tree->valid_off, tree->orig_off, ncloud);
    int levels = 0;
    {
      Stage st_levels("build.levels", st);
      // Points at a split value are rare in float data: the tie pass is
      // launched only once a level has asked for it (that level's children,
      // and so all later levels, wait for the host to notice), and then on
      // every level until four had none.
      int tied = 0;
      // The host looks every fourth level of a large build; of a smaller one
      // after four, then once the largest cloud may be down to k_block's size
      // or to leaves, and then every second level.  Kernels of a level without segments exit
      // at once.
      const bool often = nv < (1 << 21);
      int look = 2;
      while (look < 32 && (most >> look) > std::max(mid_cap, max_leaf)) look++;
      for (int lvl = 0; most > mid_cap && lvl < MAX_LEVELS; lvl++) {
        Seg<T, D>* A = lv.seg[lvl & 1];
        Seg<T, D>* B = lv.seg[(lvl + 1) & 1];
        lv.split(A, lvl, tied == 2 || lvl == 0);
        lv.tie_pass(A, lvl, tied);
        lv.children(A, lvl, tied, B);
        levels = lvl + 1;
        if (often ? levels == look || levels == 4 : levels % 4 == 0) {
          if (levels == look) look += 2;
          struct {
            int ties, big, stalled;
          } h = {0, 0, 0};
          int left = 0;
          PPTKG_CUDA(cudaMemcpyAsync(&left, &ctl->level_cnt[lvl + 1], sizeof(int), cudaMemcpyDeviceToHost, st));
          PPTKG_CUDA(cudaMemcpyAsync(&h, &ctl->ties, sizeof(h), cudaMemcpyDeviceToHost, st));
          PPTKG_CUDA(cudaStreamSynchronize(st));
          if (tied == 2 && h.big < levels - 3) tied = 1;
          if (tied == 1 && h.ties < levels - 3) tied = 0;
          if (h.stalled > 0) {
            // back to the level that waits (the later ones found no segments)
            lvl = h.stalled - 1;
            Seg<T, D>* W = lv.seg[lvl & 1];
            Seg<T, D>* X = lv.seg[(lvl + 1) & 1];
            tied = h.big == h.stalled ? 2 : 1;
            PPTKG_CUDA(cudaMemsetAsync(&ctl->stalled, 0, sizeof(int), st));
            lv.tie_pass(W, lvl, tied);
            lv.children(W, lvl, tied, X);
            levels = lvl + 1;
            continue;
          }
          if (left == 0) break;
        }
      }
    }
    if (levels >= MAX_LEVELS) throw Error(E_DEVICE, "device build: more than 4096 levels of large nodes");
    depth = levels;
    BuildCtl hctl;  // (its scalars)
    {
      Stage st_sub("build.subtree", st);
      lv.finish(most);
      PPTKG_CUDA(cudaMemcpyAsync(&hctl, ctl, offsetof(BuildCtl, level_cnt), cudaMemcpyDeviceToHost, st));
      PPTKG_CUDA(cudaStreamSynchronize(st));
      // small list too short: again with more room, from the points in their
      // input order (a split inside a run of equal values divides it by the
      // order that it finds)
      if (hctl.status == 7 && attempt < 3) continue;
      if (hctl.status)
        throw Error(E_DEVICE, "device build: check failed (code " + std::to_string(hctl.status) + ")");
    }
    tree->n_recs = hctl.rec_count;
    tree->levels = levels;
    depth = std::max(depth, hctl.depth);
    break;
  }
  if ((size_t)tree->n_recs > rec_cap) throw Error(E_DEVICE, "device build: record capacity exceeded");
  tree->depth = depth;
  std::unique_ptr<Stage> st_rec(new Stage("build.records", st));
  PPTKG_CUDA(dev_malloc(&tree->recs, std::max(tree->n_recs, 1) * sizeof(Rec<T, D>), st));
  if (tree->n_recs)
    PPTKG_CUDA(cudaMemcpyAsync(tree->recs, recs, tree->n_recs * sizeof(Rec<T, D>), cudaMemcpyDeviceToDevice, st));
  recbuf.release();
  st_rec.reset();

  // tree-ordered points and the forward map
  std::unique_ptr<Stage> st_fin(new Stage("build.finish", st));
  PointRec<T, D>* pts = nullptr;
  PPTKG_CUDA(dev_malloc((void**)&pts, std::max<int64_t>(nv, 1) * sizeof(PointRec<T, D>), st));
  tree->pts = pts;
  PPTKG_CUDA(dev_malloc((void**)&tree->fwd, std::max<int64_t>(n, 1) * sizeof(int), st));
  PPTKG_CUDA(dev_malloc((void**)&tree->ids, std::max<int64_t>(nv, 1) * sizeof(int), st));
  if (n > 0) PPTKG_CUDA(cudaMemsetAsync(tree->fwd, 0xff, n * sizeof(int), st));
  if (nv > 0) {
    k_finish<T, D><<<div_up(nv, 256), 256, 0, st>>>(soa, nv, pts, tree->fwd, tree->ids);
    PPTKG_CHECK_LAUNCH();
  }

  st_fin.reset();
  // traversal hierarchy cut at `bucket` points
  {
    Stage st_tn("build.tnodes", st);
    make_tnodes<T, D>(tree.get(), bucket, st);
  }

  if constexpr (std::is_integral<T>::value) lower_points<T, D>(tree.get(), st);
  return tree.release();
}

template <typename T, int D>
TreeBase* build_tree(const T* d_in, int64_t n, int max_leaf, double thr, int bucket, cudaStream_t st) {
  const int64_t off[2] = {0, n};
  return build_forest<T, D>(d_in, n, off, 1, max_leaf, thr, bucket, st);
}

template <typename T, int D>
void make_tnodes(TreeBase* tree, int bucket, cudaStream_t st) {
  if (tree->tnodes) {
    dev_free(tree->tnodes, st);
    tree->tnodes = nullptr;
  }
  tree->walkable = false;
  if (bucket < 1) bucket = 1;
  tree->bucket = bucket;
  const int nr = tree->n_recs;
  const Rec<T, D>* recs = (const Rec<T, D>*)tree->recs;
  BuildBuf<int> flag(nr + 1, st), tid(nr + 1, st);
  BuildBuf<double> boxbuf(8, st);
  int nt = 0, n_wide = 0;
  wide_begin<T, D>(tree, nr, st);
  PPTKG_CUDA(cudaMemcpyAsync(&n_wide, tree->wrank + (int64_t)tree->wlevels * tree->wwords, sizeof(int),
                             cudaMemcpyDeviceToHost, st));
  if (nr > 0) {
    k_tflag<T, D><<<div_up(nr, 256), 256, 0, st>>>(recs, nr, bucket, flag.get());
    PPTKG_CHECK_LAUNCH();
    exclusive_scan<int, int>(flag.get(), tid.get(), nr, tid.get() + nr, st);
    PPTKG_CUDA(cudaMemcpyAsync(&nt, tid.get() + nr, sizeof(int), cudaMemcpyDeviceToHost, st));
  }
  PPTKG_CUDA(cudaStreamSynchronize(st));
  // (a capture-ready forest's follows below from its traversal nodes' capacity)
  if (!tree->capture) {
    wide_alloc<T, D>(tree, n_wide, st);
    wide_fill<T, D>(tree, nr, false, st);
  }
  TNode<T, D>* nodes = nullptr;
  // a capture-ready forest keeps the capacity that its rebuilds fill
  const int64_t cap = tree->capture ? std::max<int64_t>(tree->cap_tnodes, (int64_t)nt + tree->ncloud)
                                    : (int64_t)nt + tree->ncloud;
  if (tree->capture) tree->cap_tnodes = cap;
  PPTKG_CUDA(dev_malloc((void**)&nodes, (size_t)cap * sizeof(TNode<T, D>), st));
  tree->tnodes = nodes;
  tree->n_tnodes = (int)cap;
  if (tree->capture) {
    wide_alloc<T, D>(tree, wide_capacity(tree), st);
    wide_fill<T, D>(tree, nr, true, st);
  }
  if (nt > 0) {
    k_tfill<T, D><<<div_up(nr, 256), 256, 0, st>>>(recs, nr, flag.get(), tid.get(), nodes);
    PPTKG_CHECK_LAUNCH();
  }
  k_troots<T, D><<<div_up(tree->ncloud, 128), 128, 0, st>>>(recs, tree->root_rec, tree->valid_off, tree->ncloud,
                                                            nr > 0 ? flag.get() : nullptr, tid.get(), nt, nodes,
                                                            tree->root_tnode, boxbuf.get());
  PPTKG_CHECK_LAUNCH();
  double box[8];
  PPTKG_CUDA(cudaMemcpyAsync(box, boxbuf.get(), sizeof(box), cudaMemcpyDeviceToHost, st));
  tree->root_tnode_h.resize(tree->ncloud);
  PPTKG_CUDA(cudaMemcpyAsync(tree->root_tnode_h.data(), tree->root_tnode, sizeof(int) * tree->ncloud,
                             cudaMemcpyDeviceToHost, st));
  if (!tree->capture) tree->tdepth = tree->depth + 2;
  if constexpr (std::is_integral<T>::value) lower_tnodes<T, D>(tree, st);
  PPTKG_CUDA(cudaStreamSynchronize(st));
  for (int d = 0; d < D; d++) {
    tree->root_lo[d] = box[d];
    tree->root_hi[d] = box[4 + d];
  }
  tree->walkable = true;
}

#ifndef PPTKG_BUILD_INT
// ------------------------------------------------------ capture mode ----
// Build status of a rebuild: the device checks of the build kernels, code
// 20 when the new data needs a deeper tree than the capacity planned for
// (large segments left after the last of the cap_levels levels, or a depth
// beyond the traversal stacks' tdepth) and 21 when it needs more records.
// meta: valid points, records, depth.
static __global__ void k_rebuild_status(const BuildCtl* ctl, int levels_cap, int tdepth, int* status, int64_t* meta,
                                        const int64_t* valid_off, int ncloud) {
  int levels = 0;
  for (int l = 0; l < levels_cap; l++)
    if (ctl->level_cnt[l] > 0) levels = l + 1;
  const int depth = ctl->depth > levels ? ctl->depth : levels;
  if (ctl->status) atomicExch(status, ctl->status == 6 ? 21 : 10 + ctl->status);
  if (ctl->level_cnt[levels_cap] > 0 || depth + 2 > tdepth) atomicExch(status, 20);
  meta[0] = valid_off[ncloud];
  meta[1] = ctl->rec_count;
  meta[2] = depth;
  meta[3] = 0;
}

template <typename T, int D>
void forest_capture_ready(TreeBase* t, cudaStream_t st) {
  if (t->capture) return;
  if (t->rec_dtype != F32 && t->rec_dtype != F64) throw Error(E_TYPE, "capture mode needs float32 or float64 points");
  const int64_t n = t->n;
  t->cap_levels = std::min(t->levels + 8, MAX_LEVELS);
  // small segments: at most two children of every larger segment of every
  // level (the planned depth is tdepth + 8), plus the clouds' roots; they are
  // disjoint
  const int64_t small = 2 * (int64_t)(t->tdepth + 8) * (mid_segments<T, D>(n, t->max_leaf) + 1) + t->ncloud + 64;
  t->cap_small = (int)std::min<int64_t>(small, n + t->ncloud + 64);
  // records and traversal nodes: twice the first build's counts (a tree
  // over n points has at most 2n - 1 records); a rebuild that needs more
  // stops with code 21
  t->cap_recs = std::min<int64_t>(2 * n + 64, 2 * (int64_t)t->n_recs + 4096);
  // (the direct build's inner traversal nodes: n_tnodes less the clouds'
  // root slots)
  const int64_t live_tnodes = std::max<int64_t>((int64_t)t->n_tnodes - t->ncloud, 0);
  t->cap_tnodes = std::min<int64_t>(t->cap_recs, 2 * live_tnodes + 4096) + t->ncloud;
  if (t->cap_recs > INT32_MAX / 2 || t->cap_tnodes > INT32_MAX / 2)
    throw Error(E_INVALID, "forest too large for capture mode");
  // capacity-sized arrays, current contents kept
  auto grow = [&](void** p, size_t have, size_t want) {
    void* q = nullptr;
    PPTKG_CUDA(dev_malloc(&q, std::max<size_t>(want, 1), st));
    if (have) PPTKG_CUDA(cudaMemcpyAsync(q, *p, have, cudaMemcpyDeviceToDevice, st));
    if (*p) dev_free(*p, st);
    *p = q;
  };
  grow(&t->pts, (size_t)t->nv * sizeof(PointRec<T, D>), (size_t)n * sizeof(PointRec<T, D>));
  grow((void**)&t->ids, (size_t)t->nv * sizeof(int), (size_t)n * sizeof(int));
  grow(&t->recs, (size_t)t->n_recs * sizeof(Rec<T, D>), (size_t)t->cap_recs * sizeof(Rec<T, D>));
  grow(&t->tnodes, (size_t)t->n_tnodes * sizeof(TNode<T, D>), (size_t)t->cap_tnodes * sizeof(TNode<T, D>));
  t->n_tnodes = (int)t->cap_tnodes;
  t->tdepth += 8;
  if (!t->dev_meta) PPTKG_CUDA(dev_malloc((void**)&t->dev_meta, 4 * sizeof(int64_t), st));
  // the map covers all input rows; the wide nodes follow from the records and
  // traversal nodes
  t->capture = true;
  t->walkable = false;
  wide_begin<T, D>(t, t->n_recs, st);
  wide_alloc<T, D>(t, wide_capacity(t), st);
  wide_fill<T, D>(t, t->n_recs, true, st);
  PPTKG_CUDA(cudaStreamSynchronize(st));
  t->walkable = true;
}

template <typename T, int D>
void rebuild_forest(TreeBase* t, const T* d_in, cudaStream_t st, int* status) {
  if (!t->capture) throw Error(E_INVALID, "rebuild needs a capture-ready forest");
  require_walkable(t);
  Stage stage("rebuild", st);
  const int64_t n = t->n;
  const int ncloud = t->ncloud;
  // valid rows and per-cloud valid offsets, all on the device
  BuildBuf<int> flag(n + 1, st), off(n + 1, st);
  if (n > 0) {
    k_valid<T, D><<<div_up(n, 256), 256, 0, st>>>(d_in, n, flag.get());
    PPTKG_CHECK_LAUNCH();
  }
  exclusive_scan<int, int>(flag.get(), off.get(), n, off.get() + n, st);
  k_cloud_off<<<div_up(ncloud + 1, 256), 256, 0, st>>>(off.get(), t->orig_off, ncloud, t->valid_off);
  PPTKG_CHECK_LAUNCH();
  BuildBuf<T> xs((size_t)D * n + 1, st);
  BuildBuf<int> ids(n + 1, st);
  SoA<T, D> soa;
  for (int d = 0; d < D; d++) soa.x[d] = xs.get() + (size_t)d * n;
  soa.id = ids.get();
  if (n > 0) {
    k_compact<T, D><<<div_up(n, 256), 256, 0, st>>>(d_in, n, flag.get(), off.get(), soa);
    PPTKG_CHECK_LAUNCH();
  }
  flag.release();
  off.release();
  const int rec_cap = (int)t->cap_recs;
  Rec<T, D>* recs = (Rec<T, D>*)t->recs;
  int64_t most = 0;  // points that the largest cloud may have
  for (int c = 0; c < ncloud; c++) most = std::max(most, t->orig_off_h[c + 1] - t->orig_off_h[c]);
  Levels<T, D> lv(t, n, n, t->cap_small, soa, recs, rec_cap, st);
  BuildCtl* ctl = lv.ctl;
  PPTKG_CUDA(cudaMemsetAsync(t->root_rec, 0xff, sizeof(int) * ncloud, st));
  lv.roots(t->valid_off, t->orig_off, ncloud);
  {
    // a fixed number of levels; the kernels of a level without segments
    // return at once
    for (int lvl = 0; lvl < t->cap_levels; lvl++) {
      Seg<T, D>* A = lv.seg[lvl & 1];
      Seg<T, D>* B = lv.seg[(lvl + 1) & 1];
      lv.split(A, lvl, true);
      lv.tie_pass(A, lvl, 2);
      lv.children(A, lvl, 2, B);
    }
  }
  // the persistent kernels take the smaller segments; blocks without work
  // return
  lv.finish(most);
  k_rebuild_status<<<1, 1, 0, st>>>(ctl, t->cap_levels, t->tdepth, status, t->dev_meta, t->valid_off, ncloud);
  PPTKG_CHECK_LAUNCH();
  // tree-ordered points and the forward map
  if (n > 0) {
    PPTKG_CUDA(cudaMemsetAsync(t->fwd, 0xff, n * sizeof(int), st));
    k_finish<T, D><<<div_up(n, 256), 256, 0, st>>>(soa, (int)n, (PointRec<T, D>*)t->pts, t->fwd,
                                                   t->ids, t->valid_off + ncloud);
    PPTKG_CHECK_LAUNCH();
  }
  // traversal hierarchy over the live records
  BuildBuf<int> tflag(rec_cap + 1, st), tid(rec_cap + 1, st);
  const int* nrec_dev = &ctl->rec_count;
  k_tflag<T, D><<<div_up(rec_cap, 256), 256, 0, st>>>(recs, rec_cap, t->bucket, tflag.get(), nrec_dev);
  PPTKG_CHECK_LAUNCH();
  exclusive_scan<int, int>(tflag.get(), tid.get(), rec_cap, tid.get() + rec_cap, st);
  TNode<T, D>* nodes = (TNode<T, D>*)t->tnodes;
  // inner nodes take the slots below cap_tnodes - ncloud, the clouds' root
  // slots the last ncloud
  const int node_lim = (int)(t->cap_tnodes - ncloud);
  k_tfill<T, D><<<div_up(rec_cap, 256), 256, 0, st>>>(recs, rec_cap, tflag.get(), tid.get(), nodes, nrec_dev,
                                                      node_lim, status);
  PPTKG_CHECK_LAUNCH();
  k_troots<T, D><<<div_up(ncloud, 128), 128, 0, st>>>(recs, t->root_rec, t->valid_off, ncloud, tflag.get(),
                                                      tid.get(), node_lim, nodes, t->root_tnode);
  PPTKG_CHECK_LAUNCH();
  wide_begin<T, D>(t, rec_cap, st, nrec_dev);
  wide_fill<T, D>(t, rec_cap, true, st, nrec_dev, status);
}

template <typename T, int D>
void forest_sync(TreeBase* t, cudaStream_t st) {
  if (!t->capture) return;
  int64_t meta[4] = {0, 0, 0, 0};
  PPTKG_CUDA(cudaMemcpyAsync(meta, t->dev_meta, sizeof(meta), cudaMemcpyDeviceToHost, st));
  t->valid_off_h.resize(t->ncloud + 1);
  PPTKG_CUDA(cudaMemcpyAsync(t->valid_off_h.data(), t->valid_off, sizeof(int64_t) * (t->ncloud + 1),
                             cudaMemcpyDeviceToHost, st));
  t->root_tnode_h.resize(t->ncloud);
  PPTKG_CUDA(cudaMemcpyAsync(t->root_tnode_h.data(), t->root_tnode, sizeof(int) * t->ncloud, cudaMemcpyDeviceToHost,
                             st));
  int root0 = -1;
  PPTKG_CUDA(cudaMemcpyAsync(&root0, t->root_rec, sizeof(int), cudaMemcpyDeviceToHost, st));
  PPTKG_CUDA(cudaStreamSynchronize(st));
  if (meta[1] > 0) {  // a rebuild ran
    t->nv = meta[0];
    t->n_recs = (int)std::min<int64_t>(meta[1], t->cap_recs);  // (a rebuild past the capacity stops there)
    t->depth = (int)meta[2];
  }
  if (root0 >= 0 && root0 < t->n_recs) {  // the first cloud's root box (saved with the tree)
    Rec<T, D> r0;
    PPTKG_CUDA(cudaMemcpyAsync(&r0, (const Rec<T, D>*)t->recs + root0, sizeof(r0), cudaMemcpyDeviceToHost, st));
    PPTKG_CUDA(cudaStreamSynchronize(st));
    for (int d = 0; d < D; d++) {
      t->root_lo[d] = (double)r0.lo[d];
      t->root_hi[d] = (double)r0.hi[d];
    }
  }
}
#endif  // PPTKG_BUILD_INT

#ifndef PPTKG_BUILD_INT
size_t TreeBase::device_bytes() const {
  size_t ps = (dtype == F64 ? 8 : 4) * dim + 4;
  ps = (ps + 15) / 16 * 16;
  return ps * nv + 4 * n;
}

TreeBase::~TreeBase() {
  // stream-ordered release on the stream the tree was built on
  if (pts) dev_free(pts, stream);
  if (recs) dev_free(recs, stream);
  if (tnodes) dev_free(tnodes, stream);
  if (fwd) dev_free(fwd, stream);
  if (wide) dev_free(wide, stream);
  if (wspan) dev_free(wspan, stream);
  if (ids) dev_free(ids, stream);
  if (wbits) dev_free(wbits, stream);
  if (wrank) dev_free(wrank, stream);
  if (root_rec) dev_free(root_rec, stream);
  if (root_tnode) dev_free(root_tnode, stream);
  if (valid_off) dev_free(valid_off, stream);
  if (orig_off) dev_free(orig_off, stream);
  if (slot_off) dev_free(slot_off, stream);
  if (warp_cloud) dev_free(warp_cloud, stream);
  if (dev_meta) dev_free(dev_meta, stream);
}

#endif  // PPTKG_BUILD_INT

#define PPTKG_INST_BUILD(T, D)                                                                                  \
  template TreeBase* build_tree<T, D>(const T*, int64_t, int, double, int, cudaStream_t);                      \
  template TreeBase* build_forest<T, D>(const T*, int64_t, const int64_t*, int, int, double, int, cudaStream_t); \
  template void make_tnodes<T, D>(TreeBase*, int, cudaStream_t);                                               \
  template void make_wide<T, D>(TreeBase*, cudaStream_t);

#define PPTKG_INST_CAPTURE(T, D)                                              \
  template void forest_capture_ready<T, D>(TreeBase*, cudaStream_t);          \
  template void rebuild_forest<T, D>(TreeBase*, const T*, cudaStream_t, int*); \
  template void forest_sync<T, D>(TreeBase*, cudaStream_t);

// This file builds float32 / float64 trees; build_int.cu includes it with
// PPTKG_BUILD_INT set and builds the eight integer point types.
#ifndef PPTKG_BUILD_INT
PPTKG_INST_CAPTURE(float, 3)
PPTKG_INST_CAPTURE(double, 3)
PPTKG_INST_CAPTURE(float, 2)
PPTKG_INST_CAPTURE(double, 2)
PPTKG_INST_CAPTURE(float, 4)
PPTKG_INST_CAPTURE(double, 4)
PPTKG_INST_BUILD(float, 3)
PPTKG_INST_BUILD(double, 3)
PPTKG_INST_BUILD(float, 2)
PPTKG_INST_BUILD(double, 2)
PPTKG_INST_BUILD(float, 4)
PPTKG_INST_BUILD(double, 4)
#else
#define PPTKG_INST_BUILD_DIMS(T) PPTKG_INST_BUILD(T, 2) PPTKG_INST_BUILD(T, 3) PPTKG_INST_BUILD(T, 4)
PPTKG_INST_BUILD_DIMS(int8_t)
PPTKG_INST_BUILD_DIMS(int16_t)
PPTKG_INST_BUILD_DIMS(int32_t)
PPTKG_INST_BUILD_DIMS(int64_t)
PPTKG_INST_BUILD_DIMS(uint8_t)
PPTKG_INST_BUILD_DIMS(uint16_t)
PPTKG_INST_BUILD_DIMS(uint32_t)
PPTKG_INST_BUILD_DIMS(uint64_t)
#endif

}  // namespace pptkg
