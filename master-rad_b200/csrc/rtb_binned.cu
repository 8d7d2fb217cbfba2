// Device BVH builder, binned mode: object SAH over B = 2..32 centroid bins per axis with the
// per-type construction weights.  This mode has no counterpart in the reference (its builder
// is the full sweep of GpuScene.java:1453-1488, restated in rtb_build.cu); it trades the
// node-for-node identity with the Java tree for a build that touches every primitive a
// constant number of times per level.
//
// Definition (restated on the CPU by the oracle, which the tests compare node for node):
//  * a node's centroid bounds, box and per-type counts are exact reductions;
//  * on every axis whose centroid extent exceeds 1e-12, bin(c) = min(B - 1,
//    (int)((c - lo) * (B / extent))); each bin keeps integer counts per primitive type and
//    the union of its primitives' float boxes;
//  * the weight of a set is ((n0 w0 + n1 w1) + n2 w2) + n3 w3 in double, w_t the per-type
//    construction weights 1 + lambda (c_t - 1): it depends only on integer counts, so the
//    result does not depend on the order in which atomics land;
//  * plane j = 1..B-1 puts bins [0, j) left; cost (A_P c_T + A_L W_L) + A_R W_R; the first
//    minimum over (axis, j) with both sides non-empty wins;
//  * leaf if count == 1, or count <= leafSize and !(cost < A_P W_P); a node whose centroids
//    coincide on every axis is a leaf when count <= leafSize and otherwise splits at
//    count / 2 in its current order;
//  * children are a stable partition of the node's primitives (left first).
//
// What bounds it: the length of the chain of levels and nodes, and atomics on few addresses, not
// bytes.  So a level goes only down to nodes of more than kSmall primitives, and by size:
//  * above kChunk ("large"), blocks of kChunk positions gather the node's bounds and then its
//    bins in shared memory and add them to the node's in global memory once a block.  A chunk
//    meets at most two such nodes, at its two ends;
//  * others, one block gathers bounds and bins and picks the split by itself;
//  * everything below a node of at most kSmall primitives is one warp's, depth first, with the
//    primitives in shared memory (k_small_binned).
// Bins are words of shared memory, one word kind apart by 32 bins, so that lanes in different
// bins meet different banks; a bound is compared before it is exchanged, since after a bin's
// first few primitives next to none moves it.  Counting by groups of equal bins
// (__match_any_sync and a reduction a group) ran the groups one after the other: 0.31 ms a level
// at 1M primitives.
// Measured, builder's clock in ms, all levels down to the leaves with those groups and a warp a
// node / this: 64 primitives 0.56 / 0.28, 1,000 1.16 / 0.51, 10k 3.47 / 0.85 (16 bins 2.89 / 0.90),
// 100k 5.69 / 1.55, 300k clustered 8.82 / 3.05, 1M clustered 17.5 / 7.25.
#include "rtb_build_common.cuh"

namespace rtb {
namespace {

constexpr int kSmall = 128;    // subtrees up to this size are built by one warp alone
constexpr int kChunk = 2048;   // positions per block in the large-node passes, largest node of one block
constexpr double kMinExtent = 1.0e-12;
constexpr unsigned kFull = 0xFFFFFFFFu;

// Inverse of order_key (double -> order-preserving 64-bit).
__device__ __forceinline__ double k2d(unsigned long long k) {
  return __longlong_as_double((long long)((k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFULL) : ~k));
}

__device__ __forceinline__ int bin_of(double c, double lo, double scale, int bins) {
  double x = c - lo;
  x = x * scale;
  int b = (int)x;
  return b < bins ? b : bins - 1;
}

// A node's bounds and type counts.
struct NodeAcc {
  unsigned long long cmin[3], cmax[3];  // order keys of the centroid bounds
  unsigned bmin[3], bmax[3];            // order bits of the box
  int cnt[4];
};

// The 32 bins of one axis: a word kind is 32 bins apart.
struct BinTable {
  unsigned cnt[4][32];
  unsigned bmin[3][32], bmax[3][32];
};
constexpr int kTableWords = sizeof(BinTable) / 4;

// What an empty table holds at word w.
__device__ __forceinline__ unsigned empty_word(int w) {
  const int kind = w / 32 % (kTableWords / 32);
  return kind >= 4 && kind < 7 ? 0xFFFFFFFFu : 0u;
}

// Per-node results of the split decision that the partition pass reads.
struct BinX {
  int* slot_of;     // large-node slot of a node of the current level, -1 for others
  int* split_bin;   // plane j: bins [0, j) go left
  double* bin_lo;   // centroid lower bound on the split axis
  double* bin_scale;
};

struct SplitCfg {
  int bins, leaf_size, weighted, roots;
  double traversal, lambda;
  double measured[4];
};

// What a level hands to the host and to the next one.
struct Round {
  int next, large;   // nodes of the next level, those of them with a slot
  int small;         // subtrees of at most kSmall primitives, of all levels
  int hand_on;       // nodes of at most kHandOn below those
  int errors;        // positions whose side disagrees with the node's bins
};

__device__ __forceinline__ void clear_acc(NodeAcc& a) {
  for (int k = 0; k < 3; ++k) {
    a.cmin[k] = ~0ULL;
    a.cmax[k] = 0ULL;
    a.bmin[k] = 0xFFFFFFFFu;
    a.bmax[k] = 0u;
  }
  for (int t = 0; t < 4; ++t) a.cnt[t] = 0;
}

// Lowers / raises a shared word; most values change nothing, which a plain read finds out (a
// word that another thread is moving is at worst read before it moved).
__device__ __forceinline__ void lower(unsigned* p, unsigned v) {
  if (v < *(volatile unsigned*)p) atomicMin(p, v);
}
__device__ __forceinline__ void raise(unsigned* p, unsigned v) {
  if (v > *(volatile unsigned*)p) atomicMax(p, v);
}

__device__ __forceinline__ unsigned long long warp_min_u64(unsigned long long v) {
  const unsigned hi = __reduce_min_sync(kFull, (unsigned)(v >> 32));
  const unsigned lo = __reduce_min_sync(kFull, (unsigned)(v >> 32) == hi ? (unsigned)v : 0xFFFFFFFFu);
  return (unsigned long long)hi << 32 | lo;
}
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
  const unsigned hi = __reduce_max_sync(kFull, (unsigned)(v >> 32));
  const unsigned lo = __reduce_max_sync(kFull, (unsigned)(v >> 32) == hi ? (unsigned)v : 0u);
  return (unsigned long long)hi << 32 | lo;
}

__device__ __forceinline__ void acc_add(NodeAcc& A, const Prims& P, int p) {
  const int t = P.type[p];
  const Box b = P.box[p];
  for (int k = 0; k < 3; ++k) {
    const unsigned long long c = order_key(P.cen[k][p]);
    A.cmin[k] = c < A.cmin[k] ? c : A.cmin[k];
    A.cmax[k] = c > A.cmax[k] ? c : A.cmax[k];
    A.bmin[k] = min(A.bmin[k], f2o(b.mn[k]));
    A.bmax[k] = max(A.bmax[k], f2o(b.mx[k]));
  }
  for (int q = 0; q < 4; ++q) A.cnt[q] += t == q;
}

// A warp's sums, by its first lane, onto an accumulator in shared or global memory.
__device__ __forceinline__ void acc_commit(const NodeAcc& v, NodeAcc* to, int lane) {
  for (int k = 0; k < 3; ++k) {
    const unsigned long long mn = warp_min_u64(v.cmin[k]), mx = warp_max_u64(v.cmax[k]);
    const unsigned lo = __reduce_min_sync(kFull, v.bmin[k]), hi = __reduce_max_sync(kFull, v.bmax[k]);
    if (lane == 0) {
      atomicMin(&to->cmin[k], mn);
      atomicMax(&to->cmax[k], mx);
      atomicMin(&to->bmin[k], lo);
      atomicMax(&to->bmax[k], hi);
    }
  }
  for (int q = 0; q < 4; ++q) {
    const int c = __reduce_add_sync(kFull, v.cnt[q]);
    if (lane == 0 && c) atomicAdd(&to->cnt[q], c);
  }
}

// Where an axis's bins lie; scale 0 where the centroids' extent is too small to split.
struct BinAxis {
  double lo, scale;
};
__device__ __forceinline__ BinAxis bin_axis(unsigned long long cmin, unsigned long long cmax, int bins) {
  BinAxis b;
  b.lo = k2d(cmin);
  const double ext = k2d(cmax) - b.lo;
  b.scale = ext > kMinExtent ? (double)bins / ext : 0.0;
  return b;
}

__device__ __forceinline__ void table_add(BinTable* tab, const BinAxis* ax, const Prims& P, int p, int bins) {
  const int t = P.type[p];
  const Box box = P.box[p];
  unsigned lo[3], hi[3];
  for (int k = 0; k < 3; ++k) {
    lo[k] = f2o(box.mn[k]);
    hi[k] = f2o(box.mx[k]);
  }
  for (int a = 0; a < 3; ++a) {
    if (ax[a].scale == 0.0) continue;
    const int b = bin_of(P.cen[a][p], ax[a].lo, ax[a].scale, bins);
    atomicAdd(&tab[a].cnt[t][b], 1u);
    for (int k = 0; k < 3; ++k) {
      lower(&tab[a].bmin[k][b], lo[k]);
      raise(&tab[a].bmax[k][b], hi[k]);
    }
  }
}

// Primitives of each type: four words, or four bytes of one word (at most kSmall of them).
struct Counts4 {
  unsigned c[4];
  __device__ __forceinline__ unsigned of(int t) const { return c[t]; }
  __device__ __forceinline__ Counts4 minus(const Counts4& o) const {
    return Counts4{{c[0] - o.c[0], c[1] - o.c[1], c[2] - o.c[2], c[3] - o.c[3]}};
  }
  __device__ __forceinline__ void scan(int off, bool take) {
    for (int t = 0; t < 4; ++t) {
      const unsigned u = __shfl_up_sync(kFull, c[t], off);
      if (take) c[t] += u;
    }
  }
};
struct CountsPacked {
  unsigned w;
  __device__ __forceinline__ unsigned of(int t) const { return w >> (8 * t) & 255u; }
  __device__ __forceinline__ CountsPacked minus(const CountsPacked& o) const { return CountsPacked{w - o.w}; }
  __device__ __forceinline__ void scan(int off, bool take) {
    const unsigned u = __shfl_up_sync(kFull, w, off);
    if (take) w += u;
  }
};
static_assert(kSmall < 256, "a type's count fits a byte");

template <class C>
__device__ __forceinline__ double set_weight(const C& c, const double* wt) {
  double w = (double)(int)c.of(0) * wt[0];
  w = w + (double)(int)c.of(1) * wt[1];
  w = w + (double)(int)c.of(2) * wt[2];
  w = w + (double)(int)c.of(3) * wt[3];
  return w;
}

__device__ __forceinline__ Box box_of(const unsigned* bmin, const unsigned* bmax) {
  Box b;
  for (int k = 0; k < 3; ++k) {
    b.mn[k] = o2f(bmin[k]);
    b.mx[k] = o2f(bmax[k]);
  }
  return b;
}

// The cost of the plane below this lane's bin on each of A axes, infinite where a side is empty;
// nl = the left side's primitives.  A warp holds an axis's bins, one a lane; the axes' scans go
// on together, so that one's shuffles fill the other's waits.
template <int A, class C>
__device__ __forceinline__ void plane_costs(const C (&own)[A], unsigned (&bmn)[A][3], unsigned (&bmx)[A][3],
                                            const C& total, double area_t, const double* wt, int bins, int lane,
                                            double (&cost)[A], int (&nl)[A]) {
  unsigned rmn[A][3], rmx[A][3];
  C upto[A];  // bins 0..lane
#pragma unroll
  for (int a = 0; a < A; ++a) {
    upto[a] = own[a];
    for (int k = 0; k < 3; ++k) {
      rmn[a][k] = bmn[a][k];
      rmx[a][k] = bmx[a][k];
    }
  }
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const bool below = lane >= off, above = lane + off < 32;
#pragma unroll
    for (int a = 0; a < A; ++a) {
      upto[a].scan(off, below);
      for (int k = 0; k < 3; ++k) {
        const unsigned u = __shfl_up_sync(kFull, bmn[a][k], off), v = __shfl_up_sync(kFull, bmx[a][k], off);
        const unsigned x = __shfl_down_sync(kFull, rmn[a][k], off), y = __shfl_down_sync(kFull, rmx[a][k], off);
        if (below) {
          bmn[a][k] = min(bmn[a][k], u);
          bmx[a][k] = max(bmx[a][k], v);
        }
        if (above) {
          rmn[a][k] = min(rmn[a][k], x);
          rmx[a][k] = max(rmx[a][k], y);
        }
      }
    }
  }
#pragma unroll
  for (int a = 0; a < A; ++a) {
    for (int k = 0; k < 3; ++k) {  // bins 0..lane - 1
      bmn[a][k] = __shfl_up_sync(kFull, bmn[a][k], 1);
      bmx[a][k] = __shfl_up_sync(kFull, bmx[a][k], 1);
    }
    const C left = upto[a].minus(own[a]), right = total.minus(left);
    nl[a] = 0;
    int nr = 0;
    for (int t = 0; t < 4; ++t) {
      nl[a] += (int)left.of(t);
      nr += (int)right.of(t);
    }
    cost[a] = CUDART_INF;
    if (lane < 1 || lane >= bins || nl[a] == 0 || nr == 0) continue;
    const double y = surface_area(box_of(bmn[a], bmx[a])) * set_weight(left, wt);
    const double z = surface_area(box_of(rmn[a], rmx[a])) * set_weight(right, wt);
    cost[a] = (area_t + y) + z;
  }
}

// First minimum over the lanes by (cost, flat); every lane gets it.
__device__ __forceinline__ void warp_first_minimum(double& cost, int& flat, int& left) {
  for (int off = 16; off > 0; off >>= 1) {
    const double oc = __shfl_xor_sync(kFull, cost, off);
    const int of = __shfl_xor_sync(kFull, flat, off), ol = __shfl_xor_sync(kFull, left, off);
    if (oc < cost || (oc == cost && of < flat)) {
      cost = oc;
      flat = of;
      left = ol;
    }
  }
}

__global__ void k_iota(int* idx, int n) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n) idx[j] = j;
}

// Clears the level's slots and what it counts for the next one.
__global__ void k_begin_level(NodeAcc* acc, unsigned* tables, int slots, Round* round) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) round->next = round->large = 0;
  if (i < slots) clear_acc(acc[i]);
  if (i < slots * 3 * kTableWords) tables[i] = empty_word(i);
}

// The slots of the large nodes that own a chunk's first and last position.  A large node is
// longer than a chunk, so a chunk meets no third one.
struct Owners {
  int slot[2];
  __device__ __forceinline__ Owners(const int* key, const int* level_of, int level, const int* slot_of, int c0,
                                    int c1) {
    const int a = key[c0], b = key[c1 - 1];
    slot[0] = level_of[a] == level ? slot_of[a] : -1;
    slot[1] = b != a && level_of[b] == level ? slot_of[b] : -1;
  }
};

// Bounds and type counts of the large nodes.
__global__ void __launch_bounds__(256) k_node_acc(const Prims P, const int* idx, const int* key,
                                                  const int* level_of, int level, const int* slot_of, int n,
                                                  NodeAcc* acc) {
  __shared__ NodeAcc sa[2];
  const int c0 = blockIdx.x * kChunk, c1 = min(n, c0 + kChunk), lane = threadIdx.x & 31;
  const Owners own(key, level_of, level, slot_of, c0, c1);
  if (own.slot[0] < 0 && own.slot[1] < 0) return;
  if (threadIdx.x < 2) clear_acc(sa[threadIdx.x]);
  __syncthreads();
  for (int w = 0; w < 2; ++w) {
    if (own.slot[w] < 0) continue;
    const int node = w == 0 ? key[c0] : key[c1 - 1];
    NodeAcc v;
    clear_acc(v);
    for (int j = c0 + threadIdx.x; j < c1; j += blockDim.x)
      if (key[j] == node) acc_add(v, P, idx[j]);
    acc_commit(v, &sa[w], lane);
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  for (int w = 0; w < 2; ++w) {
    if (own.slot[w] < 0) continue;
    NodeAcc *g = acc + own.slot[w], *s = sa + w;
    if (lane < 3) {
      atomicMin(&g->cmin[lane], s->cmin[lane]);
      atomicMax(&g->cmax[lane], s->cmax[lane]);
      atomicMin(&g->bmin[lane], s->bmin[lane]);
      atomicMax(&g->bmax[lane], s->bmax[lane]);
    }
    if (lane < 4 && s->cnt[lane]) atomicAdd(&g->cnt[lane], s->cnt[lane]);
  }
}

// Bins of the large nodes.
__global__ void __launch_bounds__(256) k_bin_large(const Prims P, const int* idx, const int* key,
                                                   const int* level_of, int level, const int* slot_of,
                                                   const NodeAcc* acc, int n, int bins, BinTable* tables) {
  __shared__ BinTable tab[2][3];
  __shared__ BinAxis ax[2][3];
  const int c0 = blockIdx.x * kChunk, c1 = min(n, c0 + kChunk);
  const Owners own(key, level_of, level, slot_of, c0, c1);
  if (own.slot[0] < 0 && own.slot[1] < 0) return;
  const int first = key[c0], last = key[c1 - 1];
  for (int i = threadIdx.x; i < 6 * kTableWords; i += blockDim.x) (&tab[0][0].cnt[0][0])[i] = empty_word(i);
  if (threadIdx.x < 6) {
    const int w = threadIdx.x / 3, a = threadIdx.x % 3;
    if (own.slot[w] >= 0) ax[w][a] = bin_axis(acc[own.slot[w]].cmin[a], acc[own.slot[w]].cmax[a], bins);
  }
  __syncthreads();
  for (int j = c0 + threadIdx.x; j < c1; j += blockDim.x) {
    const int node = key[j];
    const int w = node == first ? 0 : node == last ? 1 : -1;
    if (w >= 0 && own.slot[w] >= 0) table_add(tab[w], ax[w], P, idx[j], bins);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 6 * kTableWords; i += blockDim.x) {
    const int slot = own.slot[i / (3 * kTableWords)], at = i % (3 * kTableWords);
    const unsigned v = (&tab[0][0].cnt[0][0])[i];
    if (slot < 0 || v == empty_word(i)) continue;
    unsigned* g = &tables[(size_t)slot * 3].cnt[0][0] + at;
    const int kind = at / 32 % (kTableWords / 32);
    if (kind < 4) atomicAdd(g, v);
    else if (kind < 7) atomicMin(g, v);
    else atomicMax(g, v);
  }
}

// Split decision of every node of the level, a block a node.
__global__ void __launch_bounds__(256) k_split_binned(const Prims P, const int* idx, Nodes N, BinX X,
                                                      const int* active, SplitCfg S, const NodeAcc* acc,
                                                      const BinTable* tables, int* stats, Round* round,
                                                      int* next_active, int* small_roots, int* level_of,
                                                      int level) {
  __shared__ BinTable tab[3];
  __shared__ NodeAcc sa;
  __shared__ double best_cost[3];
  __shared__ int best_flat[3], best_left[3];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int node = active[blockIdx.x];
  const int s = N.start[node], e = N.end[node], n = e - s;
  const int slot = X.slot_of[node];
  BinAxis ax[3];
  if (slot >= 0) {
    if (threadIdx.x == 0) sa = acc[slot];
    for (int i = threadIdx.x; i < 3 * kTableWords; i += blockDim.x)
      (&tab[0].cnt[0][0])[i] = (&tables[(size_t)slot * 3].cnt[0][0])[i];
    __syncthreads();
    for (int a = 0; a < 3; ++a) ax[a] = bin_axis(sa.cmin[a], sa.cmax[a], S.bins);
  } else {
    if (threadIdx.x == 0) clear_acc(sa);
    for (int i = threadIdx.x; i < 3 * kTableWords; i += blockDim.x) (&tab[0].cnt[0][0])[i] = empty_word(i);
    __syncthreads();
    NodeAcc v;
    clear_acc(v);
    for (int j = s + threadIdx.x; j < e; j += blockDim.x) acc_add(v, P, idx[j]);
    acc_commit(v, &sa, lane);
    __syncthreads();
    for (int a = 0; a < 3; ++a) ax[a] = bin_axis(sa.cmin[a], sa.cmax[a], S.bins);
    for (int j = s + threadIdx.x; j < e; j += blockDim.x) table_add(tab, ax, P, idx[j], S.bins);
    __syncthreads();
  }
  double wt[4];
  for (int q = 0; q < 4; ++q) wt[q] = S.weighted ? 1.0 + S.lambda * (S.measured[q] - 1.0) : 1.0;
  Counts4 total;
  for (int q = 0; q < 4; ++q) total.c[q] = (unsigned)sa.cnt[q];
  const Box nb = box_of(sa.bmin, sa.bmax);
  const double area = surface_area(nb);
  if (warp < 3) {
    const int a = warp;
    double cost = CUDART_INF;
    int flat = a * 32 + lane, left = 0;
    if (ax[a].scale != 0.0) {
      Counts4 own[1];
      unsigned bmn[1][3], bmx[1][3];
      double plane[1];
      int nl[1];
      for (int t = 0; t < 4; ++t) own[0].c[t] = tab[a].cnt[t][lane];
      for (int k = 0; k < 3; ++k) {
        bmn[0][k] = tab[a].bmin[k][lane];
        bmx[0][k] = tab[a].bmax[k][lane];
      }
      plane_costs(own, bmn, bmx, total, area * S.traversal, wt, S.bins, lane, plane, nl);
      cost = plane[0];
      left = nl[0];
    }
    warp_first_minimum(cost, flat, left);
    if (lane == 0) {
      best_cost[a] = cost;
      best_flat[a] = flat;
      best_left[a] = left;
    }
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  int axis = 0;
  for (int a = 1; a < 3; ++a)
    if (best_cost[a] < best_cost[axis]) axis = a;
  const bool have = best_cost[axis] != CUDART_INF;
  const int depth = N.depth[node];
  N.bounds[node] = nb;
  if (n <= S.leaf_size && !(have && best_cost[axis] < area * set_weight(total, wt))) {
    N.leaf[node] = 1;
    N.split_axis[node] = -1;
    LeafStats st{0, 0x7FFFFFFF, 0, 0};
    st.add(n, depth);
    st.add_to(stats);
    return;
  }
  const int lc = have ? best_left[axis] : n / 2;
  const int l = child_id(S.roots, s + lc);
  write_split(N, node, l, have ? axis : 3, lc, s, e, depth);
  N.order_axis[l] = N.order_axis[l + 1] = 0;
  X.split_bin[node] = best_flat[axis] & 31;
  X.bin_lo[node] = ax[axis].lo;
  X.bin_scale[node] = ax[axis].scale;
  for (int h = 0; h < 2; ++h) {
    const int m = h ? n - lc : lc;
    level_of[l + h] = m > kSmall ? level + 1 : -1;
    if (m > kSmall) {
      X.slot_of[l + h] = m > kChunk ? atomicAdd(&round->large, 1) : -1;
      next_active[atomicAdd(&round->next, 1)] = l + h;
    } else {
      small_roots[atomicAdd(&round->small, 1)] = l + h;
    }
  }
}

// flags[j] = 1 where the primitive at j goes left.
__global__ void k_sides_binned(const Prims P, const int* idx, const Nodes N, BinX X, const int* key,
                               const int* level_of, int level, int n, int bins, int* flags) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int node = key[j];
  int axis = -1;
  if (level_of[node] == level) axis = N.split_axis[node];
  int left = 0;
  if (axis == 3)
    left = j - N.start[node] < N.split_pos[node];
  else if (axis >= 0)
    left = bin_of(P.cen[axis][idx[j]], X.bin_lo[node], X.bin_scale[node], bins) < X.split_bin[node];
  flags[j] = left;
}

// Stable partition, which checks every destination against the node's range (the left count
// comes from the bins and must equal the flags' count); a mismatch is counted in *error and the
// write is skipped.  Position j then belongs to one of the children.
__global__ void k_scatter_checked(const int* idx, const Nodes N, int* key, const int* level_of, int level,
                                  int n, const int* flags, const int* lscan, int* out, int* error) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  int node = key[j];
  int p = idx[j];
  if (!(level_of[node] == level && N.split_axis[node] >= 0)) {
    out[j] = p;
    return;
  }
  int s = N.start[node], e = N.end[node];
  int lc = N.split_pos[node];
  key[j] = j < s + lc ? N.left[node] : N.right[node];
  int lrank = lscan[j] - lscan[s];
  int rrank = (j - s) - lrank;
  const bool left = flags[j] != 0;
  int dst = left ? s + lrank : s + lc + rrank;
  bool ok = left ? lrank < lc : lc + rrank < e - s;
  if (!ok) {
    atomicAdd(error, 1);
    return;
  }
  out[dst] = p;
}

// ---- whole subtrees of at most SIZE primitives, a warp (the block) each, depth first
//
// A node is some 200 shuffles and a chain of them, and a subtree a chain of nodes, so what counts
// is how short the chain is and how many warps an SM has in flight.  A subtree of up to kSmall
// primitives hands its nodes of at most kHandOn to warps of their own (all in the second launch):
// by one warp to the leaves, an axis after the other, 129 primitives took 0.72 ms of the
// builder's clock, 10k 1.46, 1M 8.53; handed on and with the axes together 0.34, 0.85, 7.25.
// The type counts of a bin go in one word.
constexpr int kHandOn = 32;

template <int SIZE>
struct SmallSmem {
  double cen[3][SIZE];
  unsigned lo[3][SIZE], hi[3][SIZE];  // order bits of the boxes
  unsigned cnt[3][32], bmin[3][3][32], bmax[3][3][32];
  int4 stack[SIZE];  // node, start, end, depth
  int gid[SIZE];
  unsigned char type[SIZE], ord[SIZE];
};

// next: where nodes of at most kHandOn go, null to build them here.
template <int SIZE>
__global__ void __launch_bounds__(32) k_small_binned(const Prims P, int* idx, Nodes N, const int* list,
                                                     const int* count, SplitCfg S, int* stats, int* error,
                                                     int* next, int* next_count) {
  __shared__ SmallSmem<SIZE> sm;
  constexpr int kRounds = SIZE / 32;
  const int lane = threadIdx.x;
  double wt[4];
  for (int q = 0; q < 4; ++q) wt[q] = S.weighted ? 1.0 + S.lambda * (S.measured[q] - 1.0) : 1.0;
  LeafStats st{0, 0x7FFFFFFF, 0, 0};
  const int todo = *count;
  for (int at = blockIdx.x; at < todo; at += gridDim.x) {
    const int root = list[at];
    const int rs = N.start[root], M = N.end[root] - rs;
    if (next && M <= kHandOn) {
      if (lane == 0) next[atomicAdd(next_count, 1)] = root;
      continue;
    }
    for (int i = lane; i < M; i += 32) {
      const int p = idx[rs + i];
      const Box b = P.box[p];
      sm.gid[i] = p;
      sm.ord[i] = (unsigned char)i;
      sm.type[i] = (unsigned char)P.type[p];
      for (int k = 0; k < 3; ++k) {
        sm.cen[k][i] = P.cen[k][p];
        sm.lo[k][i] = f2o(b.mn[k]);
        sm.hi[k][i] = f2o(b.mx[k]);
      }
    }
    __syncwarp();
    int sp = 0;
    int4 en = make_int4(root, rs, rs + M, N.depth[root]);
    while (true) {
      const int node = en.x, s = en.y, e = en.z, m = e - s, lo = s - rs, depth = en.w;
      // bounds and type counts; this lane's primitives stay in id[]
      int id[kRounds];
      unsigned long long cmn[3], cmx[3];
      unsigned bmn[3], bmx[3];
      CountsPacked total{0u};
      for (int k = 0; k < 3; ++k) {
        cmn[k] = ~0ULL;
        cmx[k] = 0ULL;
        bmn[k] = 0xFFFFFFFFu;
        bmx[k] = 0u;
      }
#pragma unroll
      for (int q = 0; q < kRounds; ++q) {
        const int i = lane + 32 * q;
        id[q] = i < m ? sm.ord[lo + i] : -1;
        if (id[q] < 0) continue;
        total.w += 1u << (8 * sm.type[id[q]]);
        for (int k = 0; k < 3; ++k) {
          const unsigned long long c = order_key(sm.cen[k][id[q]]);
          cmn[k] = c < cmn[k] ? c : cmn[k];
          cmx[k] = c > cmx[k] ? c : cmx[k];
          bmn[k] = min(bmn[k], sm.lo[k][id[q]]);
          bmx[k] = max(bmx[k], sm.hi[k][id[q]]);
        }
      }
      total.w = __reduce_add_sync(kFull, total.w);
      BinAxis ax[3];
      for (int k = 0; k < 3; ++k) {
        bmn[k] = __reduce_min_sync(kFull, bmn[k]);
        bmx[k] = __reduce_max_sync(kFull, bmx[k]);
        ax[k] = bin_axis(warp_min_u64(cmn[k]), warp_max_u64(cmx[k]), S.bins);
      }
      const Box nb = box_of(bmn, bmx);
      const double area = surface_area(nb);
      double best = CUDART_INF;
      int flat = 0x7FFFFFFF, left = 0;
      if (m > 1) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          sm.cnt[a][lane] = 0u;
          for (int k = 0; k < 3; ++k) {
            sm.bmin[a][k][lane] = 0xFFFFFFFFu;
            sm.bmax[a][k][lane] = 0u;
          }
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < kRounds; ++q) {
          if (id[q] < 0) continue;
          for (int a = 0; a < 3; ++a) {
            if (ax[a].scale == 0.0) continue;
            const int b = bin_of(sm.cen[a][id[q]], ax[a].lo, ax[a].scale, S.bins);
            atomicAdd(&sm.cnt[a][b], 1u << (8 * sm.type[id[q]]));
            for (int k = 0; k < 3; ++k) {
              lower(&sm.bmin[a][k][b], sm.lo[k][id[q]]);
              raise(&sm.bmax[a][k][b], sm.hi[k][id[q]]);
            }
          }
        }
        __syncwarp();
        CountsPacked own[3];
        unsigned vmn[3][3], vmx[3][3];
        double cost[3];
        int nl[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          own[a].w = sm.cnt[a][lane];
          for (int k = 0; k < 3; ++k) {
            vmn[a][k] = sm.bmin[a][k][lane];
            vmx[a][k] = sm.bmax[a][k][lane];
          }
        }
        plane_costs(own, vmn, vmx, total, area * S.traversal, wt, S.bins, lane, cost, nl);
#pragma unroll
        for (int a = 0; a < 3; ++a)
          if (ax[a].scale != 0.0 && cost[a] < best) {  // an earlier axis keeps a tie
            best = cost[a];
            flat = a * 32 + lane;
            left = nl[a];
          }
      }
      warp_first_minimum(best, flat, left);
      const bool have = best != CUDART_INF;
      const bool leaf = m == 1 || (m <= S.leaf_size && !(have && best < area * set_weight(total, wt)));
      if (lane == 0) N.bounds[node] = nb;
      if (leaf) {
        if (lane == 0) {
          N.leaf[node] = 1;
          N.split_axis[node] = -1;
          st.add(m, depth);
        }
        if (sp == 0) break;
        en = sm.stack[--sp];
        __syncwarp();
        continue;
      }
      const int axis = have ? flat >> 5 : 3, plane = flat & 31, pos = have ? left : m / 2;
      const int l = child_id(S.roots, s + pos);
      if (lane == 0) {
        write_split(N, node, l, axis, pos, s, e, depth);
        N.order_axis[l] = N.order_axis[l + 1] = 0;
      }
      // stable partition; every destination is checked against the node's range
      if (have) {
        int nl = 0, nr = 0;
        const unsigned below = (1u << lane) - 1u;
        const BinAxis by = axis == 0 ? ax[0] : axis == 1 ? ax[1] : ax[2];
        __syncwarp();
#pragma unroll
        for (int q = 0; q < kRounds; ++q) {
          const bool in = id[q] >= 0;
          const bool right = in && bin_of(sm.cen[axis][in ? id[q] : 0], by.lo, by.scale, S.bins) >= plane;
          const unsigned rm = __ballot_sync(kFull, right), lm = __ballot_sync(kFull, in && !right);
          if (in) {
            const int dst = right ? pos + nr + __popc(rm & below) : nl + __popc(lm & below);
            if (right ? dst < m : dst < pos) sm.ord[lo + dst] = (unsigned char)id[q];
            else atomicAdd(error, 1);
          }
          nl += __popc(lm);
          nr += __popc(rm);
        }
      }
      const bool go_l = !next || pos > kHandOn, go_r = !next || m - pos > kHandOn;
      if (lane == 0) {
        if (go_r) sm.stack[sp] = make_int4(l + 1, s + pos, e, depth + 1);
        else next[atomicAdd(next_count, 1)] = l + 1;
        if (!go_l) next[atomicAdd(next_count, 1)] = l;
      }
      sp += go_r;
      en = make_int4(l, s, s + pos, depth + 1);
      __syncwarp();
      if (!go_l) {
        if (sp == 0) break;
        en = sm.stack[--sp];
        __syncwarp();
      }
    }
    for (int i = lane; i < M; i += 32) idx[rs + i] = sm.gid[sm.ord[i]];
    __syncwarp();
  }
  if (lane == 0) st.add_to(stats);
}

}  // namespace

rtb_status build_bvh_binned(rtb_context* ctx, const rtb_scene_desc* desc, const rtb_build_config* cfg,
                            int bins, rtb_scene** out, rtb_bvh_stats* stats) {
  if (!out) return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "null argument");
  if (bins < 2 || bins > 32) return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "binned BVH build needs 2..32 bins");
  BuildCfg c;
  bool per_type = false;
  rtb_status st = build_setup(ctx, desc, cfg, c, per_type);
  if (st != RTB_OK) return st;
  if (stats) *stats = rtb_bvh_stats{};
  if (c.total == 0) {
    rtb_status s = scene_create(ctx, desc, nullptr, nullptr, out);
    if (stats) stats->leaf_size = cfg->leaf_size;
    return s;
  }
  const int n = c.total;
  cudaStream_t sm = ctx->stream;
  Workspace W;
  W.stream = sm;
  PrimInputs in = alloc_inputs(W, c);
  Prims P = alloc_prims(W, n);
  int* idx = W.alloc<int>(n);
  int* tmp_idx = W.alloc<int>(n);
  int cap = 2 * n + 8;
  Nodes N = alloc_nodes(W, cap);
  BinX X;
  X.slot_of = W.alloc<int>(cap);
  X.split_bin = W.alloc<int>(cap);
  X.bin_lo = W.alloc<double>(cap);
  X.bin_scale = W.alloc<double>(cap);
  int max_slots = n / (kChunk + 1) + 4;
  NodeAcc* acc = W.alloc<NodeAcc>(max_slots);
  BinTable* tables = W.alloc<BinTable>((size_t)max_slots * 3);
  int* level_of = W.alloc<int>(cap);
  int* key = W.alloc<int>(n);
  int* flags = W.alloc<int>(n);
  int* lscan = W.alloc<int>(n);
  int* active = W.alloc<int>(n / kSmall + 4);
  int* next_active = W.alloc<int>(n / kSmall + 4);
  int* small_roots = W.alloc<int>(n + 4);  // a subtree holds a primitive or more
  int* hand_on = W.alloc<int>(n + 4);
  // two unused, then stats {leaves, min occupancy, max occupancy, max depth}
  int* counters = W.alloc<int>(8);
  Round* round = W.alloc<Round>(1);
  int* root_start = W.alloc<int>(4);
  int* root_end = W.alloc<int>(4);
  size_t tmp_bytes = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, flags, lscan, n);
  void* tmp = W.alloc<char>(tmp_bytes);
  if (!W.ok) return fail(ctx, RTB_ERR_OUT_OF_MEMORY, "BVH build workspace");

  cudaEventRecord(ctx->ev0, sm);
  upload_prims(desc, c, in, P, sm);
  k_iota<<<blocks(n), 256, 0, sm>>>(idx, n);

  int h_rs[4], h_re[4];
  int roots = root_ranges(c, per_type, h_rs, h_re);
  std::vector<int> h_slot(roots), h_level(roots), h_active, h_small;
  int large = 0;
  for (int r = 0; r < roots; ++r) {
    const int size = h_re[r] - h_rs[r];
    (size > kSmall ? h_active : h_small).push_back(r);
    h_level[r] = size > kSmall ? 0 : -1;
    h_slot[r] = size > kChunk ? large++ : -1;
  }
  int h_counters[8] = {0, 0, 0, 0x7FFFFFFF, 0, 0, 0, 0};
  const Round h_round{0, 0, (int)h_small.size(), 0, 0};
  cudaMemcpyAsync(root_start, h_rs, roots * 4, cudaMemcpyHostToDevice, sm);
  cudaMemcpyAsync(root_end, h_re, roots * 4, cudaMemcpyHostToDevice, sm);
  cudaMemcpyAsync(N.start, h_rs, roots * 4, cudaMemcpyHostToDevice, sm);
  cudaMemcpyAsync(N.end, h_re, roots * 4, cudaMemcpyHostToDevice, sm);
  cudaMemcpyAsync(X.slot_of, h_slot.data(), roots * 4, cudaMemcpyHostToDevice, sm);
  cudaMemcpyAsync(level_of, h_level.data(), roots * 4, cudaMemcpyHostToDevice, sm);
  if (!h_active.empty())
    cudaMemcpyAsync(active, h_active.data(), h_active.size() * 4, cudaMemcpyHostToDevice, sm);
  if (!h_small.empty())
    cudaMemcpyAsync(small_roots, h_small.data(), h_small.size() * 4, cudaMemcpyHostToDevice, sm);
  cudaMemcpyAsync(counters, h_counters, sizeof(h_counters), cudaMemcpyHostToDevice, sm);
  cudaMemcpyAsync(round, &h_round, sizeof(h_round), cudaMemcpyHostToDevice, sm);
  cudaMemsetAsync(N.order_axis, 0, (size_t)roots * 4, sm);
  cudaMemsetAsync(N.depth, 0, (size_t)roots * 4, sm);
  cudaMemsetAsync(N.leaf, 0xFF, (size_t)cap * 4, sm);  // -1: no node
  k_init_keys<<<blocks(n), 256, 0, sm>>>(key, root_start, root_end, roots, n);

  SplitCfg S;
  S.bins = bins;
  S.leaf_size = c.leaf_size;
  S.weighted = c.weighted;
  S.roots = roots;
  S.traversal = c.traversal;
  S.lambda = c.lambda;
  for (int q = 0; q < 4; ++q) S.measured[q] = c.measured[q];

  struct Back {
    Round round;
    int counters[8];
  };
  Back local;
  Back* back = landing(ctx, local);
  back->round = h_round;
  int k = (int)h_active.size(), level = 0;
  while (k > 0) {
    k_begin_level<<<blocks((long long)large * 3 * kTableWords + 1), 256, 0, sm>>>(acc, (unsigned*)tables, large, round);
    if (large > 0) {
      k_node_acc<<<blocks(n, kChunk), 256, 0, sm>>>(P, idx, key, level_of, level, X.slot_of, n, acc);
      k_bin_large<<<blocks(n, kChunk), 256, 0, sm>>>(P, idx, key, level_of, level, X.slot_of, acc, n, bins, tables);
    }
    k_split_binned<<<k, 256, 0, sm>>>(P, idx, N, X, active, S, acc, tables, counters + 2, round, next_active,
                                      small_roots, level_of, level);
    k_sides_binned<<<blocks(n), 256, 0, sm>>>(P, idx, N, X, key, level_of, level, n, bins, flags);
    size_t tb = tmp_bytes;
    cub::DeviceScan::ExclusiveSum(tmp, tb, flags, lscan, n, sm);
    k_scatter_checked<<<blocks(n), 256, 0, sm>>>(idx, N, key, level_of, level, n, flags, lscan, tmp_idx,
                                                 &round->errors);
    std::swap(idx, tmp_idx);
    cudaMemcpyAsync(&back->round, round, sizeof(Round), cudaMemcpyDeviceToHost, sm);
    cudaError_t e = cudaStreamSynchronize(sm);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "binned BVH build level");
    if (back->round.errors != 0) return fail(ctx, RTB_ERR_DEVICE_CHECK, "binned BVH partition disagrees with its bins");
    std::swap(active, next_active);
    large = back->round.large;
    k = back->round.next;
    level++;
  }
  // ---- the subtrees below the level loop
  const int max_blocks = ctx->sm_count * 32;
  if (back->round.small > 0) {
    k_small_binned<kSmall><<<std::min(back->round.small, max_blocks), 32, 0, sm>>>(
        P, idx, N, small_roots, &round->small, S, counters + 2, &round->errors, hand_on, &round->hand_on);
    k_small_binned<kHandOn><<<std::min(n, max_blocks), 32, 0, sm>>>(
        P, idx, N, hand_on, &round->hand_on, S, counters + 2, &round->errors, nullptr, nullptr);
  }
  cudaMemcpyAsync(&back->round, round, sizeof(Round), cudaMemcpyDeviceToHost, sm);
  cudaMemcpyAsync(back->counters, counters, sizeof(back->counters), cudaMemcpyDeviceToHost, sm);
  cudaError_t e = cudaStreamSynchronize(sm);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(ctx, e, "binned BVH subtrees");
  if (back->round.errors != 0) return fail(ctx, RTB_ERR_DEVICE_CHECK, "binned BVH partition disagrees with its bins");
  const int total_nodes = 2 * back->counters[2] - roots;  // a full binary forest of that many leaves
  if (back->counters[2] < 1 || total_nodes > cap) return fail(ctx, RTB_ERR_DEVICE_CHECK, "BVH node count out of range");
  IdxSet I;
  for (int a = 0; a < 3; ++a) I.a[a] = idx;
  return finish_build(ctx, desc, cfg, W, c, in, P, I, N, roots, cap, total_nodes, counters, out, stats);
}

}  // namespace rtb
