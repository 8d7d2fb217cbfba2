// Device BVH builder: the reference's full-sweep, primitive-cost-weighted object SAH
// (gfxlab/gpu/GpuScene.java BvhBuildState, 1414-1499) executed level by level on the GPU,
// producing the same tree node for node and the same flattened arrays
// (flattenBvh / leafKind, GpuScene.java:772-808).
//
// How the Java recursion maps onto data-parallel passes:
//  * bestSplit sorts a node's primitives on each axis by (centroid, order) with
//    Double.compare.  That order restricted to any subset is the global order restricted
//    to it, so the three axis orders are sorted ONCE (radix sort on an order-preserving
//    64-bit image of the double centroid, stable for the order tie-break) and every split
//    stable-partitions each axis array inside the node's range.
//  * Prefix and suffix bounds are exact min/max unions: segmented scans.
//  * Prefix and suffix weights are SEQUENTIAL double sums in the reference; with
//    non-dyadic weights (1.3, 2.1) their rounding depends on the order.  With unit weights
//    the sums are exact integers and are written directly.  Otherwise a node of more than
//    kSubtreeSize primitives takes its weights from per-type counts (a segmented integer
//    scan), summed exactly and rounded once, and its costs carry a rigorous bound on how far
//    the reference's sequentially rounded costs can be from them; its argmin is the
//    reference's whenever every other candidate's cost minus its bound exceeds the winner's
//    cost plus its bound.  Smaller nodes, and the few large ones whose winner is not that
//    clear, sum their weights sequentially per (node, axis, direction), the reference's own
//    additions in its own order.
//  * Costs are evaluated in double with the reference's expression order
//    (nodeArea*cT + A_L*W_L) + A_R*W_R; the argmin keeps the first minimum in
//    (axis, position) order, as the strict '<' does.
//  * The leaf test (count <= leafSize and !(cost < area * sequential weight sum in the
//    node's current order)) uses the parent's split-axis order, which is the order the
//    Java primitives array holds when build() reaches the node.
// The file is compiled with -fmad=false: no double expression is contracted.
#include "rtb_build_common.cuh"

namespace rtb {
namespace {

// ---- the three axis orders by one sort
//
// All 3n (centroid key, axis << 30 | primitive) pairs are sorted by key in one call, eight passes
// for the three axes together (a pass over few keys costs its launch and little else: 33 launches
// became 15, 10k primitives 1.25 -> 1.04 ms), then stably by (axis, type) in one pass more,
// which puts each axis's order in one piece, per type in a per-type forest.
//
// Up to kTileSort primitives the sort is one launch an axis by itself and stays so (builds by
// three sorts / one, ms: 1,000 primitives 0.54 / 0.60, 2,000 0.69 / 0.76, 3,000 1.01 / 0.84).
constexpr int kAxisShift = 30;  // primitives are fewer than 2^30
constexpr int kTileSort = 2048;

__global__ void k_keys(const Prims P, int n, unsigned long long* keys, unsigned* vals) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int a = blockIdx.y;
  keys[(size_t)a * n + p] = order_key(P.cen[a][p]);
  vals[(size_t)a * n + p] = (unsigned)a << kAxisShift | (unsigned)p;
}

__global__ void k_axis_tags(const Prims P, const unsigned* vals, int n3, int per_type, unsigned char* tags) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n3) return;
  const unsigned v = vals[t], p = v & ((1u << kAxisShift) - 1u);
  tags[t] = (unsigned char)((v >> kAxisShift) << 2 | (per_type ? (unsigned)P.type[p] : 0u));
}

__global__ void k_axis_orders(const unsigned* vals, int n, IdxSet I) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n) I.a[blockIdx.y][j] = (int)(vals[(size_t)blockIdx.y * n + j] & ((1u << kAxisShift) - 1u));
}

__global__ void k_gather_weights(const Prims P, const int* idx, int n, double* wpos) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n) wpos[j] = P.w[idx[j]];
}

// Weighted prefix / suffix sums in the reference's sequential order, one warp per
// (node, axis, direction), all three axes in one launch: the warp loads 32 weights at a
// time (coalesced, the next chunk prefetched), broadcasts them to every lane with all 32
// shuffles issued ahead, and every lane then runs the same strictly sequential chain of 32
// additions, lane j keeping the running sum after element j.  The additions happen in
// exactly the Java loop's order (0 + w0 = w0 exactly, then one add per element), so every
// partial sum is bit-identical to it; only the loads and shuffles are parallel.
struct WeightChains {
  const double* w[3];  // weights in each axis order
  double* pw[3];
  double* sw[3];
};

// `nodes` lists the nodes to sum; their number is *count when count is given (a list built
// on the device; k is then only the grid's bound), else k.
__global__ void __launch_bounds__(128) k_weights_seq(const WeightChains C, const Nodes N, const int* nodes,
                                                     int k, const int* count) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  if (count) k = min(k, *count);
  if (warp >= 6 * k) return;
  const int* active = nodes;
  int node = active[warp / 6];
  int axis = (warp >> 1) % 3;
  bool suffix = warp & 1;
  int s = N.start[node], e = N.end[node];
  int n = e - s;
  if (n < 2) return;
  const double* wp = C.w[axis];
  double* out = suffix ? C.sw[axis] : C.pw[axis];
  double acc = 0.0;
  double w = lane < n ? wp[suffix ? e - 1 - lane : s + lane] : 0.0;
  for (int base = 0; base < n; base += 32) {
    int j = base + lane;
    int pos = suffix ? e - 1 - j : s + j;
    int jn = j + 32;
    double wn = jn < n ? wp[suffix ? e - 1 - jn : s + jn] : 0.0;  // next chunk
    double mine = 0.0;
    if (n - base >= 32) {
      double v[32];
#pragma unroll
      for (int q = 0; q < 32; ++q) v[q] = __shfl_sync(0xFFFFFFFFu, w, q);
#pragma unroll
      for (int q = 0; q < 32; ++q) {
        acc = acc + v[q];
        mine = q == lane ? acc : mine;
      }
    } else {
      int m = n - base;
      for (int q = 0; q < m; ++q) {
        double v = __shfl_sync(0xFFFFFFFFu, w, q);
        acc = acc + v;
        if (q == lane) mine = acc;
      }
    }
    if (j < n) out[pos] = mine;
    w = wn;
  }
}

// ---- certified weights for large nodes
//
// Nodes above kSubtreeSize primitives: prefix weight of positions [s, j] = sum over the four
// primitive types of (count of that type in [s, j]) x (its construction weight), from a
// segmented inclusive scan of per-type counts, summed in double-double (each product split
// exactly with fma) and rounded once.  The reference's sequential sum of the same k weights
// (all positive) is within (k - 1) u of the exact sum relatively (u = 2^-53, the standard
// bound for recursive summation), so each cost gets a bound on its distance from the
// reference's: the weight errors times the areas, plus the cost expression's own roundings
// in both evaluations, doubled for margin.
struct TypeCounts {
  unsigned long long a, b;  // (sphere | box << 32), (affine sphere | affine box << 32)
};
// sum_t c_t w_t, exact in double-double, rounded once: within one rounding of the true sum.
__device__ __forceinline__ double counts_weight(TypeCounts c, const double* wt) {
  double cnt[4] = {(double)(c.a & 0xFFFFFFFFULL), (double)(c.a >> 32), (double)(c.b & 0xFFFFFFFFULL),
                   (double)(c.b >> 32)};
  double hi = 0.0, lo = 0.0;
  for (int t = 0; t < 4; ++t) {
    double p = cnt[t] * wt[t];
    double pe = fma(cnt[t], wt[t], -p);  // exact: cnt < 2^32 is an integer
    double s = hi + p;                    // two-sum of hi and p
    double bp = s - hi;
    double se = (hi - (s - bp)) + (p - bp);
    hi = s;
    lo = lo + (se + pe);
  }
  return hi + lo;
}

struct TypeWeights {
  double w[4];
};

// ---- segmented scans over node-sorted positions
//
// The positions are sorted by node (key[j]), every node one contiguous segment.  For every
// position j of a node at the current level, the forward scan gives the combination of the
// values over [start of j's node, j] and the backward scan over [j, end of j's node].  Three
// launches cover all three axes: every chunk of kSegChunk positions reduces to its partial
// aggregates in both directions (k_seg_chunks); one block per (axis, direction) carries
// them across the chunks (k_seg_carries); every chunk then scans again with its carries and
// hands each position's results to a consumer (k_seg_apply) that evaluates the split costs
// or the count-based weights in place, so no scanned array is written.  Chunks holding no
// position of a node at the current level do no work (a node at the level never spans
// such a chunk).  Box unions (min / max) and integer sums are exact, so any association of
// them gives the sequential result bit for bit.
// Two items a thread against four, builder's clock in ms: 1M clustered primitives 10.1-10.2 / 10.4-10.5,
// 10k to 300k within 1 %.
#ifndef RTB_SEG_ITEMS
#define RTB_SEG_ITEMS 2
#endif
constexpr int kSegThreads = 256, kSegItems = RTB_SEG_ITEMS, kSegChunk = kSegThreads * kSegItems;
constexpr int kSegWarps = kSegThreads / 32, kCarryThreads = 1024;

template <class V>
struct Seg {
  int flag;  // a segment starts inside the span (in scan order): v starts there
  V v;
};

template <bool DOWN, class V>
__device__ __forceinline__ V shfl_v(V x, int d) {
  static_assert(sizeof(V) % 4 == 0, "values of whole words");
  constexpr int kWords = sizeof(V) / 4;
  int w[kWords];
  memcpy(w, &x, sizeof(V));
#pragma unroll
  for (int q = 0; q < kWords; ++q)
    w[q] = DOWN ? __shfl_down_sync(0xFFFFFFFFu, w[q], d) : __shfl_up_sync(0xFFFFFFFFu, w[q], d);
  memcpy(&x, w, sizeof(V));
  return x;
}

// Segmented scan of a block's items in scan order: thread by thread, ITEMS consecutive
// positions each; REV runs from the block's last position down.  flag[i] marks the first
// position of a segment in scan order.  before[i] / incl[i] combine the segment's values up
// to item i, excluding / including it, with `carry` standing for all positions ahead of
// the block.  Returns the block's own aggregate (carry left out).
template <class O, bool REV, int ITEMS, int WARPS>
__device__ __forceinline__ Seg<typename O::V> seg_scan_block(const int (&flag)[ITEMS],
                                                             const typename O::V (&v)[ITEMS],
                                                             typename O::V carry,
                                                             typename O::V (&before)[ITEMS],
                                                             typename O::V (&incl)[ITEMS],
                                                             Seg<typename O::V>* s_warp) {
  using V = typename O::V;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int tf = 0;
  V tv = O::identity();
#pragma unroll
  for (int q = 0; q < ITEMS; ++q) {
    const int i = REV ? ITEMS - 1 - q : q;
    tv = flag[i] ? v[i] : O::combine(tv, v[i]);
    tf |= flag[i];
  }
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    int of = REV ? __shfl_down_sync(0xFFFFFFFFu, tf, d) : __shfl_up_sync(0xFFFFFFFFu, tf, d);
    V ov = shfl_v<REV>(tv, d);
    if (REV ? lane + d < 32 : lane >= d) {
      if (!tf) tv = O::combine(ov, tv);
      tf |= of;
    }
  }
  int ef = REV ? __shfl_down_sync(0xFFFFFFFFu, tf, 1) : __shfl_up_sync(0xFFFFFFFFu, tf, 1);
  V ev = shfl_v<REV>(tv, 1);
  if (REV ? lane == 31 : lane == 0) {
    ef = 0;
    ev = O::identity();
  }
  if (REV ? lane == 0 : lane == 31) s_warp[w] = Seg<V>{tf, tv};
  __syncthreads();
  V acc = carry;
  Seg<V> agg{0, O::identity()};
  for (int q = 0; q < WARPS; ++q) {
    const int u = REV ? WARPS - 1 - q : q;
    const Seg<V> s = s_warp[u];
    if (REV ? u > w : u < w) acc = s.flag ? s.v : O::combine(acc, s.v);
    agg.v = s.flag ? s.v : O::combine(agg.v, s.v);
    agg.flag |= s.flag;
  }
  V run = ef ? ev : O::combine(acc, ev);
#pragma unroll
  for (int q = 0; q < ITEMS; ++q) {
    const int i = REV ? ITEMS - 1 - q : q;
    before[i] = run;
    run = flag[i] ? v[i] : O::combine(run, v[i]);
    incl[i] = run;
  }
  __syncthreads();  // s_warp is free again
  return agg;
}

// One thread's kSegItems positions from j0: segment starts (head) and ends (tail), node
// ids, and values (the identity outside the loader's active nodes); bit i of the result is
// set when position j0 + i is active.  Positions past n are segments of their own.
template <class L>
__device__ __forceinline__ int seg_load(const L& load, const int* key, int n, int a, int j0,
                                        int (&head)[kSegItems], int (&tail)[kSegItems],
                                        int (&node)[kSegItems], typename L::V (&v)[kSegItems]) {
  int act = 0;
  int kp = j0 > 0 && j0 <= n ? key[j0 - 1] : -1;
#pragma unroll
  for (int i = 0; i < kSegItems; ++i) {
    const int j = j0 + i;
    const int kj = j < n ? key[j] : -1;
    const int kn = j + 1 < n ? key[j + 1] : -1;
    node[i] = kj;
    head[i] = j >= n || j == 0 || kj != kp;
    tail[i] = j >= n || j == n - 1 || kj != kn;
    const bool on = j < n && load.active(kj);
    v[i] = on ? load(a, j) : L::identity();
    act |= (int)on << i;
    kp = kj;
  }
  return act;
}

// Per (chunk, axis): the chunk's aggregate in both directions, the values from its last segment
// start on and those up to its first segment end.  Bounds are minima and maxima and counts
// integers, so each is a plain reduction, by word: 20 reductions a warp.  (Two whole scans,
// some 110 shuffles a warp, of which only the end was kept, took the builder 3.75 ms at 300k
// clustered primitives and 11.0 at 1M, reductions 3.56 and 10.2 to 10.6.)
template <class L>
__global__ void __launch_bounds__(kSegThreads) k_seg_chunks(const L load, const int* key, int n, int nc,
                                                            Seg<typename L::V>* fwd,
                                                            Seg<typename L::V>* bwd) {
  using V = typename L::V;
  __shared__ V s_f[kSegWarps], s_b[kSegWarps];
  __shared__ int s_head[kSegWarps], s_tail[kSegWarps];
  const int a = blockIdx.y, c = blockIdx.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int at = threadIdx.x * kSegItems;
  int head[kSegItems], tail[kSegItems], node[kSegItems];
  V v[kSegItems];
  const int act = seg_load(load, key, n, a, c * kSegChunk + at, head, tail, node, v);
  int last = -1, first = kSegChunk;
#pragma unroll
  for (int i = 0; i < kSegItems; ++i) {
    if (head[i]) last = at + i;
    if (tail[kSegItems - 1 - i]) first = at + kSegItems - 1 - i;
  }
  last = __reduce_max_sync(0xFFFFFFFFu, last);
  first = __reduce_min_sync(0xFFFFFFFFu, first);
  if (lane == 0) {
    s_head[w] = last;
    s_tail[w] = first;
  }
  const size_t slot = (size_t)a * nc + c;
  if (!__syncthreads_or(act)) {
    if (threadIdx.x == 0) fwd[slot] = bwd[slot] = Seg<V>{1, L::identity()};
    return;
  }
  for (int q = 0; q < kSegWarps; ++q) {
    last = max(last, s_head[q]);
    first = min(first, s_tail[q]);
  }
  V vf = L::identity(), vb = L::identity();
#pragma unroll
  for (int i = 0; i < kSegItems; ++i) {
    if (at + i >= last) vf = L::combine(vf, v[i]);
    if (at + i <= first) vb = L::combine(vb, v[i]);
  }
  vf = L::warp_all(vf);
  vb = L::warp_all(vb);
  if (lane == 0) {
    s_f[w] = vf;
    s_b[w] = vb;
  }
  __syncthreads();
  if (threadIdx.x != 0 && threadIdx.x != 32) return;
  const bool rev = threadIdx.x != 0;
  V r = L::identity();
  for (int q = 0; q < kSegWarps; ++q) r = L::combine(r, rev ? s_b[q] : s_f[q]);
  (rev ? bwd : fwd)[slot] = Seg<V>{rev ? first < kSegChunk : last >= 0, r};
}

// Per (axis, direction): chunk aggregates scanned in place over all chunks, 1024 at a time
// with a running carry; afterwards fwd[c] holds the forward result at chunk c's last
// position and bwd[c] the backward result at its first.
template <class O>
__global__ void __launch_bounds__(kCarryThreads) k_seg_carries(int nc, Seg<typename O::V>* fwd,
                                                               Seg<typename O::V>* bwd) {
  using V = typename O::V;
  __shared__ Seg<V> s_warp[kCarryThreads / 32];
  const bool rev = blockIdx.y != 0;
  Seg<V>* s = (rev ? bwd : fwd) + (size_t)blockIdx.x * nc;
  V carry = O::identity();
  const int tiles = (nc + kCarryThreads - 1) / kCarryThreads;
  for (int t = 0; t < tiles; ++t) {
    const int c = (rev ? tiles - 1 - t : t) * kCarryThreads + threadIdx.x;
    const Seg<V> x = c < nc ? s[c] : Seg<V>{1, O::identity()};
    int flag[1] = {x.flag};
    V v[1] = {x.v}, before[1], incl[1];
    Seg<V> agg = rev ? seg_scan_block<O, true, 1, kCarryThreads / 32>(flag, v, carry, before, incl, s_warp)
                     : seg_scan_block<O, false, 1, kCarryThreads / 32>(flag, v, carry, before, incl, s_warp);
    if (c < nc) s[c] = Seg<V>{x.flag, incl[0]};
    carry = agg.flag ? agg.v : O::combine(carry, agg.v);
  }
}

// Per (chunk, axis): both scans with the carries; every active position's split cost by `use`, and
// each node's least cost over the axis's positions.  The minima of a thread's, a warp's and the
// block's positions of one node meet before the one atomic: the nodes' costs are non-negative,
// so their bit patterns order like the values.
template <class L, class U>
__global__ void __launch_bounds__(kSegThreads) k_seg_costs(const L load, const U use, const int* key, int n,
                                                           int nc, const Seg<typename L::V>* fwd,
                                                           const Seg<typename L::V>* bwd,
                                                           unsigned long long* best_bits) {
  using V = typename L::V;
  __shared__ Seg<V> s_warp[kSegWarps];
  __shared__ unsigned long long s_best[kSegWarps];
  __shared__ int s_node[kSegWarps];
  const unsigned long long inf = 0x7FF0000000000000ULL;
  const int a = blockIdx.y, c = blockIdx.x;
  const int j0 = c * kSegChunk + threadIdx.x * kSegItems;
  int head[kSegItems], tail[kSegItems], node[kSegItems];
  V v[kSegItems], fb[kSegItems], fi[kSegItems], bb[kSegItems], bi[kSegItems];
  const int act = seg_load(load, key, n, a, j0, head, tail, node, v);
  if (!__syncthreads_or(act)) return;
  const size_t slot = (size_t)a * nc + c;
  const V cf = c > 0 ? fwd[slot - 1].v : L::identity();
  const V cb = c + 1 < nc ? bwd[slot + 1].v : L::identity();
  seg_scan_block<L, false, kSegItems, kSegWarps>(head, v, cf, fb, fi, s_warp);
  seg_scan_block<L, true, kSegItems, kSegWarps>(tail, v, cb, bb, bi, s_warp);
  int mine = -1;  // the node of the thread's last active positions and their least cost
  unsigned long long least = inf;
#pragma unroll
  for (int i = 0; i < kSegItems; ++i) {
    if (!(act >> i & 1)) continue;
    const unsigned long long bits =
        (unsigned long long)__double_as_longlong(use(a, j0 + i, node[i], tail[i], fb[i], fi[i], bi[i]));
    if (node[i] != mine) {
      if (least != inf) atomicMin(best_bits + mine, least);
      mine = node[i];
      least = inf;
    }
    least = min(least, bits);
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int same = 0;
  __match_all_sync(0xFFFFFFFFu, mine, &same);
  if (same) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) least = min(least, __shfl_xor_sync(0xFFFFFFFFu, least, off));
  } else if (least != inf) {
    atomicMin(best_bits + mine, least);
  }
  if (lane == 0) {
    s_best[w] = same ? least : inf;
    s_node[w] = mine;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    mine = -1;
    least = inf;
    for (int q = 0; q <= kSegWarps; ++q) {
      const int node_q = q < kSegWarps ? s_node[q] : -1;
      if (node_q != mine) {
        if (least != inf) atomicMin(best_bits + mine, least);
        mine = node_q;
        least = inf;
      }
      if (q < kSegWarps) least = min(least, s_best[q]);
    }
  }
}

struct BoxOp {
  using V = Box;
  __device__ static Box identity() {
    Box b;
    for (int k = 0; k < 3; ++k) {
      b.mn[k] = CUDART_INF_F;
      b.mx[k] = -CUDART_INF_F;
    }
    return b;
  }
  __device__ static Box combine(const Box& x, const Box& y) { return BoxUnion()(x, y); }
  // The whole warp's union.
  __device__ static Box warp_all(const Box& x) {
    Box b;
    for (int k = 0; k < 3; ++k) {
      b.mn[k] = o2f(__reduce_min_sync(0xFFFFFFFFu, f2o(x.mn[k])));
      b.mx[k] = o2f(__reduce_max_sync(0xFFFFFFFFu, f2o(x.mx[k])));
    }
    return b;
  }
};

struct CountOp {
  using V = TypeCounts;
  __device__ static TypeCounts identity() { return TypeCounts{0ULL, 0ULL}; }
  __device__ static TypeCounts combine(const TypeCounts& x, const TypeCounts& y) {
    return TypeCounts{x.a + y.a, x.b + y.b};
  }
  // A half's sum stays below 2^32: there are fewer primitives than that.
  __device__ static unsigned long long warp_sum(unsigned long long x) {
    const unsigned lo = __reduce_add_sync(0xFFFFFFFFu, (unsigned)x), hi = __reduce_add_sync(0xFFFFFFFFu, (unsigned)(x >> 32));
    return (unsigned long long)hi << 32 | lo;
  }
  __device__ static TypeCounts warp_all(const TypeCounts& x) { return TypeCounts{warp_sum(x.a), warp_sum(x.b)}; }
};

// Primitive boxes in each axis order, for the nodes at the level.
struct BoxLoad : BoxOp {
  Prims P;
  IdxSet I;
  const int* level_of;
  int level;
  __device__ bool active(int node) const { return level_of[node] == level; }
  __device__ Box operator()(int a, int j) const { return P.box[I.a[a][j]]; }
};

struct BoxCounts {
  Box box;
  TypeCounts counts;
};

struct BoxCountsOp {
  using V = BoxCounts;
  __device__ static BoxCounts identity() {
    BoxCounts r;
    r.box = BoxOp::identity();
    r.counts = CountOp::identity();
    return r;
  }
  __device__ static BoxCounts combine(const BoxCounts& x, const BoxCounts& y) {
    BoxCounts r;
    r.box = BoxOp::combine(x.box, y.box);
    r.counts = CountOp::combine(x.counts, y.counts);
    return r;
  }
  __device__ static BoxCounts warp_all(const BoxCounts& x) {
    BoxCounts r;
    r.box = BoxOp::warp_all(x.box);
    r.counts = CountOp::warp_all(x.counts);
    return r;
  }
};

// Boxes and one-hot type counts in each axis order, for the nodes at the level.
struct BoxCountsLoad : BoxCountsOp {
  Prims P;
  IdxSet I;
  const int* level_of;
  int level;
  __device__ bool active(int node) const { return level_of[node] == level; }
  __device__ BoxCounts operator()(int a, int j) const {
    const int p = I.a[a][j], t = P.type[p];
    const unsigned long long one = 1ULL << (32 * (t & 1));
    BoxCounts r;
    r.box = P.box[p];
    r.counts = t < 2 ? TypeCounts{one, 0ULL} : TypeCounts{0ULL, one};
    return r;
  }
};

// Split cost of every position (GpuScene.java:1482-1485): cost[j] is the cost of putting
// positions [s, j) left; +inf marks positions that are not candidates.  The left bounds
// are the forward scan before j, the right bounds the backward scan at j, and the node's
// bounds their union (written once per node, at its last position, for the axis-0 pass).
struct CostArgs {
  Prims P;
  IdxSet I;
  Nodes N;
  double traversal;
  double* cost[3];
  Box* node_box;  // node bounds at each node's last position
  // Bounds, and whether j is a candidate of node (then with its range).
  __device__ bool candidate(int a, int j, int node, int* s, int* e) const {
    *s = N.start[node];
    *e = N.end[node];
    if (!(j > *s && *e - *s > 1)) return false;
    const int* idx = I.a[a];
    return P.cen[a][idx[*e - 1]] - P.cen[a][idx[*s]] > 1.0e-12;
  }
  __device__ double split(double an, double al, double ar, double wl, double wr) const {
    const double b = al * wl;
    const double d = ar * wr;
    return (an + b) + d;
  }
};

// Unit weights: the sums are exact integers.
struct UnitCosts : CostArgs {
  __device__ double operator()(int a, int j, int node, int tail, const Box& left, const Box& upto,
                               const Box& right) const {
    if (a == 0 && tail) node_box[j] = upto;
    int s, e;
    double c = CUDART_INF;
    if (candidate(a, j, node, &s, &e))
      c = split(surface_area(BoxUnion()(left, right)) * traversal, surface_area(left), surface_area(right),
                (double)(j - s), (double)(e - j));
    cost[a][j] = c;
    return c;
  }
};

// Other weights: from the counts, with bound[j] limiting |cost[j] - the reference's cost|, or for a
// node marked in `seq` from its sequential sums.
struct CountedCosts : CostArgs {
  TypeWeights tw;
  const int* seq;
  const double* pw[3];
  const double* sw[3];
  double* bound[3];
  __device__ double operator()(int a, int j, int node, int tail, const BoxCounts& left, const BoxCounts& upto,
                               const BoxCounts& right) const {
    if (a == 0 && tail) node_box[j] = upto.box;
    int s, e;
    double c = CUDART_INF;
    if (candidate(a, j, node, &s, &e)) {
      const double an = surface_area(BoxUnion()(left.box, right.box)) * traversal;
      const double al = surface_area(left.box), ar = surface_area(right.box);
      if (seq[node]) {
        c = split(an, al, ar, pw[a][j - 1], sw[a][j]);
      } else {
        const double wl = counts_weight(left.counts, tw.w), wr = counts_weight(right.counts, tw.w);
        c = split(an, al, ar, wl, wr);
        const double u = 0x1p-53;
        const double kl = (double)(j - s), kr = (double)(e - j);
        bound[a][j] = 2.0 * (al * wl * (kl * u) + ar * wr * (kr * u) + 8.0 * u * c);
      }
    }
    cost[a][j] = c;
    return c;
  }
};

// A node's winner: the first minimum over (axis, position), by node id.
struct Winners {
  double* cost;     // least cost, +inf with no candidate
  long long* flat;  // axis * count + position of the first candidate that has it
  int* failed;      // the certificate failed
  int* seq;         // weights from sequential sums
};

__device__ __forceinline__ void clear_winner(const Winners& W, int node, int seq) {
  W.cost[node] = CUDART_INF;
  W.flat[node] = 0x7FFFFFFFFFFFFFFFLL;
  W.failed[node] = 0;
  W.seq[node] = seq;
}

__global__ void k_clear_winners(Winners W, int nodes) {
  const int node = blockIdx.x * blockDim.x + threadIdx.x;
  if (node < nodes) clear_winner(W, node, 0);
}

// The strict '<' of the reference's loop keeps the first of equal costs.
__global__ void k_first_minimum(const Nodes N, const int* key, const int* level_of, int level, int n,
                                const CostArgs C, Winners W) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int a = blockIdx.y, node = key[j];
  if (level_of[node] != level) return;
  const double c = C.cost[a][j];
  if (c == CUDART_INF || c != W.cost[node]) return;
  const int s = N.start[node], len = N.end[node] - s;
  atomicMin(W.flat + node, (long long)a * len + (j - s));
}

// A node with count-based weights fails when some other candidate could, in the reference's
// rounding, cost as little as the winner; it is listed once.  A node without a winner (weights
// whose sums overflow leave no cost but NaN) becomes a leaf; it has no position to compare with.
__global__ void k_certify(const Nodes N, const int* key, const int* level_of, int level, int n,
                          const CountedCosts C, Winners W, int* list, int* count) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int a = blockIdx.y, node = key[j];
  if (level_of[node] != level || C.seq[node]) return;
  const double c = C.cost[a][j], best = W.cost[node];
  if (c == CUDART_INF || best == CUDART_INF) return;
  const int s = N.start[node], len = N.end[node] - s;
  const long long flat = W.flat[node];
  if ((long long)a * len + (j - s) == flat) return;
  const int wa = (int)(flat / len), wp = (int)(flat - (long long)wa * len);
  if (c - C.bound[a][j] <= best + C.bound[wa][s + wp] && atomicExch(W.failed + node, 1) == 0)
    list[atomicAdd(count, 1)] = node;
}

// ---- whole subtrees of at most kSubtreeSize primitives, one block each
//
// The recursion of BvhBuildState.build (GpuScene.java:1424-1447) below such a node, depth first,
// with the node's three axis orders in shared memory: per node and axis the suffix boxes and
// weights (weights summed one by one in the reference's order, the same additions as its loop),
// then the prefix pass evaluating every split's cost in the reference's expression order, the
// first minimum over (axis, position), the leaf rule in the node's current order, and a stable
// partition of the other two axis orders.  Every number is the one the level loop would compute
// for the same node; the subtree only saves the per-level passes over all primitives (scans,
// gathers, argmin blocks) that dominate the deep levels.
//
// k_subtrees builds the nodes of more than kWarpNode primitives, one block of three warps a
// subtree and one warp an axis; what is left, nodes of at most kWarpNode, is listed for
// k_small_subtrees, where one warp builds all below one of them with no barrier.  Of at most
// kPackNode primitives the three axes share the warp, eight lanes each: most nodes of a tree are
// that small, and as the block's they were mostly idle lanes and barriers.  10k primitives: 950 ->
// 94 + 68 us, with the ids above (a split took a round trip to a global counter) and centroids
// from the staged boxes; the whole build 2.60 -> 1.65 ms, of 1M 14.9 -> 11.5 ms.
// k_small_subtrees' blocks are single warps so that every branch lies on a value that the compiler
// knows is the same in all lanes (read from shared memory at one address): where it does not,
// each shuffle gets a branch of its own, and the same code inside the three-warp block took 1.6 ms.
constexpr int kSubtreeSize = 512;  // 256: one level-loop round more, 10k 1.69 against 1.65 ms, 1M 11.7 against 11.5
constexpr int kSubtreeThreads = 96;  // one warp per axis
constexpr int kWarpNode = 32, kPackNode = 8;
#ifndef RTB_SUBTREE_BLOCKS_PER_SM
#define RTB_SUBTREE_BLOCKS_PER_SM 5  // 37 KB of shared memory and 80 registers each
#endif
constexpr int kSmallBlocksPerSm = 32;

struct SubtreeSmem {
  // The subtree's primitives get local slots 0..M-1 (axis 0's order at the root); the
  // axis orders hold slots, and the primitives' boxes and weights are staged by slot, so
  // the sweeps read shared memory only.
  int gid[kSubtreeSize];        // slot -> primitive
  Box lbox[kSubtreeSize];
  double lw[kSubtreeSize];
  unsigned char lside[kSubtreeSize];
  int idx[3][kSubtreeSize];     // the subtree's three axis orders (slots)
  union {  // the sweeps' terms, then (the sweeps done) the partition's scratch
    double sterm[3][kSubtreeSize];  // per axis: suffix area x suffix weight of the current node
    int tmp[3][kSubtreeSize];       // per axis: partition scratch
  };
  // Pending nodes, disjoint ranges of more than kWarpNode positions: node, start, end,
  // depth << 2 | (order axis + 1).
  int4 stack[kSubtreeSize / kWarpNode];
  double best_cost[3];
  int best_flat[3];
  int sp;
};

struct SmallSmem {
  Box lbox[kWarpNode];  // by slot, as in SubtreeSmem
  double lw[kWarpNode];
  int gid[kWarpNode];
  int idx[3][kWarpNode];
  unsigned char lside[kWarpNode];
  int4 stack[kWarpNode];
  int leaf, flat;
};

__device__ __forceinline__ Box empty_box() {
  Box b;
  for (int k = 0; k < 3; ++k) {
    b.mn[k] = CUDART_INF_F;
    b.mx[k] = -CUDART_INF_F;
  }
  return b;
}

// Inclusive union over lanes 0..lane (min / max are exact in any order), for the lanes
// below `count` (warp-uniform); lanes from `count` up hold empty boxes and are not needed.
__device__ __forceinline__ Box warp_union_scan(Box b, int lane, int count) {
  for (int off = 1; off < count; off <<= 1) {
    Box o;
    for (int k = 0; k < 3; ++k) {
      o.mn[k] = __shfl_up_sync(0xFFFFFFFFu, b.mn[k], off);
      o.mx[k] = __shfl_up_sync(0xFFFFFFFFu, b.mx[k], off);
    }
    if (lane >= off) b = BoxUnion()(b, o);
  }
  return b;
}

__device__ __forceinline__ Box warp_bcast(const Box& b, int src) {
  Box r;
  for (int k = 0; k < 3; ++k) {
    r.mn[k] = __shfl_sync(0xFFFFFFFFu, b.mn[k], src);
    r.mx[k] = __shfl_sync(0xFFFFFFFFu, b.mx[k], src);
  }
  return r;
}

// Running sums of the lanes' weights in lane order, continuing `acc`: lane q gets
// acc + w_0 + ... + w_q added one by one, for the lanes below `count` (warp-uniform).  The
// chain runs in groups of four lanes, each group's shuffles issued ahead of its additions;
// lanes past the node's end carry w = 0, and adding +0 to a non-negative sum leaves it
// unchanged, so the last group may run past `count`.
__device__ __forceinline__ double warp_sequential_sum(double w, double& acc, int lane, int count) {
  double mine = 0.0;
  for (int g = 0; g < count; g += 4) {
    double v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = __shfl_sync(0xFFFFFFFFu, w, g + q);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      acc = acc + v[q];
      mine = g + q == lane ? acc : mine;
    }
  }
  return mine;
}

__device__ __forceinline__ bool lex_less(double c, int f, double bc, int bf) {
  return c < bc || (c == bc && f < bf);
}

// A staged primitive's centroid, as k_prims computes it from the same bounds.
__device__ __forceinline__ double box_centroid(const Box& b, int axis) {
  return ((double)b.mn[axis] + (double)b.mx[axis]) * 0.5;
}

// Splits of a node of m <= W positions on the axis of this lane's group of W lanes: the best
// (cost, axis * m + position) of the group's positions in *best and *flat, lane by lane, and the
// node's bounds.  W = 8: groups 0..2 are the axes, group 3 has none (axis < 0).
template <int W>
__device__ __forceinline__ Box group_sweep(const SmallSmem& sm, int axis, int lo, int m, double traversal,
                                           double* best, int* flat) {
  const int i = (int)(threadIdx.x & 31) & (W - 1);
  const bool in = i < m && axis >= 0;
  const int slot = in ? sm.idx[axis][lo + i] : 0;
  Box pre = in ? sm.lbox[slot] : empty_box();
  Box suf = pre;
  const double w = in ? sm.lw[slot] : 0.0;
  // suffix sums from the last position down (GpuScene.java:1476-1480) and prefix sums (1470-1475),
  // two chains of additions side by side; positions from m up carry 0, which changes no sum
  double sw = 0.0, pw = 0.0, down = 0.0, up = 0.0;
  const int steps = W == 8 ? 8 : (m + 3) & ~3;
#pragma unroll
  for (int g0 = 0; g0 < W; g0 += 4) {
    if (W > 8 && g0 >= steps) break;
    double vu[4], vd[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      vu[q] = __shfl_sync(0xFFFFFFFFu, w, g0 + q, W);
      vd[q] = __shfl_sync(0xFFFFFFFFu, w, steps - 1 - g0 - q, W);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      up = up + vu[q];
      pw = g0 + q == i - 1 ? up : pw;  // of the positions before i
      down = down + vd[q];
      sw = steps - 1 - g0 - q == i ? down : sw;
    }
  }
#pragma unroll
  for (int off = 1; off < W; off <<= 1) {
    Box u, d;
    for (int k = 0; k < 3; ++k) {
      u.mn[k] = __shfl_up_sync(0xFFFFFFFFu, pre.mn[k], off, W);
      u.mx[k] = __shfl_up_sync(0xFFFFFFFFu, pre.mx[k], off, W);
      d.mn[k] = __shfl_down_sync(0xFFFFFFFFu, suf.mn[k], off, W);
      d.mx[k] = __shfl_down_sync(0xFFFFFFFFu, suf.mx[k], off, W);
    }
    if (i >= off) pre = BoxUnion()(pre, u);
    if (i + off < W) suf = BoxUnion()(suf, d);
  }
  const Box node = warp_bcast(suf, 0);  // group 0's first suffix: everything
  Box left;
  for (int k = 0; k < 3; ++k) {
    left.mn[k] = __shfl_up_sync(0xFFFFFFFFu, pre.mn[k], 1, W);
    left.mx[k] = __shfl_up_sync(0xFFFFFFFFu, pre.mx[k], 1, W);
  }
  *best = CUDART_INF;
  *flat = 0x7FFFFFFF;
  if (in && i > 0) {
    const int f = sm.idx[axis][lo], l = sm.idx[axis][lo + m - 1];
    if (box_centroid(sm.lbox[l], axis) - box_centroid(sm.lbox[f], axis) > 1.0e-12) {
      const double node_a = surface_area(node) * traversal;
      const double bl = surface_area(left) * pw;
      const double d = surface_area(suf) * sw;
      *best = (node_a + bl) + d;
      *flat = axis * m + i;
    }
  }
  return node;
}

// The leaf rule's sequential weight sum, in the node's current order (GpuScene.java:1435-1441).
template <class Smem>
__device__ __forceinline__ double order_weight(const Smem& sm, const Prims& P, int oa, int s, int lo, int m) {
  double sum = 0.0;
  for (int j = 0; j < m; ++j) sum = sum + (oa < 0 ? P.w[s + j] : sm.lw[sm.idx[oa][lo + j]]);
  return sum;
}

// Everything below each listed node of at most kWarpNode primitives, a warp (the block) a node,
// depth first.
__global__ void __launch_bounds__(32, kSmallBlocksPerSm) k_small_subtrees(const Prims P, IdxSet I, Nodes N,
                                                                         const int4* list, const int* count,
                                                                         int roots, int leaf_size,
                                                                         double traversal, int* stats) {
  __shared__ SmallSmem sm;
  const int lane = threadIdx.x;
  LeafStats st{0, 0x7FFFFFFF, 0, 0};
  const int listed = *count;
  for (int k = blockIdx.x; k < listed; k += gridDim.x) {
    int4 en = list[k];
    const int rs = en.y, M = en.z - en.y;
    {
      int p[3];
      for (int a = 0; a < 3; ++a) p[a] = lane < M ? I.a[a][rs + lane] : -1 - a;
      if (lane < M) {
        sm.gid[lane] = p[0];
        sm.lbox[lane] = P.box[p[0]];
        sm.lw[lane] = P.w[p[0]];
        sm.idx[0][lane] = lane;
      }
      int s1 = 0, s2 = 0;
      for (int j = 0; j < M; ++j) {
        const int q = __shfl_sync(0xFFFFFFFFu, p[0], j);
        s1 = q == p[1] ? j : s1;
        s2 = q == p[2] ? j : s2;
      }
      if (lane < M) sm.idx[1][lane] = s1, sm.idx[2][lane] = s2;
    }
    __syncwarp();
    int sp = 0;
    while (true) {
      const int node = en.x, s = en.y, e = en.z, m = e - s, lo = s - rs;
      const int oa = (en.w & 3) - 1, depth = en.w >> 2;
      double best = CUDART_INF;
      int flat = 0x7FFFFFFF;
      Box nb;
      if (m == 1) {
        nb = sm.lbox[sm.idx[0][lo]];
      } else if (m <= kPackNode) {
        nb = group_sweep<kPackNode>(sm, lane < 24 ? lane >> 3 : -1, lo, m, traversal, &best, &flat);
      } else {
        for (int a = 0; a < 3; ++a) {
          double c;
          int f;
          nb = group_sweep<32>(sm, a, lo, m, traversal, &c, &f);
          if (lex_less(c, f, best, flat)) best = c, flat = f;
        }
      }
      if (m > 1) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
          const double oc = __shfl_xor_sync(0xFFFFFFFFu, best, off);
          const int of = __shfl_xor_sync(0xFFFFFFFFu, flat, off);
          if (lex_less(oc, of, best, flat)) best = oc, flat = of;
        }
      }
      if (lane == 0) {
        int leaf = m == 1 || best == CUDART_INF;
        if (!leaf && m <= leaf_size && !(best < surface_area(nb) * order_weight(sm, P, oa, s, lo, m))) leaf = 1;
        sm.leaf = leaf;
        sm.flat = flat;
        N.bounds[node] = nb;
        N.split_axis[node] = -1;
        if (leaf) {
          N.leaf[node] = 1;
          st.add(m, depth);
        }
      }
      __syncwarp();
      if (sm.leaf) {
        if (sp == 0) break;
        en = sm.stack[--sp];
        __syncwarp();
        continue;
      }
      const int axis = sm.flat / m, pos = sm.flat - axis * m;
      const int l = child_id(roots, s + pos);
      if (lane == 0) write_split(N, node, l, axis, pos, s, e, depth);
      // stable partition of the other two axis orders by side
      if (lane < m) sm.lside[sm.idx[axis][lo + lane]] = lane >= pos ? 1 : 0;
      __syncwarp();
      for (int q = 1; q < 3; ++q) {
        int* ix = sm.idx[axis + q < 3 ? axis + q : axis + q - 3] + lo;
        const int p = lane < m ? ix[lane] : 0;
        const bool right = lane < m && sm.lside[p] != 0;
        const unsigned rm = __ballot_sync(0xFFFFFFFFu, right), below = (1u << lane) - 1u;
        const int rank = __popc(rm & below);
        if (lane < m) ix[right ? pos + rank : lane - rank] = p;
      }
      const int meta = ((depth + 1) << 2) | (axis + 1);
      if (lane == 0) sm.stack[sp] = make_int4(l + 1, s + pos, e, meta);
      sp++;
      en = make_int4(l, s, s + pos, meta);
      __syncwarp();
    }
    // the axis orders back in place: finishing reads a leaf's references in its order axis
    for (int a = 0; a < 3; ++a)
      if (lane < M) I.a[a][rs + lane] = sm.gid[sm.idx[a][lane]];
    __syncwarp();
  }
  if (lane == 0) st.add_to(stats);
}

__global__ void __launch_bounds__(kSubtreeThreads, RTB_SUBTREE_BLOCKS_PER_SM) k_subtrees(
    const Prims P, IdxSet I, Nodes N, const int* roots_list, const int* root_count, int roots, int leaf_size,
    double traversal, int* stats, int* slot_of, int4* small, int* small_count) {
  __shared__ SubtreeSmem sm;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if ((int)blockIdx.x >= *root_count) return;
  const int root = roots_list[blockIdx.x];
  const int rs = N.start[root], re = N.end[root], M = re - rs;
  for (int i = threadIdx.x; i < M; i += kSubtreeThreads) {
    int p = I.a[0][rs + i];
    sm.gid[i] = p;
    sm.lbox[i] = P.box[p];
    sm.lw[i] = P.w[p];
    slot_of[p] = i;  // each primitive belongs to one subtree
    sm.idx[0][i] = i;
  }
  __syncthreads();
  for (int a = 1; a < 3; ++a)
    for (int i = threadIdx.x; i < M; i += kSubtreeThreads) sm.idx[a][i] = slot_of[I.a[a][rs + i]];
  if (threadIdx.x == 0) {
    const int4 en = make_int4(root, rs, re, (N.depth[root] << 2) | (N.order_axis[root] + 1));
    sm.stack[0] = en;
    sm.sp = M > kWarpNode ? 1 : 0;
    if (M <= kWarpNode) small[atomicAdd(small_count, 1)] = en;
  }
  // the subtree's statistics, kept by thread 0 and added to the build's once at the end
  LeafStats st{0, 0x7FFFFFFF, 0, 0};
  __syncthreads();
  // ---- the block's nodes: warp a sweeps axis a, the block takes the first minimum over the three
  // axes' winners, and the warps of the two other axes partition their orders.  Every decision is
  // computed identically by all threads (or broadcast through shared memory), so the block's
  // barriers are uniform.
  while (sm.sp > 0) {
    const int4 en = sm.stack[sm.sp - 1];
    __syncthreads();
    if (threadIdx.x == 0) sm.sp--;
    const int node = en.x, s = en.y, e = en.z, m = e - s, lo = s - rs;
    const int oa = (en.w & 3) - 1, depth = en.w >> 2;
    // node bounds (every warp computes the same union)
    Box nb = empty_box();
    for (int i = lane; i < m; i += 32) nb = BoxUnion()(nb, sm.lbox[sm.idx[0][lo + i]]);
    for (int off = 1; off < 32; off <<= 1) {
      Box o;
      for (int k = 0; k < 3; ++k) {
        o.mn[k] = __shfl_xor_sync(0xFFFFFFFFu, nb.mn[k], off);
        o.mx[k] = __shfl_xor_sync(0xFFFFFFFFu, nb.mx[k], off);
      }
      nb = BoxUnion()(nb, o);
    }
    const double node_a = surface_area(nb) * traversal;
    // this warp's axis
    double best = CUDART_INF;
    int best_flat = 0x7FFFFFFF;
    const int a = warp;
    const int* ix = sm.idx[a] + lo;
    if (box_centroid(sm.lbox[ix[m - 1]], a) - box_centroid(sm.lbox[ix[0]], a) > 1.0e-12) {
      // suffix boxes and weights, from the last position down (GpuScene.java:1476-1480)
      Box carry = empty_box();
      double acc = 0.0;
      for (int base = 0; base < m; base += 32) {
        const int cnt = min(32, m - base);
        int q = m - 1 - (base + lane);
        Box b = q >= 0 ? sm.lbox[ix[q]] : empty_box();
        double w = q >= 0 ? sm.lw[ix[q]] : 0.0;
        b = BoxUnion()(warp_union_scan(b, lane, cnt), carry);
        double sw = warp_sequential_sum(w, acc, lane, cnt);
        if (q >= 0) sm.sterm[a][lo + q] = surface_area(b) * sw;
        carry = warp_bcast(b, cnt - 1);
      }
      __syncwarp();
      // prefix pass and the cost of putting local positions [0, i) left (1470-1475, 1482-1485)
      carry = empty_box();
      acc = 0.0;
      for (int base = 0; base < m; base += 32) {
        const int cnt = min(32, m - base);
        int li = base + lane;
        Box b = li < m ? sm.lbox[ix[li]] : empty_box();
        double w = li < m ? sm.lw[ix[li]] : 0.0;
        b = BoxUnion()(warp_union_scan(b, lane, cnt), carry);
        double pw = warp_sequential_sum(w, acc, lane, cnt);
        int i = li + 1;  // split after li
        if (i < m) {
          double bl = surface_area(b) * pw;
          double d = sm.sterm[a][lo + i];
          double c = (node_a + bl) + d;
          const int flat = a * m + i;
          if (lex_less(c, flat, best, best_flat)) {
            best = c;
            best_flat = flat;
          }
        }
        carry = warp_bcast(b, cnt - 1);
      }
      for (int off = 16; off > 0; off >>= 1) {
        double oc = __shfl_xor_sync(0xFFFFFFFFu, best, off);
        int of = __shfl_xor_sync(0xFFFFFFFFu, best_flat, off);
        if (lex_less(oc, of, best, best_flat)) {
          best = oc;
          best_flat = of;
        }
      }
    }
    if (lane == 0) {
      sm.best_cost[a] = best;
      sm.best_flat[a] = best_flat;
    }
    __syncthreads();
    best = sm.best_cost[0];
    best_flat = sm.best_flat[0];
    for (int k = 1; k < 3; ++k)
      if (lex_less(sm.best_cost[k], sm.best_flat[k], best, best_flat)) {
        best = sm.best_cost[k];
        best_flat = sm.best_flat[k];
      }
    bool leaf = best == CUDART_INF;
    if (!leaf && m <= leaf_size && !(best < surface_area(nb) * order_weight(sm, P, oa, s, lo, m))) leaf = true;
    if (threadIdx.x == 0) {
      N.bounds[node] = nb;
      N.split_axis[node] = -1;
    }
    if (leaf) {
      if (threadIdx.x == 0) {
        N.leaf[node] = 1;
        st.add(m, depth);
      }
      __syncthreads();
      continue;
    }
    const int axis = best_flat / m, pos = best_flat % m;
    if (threadIdx.x == 0) {
      const int l = child_id(roots, s + pos);
      write_split(N, node, l, axis, pos, s, e, depth);
      const int meta = ((depth + 1) << 2) | (axis + 1);
      const int4 kids[2] = {make_int4(l + 1, s + pos, e, meta), make_int4(l, s, s + pos, meta)};
      for (int h = 0; h < 2; ++h) {
        if (kids[h].z - kids[h].y > kWarpNode) sm.stack[sm.sp++] = kids[h];
        else small[atomicAdd(small_count, 1)] = kids[h];
      }
    }
    // stable partition of the other two axis orders by side
    if (warp == axis)
      for (int i = lane; i < m; i += 32) sm.lside[sm.idx[axis][lo + i]] = i >= pos ? 1 : 0;
    __syncthreads();
    if (warp != axis) {
      int* t = sm.tmp[a];
      int nl = 0, nr = 0;
      for (int base = 0; base < m; base += 32) {
        int li = base + lane;
        bool in = li < m;
        int p = in ? sm.idx[a][lo + li] : 0;
        const bool right = in && sm.lside[p] != 0;
        const unsigned rm = __ballot_sync(0xFFFFFFFFu, right);
        const unsigned lm = __ballot_sync(0xFFFFFFFFu, in && !right);
        const unsigned below = (1u << lane) - 1u;
        if (in) t[right ? pos + nr + __popc(rm & below) : nl + __popc(lm & below)] = p;
        nl += __popc(lm);
        nr += __popc(rm);
      }
      __syncwarp();
      for (int i = lane; i < m; i += 32) sm.idx[a][lo + i] = t[i];
    }
    __syncthreads();
  }
  for (int a = 0; a < 3; ++a)
    for (int i = threadIdx.x; i < M; i += kSubtreeThreads) I.a[a][rs + i] = sm.gid[sm.idx[a][i]];
  if (threadIdx.x == 0) st.add_to(stats);
}

// Leaf-or-split decision per active node (GpuScene.java:1424-1447).  A node whose certificate
// failed stays for the next round, with sequential weights.
__global__ void k_decide(const Prims P, IdxSet I, Nodes N, const int* active, int k, Winners W,
                         const Box* node_box, int leaf_size, int roots, int* next_active, int* next_count,
                         int* level_of, int level, int* stats, int* small_roots, int* small_count) {
  int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= k) return;
  int node = active[g];
  int s = N.start[node], e = N.end[node];
  int n = e - s;
  N.split_axis[node] = -1;
  if (W.failed[node]) {
    clear_winner(W, node, 1);
    level_of[node] = level + 1;
    next_active[atomicAdd(next_count, 1)] = node;
    return;
  }
  Box bounds = node_box[e - 1];
  N.bounds[node] = bounds;
  const double best = W.cost[node];
  bool leaf = n == 1 || best == CUDART_INF;
  if (!leaf && n <= leaf_size) {
    double wsum = 0.0;
    for (int j = s; j < e; ++j) wsum = wsum + P.w[current_prim(I.a, N.order_axis[node], j)];
    double leaf_cost = surface_area(bounds) * wsum;
    if (!(best < leaf_cost)) leaf = true;
  }
  if (leaf) {
    N.leaf[node] = 1;
    atomicAdd(stats + 0, 1);                 // leaves
    atomicMin(stats + 1, n);                 // min occupancy
    atomicMax(stats + 2, n);                 // max occupancy
    atomicMax(stats + 3, N.depth[node]);     // max depth
    return;
  }
  const long long flat = W.flat[node];
  const int axis = (int)(flat / n), pos = (int)(flat % n);
  const int l = child_id(roots, s + pos);
  write_split(N, node, l, axis, pos, s, e, N.depth[node]);
  // children of at most kSubtreeSize primitives leave the level loop: k_subtrees builds
  // their whole subtrees later (level_of -1 keeps the level kernels off their positions)
  const int sizes[2] = {pos, n - pos};
  for (int h = 0; h < 2; ++h) {
    if (sizes[h] <= kSubtreeSize) {
      level_of[l + h] = -1;
      small_roots[atomicAdd(small_count, 1)] = l + h;
    } else {
      level_of[l + h] = level + 1;
      clear_winner(W, l + h, 0);
      next_active[atomicAdd(next_count, 1)] = l + h;
    }
  }
}

// Stable partition of the three axis orders of every node split at this level, one axis per
// blockIdx.y: left flags, one exclusive sum over all 3n of them (a node's left rank is a difference
// inside its own axis range, so the other axes' counts cancel), then the scatter, which also gives
// the positions of split nodes their children's keys.  (Flags made as the scan reads them: the
// scan's few threads wait for the chain of gathers, 1.6 ms for 0.42 + 0.2 at 1M.)
__global__ void k_left_flags3(IdxSet I, const Nodes N, const int* key, const int* level_of, int level,
                              int n, const unsigned char* side, int* flags) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int a = blockIdx.y;
  const int node = key[j];
  const bool split = level_of[node] == level && N.split_axis[node] >= 0;
  flags[(size_t)a * n + j] = split ? (side[I.a[a][j]] == 0) : 0;
}

__global__ void k_scatter3(IdxSet I, IdxSet T, const Nodes N, const int* key, int* key_out, const int* level_of,
                           int level, int n, const unsigned char* side, const int* lscan) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int a = blockIdx.y;
  const int node = key[j];
  const int p = I.a[a][j];
  int* out = T.a[a];
  if (!(level_of[node] == level && N.split_axis[node] >= 0)) {
    out[j] = p;
    if (a == 0) key_out[j] = node;
    return;
  }
  const int* ls = lscan + (size_t)a * n;
  const int s = N.start[node], pos = N.split_pos[node];
  const int lrank = ls[j] - ls[s];
  out[side[p] == 0 ? s + lrank : s + pos + ((j - s) - lrank)] = p;
  if (a == 0) key_out[j] = N.left[node] + (j < s + pos ? 0 : 1);
}

__global__ void k_sides(IdxSet I, const Nodes N, const int* key, const int* level_of, int level, int n,
                        unsigned char* side) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  int node = key[j];
  if (level_of[node] != level) return;
  int axis = N.split_axis[node];
  if (axis < 0) return;
  int p = I.a[axis][j];
  side[p] = (j - N.start[node]) >= N.split_pos[node] ? 1 : 0;
}



// ---- BvhRotator (GpuScene.java:968-1057) on the device
//
// A pass visits the tree bottom-up; at each interior node it compares the current node
// with the four rotations that swap a grandchild with the uncle, by areaCost (surface area
// times c_T per interior node plus surface area times the leaf's sequential weight sum per
// leaf), and keeps the first one cheaper by more than 1e-12.  The decision at a node only
// reads its own subtree, which the deeper levels have already settled, so each level runs
// in parallel.  The reference recomputes areaCost recursively for every candidate; here each
// node keeps its settled subtree's cost, and a candidate's cost adds the same terms in the
// same order ((A_node c_T + cost(left)) + cost(right)), so every comparison is the
// reference's to the bit.  A rotation reuses the child slot it restructures.

// Breadth-first levels of the current tree: children of the frontier.
__global__ void k_next_level(const Nodes N, const int* frontier, int k, int* next, int* next_count) {
  int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= k) return;
  int node = frontier[g];
  if (N.leaf[node]) return;
  int q = atomicAdd(next_count, 2);
  next[q] = N.left[node];
  next[q + 1] = N.right[node];
}

__global__ void k_leaf_area_cost(const Prims P, IdxSet I, const Nodes N, const int* nodes, int k,
                                 double* rcost) {
  int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= k) return;
  int node = nodes[g];
  if (!N.leaf[node]) return;
  double w = 0.0;
  for (int j = N.start[node]; j < N.end[node]; ++j) w = w + P.w[current_prim(I.a, N.order_axis[node], j)];
  rcost[node] = surface_area(N.bounds[node]) * w;
}

__device__ __forceinline__ Box box_union(const Box& a, const Box& b) { return BoxUnion()(a, b); }

__global__ void k_rotate_level(Nodes N, const int* nodes, int k, double traversal, double* rcost,
                               int* rotations) {
  int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= k) return;
  int n = nodes[g];
  if (N.leaf[n]) return;
  const double eps = 1.0e-12;
  int L = N.left[n], R = N.right[n];
  double top = surface_area(N.bounds[n]) * traversal;
  double x = top + rcost[L];
  double best = x + rcost[R];
  int choice = 0;
  double inner_best = 0.0;
  if (!N.leaf[L]) {
    int a = N.left[L], b = N.right[L], c = R;
    // join(a, join(b, c))
    double in1 = surface_area(box_union(N.bounds[b], N.bounds[c])) * traversal;
    in1 = in1 + rcost[b];
    in1 = in1 + rcost[c];
    double c1 = top + rcost[a];
    c1 = c1 + in1;
    if (c1 < best - eps) {
      best = c1;
      choice = 1;
      inner_best = in1;
    }
    // join(b, join(a, c))
    double in2 = surface_area(box_union(N.bounds[a], N.bounds[c])) * traversal;
    in2 = in2 + rcost[a];
    in2 = in2 + rcost[c];
    double c2 = top + rcost[b];
    c2 = c2 + in2;
    if (c2 < best - eps) {
      best = c2;
      choice = 2;
      inner_best = in2;
    }
  }
  if (!N.leaf[R]) {
    int a = L, b = N.left[R], c = N.right[R];
    // join(join(a, c), b)
    double in3 = surface_area(box_union(N.bounds[a], N.bounds[c])) * traversal;
    in3 = in3 + rcost[a];
    in3 = in3 + rcost[c];
    double c3 = top + in3;
    c3 = c3 + rcost[b];
    if (c3 < best - eps) {
      best = c3;
      choice = 3;
      inner_best = in3;
    }
    // join(join(a, b), c)
    double in4 = surface_area(box_union(N.bounds[a], N.bounds[b])) * traversal;
    in4 = in4 + rcost[a];
    in4 = in4 + rcost[b];
    double c4 = top + in4;
    c4 = c4 + rcost[c];
    if (c4 < best - eps) {
      best = c4;
      choice = 4;
      inner_best = in4;
    }
  }
  if (choice == 1 || choice == 2) {
    int a = N.left[L], b = N.right[L], c = R;
    int outer = choice == 1 ? a : b, p = choice == 1 ? b : a;
    N.left[n] = outer;
    N.right[n] = L;
    N.left[L] = p;
    N.right[L] = c;
    N.bounds[L] = box_union(N.bounds[p], N.bounds[c]);
    rcost[L] = inner_best;
  } else if (choice == 3 || choice == 4) {
    int a = L, b = N.left[R], c = N.right[R];
    int q = choice == 3 ? c : b, outer = choice == 3 ? b : c;
    N.left[n] = R;
    N.right[n] = outer;
    N.left[R] = a;
    N.right[R] = q;
    N.bounds[R] = box_union(N.bounds[a], N.bounds[q]);
    rcost[R] = inner_best;
  }
  rcost[n] = best;
  if (choice) atomicAdd(rotations, 1);
}

// Breadth-first levels of the tree under `roots`: nodes level by level in `all_nodes`,
// level starts in level_begin.  Returns false on a CUDA error.
bool tree_levels(const Nodes& N, int roots, int* all_nodes, int* counter, std::vector<int>& level_begin,
                 cudaStream_t sm) {
  std::vector<int> h(roots);
  for (int r = 0; r < roots; ++r) h[r] = r;
  cudaMemcpyAsync(all_nodes, h.data(), roots * 4, cudaMemcpyHostToDevice, sm);
  level_begin.assign(1, 0);
  int begin = 0, k = roots;
  while (k > 0) {
    level_begin.push_back(begin + k);
    cudaMemsetAsync(counter, 0, 4, sm);
    k_next_level<<<blocks(k), 256, 0, sm>>>(N, all_nodes + begin, k, all_nodes + begin + k, counter);
    int next = 0;
    cudaMemcpyAsync(&next, counter, 4, cudaMemcpyDeviceToHost, sm);
    if (cudaStreamSynchronize(sm) != cudaSuccess) return false;
    begin += k;
    k = next;
  }
  return true;
}

}  // namespace

rtb_status build_bvh(rtb_context* ctx, const rtb_scene_desc* desc, const rtb_build_config* cfg,
                     rtb_scene** out, rtb_bvh_stats* stats) {
  return build_bvh_options(ctx, desc, cfg, nullptr, out, stats);
}

rtb_status build_bvh_options(rtb_context* ctx, const rtb_scene_desc* desc, const rtb_build_config* cfg,
                             const rtb_build_options* options, rtb_scene** out, rtb_bvh_stats* stats) {
  if (!out) return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "null argument");
  if (cfg && (cfg->mode == 4 || cfg->mode == 5)) return build_bvh_sbvh(ctx, desc, cfg, options, out, stats);
  BuildCfg c;
  bool per_type = false;
  rtb_status st = build_setup(ctx, desc, cfg, c, per_type, true);
  if (st != RTB_OK) return st;
  int rotation_passes = options ? options->rotation_passes : 4;  // BvhBuildOptions.defaults
  bool rotate = cfg->mode == 6 || cfg->mode == 7;
  if (rotate && rotation_passes < 1)
    return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "rotationPasses must be positive.");
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
  IdxSet I, T;
  for (int k = 0; k < 3; ++k) {
    I.a[k] = W.alloc<int>(n);
    T.a[k] = W.alloc<int>(n);
  }
  int cap = 2 * n + 8;
  Nodes N = alloc_nodes(W, cap);
  int* level_of = W.alloc<int>(cap);
  int* key = W.alloc<int>(n);
  int* key2 = W.alloc<int>(n);
  Box* node_box = W.alloc<Box>(n);  // a node's bounds at its last position
  const int nc = (n + kSegChunk - 1) / kSegChunk;
  const size_t seg = c.weighted ? sizeof(Seg<BoxCounts>) : sizeof(Seg<Box>);
  char* seg_fwd = W.alloc<char>(3 * (size_t)nc * seg);
  char* seg_bwd = W.alloc<char>(3 * (size_t)nc * seg);
  WeightChains chains;
  double* cost[3];
  double* bound[3];
  for (int a = 0; a < 3; ++a) {
    chains.w[a] = c.weighted ? W.alloc<double>(n) : nullptr;
    chains.pw[a] = c.weighted ? W.alloc<double>(n) : nullptr;
    chains.sw[a] = c.weighted ? W.alloc<double>(n) : nullptr;
    cost[a] = W.alloc<double>(n);
    bound[a] = c.weighted ? W.alloc<double>(n) : nullptr;
  }
  Winners win{W.alloc<double>(cap), W.alloc<long long>(cap), W.alloc<int>(cap), W.alloc<int>(cap)};
  int* failed_list = W.alloc<int>(cap);
  int* lists = W.alloc<int>(2);  // next round's nodes, failed nodes
  int* sub_roots = W.alloc<int>(cap);  // nodes whose subtrees k_subtrees builds
  unsigned char* side = W.alloc<unsigned char>(n);
  int* flags = W.alloc<int>(3 * (size_t)n);  // left flags of the three axis orders
  int* lscan = W.alloc<int>(3 * (size_t)n);
  const int n3 = 3 * n;
  unsigned long long* skeys = W.alloc<unsigned long long>(n3);
  unsigned long long* skeys2 = W.alloc<unsigned long long>(n3);
  unsigned* svals = W.alloc<unsigned>(n3);
  unsigned* svals2 = W.alloc<unsigned>(n3);
  unsigned char* tags = W.alloc<unsigned char>(n3);
  unsigned char* tags2 = W.alloc<unsigned char>(n3);
  int* active = W.alloc<int>(cap);
  int* next_active = W.alloc<int>(cap);
  int4* small_list = W.alloc<int4>(n);  // nodes that k_small_subtrees builds
  int* counters = W.alloc<int>(8);  // their number, -, stats[4], -, subtrees
  int* root_start = W.alloc<int>(4);
  int* root_end = W.alloc<int>(4);
  size_t tmp_bytes = 0, b1 = 0, b3 = 0, b4 = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, b1, skeys, skeys2, svals, svals2, n3);
  cub::DeviceScan::ExclusiveSum(nullptr, b3, flags, lscan, 3 * n);
  cub::DeviceRadixSort::SortPairs(nullptr, b4, tags, tags2, svals2, svals, n3, 0, 4);
  tmp_bytes = std::max(b1, std::max(b3, b4));
  void* tmp = W.alloc<char>(tmp_bytes);
  if (!W.ok) return fail(ctx, RTB_ERR_OUT_OF_MEMORY, "BVH build workspace");

  cudaEventRecord(ctx->ev0, sm);
  upload_prims(desc, c, in, P, sm);

  // ---- axis orders: (centroid, order), then (type, centroid, order) for per-type forests
  {
    const dim3 per_axis(blocks(n), 3);
    k_keys<<<per_axis, 256, 0, sm>>>(P, n, skeys, svals);
    const int groups = n <= kTileSort ? 3 : 1, each = n3 / groups;
    size_t tb = tmp_bytes;
    for (int g = 0; g < groups; ++g)
      cub::DeviceRadixSort::SortPairs(tmp, tb, skeys + (size_t)g * each, skeys2 + (size_t)g * each,
                                      svals + (size_t)g * each, svals2 + (size_t)g * each, each, 0, 64, sm);
    const unsigned* ordered = svals2;
    if (groups == 1 || per_type) {
      k_axis_tags<<<blocks(n3), 256, 0, sm>>>(P, svals2, n3, per_type ? 1 : 0, tags);
      tb = tmp_bytes;
      cub::DeviceRadixSort::SortPairs(tmp, tb, tags, tags2, svals2, svals, n3, 0, 4, sm);
      ordered = svals;
    }
    k_axis_orders<<<per_axis, 256, 0, sm>>>(ordered, n, I);
  }

  // ---- roots
  int h_rs[4], h_re[4];
  int roots = root_ranges(c, per_type, h_rs, h_re);
  int h_counters[8] = {0, 0, 0, 0x7FFFFFFF, 0, 0, 0, 0};
  cudaMemcpyAsync(root_start, h_rs, roots * 4, cudaMemcpyHostToDevice, sm);
  cudaMemcpyAsync(root_end, h_re, roots * 4, cudaMemcpyHostToDevice, sm);
  cudaMemcpyAsync(N.start, h_rs, roots * 4, cudaMemcpyHostToDevice, sm);
  cudaMemcpyAsync(N.end, h_re, roots * 4, cudaMemcpyHostToDevice, sm);
  // roots of at most kSubtreeSize primitives go straight to the subtree kernel
  std::vector<int> h_big, h_small, h_level(roots);
  for (int r = 0; r < roots; ++r) {
    bool small = h_re[r] - h_rs[r] <= kSubtreeSize;
    (small ? h_small : h_big).push_back(r);
    h_level[r] = small ? -1 : 0;
  }
  h_counters[7] = (int)h_small.size();
  if (!h_big.empty())
    cudaMemcpyAsync(active, h_big.data(), h_big.size() * 4, cudaMemcpyHostToDevice, sm);
  if (!h_small.empty())
    cudaMemcpyAsync(sub_roots, h_small.data(), h_small.size() * 4, cudaMemcpyHostToDevice, sm);
  cudaMemcpyAsync(counters, h_counters, sizeof(h_counters), cudaMemcpyHostToDevice, sm);
  cudaMemsetAsync(N.order_axis, 0xFF, (size_t)roots * 4, sm);  // -1: input order
  cudaMemsetAsync(N.depth, 0, (size_t)roots * 4, sm);
  cudaMemsetAsync(N.leaf, 0xFF, (size_t)cap * 4, sm);  // -1: no node
  cudaMemcpyAsync(level_of, h_level.data(), roots * 4, cudaMemcpyHostToDevice, sm);
  k_init_keys<<<blocks(n), 256, 0, sm>>>(key, root_start, root_end, roots, n);

  // ---- level loop
  TypeWeights tw;
  for (int t = 0; t < 4; ++t) tw.w[t] = c.weighted ? 1.0 + c.lambda * (c.measured[t] - 1.0) : 1.0;
  int sequential_nodes = 0;
  int k = (int)h_big.size(), level = 0, total_nodes = roots;
  const dim3 seg_grid(nc, 3), carry_grid(3, 2), axes_grid(blocks(n), 3);
  k_clear_winners<<<1, 32, 0, sm>>>(win, roots);
  struct Round {
    int next, failed;  // next round's nodes, this round's failed ones
  } local;
  Round* round = landing(ctx, local);
  while (k > 0) {
    // Every node of the level loop holds more than kSubtreeSize primitives
    // (smaller ones go to k_subtrees), so with non-unit weights all of them take the certified
    // count-based weights; one whose certificate fails comes back in the next round with its
    // sequential sums.  A round is one wait for the host.
    CostArgs A{P, I, N, c.traversal, {cost[0], cost[1], cost[2]}, node_box};
    CountedCosts U;
    if (c.weighted) {
      static_cast<CostArgs&>(U) = A;
      U.tw = tw;
      U.seq = win.seq;
      for (int a = 0; a < 3; ++a) {
        U.pw[a] = chains.pw[a];
        U.sw[a] = chains.sw[a];
        U.bound[a] = bound[a];
      }
      BoxCountsLoad L;
      L.P = P;
      L.I = I;
      L.level_of = level_of;
      L.level = level;
      auto *fwd = (Seg<BoxCounts>*)seg_fwd, *bwd = (Seg<BoxCounts>*)seg_bwd;
      k_seg_chunks<<<seg_grid, kSegThreads, 0, sm>>>(L, key, n, nc, fwd, bwd);
      k_seg_carries<BoxCountsOp><<<carry_grid, kCarryThreads, 0, sm>>>(nc, fwd, bwd);
      k_seg_costs<<<seg_grid, kSegThreads, 0, sm>>>(L, U, key, n, nc, fwd, bwd, (unsigned long long*)win.cost);
    } else {
      BoxLoad L;
      L.P = P;
      L.I = I;
      L.level_of = level_of;
      L.level = level;
      UnitCosts UU;
      static_cast<CostArgs&>(UU) = A;
      auto *fwd = (Seg<Box>*)seg_fwd, *bwd = (Seg<Box>*)seg_bwd;
      k_seg_chunks<<<seg_grid, kSegThreads, 0, sm>>>(L, key, n, nc, fwd, bwd);
      k_seg_carries<BoxOp><<<carry_grid, kCarryThreads, 0, sm>>>(nc, fwd, bwd);
      k_seg_costs<<<seg_grid, kSegThreads, 0, sm>>>(L, UU, key, n, nc, fwd, bwd, (unsigned long long*)win.cost);
    }
    cudaMemsetAsync(lists, 0, 2 * sizeof(int), sm);
    k_first_minimum<<<axes_grid, 256, 0, sm>>>(N, key, level_of, level, n, A, win);
    if (c.weighted)
      k_certify<<<axes_grid, 256, 0, sm>>>(N, key, level_of, level, n, U, win, failed_list, lists + 1);
    k_decide<<<blocks(k), 256, 0, sm>>>(P, I, N, active, k, win, node_box, c.leaf_size, roots, next_active, lists,
                                        level_of, level, counters + 2, sub_roots, counters + 7);
    k_sides<<<blocks(n), 256, 0, sm>>>(I, N, key, level_of, level, n, side);
    {
      k_left_flags3<<<axes_grid, 256, 0, sm>>>(I, N, key, level_of, level, n, side, flags);
      size_t tb = tmp_bytes;
      cub::DeviceScan::ExclusiveSum(tmp, tb, flags, lscan, 3 * n, sm);
      k_scatter3<<<axes_grid, 256, 0, sm>>>(I, T, N, key, key2, level_of, level, n, side, lscan);
      for (int a = 0; a < 3; ++a) std::swap(I.a[a], T.a[a]);
      std::swap(key, key2);
    }
    cudaMemcpyAsync(round, lists, sizeof(Round), cudaMemcpyDeviceToHost, sm);
    cudaError_t e = cudaStreamSynchronize(sm);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "BVH build level");
    const int next = round->next, nfail = round->failed;
    if (nfail > 0) {
      for (int a = 0; a < 3; ++a)
        k_gather_weights<<<blocks(n), 256, 0, sm>>>(P, I.a[a], n, const_cast<double*>(chains.w[a]));
      k_weights_seq<<<blocks(6LL * 32 * nfail, 128), 128, 0, sm>>>(chains, N, failed_list, nfail, nullptr);
      sequential_nodes += nfail;
    }
    std::swap(active, next_active);
    k = next;
    level++;
  }
  // ---- the subtrees below the level loop
  {
    int h[8];
    cudaMemcpyAsync(h, counters, sizeof(h), cudaMemcpyDeviceToHost, sm);
    cudaError_t e = cudaStreamSynchronize(sm);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "BVH build levels");
    if (h[7] > 0) {
      k_subtrees<<<(unsigned)h[7], kSubtreeThreads, 0, sm>>>(
          P, I, N, sub_roots, counters + 7, roots, c.leaf_size, c.traversal, counters + 2, lscan, small_list, counters);
      k_small_subtrees<<<ctx->sm_count * kSmallBlocksPerSm, 32, 0, sm>>>(P, I, N, small_list, counters, roots, c.leaf_size,
                                                                        c.traversal, counters + 2);
    }
    cudaMemcpyAsync(h, counters, sizeof(h), cudaMemcpyDeviceToHost, sm);
    e = cudaStreamSynchronize(sm);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(ctx, e, "BVH subtrees");
    total_nodes = 2 * h[2] - roots;  // a full binary forest of h[2] leaves
    if (h[2] < 1 || total_nodes > cap) return fail(ctx, RTB_ERR_DEVICE_CHECK, "BVH node count out of range");
  }
  int rotation_count = 0;
  if (rotate) {
    std::vector<int> level_begin;
    int* all_nodes = W.alloc<int>(cap);
    double* rcost = W.alloc<double>(cap);
    int* rot = W.alloc<int>(2);
    if (!W.ok) return fail(ctx, RTB_ERR_OUT_OF_MEMORY, "BVH rotation workspace");
    bool leaves_done = false;
    for (int pass = 0; pass < rotation_passes; ++pass) {
      if (!tree_levels(N, roots, all_nodes, rot + 1, level_begin, sm))
        return cuda_fail(ctx, cudaGetLastError(), "BVH levels");
      int levels = (int)level_begin.size() - 1;
      if (!leaves_done) {
        k_leaf_area_cost<<<blocks(total_nodes), 256, 0, sm>>>(P, I, N, all_nodes, total_nodes, rcost);
        leaves_done = true;
      }
      cudaMemsetAsync(rot, 0, 4, sm);
      for (int L = levels - 1; L >= 0; --L) {
        int b = level_begin[L], cnt = level_begin[L + 1] - b;
        k_rotate_level<<<blocks(cnt), 256, 0, sm>>>(N, all_nodes + b, cnt, c.traversal, rcost, rot);
      }
      int h_rot = 0;
      cudaMemcpyAsync(&h_rot, rot, 4, cudaMemcpyDeviceToHost, sm);
      cudaError_t e = cudaStreamSynchronize(sm);
      if (e != cudaSuccess) return cuda_fail(ctx, e, "BVH rotation pass");
      rotation_count += h_rot;
      if (h_rot == 0) break;
    }
    if (!tree_levels(N, roots, all_nodes, rot + 1, level_begin, sm))
      return cuda_fail(ctx, cudaGetLastError(), "BVH levels");
    // the rotated tree's depth replaces the build's
    int depth = (int)level_begin.size() - 2;
    cudaMemcpyAsync(counters + 5, &depth, 4, cudaMemcpyHostToDevice, sm);
    cudaStreamSynchronize(sm);
  }
  rtb_status fs = finish_build(ctx, desc, cfg, W, c, in, P, I, N, roots, cap, total_nodes, counters, out, stats);
  if (fs == RTB_OK && stats) {
    stats->rotation_count = rotation_count;
    stats->sequential_nodes = sequential_nodes;
  }
  return fs;
}

}  // namespace rtb
