// Pieces shared by the device BVH builders (full sweep in rtb_build.cu, binned in
// rtb_binned.cu): primitive bounds and weights, the node arrays of a level-synchronous
// build, the stable partition of a level, and the bottom-up / preorder / flatten passes
// that turn the node arrays into the reference's flattened layout (GpuScene.java:772-838).
// Every symbol has internal linkage; each builder's translation unit gets its own copy.
// Compiled with -fmad=false: no double expression is contracted.
#pragma once

#include <cub/cub.cuh>

#include <algorithm>
#include <vector>

#include "rtb_internal.h"

namespace rtb {
namespace {

struct Box {
  float mn[3], mx[3];
};

struct BoxUnion {
  __device__ __forceinline__ Box operator()(const Box& a, const Box& b) const {
    Box r;
    for (int k = 0; k < 3; ++k) {
      r.mn[k] = fminf(a.mn[k], b.mn[k]);
      r.mx[k] = fmaxf(a.mx[k], b.mx[k]);
    }
    return r;
  }
};

// Aabb.surfaceArea (GpuScene.java:70-74) on float-valued bounds, in double.
__device__ __forceinline__ double surface_area(const Box& b) {
  double dx = (double)b.mx[0] - (double)b.mn[0];
  double dy = (double)b.mx[1] - (double)b.mn[1];
  double dz = (double)b.mx[2] - (double)b.mn[2];
  double s = dx * dy + dx * dz;
  s = s + dy * dz;
  return 2.0 * s;
}

__device__ __forceinline__ float down2(float v) {
  return nextafterf(nextafterf(v, -CUDART_INF_F), -CUDART_INF_F);
}
__device__ __forceinline__ float up2(float v) {
  return nextafterf(nextafterf(v, CUDART_INF_F), CUDART_INF_F);
}

// Double.compare order as an unsigned key (-0.0 before +0.0, finite values in order).
__device__ __forceinline__ unsigned long long order_key(double v) {
  unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ULL);
}

// float <-> order-preserving unsigned, so that integer minima and maxima order float values.
__device__ __forceinline__ unsigned f2o(float f) {
  unsigned b = __float_as_uint(f);
  return (b >> 31) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float o2f(unsigned o) {
  return __uint_as_float((o >> 31) ? (o & 0x7FFFFFFFu) : ~o);
}

struct Prims {
  float* lo[3];
  float* hi[3];
  Box* box;          // the same bounds, one 24-byte record per primitive (gathers)
  double* cen[3];
  double* w;         // construction weight q = 1 + lambda (c - 1), or 1
  double* measured;  // c
  int* ref;
  int* type;
};

struct BuildCfg {
  int n[4];
  int total;
  int leaf_size;
  int weighted;
  double traversal, lambda;
  double measured[4];
};

// Primitive bounds (GpuScene.java:626-649, 877-903) and weights.
__global__ void k_prims(const float* spheres, const float* boxes, const float* ab, const float* bb,
                        BuildCfg c, Prims P) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= c.total) return;
  int t = 0, i = p;
  while (t < 3 && i >= c.n[t]) {
    i -= c.n[t];
    ++t;
  }
  float lo[3], hi[3];
  if (t == 0) {
    const float* s = spheres + 5 * (size_t)i;
    float r = s[3];
    for (int k = 0; k < 3; ++k) {
      lo[k] = down2(s[k] - r);
      hi[k] = up2(s[k] + r);
    }
  } else if (t == 1) {
    const float* b = boxes + 7 * (size_t)i;
    for (int k = 0; k < 3; ++k) {
      lo[k] = down2(b[k]);
      hi[k] = up2(b[3 + k]);
    }
  } else {
    const float* b = (t == 2 ? ab : bb) + 6 * (size_t)i;
    for (int k = 0; k < 3; ++k) {
      lo[k] = down2(b[k]);
      hi[k] = up2(b[3 + k]);
    }
  }
  Box bx;
  for (int k = 0; k < 3; ++k) {
    P.lo[k][p] = lo[k];
    P.hi[k][p] = hi[k];
    P.cen[k][p] = ((double)lo[k] + (double)hi[k]) * 0.5;
    bx.mn[k] = lo[k];
    bx.mx[k] = hi[k];
  }
  P.box[p] = bx;
  double m = c.measured[t];
  P.measured[p] = m;
  P.w[p] = c.weighted ? 1.0 + c.lambda * (m - 1.0) : 1.0;
  P.ref[p] = (int)((unsigned)t << kTypeShift) | i;
  P.type[p] = t;
}


struct Nodes {
  int* start;
  int* end;
  int* order_axis;  // axis array holding the node's current order; -1: input order
  int* depth;
  int* left;
  int* right;
  int* leaf;        // 1 leaf, 0 interior, -1 no node of this id
  int* split_axis;  // this level's decision (-1: none)
  int* split_pos;
  Box* bounds;
  int* size;
  int* parent;  // -1 at a root
  int* visits;  // of the bottom-up pass
  int* rsize;   // primitive references under the node
  double* sah[3];   // generalized, uniform, weighted
};

// key[j] = the root whose range [start, end) holds position j (at most four roots).
__global__ void k_init_keys(int* key, const int* start, const int* end, int roots, int n) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  for (int r = 0; r < roots; ++r)
    if (j >= start[r] && j < end[r]) key[j] = r;
}

__device__ __forceinline__ int current_prim(const int* const* idx, int order_axis, int j) {
  return order_axis < 0 ? j : idx[order_axis][j];
}

struct IdxSet {
  int* a[3];
};

// A split puts a boundary between two positions that no other split of the tree uses, so the
// children of a node split at position q are nodes roots + 2 q and the next: ids need no counter.
// They are sparse; N.leaf is -1 where there is no node.
__device__ __forceinline__ int child_id(int roots, int split) { return roots + 2 * split; }

// The leaves one thread or warp has made, added to the build's statistics once at its end.
struct LeafStats {
  int leaves, min_occ, max_occ, max_depth;
  __device__ __forceinline__ void add(int m, int depth) {
    leaves++;
    min_occ = min(min_occ, m);
    max_occ = max(max_occ, m);
    max_depth = max(max_depth, depth);
  }
  __device__ __forceinline__ void add_to(int* stats) const {
    if (leaves == 0) return;
    atomicAdd(stats + 0, leaves);
    atomicMin(stats + 1, min_occ);
    atomicMax(stats + 2, max_occ);
    atomicMax(stats + 3, max_depth);
  }
};

// A split node's record and its children's, by one thread.
__device__ __forceinline__ void write_split(const Nodes& N, int node, int l, int axis, int pos, int s, int e,
                                            int depth) {
  const int r = l + 1;
  N.leaf[node] = 0;
  N.left[node] = l;
  N.right[node] = r;
  N.split_axis[node] = axis;
  N.split_pos[node] = pos;
  N.start[l] = s;
  N.end[l] = s + pos;
  N.start[r] = s + pos;
  N.end[r] = e;
  N.order_axis[l] = N.order_axis[r] = axis;
  N.depth[l] = N.depth[r] = depth + 1;
}

// ---- finishing passes: three launches over all nodes, whatever the tree's depth (a launch per
// level took 34 launches of some 5 us each at 10k primitives, 58 at 1M)

__global__ void k_parents(Nodes N, int count, int roots) {
  int node = blockIdx.x * blockDim.x + threadIdx.x;
  if (node >= count || N.leaf[node] < 0) return;
  if (node < roots) N.parent[node] = -1;
  N.visits[node] = 0;
  if (N.leaf[node]) return;
  N.parent[N.left[node]] = node;
  N.parent[N.right[node]] = node;
}

// Subtree sizes and SAH statistics (GpuScene.java:810-838): every leaf's thread climbs, and of
// a node's two children the one that arrives last goes on with the node, whose values are the
// same expression of both children's whichever that is.  The children's values pass between
// SMs: written before a fence and the visit, read past the L1 cache after it.
__global__ void k_bottom_up(const Prims P, IdxSet I, Nodes N, int count, double traversal) {
  int node = blockIdx.x * blockDim.x + threadIdx.x;
  if (node >= count || N.leaf[node] != 1) return;
  N.size[node] = 1;
  N.rsize[node] = N.end[node] - N.start[node];
  double c0 = 0.0, c1 = 0.0, c2 = 0.0;
  for (int j = N.start[node]; j < N.end[node]; ++j) {
    int p = current_prim(I.a, N.order_axis[node], j);
    c0 = c0 + P.w[p];
    c1 = c1 + 1.0;
    c2 = c2 + P.measured[p];
  }
  N.sah[0][node] = c0;
  N.sah[1][node] = c1;
  N.sah[2][node] = c2;
  while ((node = N.parent[node]) >= 0) {
    __threadfence();
    if (atomicAdd(N.visits + node, 1) == 0) return;
    __threadfence();
    const int l = N.left[node], r = N.right[node];
    N.size[node] = 1 + __ldcg(N.size + l) + __ldcg(N.size + r);
    N.rsize[node] = __ldcg(N.rsize + l) + __ldcg(N.rsize + r);
    const double area = surface_area(N.bounds[node]);
    const double al = surface_area(N.bounds[l]), ar = surface_area(N.bounds[r]);
    for (int m = 0; m < 3; ++m) {
      const double sl = __ldcg(N.sah[m] + l), sr = __ldcg(N.sah[m] + r);
      double v;
      if (!(area > 0.0)) {
        v = sl + sr;
      } else {
        double x = al / area * sl;
        double y = ar / area * sr;
        v = (traversal + x) + y;
      }
      N.sah[m][node] = v;
    }
  }
}

// What the host reads back of a finished build.
struct BuildResult {
  double sah[4][3];  // per root
  int nodes, refs;   // below all roots, by the climb: every node and primitive, if none was lost
};

// The flattened reference layout (flattenBvh / leafKind, GpuScene.java:772-808).  A node's preorder
// index and first reference are sums over the path to its root: one for every step down, the
// left sibling's sizes for every step to the right, the earlier trees' sizes at the root.  A full
// binary tree of s nodes has (s + 1) / 2 leaves, so the same walk gives an interior node's rank
// among the interior nodes.  The arrays are sized by the leaves that the build counted, not by
// these sums: nothing is written past total_nodes and total_refs, and the host compares.
__global__ void k_flatten(const Prims P, IdxSet I, const Nodes N, int count, int roots, int total_nodes,
                          int total_refs, float* node_bounds, int* node_data, int* refs, int* ranks,
                          int* root_out, BuildResult* result) {
  const int node = blockIdx.x * blockDim.x + threadIdx.x;
  if (node == 0) {
    int nodes = 0, prims = 0;
    for (int r = 0; r < roots; ++r) {
      nodes += N.size[r];
      prims += N.rsize[r];
    }
    result->nodes = nodes;
    result->refs = prims;
  }
  if (node >= count || N.leaf[node] < 0) return;
  int at = 0, f = 0, leaves = 0, c = node;
  for (int p = N.parent[c]; p >= 0; c = p, p = N.parent[c]) {
    const int l = N.left[p];
    at += 1;
    if (c != l) {
      const int size = N.size[l];
      at += size;
      leaves += (size + 1) >> 1;
      f += N.rsize[l];
    }
  }
  for (int r = 0; r < c; ++r) {  // c is the root now, and the roots are the first nodes
    const int size = N.size[r];
    at += size;
    leaves += (size + 1) >> 1;
    f += N.rsize[r];
  }
  if ((unsigned)at >= (unsigned)total_nodes) return;
  if (node < roots) {
    root_out[node] = at;
    for (int m = 0; m < 3; ++m) result->sah[node][m] = N.sah[m][node];
  }
  Box b = N.bounds[node];
  for (int k = 0; k < 3; ++k) {
    node_bounds[6 * (size_t)at + k] = b.mn[k];
    node_bounds[6 * (size_t)at + 3 + k] = b.mx[k];
  }
  int* d = node_data + 4 * (size_t)at;
  ranks[at] = at - leaves;
  if (!N.leaf[node]) {
    d[0] = at + 1;
    d[1] = at + 1 + N.size[N.left[node]];
    d[2] = -1;
    d[3] = 0;
    return;
  }
  // references in preorder of the leaves (after rotations that differs from array order)
  int s = N.start[node], e = N.end[node];
  if (f < 0 || e - s > total_refs - f) return;
  int t0 = -1;
  bool mixed = false;
  for (int j = s; j < e; ++j) {
    int p = current_prim(I.a, N.order_axis[node], j);
    refs[f + (j - s)] = P.ref[p];
    int t = P.type[p];
    if (t0 < 0) t0 = t;
    else if (t != t0) mixed = true;
  }
  d[0] = mixed ? -1 : -2 - t0;
  d[1] = -1;
  d[2] = f;
  d[3] = e - s;
}

inline unsigned blocks(long long n, int b = 256) { return (unsigned)std::max<long long>(1, (n + b - 1) / b); }

// Build workspace from the device's stream-ordered pool: after the first build the pool
// holds the memory, so later builds allocate without a device-wide synchronisation.
struct Workspace {
  std::vector<void*> ptrs;
  cudaStream_t stream = nullptr;
  bool ok = true;
  template <typename T>
  T* alloc(size_t n) {
    void* p = nullptr;
    if (cudaMallocAsync(&p, std::max<size_t>(n, 1) * sizeof(T), stream) != cudaSuccess) {
      cudaGetLastError();
      ok = false;
      return nullptr;
    }
    ptrs.push_back(p);
    return (T*)p;
  }
  ~Workspace() {
    for (void* p : ptrs) cudaFreeAsync(p, stream);
  }
};

// ---- host side shared by the builders

// Validates a build request and fills the per-build constants.
// allow_rotations: the full-sweep builder also takes the rotation modes (6, 7).
inline rtb_status build_setup(rtb_context* ctx, const rtb_scene_desc* desc, const rtb_build_config* cfg,
                              BuildCfg& c, bool& per_type, bool allow_rotations = false) {
  if (!desc || !cfg) return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "null argument");
  if (cfg->mode < 0 || cfg->mode > 7) return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "unknown BVH build mode");
  if (cfg->mode == 4 || cfg->mode == 5)
    return fail(ctx, RTB_ERR_UNSUPPORTED, "the SBVH modes have their own builder (rtb_scene_build)");
  if (cfg->mode > 5 && !allow_rotations)
    return fail(ctx, RTB_ERR_UNSUPPORTED, "rotation modes apply to the full-sweep builder");
  if (cfg->leaf_size < 1) return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "BVH leaf size must be positive.");
  bool weighted = cfg->mode == 1 || cfg->mode == 3 || cfg->mode == 7;
  per_type = cfg->mode == 2 || cfg->mode == 3;
  c.n[0] = desc->sphere_count;
  c.n[1] = desc->box_count;
  c.n[2] = desc->affine_sphere_count;
  c.n[3] = desc->affine_box_count;
  for (int t = 0; t < 4; ++t)
    if (c.n[t] < 0) return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "negative primitive count");
  if ((c.n[2] > 0 && !desc->affine_sphere_bounds) || (c.n[3] > 0 && !desc->affine_box_bounds))
    return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "affine bounds are required to build a BVH");
  long long total = (long long)c.n[0] + c.n[1] + c.n[2] + c.n[3];
  if (total > (1LL << 30) - 1) return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "too many primitives");
  c.total = (int)total;
  c.leaf_size = cfg->leaf_size;
  c.weighted = weighted ? 1 : 0;
  c.traversal = cfg->traversal_weight;
  c.lambda = weighted ? cfg->lambda : 0.0;
  c.measured[0] = cfg->sphere_weight;
  c.measured[1] = cfg->box_weight;
  c.measured[2] = cfg->affine_sphere_weight;
  c.measured[3] = cfg->affine_box_weight;
  return RTB_OK;
}

// Primitive arrays of one build, allocated from the workspace.
inline Prims alloc_prims(Workspace& W, int n) {
  Prims P;
  for (int k = 0; k < 3; ++k) {
    P.lo[k] = W.alloc<float>(n);
    P.hi[k] = W.alloc<float>(n);
    P.cen[k] = W.alloc<double>(n);
  }
  P.box = W.alloc<Box>(n);
  P.w = W.alloc<double>(n);
  P.measured = W.alloc<double>(n);
  P.ref = W.alloc<int>(n);
  P.type = W.alloc<int>(n);
  return P;
}

struct PrimInputs {
  float *sph, *box, *ab, *bb;
};

inline PrimInputs alloc_inputs(Workspace& W, const BuildCfg& c) {
  return PrimInputs{W.alloc<float>((size_t)c.n[0] * 5), W.alloc<float>((size_t)c.n[1] * 7),
                    W.alloc<float>((size_t)c.n[2] * 6), W.alloc<float>((size_t)c.n[3] * 6)};
}

// Copies the packed host arrays in and computes bounds, centroids and weights.
inline void upload_prims(const rtb_scene_desc* desc, const BuildCfg& c, const PrimInputs& in,
                         const Prims& P, cudaStream_t sm) {
  if (c.n[0]) cudaMemcpyAsync(in.sph, desc->spheres, (size_t)c.n[0] * 20, cudaMemcpyHostToDevice, sm);
  if (c.n[1]) cudaMemcpyAsync(in.box, desc->boxes, (size_t)c.n[1] * 28, cudaMemcpyHostToDevice, sm);
  if (c.n[2])
    cudaMemcpyAsync(in.ab, desc->affine_sphere_bounds, (size_t)c.n[2] * 24, cudaMemcpyHostToDevice, sm);
  if (c.n[3])
    cudaMemcpyAsync(in.bb, desc->affine_box_bounds, (size_t)c.n[3] * 24, cudaMemcpyHostToDevice, sm);
  k_prims<<<blocks(c.total), 256, 0, sm>>>(in.sph, in.box, in.ab, in.bb, c, P);
}

inline Nodes alloc_nodes(Workspace& W, int cap) {
  Nodes N;
  N.start = W.alloc<int>(cap);
  N.end = W.alloc<int>(cap);
  N.order_axis = W.alloc<int>(cap);
  N.depth = W.alloc<int>(cap);
  N.left = W.alloc<int>(cap);
  N.right = W.alloc<int>(cap);
  N.leaf = W.alloc<int>(cap);
  N.split_axis = W.alloc<int>(cap);
  N.split_pos = W.alloc<int>(cap);
  N.bounds = W.alloc<Box>(cap);
  N.size = W.alloc<int>(cap);
  N.parent = W.alloc<int>(cap);
  N.visits = W.alloc<int>(cap);
  N.rsize = W.alloc<int>(cap);
  for (int m = 0; m < 3; ++m) N.sah[m] = W.alloc<double>(cap);
  return N;
}

// Root ranges: one tree over all primitives, or one per non-empty type (per-type forests,
// GpuScene.java:702-720); primitives are laid out type by type.
inline int root_ranges(const BuildCfg& c, bool per_type, int* rs, int* re) {
  if (!per_type) {
    rs[0] = 0;
    re[0] = c.total;
    return 1;
  }
  int roots = 0, off = 0;
  for (int t = 0; t < 4; ++t) {
    if (c.n[t] > 0) {
      rs[roots] = off;
      re[roots] = off + c.n[t];
      roots++;
    }
    off += c.n[t];
  }
  return roots;
}

// Sizes and SAH statistics, the flattened arrays and the resident scene, of total_nodes nodes
// whose ids lie below `ids`, the roots first.  counters + 2 holds
// {leaves, min occupancy, max occupancy, max depth}.
inline rtb_status finish_build(rtb_context* ctx, const rtb_scene_desc* desc, const rtb_build_config* cfg,
                               Workspace& W, const BuildCfg& c, const PrimInputs& in, const Prims& P,
                               const IdxSet& I, const Nodes& N, int roots, int ids, int total_nodes,
                               const int* counters,
                               rtb_scene** out, rtb_bvh_stats* stats) {
  cudaStream_t sm = ctx->stream;
  const int n = c.total;
  float* o_nb = W.alloc<float>((size_t)total_nodes * 6);
  int* o_nd = W.alloc<int>((size_t)total_nodes * 4);
  int* o_rank = W.alloc<int>(total_nodes);
  int* o_refs = W.alloc<int>(n);
  int* o_roots = W.alloc<int>(4);
  BuildResult* o_result = W.alloc<BuildResult>(1);
  if (!W.ok) return fail(ctx, RTB_ERR_OUT_OF_MEMORY, "BVH output");
  k_parents<<<blocks(ids), 256, 0, sm>>>(N, ids, roots);
  k_bottom_up<<<blocks(ids, 128), 128, 0, sm>>>(P, I, N, ids, c.traversal);
  k_flatten<<<blocks(ids, 128), 128, 0, sm>>>(P, I, N, ids, roots, total_nodes, n, o_nb, o_nd, o_refs, o_rank,
                                              o_roots, o_result);
  cudaEventRecord(ctx->ev1, sm);
  // Read back through pinned memory, so that the host goes on; scene_create waits for the stream.
  struct Back {
    int stats[4];
    BuildResult result;
  };
  Back local;
  Back* back = landing(ctx, local);
  cudaMemcpyAsync(back->stats, counters + 2, sizeof(back->stats), cudaMemcpyDeviceToHost, sm);
  cudaMemcpyAsync(&back->result, o_result, sizeof(BuildResult), cudaMemcpyDeviceToHost, sm);
  BuiltTree tree{o_nb, o_nd, total_nodes, o_refs, n, o_roots, roots, o_rank, (total_nodes - roots) / 2, in.sph, in.box};
  rtb_status s = scene_create(ctx, desc, nullptr, &tree, out);
  if (s != RTB_OK) return s;
  const int* h_stats = back->stats;
  const BuildResult& h_result = back->result;
  float ms = 0.0f;
  cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
  if (h_result.nodes != total_nodes || h_result.refs != n) {
    scene_free(*out, sm);
    *out = nullptr;
    return fail(ctx, RTB_ERR_DEVICE_CHECK,
                "A binary BVH forest must contain 2 * leafCount - rootCount nodes and every primitive.");
  }
  if (stats) {
    stats->node_count = total_nodes;
    stats->root_count = roots;
    stats->leaf_count = h_stats[0];
    stats->max_depth = h_stats[3];
    stats->primitive_ref_count = n;
    stats->leaf_size = cfg->leaf_size;
    stats->min_leaf_occupancy = h_stats[1];
    stats->max_leaf_occupancy = h_stats[2];
    double g = 0.0, u = 0.0, w = 0.0;
    for (int r = 0; r < roots; ++r) {
      u = u + h_result.sah[r][1];
      w = w + h_result.sah[r][2];
      g = g + h_result.sah[r][0];
    }
    stats->generalized_sah_cost = g;
    stats->uniform_sah_cost = u;
    stats->weighted_sah_cost = w;
    stats->bytes = (long long)total_nodes * 24 + ((long long)total_nodes * 4 + n + roots) * 4;
    stats->build_ms = ms;
    stats->sequential_nodes = 0;
    stats->rotation_count = 0;
  }
  return RTB_OK;
}

}  // namespace
}  // namespace rtb
