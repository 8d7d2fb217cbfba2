// Paths on the device: their arguments, seeds, camera rays and shading, and the two-phase form
// in which the frame and adjoint kernels run many of them per lane.
#pragma once
#include "rtb_internal.h"
#include "rtb_plan.h"

namespace rtb {
namespace {

struct RenderArgs {
  DevScene S;
  float3 cam_pos, cam_f, cam_r, cam_u;
  int width, height, spp, max_depth;
  float aspect, step_x, step_y;    // width / height, 2 / width, 2 / height
  float inv_spp;                   // 1 / spp
  uint32_t frame_hash;             // the frame's part of every pixel's seed
  unsigned long long spp_magic, width_magic;  // of fast_div
  float* out;
  long long pixels;                // pixels of the output (the frame, or a set of its rows)
  int row0, row_stride;            // output row k is frame row row0 + k * row_stride
  long long split;                 // pixels [split, pixels) are queued one sample per item
  long long items;                 // split + (pixels - split) * spp queue items
  void* paths;                     // the blocks' path slots
  int slots;                       // path slots a block uses; k_render_small: lanes a warp uses
  float* tail;                     // RGB of each tail item, item - split order
  unsigned long long* queue;       // work queue head
  int* abort_flag;                 // the context's abort words (abort_raised)
  unsigned long long* counters;    // 14 counters (metrics build) + overflow count
};

__device__ __forceinline__ float luminance(float3 c) {  // K:181-183
  return c.x * 0.212655f + c.y * 0.715158f + c.z * 0.072187f;
}
__device__ __forceinline__ float3 reflect_dir(float3 n, float3 i) {  // K:1022-1024
  return sub(mul(n, 2.0f * dot(i, n)), i);
}
// Out of line: the refraction lobe is rare, and its code stays out of the frame loop.
static __device__ __noinline__ float3 refract_dir(float3 incoming, float3 n, float eta) {  // K:1026-1039
  float3 i = normalize_safe(incoming);
  float c1 = dot(i, n);
  float ri = (c1 >= 0.0f) ? eta : -1.0f / eta;
  float inv_ri2 = 1.0f / (ri * ri);
  float c2 = 1.0f - (1.0f - c1 * c1) * inv_ri2;
  if (c2 <= 0.0f) return normalize_safe(reflect_dir(n, i));
  float sq = sqrtf(c2);
  return normalize_safe(sub(mul(n, c1 - sq * ri), i));
}

// K:1231-1236; the part that every pixel of the frame shares is hashed on the host.
__device__ __forceinline__ uint32_t pixel_base_seed(uint32_t frame_hash, uint32_t pixel) {
  return hash_u32(frame_hash ^ hash_u32(pixel));
}

// n / d for 32-bit n by the divisor's magic number floor((2^64 - 1) / d) + 1 (0 for d = 1): the
// quotient n M / 2^64 exceeds n / d by less than n / 2^64 < 1 / d, so its floor is exact.
inline unsigned long long div_magic(unsigned d) { return ~0ULL / d + 1ULL; }
__device__ __forceinline__ unsigned fast_div(unsigned n, unsigned long long magic) {
  return magic ? (unsigned)__umul64hi((unsigned long long)n, magic) : n;
}

// One path segment after its closest-hit query (tracePath loop body, K:1098-1162), in two
// parts.  hit_vertex: the hit's material and emission; scatter: the lobe chosen by luminance
// and the next ray.  The frame kernels and the adjoint shade through them.
struct Vertex {
  int material;
  float3 pos, n;
  float4 m0, m1, m2;  // diffuse + ior, reflective, refractive
  float3 emission;
};
__device__ __forceinline__ Vertex hit_vertex(const DevScene& S, const Best& b, float3 o, float3 d) {
  Vertex v;
  v.pos = add(o, mul(d, b.t));
  const HitRecord hr = hit_record_inline(S, b, o, d, v.pos);
  v.n = hr.n;
  v.material = hr.material;
  float4 m3 = make_float4(0, 0, 0, 0);
  v.m0 = v.m1 = v.m2 = m3;
  if (v.material >= 0) {
    const float4* mp = S.materials + 4 * v.material;
    v.m0 = __ldg(mp);
    v.m1 = __ldg(mp + 1);
    v.m2 = __ldg(mp + 2);
    m3 = __ldg(mp + 3);
  }
  v.emission = v3(m3.x, m3.y, m3.z);
  return v;
}

// Returns false where the path ends here; else the next ray (o, d), the lobe's weight colour
// `wc`, its probability `pc`, and whether it is the diffuse one.
__device__ __forceinline__ bool scatter(const Vertex& v, float3& o, float3& d, uint32_t& rng, float3& wc,
                                        float& pc, bool& diffuse) {
  const float3 cd = v3(v.m0.x, v.m0.y, v.m0.z), cr = v3(v.m1.x, v.m1.y, v.m1.z), ct = v3(v.m2.x, v.m2.y, v.m2.z);
  const float3 inc = neg(d);
  const float wd = luminance(cd), wr = luminance(cr), wt = luminance(ct);
  const float sum = wd + wr + wt;
  if (sum <= 0.0f) return false;
  const float xi = rand01(&rng) * sum;
  diffuse = xi < wd;
  float3 nd;
  if (diffuse) {
    pc = wd / sum;
    float z = rand01(&rng) * 2.0f - 1.0f;
    float t = rand01(&rng) * 2.0f * CUDART_PI_F;
    float r = sqrtf(fmaxf(0.0f, 1.0f - z * z));
    // one range reduction; equal to sinf and cosf bit for bit on all 2^24 values of t
    float st, ct2;
    sincosf(t, &st, &ct2);
    nd = add(v3(r * ct2, r * st, z), v.n);
    wc = divs(cd, pc);
  } else if (xi < wd + wr) {
    pc = wr / sum;
    nd = reflect_dir(v.n, inc);
    wc = divs(cr, pc);
  } else {
    pc = wt / sum;
    nd = refract_dir(inc, v.n, v.m0.w);
    wc = divs(ct, pc);
  }
  o = add(v.pos, mul(nd, kEps));
  d = nd;
  return true;
}

// Returns true when the path ends.
__device__ __forceinline__ bool shade_segment(const DevScene& S, bool hit, const Best& b, float3& o,
                                              float3& d, float3& thr, float3& rad, uint32_t& rng,
                                              int& depth, int max_depth) {
  if (!hit) {
    rad = add(rad, mulv(thr, S.background));
    return true;
  }
  const Vertex v = hit_vertex(S, b, o, d);
  rad = add(rad, mulv(thr, v.emission));
  float3 wc;
  float pc;
  bool diffuse;
  if (!scatter(v, o, d, rng, wc, pc, diffuse)) return true;
  thr = mulv(thr, wc);
  depth++;
  return depth >= max_depth;
}

// The camera ray of sample `so` of pixel (x, y) and its random stream (renderKernel
// prologue, K:1251-1264), for every form of the frame and the replay.
__device__ __forceinline__ void camera_sample(const RenderArgs& a, int x, int y, int so, uint32_t& rng,
                                              float3& o, float3& d) {
  uint32_t seed = pixel_base_seed(a.frame_hash, (uint32_t)y * (uint32_t)a.width + (uint32_t)x) ^ hash_u32((uint32_t)so);
  seed ^= hash_u32((uint32_t)(so * 0x9E3779B9u));
  rng = hash_u32(seed);
  float jx = rand01(&rng) - 0.5f;
  float jy = rand01(&rng) - 0.5f;
  float u = ((((float)x + 0.5f) + jx) * a.step_x - 1.0f) * a.aspect;
  float v = 1.0f - ((((float)y + 0.5f) + jy) * a.step_y);
  o = a.cam_pos;
  d = add(add(a.cam_f, mul(a.cam_r, u)), mul(a.cam_u, v));
}

// Queue entry p as a work item: a whole pixel from its first sample, or ~(tail item), one sample.
__device__ __forceinline__ void take_item(const RenderArgs& a, long long p, long long& item,
                                          long long& pixel, int& so) {
  if (p < a.split) {
    item = pixel = p;
    so = 0;
  } else {
    const unsigned t = (unsigned)(p - a.split);  // at most kMaxTailItems
    const unsigned q = fast_div(t, a.spp_magic);
    item = ~(long long)t;
    pixel = a.split + q;
    so = (int)(t - q * (unsigned)a.spp);
  }
}

// The camera ray and random stream of sample `so` of an output pixel.
__device__ __forceinline__ void start_sample(const RenderArgs& a, long long pixel, int so, uint32_t& rng,
                                             float3& o, float3& d) {
  int x, y;
  if (a.pixels <= 0xFFFFFFFFLL) {
    const unsigned row = fast_div((unsigned)pixel, a.width_magic);
    x = (int)((unsigned)pixel - row * (unsigned)a.width);
    y = (int)row;
  } else {
    x = (int)(pixel % a.width);
    y = (int)(pixel / a.width);
  }
  camera_sample(a, x, a.row0 + y * a.row_stride, so, rng, o, d);
}

// ---- the persistent frame kernel
//
// Every block owns path slots in global memory, several per lane; a slot holds a path (ray,
// throughput, radiance, random stream) and the work item it belongs to.  The block runs two
// alternating phases over its slots:
//
//  trace  lanes take the slots' rays in order; when at least kRefillLanes lanes of a warp
//         have finished their rays they store the hits and take the next ones, so a lane
//         whose ray needs few nodes does not idle until the warp's longest ray ends;
//  shade  every traced path is shaded, 32 per warp; a path that ends is replaced by its
//         item's next sample or the next item of the frame's queue.
//
// When the queue is empty and paths end, two lists name the slots that still hold one, the
// list that the phases read and the list that the shading writes, so that the paths that are
// left keep full warps; until then a block's slots are all in use and need no list.
//
// The phases are the block's, not the warp's, for the instruction cache: the walk's loop is
// small and the shading long and straight, and warps in both at once evict each other's
// code (no_instruction stalls 7 per issue with a pool per warp, against 0.4 in a kernel that
// only traces).  A block's slots are read and written once a phase, in order, mostly in L2.
// The order in which paths are traced and shaded changes nothing in a path: its random
// stream, its arithmetic and the sample order of a pixel's sum stay the same.
//
// Measured against one path a lane (k_render_small's form, as it was), where a warp's lanes wait
// for its longest ray (9.65 active lanes, 12.56 G
// warp instructions for 4.2 M samples of the 10k scene): 14.3 lanes, 8.45 G instructions; 10k
// scene 1024x1024, 16 spp 68.5 -> 49.1 ms, 1M scene 1920x1080, 4 spp 56.0 -> 45.2 ms.
//
// A block of 1,024 threads keeps a whole SM in one phase: 10k scene 49.1 ms, with two blocks of
// 512 52.4, with four of 256 56.8 (the same kernel's first form).
//
// k_render_small, in which every lane runs its own path's segments one after the other, has no
// phases to wait for and keeps the path in registers; it is the faster one where the frame is
// small or its rays meet next to no nodes (phases / lanes, ms): 65 spheres 256x256, 16 spp
// 0.379 / 0.353 and 1024x1024 11.1 / 10.9, four glass spheres 1024x768, 16 spp, 24 segments
// deep 6.21 / 4.56; but 300 mixed primitives 512x512, 16 spp 2.90 / 3.68, 10k 256x256 at 4 spp
// 1.121 / 1.125, 8 spp 1.75 / 1.97.  So the phases take frames of kPhaseItems samples per
// resident thread over a tree of kPhaseNodes nodes, and paths of kPhaseDepth segments: camera rays
// walk the tree together as neighbours and gain nothing from being taken singly.  Three segments
// is where the forms meet.  Phases' time over lanes', 15 whole frames (300 to 1M primitives,
// 400x401 to 1024x1024, 1 / 4 / 16 spp) and 12 ranks' rows of 10k and 120k primitives:
//
//   segments        2                 3                 4              5
//   whole frames    1.00-1.25         0.95-1.11         0.90-1.07      0.84-1.02
//   rows            0.96-1.29         0.82-1.10         0.76-1.02      -
//   at 3, by samples a pixel (means): 1 spp 1.05, 4 spp 1.05, 16 spp 1.00; rows 0.99
//
// Wide frames, whose camera rays are far apart (1834x219: 0.82 and 0.87), gain most at three, square
// ones of few samples lose most (10k 1024x1024, 1 spp: 1.22 / 1.10 ms), so neither side of the line
// has three segments to itself; from three on both are faster than the form before this walk in
// every cell.  Refilling only whole warps in phases of mostly camera rays took back between none and
// four tenths of the difference at one segment and cost 1 % at depth 8.
constexpr int kPhaseItems = 2, kPhaseNodes = 64, kPhaseDepth = 3;
constexpr int kRefillLanes = 8;    // 4 and 12 within 1 %
constexpr int kPoolLeafLanes = 8;  // 4 and 12 within 1 %

// A path slot in global memory, by groups of 32 slots: the group's origins, directions,
// throughputs, radiances, sums (16 bytes a slot), hits and items (8 bytes a slot).  A warp
// that takes a group reads whole lines, and one base address serves every field.
struct Slot {
  char* p;   // the slot's 16-byte column
  char* p8;  // its 8-byte column
  __device__ __forceinline__ Slot(char* base, int s) {
    char* g = base + (size_t)((unsigned)s >> 5) * kGroupBytes;
    p = g + (s & 31) * 16;
    p8 = g + (s & 31) * 8;
  }
  __device__ __forceinline__ float4& o() const { return *(float4*)p; }             // w: random stream's state
  __device__ __forceinline__ float4& d() const { return *(float4*)(p + 512); }     // w: depth
  __device__ __forceinline__ float4& thr() const { return *(float4*)(p + 1024); }  // w unused
  __device__ __forceinline__ float4& rad() const { return *(float4*)(p + 1536); }  // w: sample index
  // a whole pixel's running sum; read and written once a sample
  __device__ __forceinline__ float4& acc() const { return *(float4*)(p + 2048); }
  // closest bounded hit: distance, and type << 30 | index or one of the constants below
  __device__ __forceinline__ float2& hit() const { return *(float2*)(p8 + 2560); }
  // the work item: a whole pixel, or ~(tail item) of a single sample
  __device__ __forceinline__ long long& item() const { return *(long long*)(p8 + 2816); }
};
// In a slot's hit: no traversal result (linear mode, stack overflow), the shade phase tests every
// primitive.  Storage indices stay below kIndexMask - 1, so it is no reference.
constexpr int kExhaustive = -2;

__device__ __forceinline__ char* block_slots(const RenderArgs& a) {
  return (char*)a.paths + (size_t)blockIdx.x * (((a.slots + 31) / 32) * (kGroupBytes + 256));
}

// How many slots of the block hold a path: all of them, or those of list[cur].  The trace loop
// reads its block's addresses here where it needs them, a few times per ray, and not from
// registers that the walk has no room for.
struct SlotLists {
  int count[2];
  int head;  // the next entry to trace
  int n;     // entries to trace
  char* slots;
  const int* list;  // the entries' slots, null: entry e is slot e
};
__device__ __forceinline__ int* slot_list(const RenderArgs& a, char* base, int which) {
  const int padded = (a.slots + 31) / 32 * 32;
  return (int*)(base + (size_t)padded / 32 * kGroupBytes) + which * padded;
}

// Between the shade and the trace phase: the block's one thread that calls it sets up the list
// that the shading wrote, before a barrier.
__device__ __forceinline__ void begin_trace(const RenderArgs& a, SlotLists& L, int cur) {
  char* base = block_slots(a);
  L.head = 0;
  L.n = L.count[cur];
  L.slots = base;
  L.list = L.n == a.slots ? nullptr : slot_list(a, base, cur);
}

// The trace phase over the block's listed paths: the closest bounded hit of each goes to its
// slot.  All threads of the block call it.
template <bool METRICS, int SDEPTH>
__device__ __forceinline__ void trace_phase(const RenderArgs& a, const volatile SlotLists& L, int* head, int2* s_col,
                                            TraceCounters* c) {
  const DevScene& S = a.S;
  const int lane = threadIdx.x & 31;
  const bool bvh = S.use_bvh && S.node_count > 0;
  int slot = -1;
  float3 o = v3(0, 0, 0), d = v3(0, 0, 0), inv = v3(0, 0, 0);
  Hit b = no_hit();
  Walk w;
  WalkStack<SDEPTH> ws;
  w.begin(S, false);
  bool more = true;  // warp-uniform: slots may be left to take
  while (true) {
    const unsigned walk = __ballot_sync(0xFFFFFFFFu, w.can_walk());
    const unsigned waiting = __ballot_sync(0xFFFFFFFFu, w.waiting());
    const unsigned busy = walk | waiting;
    const int idle = 32 - __popc(busy);
    if (busy == 0u || (more && idle >= kRefillLanes)) {
      const bool free_lane = !(busy >> lane & 1u);
      if (free_lane && slot >= 0) {
        Slot(L.slots, slot).hit() =
            make_float2(b.t, __int_as_float(!bvh || w.overflow() ? kExhaustive : b.ref));
        slot = -1;
      }
      if (!more) break;
      int next = 0;
      if (lane == 0) next = atomicAdd(head, idle);
      next = __shfl_sync(0xFFFFFFFFu, next, 0);
      const int n = L.n;
      more = next + idle < n;
      const int e = next + __popc(~busy & ((1u << lane) - 1u));
      if (free_lane && e < n) {
        const int* list = L.list;
        slot = list ? list[e] : e;
        const Slot Q(L.slots, slot);
        const float4 o4 = Q.o(), d4 = Q.d();
        o = v3(o4.x, o4.y, o4.z);
        d = v3(d4.x, d4.y, d4.z);
        inv = ray_inverse(d);
        b = no_hit();
        w.begin(S, bvh);
      }
      continue;
    }
    if (__popc(walk) <= kPoolLeafLanes && waiting != 0u) {
      test_recorded<METRICS>(S, w, o, d, b, c);
      continue;
    }
    if (w.can_walk())
      walk_node<METRICS, SDEPTH, kBlock>(S, w, ws, o, inv, b, c, s_col);
  }
}

// The closest hit of a slot's segment: the traced bounded hit (every primitive tested where
// there is none to go by), then the planes.
template <bool METRICS>
__device__ __forceinline__ Best slot_hit(const DevScene& S, float2 h2, float3 o, float3 d, TraceCounters* c) {
  Hit b{h2.x, __float_as_int(h2.y)};
  if (b.ref == kExhaustive) {
    const bool bvh = S.use_bvh && S.node_count > 0;
    if (METRICS && bvh) c->overflow++;
    b = bvh ? test_all_refs<METRICS>(S, o, d, dot(d, d), no_hit(), c)
            : test_all_primitives<METRICS>(S, o, d, dot(d, d), no_hit(), c);
  }
  Best h = best_of(b);
  if (METRICS) c->rays++;
  test_planes<METRICS>(S, o, d, h, c);
  return h;
}

// The arguments that a scene, a camera and render parameters give; output, items, buffers and
// queue are the caller's.
inline RenderArgs frame_args(const rtb_scene* scene, const rtb_camera* cam, const rtb_render_params* p) {
  RenderArgs a{};
  a.S = scene->dev;
  a.S.use_bvh = (p->use_bvh && scene->has_bvh) ? 1 : 0;
  a.cam_pos = make_float3(cam->position[0], cam->position[1], cam->position[2]);
  a.cam_f = make_float3(cam->forward[0], cam->forward[1], cam->forward[2]);
  a.cam_r = make_float3(cam->right[0], cam->right[1], cam->right[2]);
  a.cam_u = make_float3(cam->up[0], cam->up[1], cam->up[2]);
  a.width = p->width;
  a.height = p->height;
  a.spp = p->samples_per_frame;
  a.aspect = (float)a.width / (float)a.height;  // IEEE quotients, the same on host and device
  a.step_x = 2.0f / (float)a.width;
  a.step_y = 2.0f / (float)a.height;
  a.inv_spp = 1.0f / (float)a.spp;
  a.spp_magic = div_magic((unsigned)a.spp);
  a.width_magic = div_magic((unsigned)a.width);
  a.max_depth = p->max_depth;
  a.frame_hash = hash_u32((uint32_t)(p->frame_seed & 0xFFFFFFFFULL)) ^
                 hash_u32((uint32_t)(p->frame_seed >> 32)) ^ hash_u32((uint32_t)p->frame_index);
  a.row_stride = 1;
  a.pixels = (long long)p->width * p->height;
  return a;
}

// Whether the two-phase form is the faster one (see above).
inline bool use_phases(const RenderArgs& a, int sm_count) {
  return a.max_depth >= kPhaseDepth && a.S.use_bvh && a.S.node_count >= kPhaseNodes &&
         a.pixels * a.spp >= (long long)kPhaseItems * 1024 * sm_count;
}

}  // namespace
}  // namespace rtb
