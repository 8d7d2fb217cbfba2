// Path-tracing and closest-hit kernels.
//
// Render: one persistent launch per frame (the reference issues one launch per sample and
// tile, GpuRayTracer.java:356-376), which takes work items from a warp-aggregated queue: a
// whole pixel, its samples in order, or a single sample.  A path that ends is followed by its
// pixel's next sample or the queue's next item while the others continue, so warps stay full
// across uneven path lengths.  The per-pixel sum is the reference's FP32 running sum over
// samples 0..spp-1 scaled by 1/spp after the last one (GpuKernelSources.java:1284-1293), and
// each sample consumes the reference's random stream (seed K:1231-1254, jitter and camera
// K:1256-1264, tracePath K:1061-1165), so the image matches the reference's renderKernel bit
// for bit under the same arithmetic.
//
// The frame's last pixels (about four per resident thread, or all of a small frame) are
// handed out one sample per queue item instead, so the end of the frame does not wait on
// a few lanes that each still hold a whole pixel.  Those samples' radiance goes to a
// buffer in item order and k_sum_tail adds each pixel's samples in sample order, the same
// FP32 additions as the in-register sum.
#include "rtb_internal.h"
#include "rtb_paths.cuh"

namespace rtb {
namespace {

__device__ void add_counters(unsigned long long* k, const TraceCounters& c) {
  atomicAdd(k + 0, c.rays);
  atomicAdd(k + 1, c.aabb);
  atomicAdd(k + 2, c.prim);
  atomicAdd(k + 3, c.type[0]);
  atomicAdd(k + 4, c.type[1]);
  atomicAdd(k + 5, c.type[2]);
  atomicAdd(k + 6, c.type[3]);
  atomicAdd(k + 7, c.type[4]);
  atomicAdd(k + 8, c.overflow);
  atomicMax(k + 9, c.maxstack);
  atomicAdd(k + 10, c.internal);
  atomicAdd(k + 11, c.leaf);
  atomicAdd(k + 12, c.homo);
  atomicAdd(k + 13, c.mixed);
}

// The shade phase.  Out of line, so that the trace loop has the registers to itself.
template <bool METRICS>
static __device__ __noinline__ void shade_phase(const RenderArgs& a, SlotLists& L, int cur, bool first,
                                                TraceCounters* c) {
  const DevScene& S = a.S;
  char* const base_q = block_slots(a);
  const int lane = threadIdx.x & 31;
  const int n = L.count[cur];
  const int* list = slot_list(a, base_q, cur);
  int* out_list = slot_list(a, base_q, cur ^ 1);
  for (int e0 = threadIdx.x - lane; e0 < n; e0 += kBlock) {
    const bool in = e0 + lane < n;
    const int s = !in ? 0 : n == a.slots ? e0 + lane : list[e0 + lane];
    const Slot Q(base_q, s);
    uint32_t rng = 0;
    int depth = 0, so = -1;
    float3 o = v3(0, 0, 0), d = v3(0, 0, 0), thr = v3(0, 0, 0), rad = v3(0, 0, 0);
    bool finished = false, alive = in, need = first && in;
    long long item = 0, pixel = 0;
    if (in && !first) {
      const float4 o4 = Q.o(), d4 = Q.d(), t4 = Q.thr(), r4 = Q.rad();
      const float2 h2 = Q.hit();
      o = v3(o4.x, o4.y, o4.z);
      rng = __float_as_uint(o4.w);
      d = v3(d4.x, d4.y, d4.z);
      depth = __float_as_int(d4.w);
      thr = v3(t4.x, t4.y, t4.z);
      rad = v3(r4.x, r4.y, r4.z);
      so = __float_as_int(r4.w);
      const Best h = slot_hit<METRICS>(S, h2, o, d, c);
      finished = shade_segment(S, h.type >= 0, h, o, d, thr, rad, rng, depth, a.max_depth);
    }
    if (finished) {
      item = pixel = Q.item();
      if (item < 0) {
        float* t = a.tail + 3 * (size_t)~item;
        t[0] = rad.x;
        t[1] = rad.y;
        t[2] = rad.z;
        need = true;
      } else {
        float3 acc = rad;
        if (so > 0) {
          const float4 a4 = Q.acc();
          acc = add(v3(a4.x, a4.y, a4.z), rad);
        }
        so++;
        if (so == a.spp) {
          acc = mul(acc, a.inv_spp);
          float* out = a.out + 3 * item;
          out[0] = acc.x;
          out[1] = acc.y;
          out[2] = acc.z;
          need = true;
        } else {
          Q.acc() = make_float4(acc.x, acc.y, acc.z, 0.0f);
        }
      }
    }
    // An abort ends every path at its sample's end: pixels with samples left stay unwritten.
    if (__any_sync(0xFFFFFFFFu, finished || need) && abort_raised(a.abort_flag) && (finished || need))
      alive = finished = need = false;
    // ---- fetch an item (warp-aggregated) for slots that need one
    const unsigned need_mask = __ballot_sync(0xFFFFFFFFu, need);
    if (need_mask) {
      unsigned long long basep = 0;
      const int leader = __ffs(need_mask) - 1;
      if (lane == leader) basep = atomicAdd(a.queue, (unsigned long long)__popc(need_mask));
      basep = __shfl_sync(0xFFFFFFFFu, basep, leader);
      if (need) {
        const long long p = (long long)basep + __popc(need_mask & ((1u << lane) - 1u));
        finished = alive = p < a.items;
        take_item(a, p, item, pixel, so);
        if (alive) Q.item() = item;
      }
    }
    // ---- start a sample (renderKernel prologue, K:1251-1264)
    if (alive) {
      if (finished) {
        start_sample(a, pixel, so, rng, o, d);
        thr = v3(1.0f, 1.0f, 1.0f);
        rad = v3(0.0f, 0.0f, 0.0f);
        depth = 0;
      }
      Q.o() = make_float4(o.x, o.y, o.z, __uint_as_float(rng));
      Q.d() = make_float4(d.x, d.y, d.z, __int_as_float(depth));
      Q.thr() = make_float4(thr.x, thr.y, thr.z, 0.0f);
      Q.rad() = make_float4(rad.x, rad.y, rad.z, __int_as_float(so));
    }
    const unsigned alive_mask = __ballot_sync(0xFFFFFFFFu, alive);
    int base = 0;
    if (lane == 0 && alive_mask) base = atomicAdd(&L.count[cur ^ 1], __popc(alive_mask));
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    if (alive) out_list[base + __popc(alive_mask & ((1u << lane) - 1u))] = s;
  }
}

template <bool METRICS, int SDEPTH>
__global__ void __launch_bounds__(kBlock, 1) k_render(const __grid_constant__ RenderArgs a) {
  extern __shared__ int2 s_stack[];  // [SDEPTH][kBlock]
  __shared__ SlotLists L;
  TraceCounters c{};
  if (threadIdx.x == 0) {
    L.count[0] = a.slots;
    L.count[1] = 0;
  }
  int cur = 0;
  bool first = true;
  while (true) {
    __syncthreads();
    shade_phase<METRICS>(a, L, cur, first, METRICS ? &c : nullptr);
    first = false;
    __syncthreads();
    const int n = L.count[cur ^ 1];
    if (threadIdx.x == 0) {
      L.count[cur] = 0;
      begin_trace(a, L, cur ^ 1);
    }
    cur ^= 1;
    __syncthreads();
    if (n == 0) break;
    trace_phase<METRICS, SDEPTH>(a, L, &L.head, s_stack + threadIdx.x, METRICS ? &c : nullptr);
  }
  if (METRICS) add_counters(a.counters, c);
}

// Each lane holds one item at a time: a whole pixel, its samples in order, or a single sample.
template <bool METRICS, int SDEPTH>
__global__ void __launch_bounds__(kSmallBlock, 1024 / kSmallBlock) k_render_small(const __grid_constant__ RenderArgs a) {
  extern __shared__ int2 s_stack[];  // [SDEPTH][kSmallBlock]
  const DevScene& S = a.S;
  const int lane = threadIdx.x & 31;
  if (a.max_depth <= 0) {  // every sample is black
    for (long long p = (long long)blockIdx.x * kSmallBlock + threadIdx.x; p < 3 * a.pixels;
         p += (long long)gridDim.x * kSmallBlock)
      a.out[p] = 0.0f;
    return;
  }
  TraceCounters c{};
  long long item = 0, pixel = 0;
  int so = 0, depth = 0;
  uint32_t rng = 0;
  float3 acc = v3(0, 0, 0), thr = v3(0, 0, 0), rad = v3(0, 0, 0), o = v3(0, 0, 0), d = v3(0, 0, 0);
  bool alive = lane < a.slots, need = alive, start = true;
  while (true) {
    // ---- fetch an item (warp-aggregated) for lanes that need one
    const unsigned need_mask = __ballot_sync(0xFFFFFFFFu, need);
    if (need_mask) {
      unsigned long long basep = 0;
      const int leader = __ffs(need_mask) - 1;
      if (lane == leader)
        basep = abort_raised(a.abort_flag) ? (unsigned long long)a.items
                                           : atomicAdd(a.queue, (unsigned long long)__popc(need_mask));
      basep = __shfl_sync(0xFFFFFFFFu, basep, leader);
      if (need) {
        const long long p = (long long)basep + __popc(need_mask & ((1u << lane) - 1u));
        alive = p < a.items;
        need = false;
        take_item(a, p, item, pixel, so);
      }
      if (!__any_sync(0xFFFFFFFFu, alive)) break;
    }
    if (alive && start) {
      start_sample(a, pixel, so, rng, o, d);
      thr = v3(1.0f, 1.0f, 1.0f);
      rad = v3(0.0f, 0.0f, 0.0f);
      depth = 0;
      start = false;
    }
    Best b;
    const bool hit = trace_closest<METRICS, SDEPTH, kSmallBlock>(S, o, d, alive, b, METRICS ? &c : nullptr, nullptr,
                                                                  s_stack + threadIdx.x);
    if (alive) {
      if (METRICS) c.rays++;
      if (shade_segment(S, hit, b, o, d, thr, rad, rng, depth, a.max_depth)) {
        start = true;
        if (item < 0) {
          float* t = a.tail + 3 * (size_t)~item;
          t[0] = rad.x;
          t[1] = rad.y;
          t[2] = rad.z;
          need = true;
        } else {
          acc = so == 0 ? rad : add(acc, rad);
          so++;
          if (so == a.spp) {
            acc = mul(acc, a.inv_spp);
            float* out = a.out + 3 * item;
            out[0] = acc.x;
            out[1] = acc.y;
            out[2] = acc.z;
            need = true;
          }
        }
      }
    }
  }
  if (METRICS) add_counters(a.counters, c);
}

// One thread per tail pixel: the in-order FP32 sum of its samples, scaled as in k_render.
// A frame whose render stopped on an abort leaves tail pixels unwritten, like the pixels it
// never fetched.
__global__ void __launch_bounds__(256) k_sum_tail(const float* __restrict__ tail, float* out,
                                                 long long split, int tail_pixels, int spp,
                                                 const int* abort_flag) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= tail_pixels || abort_stopped(abort_flag)) return;
  const float* s = tail + 3 * (size_t)q * spp;
  float3 acc = v3(s[0], s[1], s[2]);
  for (int i = 1; i < spp; i++) acc = add(acc, v3(s[3 * i], s[3 * i + 1], s[3 * i + 2]));
  acc = mul(acc, 1.0f / (float)spp);
  float* o = out + 3 * (split + q);
  o[0] = acc.x;
  o[1] = acc.y;
  o[2] = acc.z;
}

constexpr int kTraceBlock = 128;

// `per_warp` rays a warp, in its first lanes.
template <bool METRICS>
__global__ void __launch_bounds__(kTraceBlock) k_trace(const __grid_constant__ DevScene S, const float* rays, int n,
                                                       int per_warp, int* flags, float* dist, int* order, int* mat,
                                                       float* normal, unsigned long long* counters) {
  const int lane = threadIdx.x & 31;
  const long long at = ((long long)blockIdx.x * (kTraceBlock / 32) + (threadIdx.x >> 5)) * per_warp + lane;
  const bool active = lane < per_warp && at < n;  // every lane stays for the warp-cooperative traversal
  const int r = active ? (int)at : 0;
  float3 o = v3(0.0f, 0.0f, 0.0f), d = v3(0.0f, 0.0f, 1.0f);
  if (active) {
    const float* ry = rays + 6 * (size_t)r;
    o = v3(ry[0], ry[1], ry[2]);
    d = v3(ry[3], ry[4], ry[5]);
  }
  TraceCounters c{};
  Best b;
  bool hit = trace_closest<METRICS>(S, o, d, active, b, &c, nullptr);
  if (!active) return;
  float3 nn = v3(0, 0, 0);
  int mi = -1;
  if (hit) {
    const HitRecord hr = hit_record(S, b, o, d, add(o, mul(d, b.t)));
    nn = hr.n;
    mi = hr.material;
  }
  flags[r] = hit ? 1 : 0;
  dist[r] = hit ? b.t : CUDART_INF_F;
  order[r] = hit ? order_of(S, b.type, b.index) : -1;
  mat[r] = hit ? mi : -1;
  normal[3 * (size_t)r] = nn.x;
  normal[3 * (size_t)r + 1] = nn.y;
  normal[3 * (size_t)r + 2] = nn.z;
  if (METRICS) {
    atomicAdd(counters + 0, 1ULL);
    atomicAdd(counters + 1, c.aabb);
    atomicAdd(counters + 2, c.prim);
    atomicAdd(counters + 3, c.type[0]);
    atomicAdd(counters + 4, c.type[1]);
    atomicAdd(counters + 5, c.type[2]);
    atomicAdd(counters + 6, c.type[3]);
    atomicAdd(counters + 7, c.type[4]);
    atomicAdd(counters + 8, c.overflow);
    atomicMax(counters + 9, c.maxstack);
    atomicAdd(counters + 10, c.internal);
    atomicAdd(counters + 11, c.leaf);
    atomicAdd(counters + 12, c.homo);
    atomicAdd(counters + 13, c.mixed);
  }
}

// Scenes whose traversal data (nodes, references, primitive records) exceed this many bytes
// use the shared-memory stack: on the 1M-primitive scene (about 150 MB) it was 5 % faster,
// on the 10k scene (about 2 MB) 1.7 % slower.
constexpr long long kSharedStackSceneBytes = 16LL << 20;
constexpr int kSharedStackDepth = 16;

#ifndef RTB_TAIL_FACTOR
#define RTB_TAIL_FACTOR 4.0
#endif
// At most 64M tail samples (768 MB of radiance, held by the context); frames whose last
// four pixels per resident thread hold more samples split fewer pixels.
constexpr long long kMaxTailItems = 1LL << 26;

// ---- the wavefront form of a frame (rtb_render_device_wavefront)
//
// One wave per sample index over every pixel of the frame; per bounce, k_wf_trace runs the
// closest-hit query of every live path of the wave (the compacted list) and k_wf_shade
// shades it through shade_segment (k_render's segment statements), appending the paths
// that go on to the next list.  Path state lives in HBM, 16-byte records per path: origin, direction,
// throughput with the random stream's state, radiance with the depth, and the hit.  A
// pixel's samples are summed in sample order, one wave after the other, as k_render sums
// them, so the image is bit-identical.  It exists as the A/B counterpart of the persistent
// kernel: on the B200 it is slower (the state round trips and the per-bounce launches cost
// more than the warps' coherence buys).
struct WaveState {
  float4* o;    // origin (w unused)
  float4* d;    // direction (w unused)
  float4* thr;  // throughput; w holds the random stream's state
  float4* rad;  // radiance; w holds the depth
  Best* hit;
  int* list[2];
  int* count;   // sizes of list[0] and list[1]
};

__global__ void __launch_bounds__(256) k_wf_start(RenderArgs a, WaveState W, int so, int cur) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= a.pixels) return;
  const int x = (int)(p % a.width), y = (int)(p / a.width);
  if (p == 0) W.count[cur] = (a.max_depth > 0 && !abort_raised(a.abort_flag)) ? (int)a.pixels : 0;
  if (a.max_depth <= 0) {  // a black sample, summed like k_render's
    float* out = a.out + 3 * p;
    float3 acc = so == 0 ? v3(0, 0, 0) : add(v3(out[0], out[1], out[2]), v3(0, 0, 0));
    if (so + 1 == a.spp) acc = mul(acc, 1.0f / (float)a.spp);
    out[0] = acc.x;
    out[1] = acc.y;
    out[2] = acc.z;
    return;
  }
  uint32_t rng;
  float3 o, d;
  camera_sample(a, x, y, so, rng, o, d);
  W.o[p] = make_float4(o.x, o.y, o.z, 0.0f);
  W.d[p] = make_float4(d.x, d.y, d.z, 0.0f);
  W.thr[p] = make_float4(1.0f, 1.0f, 1.0f, __uint_as_float(rng));
  W.rad[p] = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(0));
  W.list[cur][p] = (int)p;
}

template <int SDEPTH>
__global__ void __launch_bounds__(128, 8) k_wf_trace(const __grid_constant__ RenderArgs a, WaveState W,
                                                                           int cur) {
  __shared__ int2 s_stack[SDEPTH > 0 ? SDEPTH : 1][128];
  const int n = W.count[cur];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if ((i & ~31) >= n) return;  // whole warps only: the traversal is warp-cooperative
  const bool active = i < n;
  const int p = active ? W.list[cur][i] : 0;
  float3 o = v3(0, 0, 0), d = v3(0, 0, 0);
  if (active) {
    const float4 o4 = W.o[p], d4 = W.d[p];
    o = v3(o4.x, o4.y, o4.z);
    d = v3(d4.x, d4.y, d4.z);
  }
  Best b;
  TraceCounters c{};
  const bool hit = trace_closest<false, SDEPTH, 128>(a.S, o, d, active, b, &c, nullptr,
                                                    &s_stack[0][threadIdx.x]);
  if (active) {
    if (!hit) b.type = -1;
    W.hit[p] = b;
  }
}

__global__ void __launch_bounds__(256) k_wf_shade(const __grid_constant__ RenderArgs a, WaveState W, int so, int cur) {
  const int n = W.count[cur];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  if ((i & ~31) >= n) return;
  bool more = false;
  int p = 0;
  if (i < n) {
    p = W.list[cur][i];
    const float4 o4 = W.o[p], d4 = W.d[p], t4 = W.thr[p], r4 = W.rad[p];
    float3 o = v3(o4.x, o4.y, o4.z), d = v3(d4.x, d4.y, d4.z);
    float3 thr = v3(t4.x, t4.y, t4.z), rad = v3(r4.x, r4.y, r4.z);
    uint32_t rng = __float_as_uint(t4.w);
    int depth = __float_as_int(r4.w);
    const Best b = W.hit[p];
    if (shade_segment(a.S, b.type >= 0, b, o, d, thr, rad, rng, depth, a.max_depth)) {
      float* out = a.out + 3 * (size_t)p;
      float3 acc = so == 0 ? rad : add(v3(out[0], out[1], out[2]), rad);
      if (so + 1 == a.spp) acc = mul(acc, 1.0f / (float)a.spp);
      out[0] = acc.x;
      out[1] = acc.y;
      out[2] = acc.z;
    } else {
      W.o[p] = make_float4(o.x, o.y, o.z, 0.0f);
      W.d[p] = make_float4(d.x, d.y, d.z, 0.0f);
      W.thr[p] = make_float4(thr.x, thr.y, thr.z, __uint_as_float(rng));
      W.rad[p] = make_float4(rad.x, rad.y, rad.z, __int_as_float(depth));
      more = true;
    }
  }
  // warp-aggregated append to the next bounce's list
  const unsigned m = __ballot_sync(0xFFFFFFFFu, more);
  if (m) {
    const int leader = __ffs(m) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(W.count + (cur ^ 1), __popc(m));
    base = __shfl_sync(0xFFFFFFFFu, base, leader);
    if (more) W.list[cur ^ 1][base + __popc(m & ((1u << lane) - 1u))] = p;
  }
}

}  // namespace

// One frame's launch: arguments, and how its pixels become items and blocks.  Built by
// plan_frame; the caller binds the queue, the buffers and the flags.
struct FramePlan {
  RenderArgs a;
  FrameShape shape;
  int metrics = 0;
  int shared_stack = 0;       // k_render's SDEPTH: 0, 8 or kSharedStackDepth
};

namespace {

template <bool METRICS, int SDEPTH>
const void* render_kernel_of(int block) {
  return block == kBlock ? (const void*)k_render<METRICS, SDEPTH> : (const void*)k_render_small<METRICS, SDEPTH>;
}

const void* render_kernel(int metrics, int shared_stack, int block) {
  if (shared_stack == kSharedStackDepth)
    return metrics ? render_kernel_of<true, kSharedStackDepth>(block)
                   : render_kernel_of<false, kSharedStackDepth>(block);
  if (shared_stack == 8) return metrics ? render_kernel_of<true, 8>(block) : render_kernel_of<false, 8>(block);
  return metrics ? render_kernel_of<true, 0>(block) : render_kernel_of<false, 0>(block);
}

size_t stack_smem(int shared_stack, int block) { return (size_t)shared_stack * block * sizeof(int2); }

int frame_blocks_per_sm(rtb_context* ctx, int metrics, int shared_stack, int block) {
  int& bps = ctx->frame_blocks[metrics][shared_stack == 0 ? 0 : shared_stack == 8 ? 1 : 2][block == kBlock];
  if (bps == 0) {
    const void* kernel = render_kernel(metrics, shared_stack, block);
    const size_t smem = stack_smem(shared_stack, block);
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kernel, block, smem);
    if (bps < 1) bps = 1;
    // Loads the sum's code now: loaded at its first launch, behind a running frame, it would
    // hold up an abort request until the frame ends.
    cudaFuncAttributes loaded;
    cudaFuncGetAttributes(&loaded, (const void*)k_sum_tail);
  }
  return bps;
}

long long traversal_bytes(const DevScene& S) {
  return (long long)S.node_count * 64 + (long long)S.ref_count * 4 + (long long)S.count[kSphere] * 16 +
         (long long)S.count[kBox] * 32 + ((long long)S.count[kAffineSphere] + S.count[kAffineBox]) * 48;
}

long long resident_threads(rtb_context* ctx, const FramePlan* f, int block) {
  return (long long)ctx->sm_count * frame_blocks_per_sm(ctx, f->metrics, f->shared_stack, block) * block;
}

}  // namespace

rtb_status plan_frame(rtb_context* ctx, rtb_scene* scene, const rtb_camera* cam,
                      const rtb_render_params* p, float* d_rgb, FramePlan* f, int row0,
                      int row_stride, int tail_per_thread) {
  if (!scene || !cam || !p || !d_rgb) return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "null argument");
  if (p->width < 1 || p->height < 1 || p->samples_per_frame < 1)
    return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "image size and samples must be positive");
  if (p->max_depth < 0 || p->max_depth > 32)
    return fail(ctx, RTB_ERR_INVALID_ARGUMENT,
                "GPU full-path depth must be in [0, 32] but was " + std::to_string(p->max_depth));
  RenderArgs& a = f->a;
  a = frame_args(scene, cam, p);
  if (row0 < 0 || row0 >= p->height || row_stride < 1)
    return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "first row must be in [0, height) and the stride positive");
  a.out = d_rgb;
  a.row0 = row0;
  a.row_stride = row_stride;
  a.pixels = (long long)p->width * ((p->height - row0 + row_stride - 1) / row_stride);
  f->metrics = p->collect_metrics ? 1 : 0;
  // rtb_render_params.shared_stack_entries: 0 picks by scene size, -1 none, 8 or 16 entries
  int se = p->shared_stack_entries;
  if (se != 0 && se != -1 && se != 8 && se != kSharedStackDepth)
    return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "shared_stack_entries must be 0, -1, 8 or 16");
  f->shared_stack = se == 0 ? (traversal_bytes(a.S) > kSharedStackSceneBytes ? kSharedStackDepth : 0)
                  : se < 0 ? 0 : se;
  FrameShape& shape = f->shape;
  shape.block = use_phases(a, ctx->sm_count) ? kBlock : kSmallBlock;
  shape.sm_count = ctx->sm_count;
  shape.spp = a.spp;
  shape.pixels = a.pixels;
  shape.resident = resident_threads(ctx, f, shape.block);
  // Tail: about four pixels per resident thread are split into single samples.
  double per_thread = tail_per_thread > 0 ? (double)tail_per_thread : RTB_TAIL_FACTOR;
  long long tail_pixels = std::min<long long>(a.pixels, (long long)(per_thread * shape.resident));
  // A pixel of one sample is its own item, and a black frame has none.
  shape.set_tail(a.max_depth > 0 && a.spp > 1 ? std::min<long long>(tail_pixels, kMaxTailItems / a.spp) : 0);
  return RTB_OK;
}

size_t frame_tail_bytes(const FramePlan* f) { return f->shape.tail_bytes(); }

size_t frame_path_bytes(const FramePlan* f) { return f->shape.path_bytes(); }

void frame_without_slots(rtb_context* ctx, FramePlan* f) {
  if (f->shape.block == kBlock) f->shape.without_slots(resident_threads(ctx, f, kSmallBlock));
}

void bind_frame(FramePlan* f, unsigned long long* queue, float* tail, void* paths, int* abort_flag,
                unsigned long long* counters) {
  RenderArgs& a = f->a;
  a.split = f->shape.split;
  a.items = f->shape.items;
  a.slots = f->shape.slots;
  a.queue = queue;
  a.tail = tail;
  a.paths = paths;
  a.abort_flag = abort_flag;
  a.counters = counters;
}

int launch_frame(const FramePlan* f, cudaStream_t stream) {
  const RenderArgs& a = f->a;
  const FrameShape& shape = f->shape;
  void* args[] = {const_cast<RenderArgs*>(&a)};
  cudaLaunchKernel(render_kernel(f->metrics, f->shared_stack, shape.block), dim3((unsigned)shape.grid),
                   dim3(shape.block), args, stack_smem(f->shared_stack, shape.block), stream);
  if (shape.tail_pixels == 0) return 1;
  k_sum_tail<<<(unsigned)((shape.tail_pixels + 255) / 256), 256, 0, stream>>>(
      a.tail, a.out, a.split, (int)shape.tail_pixels, a.spp, a.abort_flag);
  return 2;
}

FramePlan* new_frame_plan() { return new FramePlan(); }
void delete_frame_plan(FramePlan* f) { delete f; }

rtb_status render_frame(rtb_context* ctx, rtb_scene* scene, const rtb_camera* cam,
                        const rtb_render_params* p, float* d_rgb, cudaStream_t stream, bool timed,
                        int row0, int row_stride) {
  FramePlan f;
  rtb_status s = plan_frame(ctx, scene, cam, p, d_rgb, &f, row0, row_stride);
  if (s != RTB_OK) return s;
  settle_frame(
      f.shape, [&](size_t bytes) { return ctx_grow(&ctx->d_tail, &ctx->tail_bytes, bytes, stream); },
      [&](size_t bytes) { return ctx_grow_paths(ctx, bytes, stream); },
      [&] { return resident_threads(ctx, &f, kSmallBlock); });
  bind_frame(&f, ctx->d_work, ctx->d_tail, ctx->d_paths, ctx->d_abort, ctx->d_work + 8);
  if (timed) cudaEventRecord(ctx->ev0, stream);
  ctx->render_launches = launch_frame(&f, stream);
  if (timed) cudaEventRecord(ctx->ev1, stream);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(ctx, e, "render launch");
  return RTB_OK;
}

struct TraceGrid {
  unsigned blocks;
  int per_warp;
};
static TraceGrid trace_grid(int n, int sm_count) {
  const int per = lanes_per_warp(n, sm_count);
  const long long per_block = (long long)per * (kTraceBlock / 32);
  return TraceGrid{(unsigned)((n + per_block - 1) / per_block), per};
}

cudaError_t launch_trace(const DevScene& scene, int use_bvh, const float* d_rays, int n, int* d_flags,
                         float* d_t, int* d_order, int* d_mat, float* d_normal, cudaStream_t stream) {
  DevScene S = scene;
  S.use_bvh = use_bvh ? scene.use_bvh : 0;
  if (n > 0) {
    int device = 0, sm_count = 1;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device);
    const TraceGrid g = trace_grid(n, sm_count);
    k_trace<false><<<g.blocks, kTraceBlock, 0, stream>>>(S, d_rays, n, g.per_warp, d_flags, d_t, d_order, d_mat,
                                                         d_normal, nullptr);
  }
  return cudaGetLastError();
}

rtb_status trace_rays(rtb_context* ctx, rtb_scene* scene, const float* d_rays, int n, int use_bvh,
                      int collect_metrics, int* d_flags, float* d_t, int* d_order, int* d_mat,
                      float* d_normal, cudaStream_t stream) {
  DevScene S = scene->dev;
  S.use_bvh = (use_bvh && scene->has_bvh) ? 1 : 0;
  unsigned long long* counters = ctx->d_work + 8;
  if (collect_metrics) cudaMemsetAsync(ctx->d_work, 0, 32 * sizeof(unsigned long long), stream);
  if (n > 0) {
    const TraceGrid g = trace_grid(n, ctx->sm_count);
    if (collect_metrics)
      k_trace<true><<<g.blocks, kTraceBlock, 0, stream>>>(S, d_rays, n, g.per_warp, d_flags, d_t, d_order, d_mat,
                                                          d_normal, counters);
    else
      k_trace<false><<<g.blocks, kTraceBlock, 0, stream>>>(S, d_rays, n, g.per_warp, d_flags, d_t, d_order, d_mat,
                                                           d_normal, counters);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(ctx, e, "trace launch");
  return RTB_OK;
}

rtb_status render_frame_wavefront(rtb_context* ctx, rtb_scene* scene, const rtb_camera* cam,
                                  const rtb_render_params* p, float* d_rgb, cudaStream_t stream) {
  FramePlan f;
  rtb_status s = plan_frame(ctx, scene, cam, p, d_rgb, &f, 0, 1);
  if (s != RTB_OK) return s;
  if (f.metrics) return fail(ctx, RTB_ERR_UNSUPPORTED, "the wavefront form has no metrics build");
  const long long P = f.a.pixels;
  if (P > 0x7FFFFFFFLL) return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "frame too large");
  // path state: four 16-byte records, the hit and two list slots per pixel, two counts
  const size_t bytes = (size_t)P * (4 * sizeof(float4) + sizeof(Best) + 2 * sizeof(int)) + 256;
  if (bytes > ctx->wave_bytes) {
    cudaStreamSynchronize(stream);  // an earlier wavefront frame may still use the buffer
    cudaFree(ctx->d_wave);
    ctx->d_wave = nullptr;
    ctx->wave_bytes = 0;
    if (cudaMalloc(&ctx->d_wave, bytes) != cudaSuccess) {
      cudaGetLastError();
      return fail(ctx, RTB_ERR_OUT_OF_MEMORY, "wavefront path state");
    }
    ctx->wave_bytes = bytes;
  }
  char* q = (char*)ctx->d_wave;
  WaveState W;
  W.o = (float4*)q;
  W.d = W.o + P;
  W.thr = W.d + P;
  W.rad = W.thr + P;
  W.hit = (Best*)(W.rad + P);
  W.list[0] = (int*)(W.hit + P);
  W.list[1] = W.list[0] + P;
  W.count = W.list[1] + P;
  f.a.abort_flag = ctx->d_abort;
  const unsigned g256 = (unsigned)((P + 255) / 256), g128 = (unsigned)((P + 127) / 128);
  int launches = 0;
  for (int so = 0; so < f.a.spp; ++so) {
    int cur = 0;
    k_wf_start<<<g256, 256, 0, stream>>>(f.a, W, so, cur);
    ++launches;
    for (int b = 0; b < f.a.max_depth; ++b) {
      if (f.shared_stack == kSharedStackDepth)
        k_wf_trace<kSharedStackDepth><<<g128, 128, 0, stream>>>(f.a, W, cur);
      else if (f.shared_stack == 8)
        k_wf_trace<8><<<g128, 128, 0, stream>>>(f.a, W, cur);
      else
        k_wf_trace<0><<<g128, 128, 0, stream>>>(f.a, W, cur);
      cudaMemsetAsync(W.count + (cur ^ 1), 0, sizeof(int), stream);
      k_wf_shade<<<g256, 256, 0, stream>>>(f.a, W, so, cur);
      launches += 2;
      cur ^= 1;
    }
  }
  ctx->render_launches = launches;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(ctx, e, "wavefront launch");
  return RTB_OK;
}

}  // namespace rtb
