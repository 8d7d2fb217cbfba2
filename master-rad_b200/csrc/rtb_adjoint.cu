// Adjoint of the path tracer with respect to per-material albedo (diffuse colour) and
// emission: path replay.  No counterpart in the reference.
//
// For one sample the kernel's radiance is  L = sum_k thr_k (*) E_k  (+ thr_K (*) background on
// a miss), with thr_{k+1} = thr_k (*) W_k and W_k the lobe weight colour (for the diffuse lobe
// W = albedo / p, p the lobe probability).  Given the image adjoint a = dLoss/dI of the
// pixel, the backward kernel re-traces each sample from its random seed -- the same traversal
// and the same random stream as the forward frame, so the same path -- keeping the vertices
// (material, thr, W, 1/p, lobe) in a per-thread stack, then walks them backward with the
// incoming radiance Li (background or 0 after the last vertex, Li <- E_k + W_k (*) Li):
//     dLoss/dE_k      += (a / spp) (*) thr_k
//     dLoss/dalbedo_k += (a / spp) (*) thr_k (*) Li_after_k / p_k      (diffuse lobe chosen)
// The lobe probability is treated as fixed (the sampling decision is not differentiated); for
// materials with only a diffuse lobe -- the differentiable workload's -- p = 1 and the result
// is the exact derivative of the rendered image.  Emission gradients are exact for all
// materials.  Gradients accumulate in FP32: first in a per-block shared-memory table keyed by
// material (walls and emitters are hit by most paths), then with one global atomic per entry.
#include <algorithm>

#include "rtb_internal.h"
#include "rtb_paths.cuh"

namespace rtb {
namespace {

constexpr int kTable = 512;       // shared-memory gradient entries per block
constexpr int kMaxVertices = 32;  // max_depth limit of the renderer

struct AdjointArgs {
  RenderArgs r;          // scene, camera, sizes, queue, path slots
  const float* adjoint;  // dLoss/dI, 3 floats per pixel
  float* grad_albedo;    // 3 per material
  float* grad_emission;  // 3 per material
  float4* vertices;      // k_adjoint: the slots' path vertices, see PathVertices
  long long samples;     // of the frame
};

struct GradTable {
  int key[kTable];
  float val[kTable][6];
};

__device__ __forceinline__ void clear_table(GradTable& T) {
  for (int i = threadIdx.x; i < kTable; i += blockDim.x) {
    T.key[i] = -1;
    for (int k = 0; k < 6; ++k) T.val[i][k] = 0.0f;
  }
}

// Adds the table to the gradients and empties it; between barriers.
__device__ __forceinline__ void flush_table(GradTable& T, const AdjointArgs& a) {
  for (int i = threadIdx.x; i < kTable; i += blockDim.x) {
    const int m = T.key[i];
    if (m < 0) continue;
    for (int k = 0; k < 3; ++k) {
      if (T.val[i][k] != 0.0f) atomicAdd(a.grad_albedo + 3 * m + k, T.val[i][k]);
      if (T.val[i][3 + k] != 0.0f) atomicAdd(a.grad_emission + 3 * m + k, T.val[i][3 + k]);
      T.val[i][k] = T.val[i][3 + k] = 0.0f;
    }
    T.key[i] = -1;
  }
}

// The albedo gradient is zero wherever the path met no light afterwards: nothing is added then.
__device__ __forceinline__ void accumulate(GradTable& T, const AdjointArgs& a, int m, float3 ga, float3 ge) {
  float* pa = a.grad_albedo + 3 * m;
  float* pe = a.grad_emission + 3 * m;
  unsigned h = ((unsigned)m * 2654435761u) & (kTable - 1);
  for (int probe = 0; probe < 8; ++probe) {
    int slot = (h + probe) & (kTable - 1);
    int k = *(volatile int*)&T.key[slot];
    if (k == -1) k = atomicCAS(&T.key[slot], -1, m);
    if (k == -1 || k == m) {
      pa = &T.val[slot][0];
      pe = &T.val[slot][3];
      break;
    }
  }
  if (ga.x != 0.0f || ga.y != 0.0f || ga.z != 0.0f) {
    atomicAdd(pa, ga.x);
    atomicAdd(pa + 1, ga.y);
    atomicAdd(pa + 2, ga.z);
  }
  atomicAdd(pe, ge.x);
  atomicAdd(pe + 1, ge.y);
  atomicAdd(pe + 2, ge.z);
}

__device__ __forceinline__ float warp_sum(float v) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, off);
  return v;
}

// accumulate() for the lanes with `valid` set, all 32 lanes calling it.  Walls and lights are hit by
// many lanes at once, and adds to one shared word run one after the other: the materials that
// most lanes share are summed over the warp first, at most two of them.
__device__ __forceinline__ void accumulate_warp(GradTable& T, const AdjointArgs& a, bool valid, int m, float3 ga,
                                                float3 ge) {
  for (int round = 0; round < 2; ++round) {
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, valid ? m : -1);
    const int share = valid ? __popc(peers) : 0;
    const int most = __reduce_max_sync(0xFFFFFFFFu, share);
    if (most < 6) break;
    const int leader = __ffs(__ballot_sync(0xFFFFFFFFu, share == most)) - 1;
    const int common = __shfl_sync(0xFFFFFFFFu, m, leader);
    const bool in = valid && m == common;
    float3 sa = v3(0, 0, 0);
    if (__any_sync(0xFFFFFFFFu, in && (ga.x != 0.0f || ga.y != 0.0f || ga.z != 0.0f)))
      sa = v3(warp_sum(in ? ga.x : 0.0f), warp_sum(in ? ga.y : 0.0f), warp_sum(in ? ga.z : 0.0f));
    const float3 se = v3(warp_sum(in ? ge.x : 0.0f), warp_sum(in ? ge.y : 0.0f), warp_sum(in ? ge.z : 0.0f));
    if ((int)(threadIdx.x & 31) == leader) accumulate(T, a, common, sa, se);
    valid = valid && !in;
  }
  if (valid) accumulate(T, a, m, ga, ge);
}

// The vertices of a block's paths: (throughput, 1 / p or 0) and (lobe weight, material), by
// vertex, then slot.
struct PathVertices {
  float4* v;
  int slots;
  __device__ __forceinline__ PathVertices(const AdjointArgs& a)
      : v(a.vertices + (size_t)blockIdx.x * a.r.slots * a.r.max_depth * 2), slots(a.r.slots) {}
  __device__ __forceinline__ float4& thr(int k, int s) const { return v[(size_t)(2 * k) * slots + s]; }
  __device__ __forceinline__ float4& w(int k, int s) const { return v[(size_t)(2 * k + 1) * slots + s]; }
};

// Queue entry p: a sample of a pixel.
__device__ __forceinline__ void sample_item(const AdjointArgs& a, long long p, long long& pixel, int& so) {
  if (a.samples <= 0xFFFFFFFFLL) {
    const unsigned q = fast_div((unsigned)p, a.r.spp_magic);
    pixel = q;
    so = (int)((unsigned)p - q * (unsigned)a.r.spp);
  } else {
    pixel = p / a.r.spp;
    so = (int)(p % a.r.spp);
  }
}

__device__ __forceinline__ float3 pixel_adjoint(const AdjointArgs& a, long long pixel) {
  const float* ap = a.adjoint + 3 * pixel;
  return v3(ap[0] * a.r.inv_spp, ap[1] * a.r.inv_spp, ap[2] * a.r.inv_spp);
}

// The shade phase of the replay: every traced path gets its vertex, and a path that ends is
// walked backward into the gradients and replaced by the queue's next sample.
static __device__ __noinline__ void replay_phase(const AdjointArgs& a, GradTable& T, SlotLists& L, int cur,
                                                 bool first) {
  const DevScene& S = a.r.S;
  char* const base_q = block_slots(a.r);
  const PathVertices V(a);
  const int lane = threadIdx.x & 31;
  const int n = L.count[cur];
  const int* list = slot_list(a.r, base_q, cur);
  int* out_list = slot_list(a.r, base_q, cur ^ 1);
  for (int e0 = threadIdx.x - lane; e0 < n; e0 += kBlock) {
    const bool in = e0 + lane < n;
    const int s = !in ? 0 : n == a.r.slots ? e0 + lane : list[e0 + lane];
    const Slot Q(base_q, s);
    uint32_t rng = 0;
    int depth = 0, nv = 0;
    float3 o = v3(0, 0, 0), d = v3(0, 0, 0), thr = v3(0, 0, 0), adj = v3(0, 0, 0), li = v3(0, 0, 0);
    bool alive = in, finished = first && in;
    if (in && !first) {
      const float4 o4 = Q.o(), d4 = Q.d(), t4 = Q.thr();
      o = v3(o4.x, o4.y, o4.z);
      rng = __float_as_uint(o4.w);
      d = v3(d4.x, d4.y, d4.z);
      depth = nv = __float_as_int(d4.w);
      thr = v3(t4.x, t4.y, t4.z);
      const Best h = slot_hit<false>(S, Q.hit(), o, d, nullptr);
      if (h.type < 0) {
        li = S.background;
        finished = true;
      } else {
        const Vertex v = hit_vertex(S, h, o, d);
        float3 wc = v3(0.0f, 0.0f, 0.0f);
        float pc = 1.0f;
        bool diffuse = false;
        finished = !scatter(v, o, d, rng, wc, pc, diffuse);
        // 1 / p of 0: no albedo gradient through this vertex
        V.thr(depth, s) = make_float4(thr.x, thr.y, thr.z, diffuse ? 1.0f / pc : 0.0f);
        V.w(depth, s) = make_float4(wc.x, wc.y, wc.z, __int_as_float(v.material));
        nv = depth + 1;
        if (!finished) {
          thr = mulv(thr, wc);
          depth++;
          finished = depth >= a.r.max_depth;
        }
      }
      if (finished) adj = pixel_adjoint(a, Q.item());
    }
    // ---- backward over the vertices of the paths that ended
    if (__any_sync(0xFFFFFFFFu, finished && nv > 0)) {
      for (int k = __reduce_max_sync(0xFFFFFFFFu, finished ? nv : 0) - 1; k >= 0; --k) {
        const bool mine = finished && k < nv;
        int m = -1;
        float3 ga = v3(0, 0, 0), base = v3(0, 0, 0);
        if (mine) {
          const float4 t4 = V.thr(k, s), w4 = V.w(k, s);
          m = __float_as_int(w4.w);
          float3 e = v3(0.0f, 0.0f, 0.0f);
          if (m >= 0) {
            const float4 m3 = __ldg(S.materials + 4 * m + 3);
            e = v3(m3.x, m3.y, m3.z);
            base = mulv(adj, v3(t4.x, t4.y, t4.z));
            ga = mul(mulv(base, li), t4.w);
          }
          li = add(e, mulv(v3(w4.x, w4.y, w4.z), li));
        }
        accumulate_warp(T, a, mine && m >= 0, m, ga, base);
      }
    }
    // ---- the queue's next sample (warp-aggregated)
    const unsigned need_mask = __ballot_sync(0xFFFFFFFFu, finished);
    if (need_mask) {
      unsigned long long basep = 0;
      const int leader = __ffs(need_mask) - 1;
      if (lane == leader)
        basep = abort_raised(a.r.abort_flag) ? (unsigned long long)a.samples
                                             : atomicAdd(a.r.queue, (unsigned long long)__popc(need_mask));
      basep = __shfl_sync(0xFFFFFFFFu, basep, leader);
      if (finished) {
        const long long p = (long long)basep + __popc(need_mask & ((1u << lane) - 1u));
        alive = p < a.samples;
        if (alive) {
          long long pixel;
          int so;
          sample_item(a, p, pixel, so);
          start_sample(a.r, pixel, so, rng, o, d);
          thr = v3(1.0f, 1.0f, 1.0f);
          depth = 0;
          Q.item() = pixel;
        }
      }
    }
    if (alive) {
      Q.o() = make_float4(o.x, o.y, o.z, __uint_as_float(rng));
      Q.d() = make_float4(d.x, d.y, d.z, __int_as_float(depth));
      Q.thr() = make_float4(thr.x, thr.y, thr.z, 0.0f);
    }
    const unsigned alive_mask = __ballot_sync(0xFFFFFFFFu, alive);
    int at = 0;
    if (lane == 0 && alive_mask) at = atomicAdd(&L.count[cur ^ 1], __popc(alive_mask));
    at = __shfl_sync(0xFFFFFFFFu, at, 0);
    if (alive) out_list[at + __popc(alive_mask & ((1u << lane) - 1u))] = s;
  }
}

// The replay in the frame kernel's two phases.  The gradients of a block meet in a shared
// table that is added to the global ones every kFlushPhases phases, so that no partial sum grows
// longer than in one pass over a small share of the frame.
constexpr int kFlushPhases = 8;
__global__ void __launch_bounds__(kBlock, 1) k_adjoint(const __grid_constant__ AdjointArgs a) {
  __shared__ SlotLists L;
  __shared__ GradTable T;
  clear_table(T);
  if (threadIdx.x == 0) {
    L.count[0] = a.r.slots;
    L.count[1] = 0;
  }
  int cur = 0, phase = 0;
  while (true) {
    __syncthreads();
    replay_phase(a, T, L, cur, phase == 0);
    __syncthreads();
    const int n = L.count[cur ^ 1];
    if (threadIdx.x == 0) {
      L.count[cur] = 0;
      begin_trace(a.r, L, cur ^ 1);
    }
    cur ^= 1;
    __syncthreads();
    if (++phase % kFlushPhases == 0 || n == 0) flush_table(T, a);
    if (n == 0) break;
    trace_phase<false, 0>(a.r, L, &L.head, nullptr, nullptr);
  }
}

// One path a lane, for what the phases are not faster at (see use_phases).
__global__ void __launch_bounds__(128, 6) k_adjoint_small(const __grid_constant__ AdjointArgs a) {
  __shared__ GradTable T;
  clear_table(T);
  __syncthreads();
  const DevScene& S = a.r.S;
  const int lane = threadIdx.x & 31;
  long long pixel = 0;
  uint32_t rng = 0;
  float3 thr = v3(0, 0, 0), o = v3(0, 0, 0), d = v3(0, 0, 0);
  bool alive = a.r.max_depth > 0, finished = true;
  int nv = 0;
  // Vertex stack of the current sample.
  int vm[kMaxVertices];
  float3 vthr[kMaxVertices], vw[kMaxVertices];
  float vinvp[kMaxVertices];
  while (true) {
    const unsigned need_mask = __ballot_sync(0xFFFFFFFFu, alive && finished);
    if (need_mask) {
      unsigned long long basep = 0;
      const int leader = __ffs(need_mask) - 1;
      if (lane == leader)
        basep = abort_raised(a.r.abort_flag) ? (unsigned long long)a.samples
                                             : atomicAdd(a.r.queue, (unsigned long long)__popc(need_mask));
      basep = __shfl_sync(0xFFFFFFFFu, basep, leader);
      if (alive && finished) {
        const long long p = (long long)basep + __popc(need_mask & ((1u << lane) - 1u));
        alive = p < a.samples;
        if (alive) {
          int so;
          sample_item(a, p, pixel, so);
          start_sample(a.r, pixel, so, rng, o, d);
          thr = v3(1.0f, 1.0f, 1.0f);
          nv = 0;
          finished = false;
        }
      }
    }
    if (!__any_sync(0xFFFFFFFFu, alive)) break;
    Best b;
    const bool hit = trace_closest<false>(S, o, d, alive, b, nullptr, nullptr);
    float3 li = v3(0.0f, 0.0f, 0.0f);
    if (alive) {
      if (!hit) {
        li = S.background;
        finished = true;
      } else {
        const Vertex v = hit_vertex(S, b, o, d);
        float3 wc = v3(0.0f, 0.0f, 0.0f);
        float pc = 1.0f;
        bool diffuse = false;
        finished = !scatter(v, o, d, rng, wc, pc, diffuse);
        vm[nv] = v.material;
        vthr[nv] = thr;
        vw[nv] = wc;
        vinvp[nv] = diffuse ? 1.0f / pc : 0.0f;  // 0: no albedo gradient through this vertex
        nv++;
        if (!finished) {
          thr = mulv(thr, wc);
          finished = nv >= a.r.max_depth;
        }
      }
    }
    if (alive && finished) {
      // Backward over the sample's vertices.
      const float3 adj = pixel_adjoint(a, pixel);
      for (int k = nv - 1; k >= 0; --k) {
        int m = vm[k];
        float3 e = v3(0.0f, 0.0f, 0.0f);
        if (m >= 0) {
          float4 m3 = __ldg(S.materials + 4 * m + 3);
          e = v3(m3.x, m3.y, m3.z);
          float3 base = mulv(adj, vthr[k]);
          accumulate(T, a, m, mul(mulv(base, li), vinvp[k]), base);
        }
        li = add(e, mulv(vw[k], li));
      }
    }
  }
  __syncthreads();
  flush_table(T, a);
}

__global__ void k_repack_materials(const float* raw, int n, float4* out) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const float* r = raw + 13 * (size_t)s;
  out[4 * s] = make_float4(r[0], r[1], r[2], r[12]);
  out[4 * s + 1] = make_float4(r[3], r[4], r[5], 0.0f);
  out[4 * s + 2] = make_float4(r[6], r[7], r[8], 0.0f);
  out[4 * s + 3] = make_float4(r[9], r[10], r[11], 0.0f);
}

}  // namespace
}  // namespace rtb

using namespace rtb;

extern "C" {

rtb_status rtb_scene_set_materials(rtb_context* ctx, rtb_scene* scene, const float* materials,
                                   int material_count) {
  if (!ctx) return RTB_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(ctx->mu);
  cudaSetDevice(ctx->device);
  if (!scene || !materials || material_count != scene->dev.material_count)
    return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "material table must keep the scene's material count");
  size_t bytes = (size_t)material_count * 13 * sizeof(float);
  float* raw = (float*)stage(ctx, bytes);
  if (!raw) return fail(ctx, RTB_ERR_OUT_OF_MEMORY, "material staging");
  cudaStream_t sm = ctx->stream;
  ctx_acquire(ctx, sm);
  cudaMemcpyAsync(raw, materials, bytes, cudaMemcpyHostToDevice, sm);
  k_repack_materials<<<(material_count + 255) / 256, 256, 0, sm>>>(
      raw, material_count, const_cast<float4*>(scene->dev.materials));
  ctx_release(ctx, sm);
  cudaError_t e = cudaStreamSynchronize(sm);
  if (e == cudaSuccess) e = cudaGetLastError();
  return e == cudaSuccess ? RTB_OK : cuda_fail(ctx, e, "material update");
}

// The backward launch; the caller holds the context lock with its device current.
static rtb_status render_backward(rtb_context* ctx, rtb_scene* scene, const rtb_camera* cam,
                                  const rtb_render_params* p, const float* adjoint_device,
                                  float* grad_albedo_device, float* grad_emission_device,
                                  cudaStream_t stream) {
  if (!scene || !cam || !p || !adjoint_device || !grad_albedo_device || !grad_emission_device)
    return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "null argument");
  if (p->width < 1 || p->height < 1 || p->samples_per_frame < 1)
    return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "image size and samples must be positive");
  if (p->max_depth < 0 || p->max_depth > kMaxVertices)
    return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "GPU full-path depth must be in [0, 32]");
  cudaStream_t sm = stream ? stream : ctx->stream;
  ctx_acquire(ctx, sm);
  AdjointArgs a{};
  a.r = frame_args(scene, cam, p);
  a.adjoint = adjoint_device;
  a.grad_albedo = grad_albedo_device;
  a.grad_emission = grad_emission_device;
  a.samples = a.r.pixels * a.r.spp;
  a.r.queue = ctx->d_work;
  a.r.abort_flag = ctx->d_abort;
  bool phases = use_phases(a.r, ctx->sm_count);
  long long grid = ctx->sm_count;
  if (phases) {
    const ReplayShape shape(a.samples, a.r.max_depth, ctx->sm_count);
    // without the memory, one path a lane
    phases = ctx_grow_paths(ctx, shape.path_bytes + shape.vertex_bytes, sm);
    if (phases) {
      grid = shape.grid;
      a.r.slots = shape.slots;
      a.r.paths = ctx->d_paths;
      a.vertices = (float4*)((char*)ctx->d_paths + shape.path_bytes);
    }
  }
  size_t gbytes = (size_t)scene->dev.material_count * 3 * sizeof(float);
  arm_abort(ctx, sm, true);
  cudaMemsetAsync(grad_albedo_device, 0, gbytes, sm);
  cudaMemsetAsync(grad_emission_device, 0, gbytes, sm);
  cudaEventRecord(ctx->ev0, sm);
  if (phases) {
    k_adjoint<<<(unsigned)grid, kBlock, 0, sm>>>(a);
  } else {
    int bps = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, (const void*)k_adjoint_small, 128, 0);
    grid = std::min<long long>(grid * std::max(bps, 1), (a.samples + 127) / 128);
    k_adjoint_small<<<(unsigned)std::max<long long>(1, grid), 128, 0, sm>>>(a);
  }
  cudaEventRecord(ctx->ev1, sm);
  ctx_release(ctx, sm);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(ctx, e, "adjoint launch");
  return RTB_OK;
}

rtb_status rtb_render_backward(rtb_context* ctx, rtb_scene* scene, const rtb_camera* cam,
                               const rtb_render_params* p, const float* adjoint_device,
                               float* grad_albedo_device, float* grad_emission_device, void* stream) {
  if (!ctx) return RTB_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(ctx->mu);
  cudaSetDevice(ctx->device);
  return render_backward(ctx, scene, cam, p, adjoint_device, grad_albedo_device,
                         grad_emission_device, (cudaStream_t)stream);
}

rtb_status rtb_render_backward_sample(rtb_context* ctx, rtb_scene* scene, const rtb_camera* cam,
                                      const rtb_render_params* p, const float* adjoint,
                                      float* grad_albedo, float* grad_emission) {
  if (!ctx) return RTB_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(ctx->mu);
  cudaSetDevice(ctx->device);
  if (!scene || !p || !adjoint || !grad_albedo || !grad_emission)
    return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "null argument");
  if (p->width < 1 || p->height < 1)
    return fail(ctx, RTB_ERR_INVALID_ARGUMENT, "image size and samples must be positive");
  size_t img = (size_t)p->width * p->height * 3 * sizeof(float);
  size_t grads = (size_t)scene->dev.material_count * 3 * sizeof(float);
  size_t img_pad = (img + 255) & ~(size_t)255, grads_pad = (grads + 255) & ~(size_t)255;
  char* d = (char*)stage(ctx, img_pad + 2 * grads_pad);
  if (!d) return fail(ctx, RTB_ERR_OUT_OF_MEMORY, "adjoint staging");
  float* d_adj = (float*)d;
  float* d_ga = (float*)(d + img_pad);
  float* d_ge = (float*)(d + img_pad + grads_pad);
  cudaStream_t sm = ctx->stream;
  ctx_acquire(ctx, sm);
  cudaMemcpyAsync(d_adj, adjoint, img, cudaMemcpyHostToDevice, sm);
  ctx_release(ctx, sm);
  rtb_status s = render_backward(ctx, scene, cam, p, d_adj, d_ga, d_ge, sm);
  if (s != RTB_OK) return s;
  // Not before the replay is done: a copy to pageable memory waits inside the driver, where it
  // holds up an abort request from another thread.
  cudaError_t e = cudaEventSynchronize(ctx->ev1);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "adjoint");
  ctx_acquire(ctx, sm);
  cudaMemcpyAsync(grad_albedo, d_ga, grads, cudaMemcpyDeviceToHost, sm);
  cudaMemcpyAsync(grad_emission, d_ge, grads, cudaMemcpyDeviceToHost, sm);
  ctx_release(ctx, sm);
  e = cudaStreamSynchronize(sm);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "adjoint");
  int aborted = 0;
  cudaMemcpy(&aborted, ctx->d_abort + 2, sizeof(int), cudaMemcpyDeviceToHost);
  if (aborted) return fail(ctx, RTB_ERR_WATCHDOG, "backward pass aborted on request");
  return RTB_OK;
}

}  // extern "C"
