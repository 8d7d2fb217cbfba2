"""What a program does with rtb200, as cases that can be timed: frames, closest-hit queries,
tree builds, batches of frames and the differentiable frame, each through the entry points
that such a program calls, from a thumbnail of a 65-sphere scene to a million primitives.

A case is a dict of plain values whose "kind" is one of

  frame    ``GpuRayTracer.render_sample`` of a resident scene into a host image;
  rows     one rank's rows of a frame split over several GPUs, into device memory;
  trace    ``GpuRayTracer.trace_replay``: closest hits of rays held on the host;
  build    the tree of a scene held on the host, built on the device and downloaded;
  open     a scene held on the host is uploaded, built and shown as one small frame;
  adjoint  a frame and its gradients by every albedo and emission (autograd);
  batch    many scenes' frames in one replayed launch.

Scenes are the synthetic ones of this repository's benchmark and tests (rtb200/synth.py):
``plain`` (small spheres in a closed room), ``glass`` (refracting and reflecting spheres in
a lit box), ``mix`` (40 % spheres, 30 % boxes, 30 % affine spheres and boxes, uniform in the
room) and ``cluster`` (the same mix, small, in 64 Gaussian clusters).
"""
import ctypes as C
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "master-rad_b200"))

from rtb200 import native, synth  # noqa: E402
from rtb200.batch import Batch  # noqa: E402
from rtb200.diff import DifferentiableScene, render_function, torch_stream_handle  # noqa: E402
from rtb200.scene import BvhBuildConfig, BvhBuildMode, GpuScene, MaterialData  # noqa: E402
from rtb200.split import band_rows, device_rows_renderer  # noqa: E402
from rtb200.tracer import Context, GpuRayTracer, ResidentScene, camera_struct  # noqa: E402

CLUSTERS = 64
PALETTE = 4096  # colours of the larger scenes; many primitives share one
BYTES_PER_PRIMITIVE = 50  # the mix's mean record: 20 to 88 bytes by type
BATCH_SIDES = (128, 256, 512)
BATCH_SPP = (4, 16)


def listed():
    return [
        # A thumbnail or a cursor preview: launches and latency, hardly any work.
        {"name": "frame thumbnail", "kind": "frame", "scene": "plain", "primitives": 64,
         "width": 64, "height": 36, "spp": 1, "depth": 4},
        # The small frame of the benchmark: 64 spheres in a room, 256 x 256.
        {"name": "frame plain", "kind": "frame", "scene": "plain", "primitives": 64,
         "width": 256, "height": 256, "spp": 16, "depth": 4},
        # Long specular paths (glass, mirrors) at an odd size.
        {"name": "frame glass odd", "kind": "frame", "scene": "glass", "primitives": 4,
         "width": 451, "height": 253, "spp": 8, "depth": 24},
        # The benchmark's headline frame: 10k mixed primitives, 1024 x 1024, 64 samples.
        {"name": "frame mix 10k", "kind": "frame", "scene": "mix", "primitives": 10000,
         "width": 1024, "height": 1024, "spp": 64, "depth": 8},
        # The largest scene: a million clustered primitives in full HD.
        {"name": "frame cluster 1M", "kind": "frame", "scene": "cluster", "primitives": 1000000,
         "width": 1920, "height": 1080, "spp": 16, "depth": 8},
        # One of four ranks' share of a frame of odd size.
        {"name": "rows of a rank", "kind": "rows", "scene": "mix", "primitives": 50000,
         "width": 777, "height": 431, "spp": 16, "depth": 6, "ranks": 4, "rank": 1},
        # Picking and visibility queries of an editor: a few hundred rays.
        {"name": "trace pick", "kind": "trace", "scene": "mix", "primitives": 4096, "rays": 257,
         "primary": False},
        # Replay of a megapixel's rays against the headline scene.
        {"name": "trace replay 1M", "kind": "trace", "scene": "mix", "primitives": 10000,
         "rays": 1 << 20, "primary": True},
        # The tree of an ordinary scene, for a program that keeps the flattened arrays.
        {"name": "build 10k", "kind": "build", "scene": "mix", "primitives": 10000, "bins": 0},
        # A large scene is loaded and shown: upload, build, first frame.
        {"name": "open cluster 1M", "kind": "open", "scene": "cluster", "primitives": 1000000,
         "width": 480, "height": 270, "spp": 1, "depth": 4},
        # One optimisation step's forward and backward pass over albedos and emissions.
        {"name": "adjoint 4k", "kind": "adjoint", "scene": "mix", "primitives": 4096,
         "width": 512, "height": 512, "spp": 32, "depth": 6},
        # A data set's views: many scenes of uneven sizes in one replayed launch.
        {"name": "batch of 16", "kind": "batch", "scene": "mix", "primitives": 20000, "scenes": 16,
         "depth": 6},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("frame", "frame", "frame", "rows", "trace", "build", "open", "adjoint", "batch"))
    if kind in ("frame", "rows"):
        scene = rng.choice(("plain", "glass", "mix", "mix", "cluster")) if kind == "frame" else "mix"
        n = 4 if scene == "glass" else 64 if scene == "plain" else _log_int(
            rng, 300, 1000000 if scene == "cluster" else 200000)
        depth = rng.randint(2, 24) if scene == "glass" else rng.randint(1, 8)
        spp = _log_int(rng, 1, 64)
        # pixels up to a full HD frame, and no more path segments than the largest listed frame
        most = min(1920 * 1080, (1920 * 1080 * 16 * 8) // (spp * depth))
        pixels = _log_int(rng, min(1500, most), most)
        width = max(8, min(4096, int(math.sqrt(pixels * rng.uniform(0.6, 2.0)))))
        c = {"kind": kind, "scene": scene, "primitives": n, "width": width,
             "height": max(8, pixels // width), "spp": spp, "depth": depth}
        if kind == "rows":
            c["ranks"] = rng.randint(2, 8)
            c["rank"] = rng.randrange(c["ranks"])
        return c
    if kind == "trace":
        return {"kind": kind, "scene": "mix", "primitives": _log_int(rng, 300, 200000),
                "rays": _log_int(rng, 64, 1 << 20), "primary": rng.random() < 0.5}
    if kind == "build":
        return {"kind": kind, "scene": rng.choice(("mix", "cluster")),
                "primitives": _log_int(rng, 64, 300000), "bins": rng.choice((0, 0, 16, 32))}
    if kind == "open":
        return {"kind": kind, "scene": rng.choice(("mix", "cluster")),
                "primitives": _log_int(rng, 300, 1000000), "width": rng.randint(100, 640),
                "height": rng.randint(60, 360), "spp": rng.randint(1, 4), "depth": rng.randint(2, 6)}
    if kind == "adjoint":
        side = _log_int(rng, 48, 512)
        return {"kind": kind, "scene": "mix", "primitives": _log_int(rng, 300, 20000),
                "width": side, "height": max(32, side - rng.randint(0, 16)), "spp": _log_int(rng, 2, 32),
                "depth": rng.randint(2, 6)}
    return {"kind": kind, "scene": "mix", "primitives": _log_int(rng, 2000, 20000),
            "scenes": rng.randint(2, 16), "depth": rng.randint(3, 6)}


# ---------------------------------------------------------------- scenes

def _palette(scene, rng, n, colours):
    rows = np.zeros((colours, 13))
    rows[:, 0:3] = rng.uniform(0.2, 0.9, (colours, 3))
    rows[:, 12] = 1.5
    ids = scene.register_materials(rows)
    return ids if colours == n else ids[rng.integers(0, colours, n)]


def _transforms(rng, centres, base):
    """Object-to-world maps: uniform random rotations, per-axis scales of 0.5 to 2 x base."""
    k = len(centres)
    q = rng.standard_normal((k, 4))
    q /= np.linalg.norm(q, axis=1)[:, None]
    w, x, y, z = q.T
    r = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                  2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                  2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], axis=1)
    t = np.zeros((k, 3, 4))
    t[:, :, :3] = r.reshape(k, 3, 3) * (rng.uniform(0.5, 2.0, (k, 3)) * base[:, None])[:, None, :]
    t[:, :, 3] = centres
    return t


def _mix(seed, n, clustered):
    """n primitives of the 40/30/15/15 mix, a light and a closed room."""
    rng = np.random.default_rng([seed, n, int(clustered)])
    scene = GpuScene(BvhBuildConfig.weighted(leaf_size=4, mode=BvhBuildMode.WEIGHTED_SAH))
    size = 0.1 if clustered else 1.0
    if clustered:
        hubs = rng.uniform(0.0, 1.0, (CLUSTERS, 3))
        centres = np.clip(hubs[rng.integers(0, CLUSTERS, n)] + 0.05 * rng.standard_normal((n, 3)), 0.0, 1.0)
    else:
        centres = rng.uniform(-1.0, 1.0, (n, 3))
    ids = _palette(scene, rng, n, min(n, PALETTE))
    ns, nb = int(round(n * 0.4)), int(round(n * 0.3))
    na = (n - ns - nb) // 2
    a, b, c = ns, ns + nb, ns + nb + na
    radii = rng.uniform(0.01, 0.05, n) * size
    scene.add_spheres(centres[:a], radii[:a], ids[:a])
    if b > a:
        half = 0.5 * size * rng.uniform(0.01, 0.1, (b - a, 3))
        scene.add_boxes(centres[a:b] - half, centres[a:b] + half, ids[a:b])
    if c > b:
        scene.add_transformed_spheres(_transforms(rng, centres[b:c], radii[b:c]), ids[b:c])
    if n > c:
        scene.add_transformed_boxes(_transforms(rng, centres[c:], radii[c:]), ids[c:])
    light = MaterialData.light((10.0, 10.0, 10.0))
    if clustered:
        scene.add_sphere((0.5, 1.3, 0.5), 0.1, light)
        synth.add_room(scene, -0.5, 1.5)
    else:
        scene.add_sphere((0.0, 2.0, 0.0), 0.3, light)
        synth.add_room(scene, -3.0, 3.0)
    return scene


def _scene(name, n, seed):
    """The scene and a camera that looks at it."""
    rng = np.random.default_rng([seed, 77])
    if name == "plain":
        return synth.plain_workload(seed).scene, synth.camera_looking_z((0.0, 0.0, -2.9))
    if name == "glass":
        scene = synth.gi_test_scene()
        return scene, synth.camera_looking_z(tuple(rng.uniform(-0.2, 0.2, 2)) + (-2.6,))
    eye = tuple(rng.uniform(-0.1, 0.1, 2))
    if name == "cluster":
        return _mix(seed, n, True), synth.camera_looking_z((0.5 + eye[0], 0.5 + eye[1], -0.45))
    return _mix(seed, n, False), synth.camera_looking_z((eye[0], eye[1], -2.9))


def _rays(case, camera, seed):
    n = case["rays"]
    if case["primary"]:
        width = max(1, int(math.sqrt(n)))
        return synth.primary_grid(camera, width, -(-n // width))[:n].copy()
    rng = np.random.default_rng([seed, n])
    o = rng.uniform(-2.5, 2.5, (n, 3))
    return np.concatenate([o, rng.uniform(-1.5, 1.5, (n, 3)) - o], axis=1).astype(np.float32)


def _batch_views(case, seed):
    """(primitives, side, spp) of each scene of a batch: counts spread over their logarithm
    from 1,000, frames of three sides and two sample counts."""
    rng = random.Random(case["scenes"] * 1000003 + case["primitives"])
    return [(_log_int(rng, 1000, case["primitives"]), rng.choice(BATCH_SIDES), rng.choice(BATCH_SPP))
            for _ in range(case["scenes"])]


# ---------------------------------------------------------------- cases

def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "batch":
        ctx = Context()
        jobs, outs, keep = [], [], []
        for k, (n, side, spp) in enumerate(_batch_views(case, seed)):
            scene, camera = _scene("mix", n, seed * 100 + k)
            res = ResidentScene.build(ctx, scene)
            out = torch.zeros(side * side * 3, dtype=torch.float32, device="cuda")
            jobs.append((res, camera, side, side, spp, case["depth"], 0, seed * 100 + k, out.data_ptr()))
            outs.append(out)
            keep.append(res)
        torch.cuda.synchronize()
        return dict(st, ctx=ctx, batch=Batch(ctx, jobs), outs=outs, keep=keep)
    scene, camera = _scene(case["scene"], case["primitives"], seed)
    if kind == "frame":
        tracer = GpuRayTracer(case["width"], case["height"], case["spp"])
        tracer.ensure_scene_resident(scene)
        return dict(st, tracer=tracer, scene=scene, camera=camera, seed=seed,
                    image=np.zeros(case["width"] * case["height"] * 3, np.float32))
    if kind == "trace":
        tracer = GpuRayTracer(1, 1, 1)
        tracer.ensure_scene_resident(scene)
        return dict(st, tracer=tracer, scene=scene, rays=_rays(case, camera, seed))
    ctx = Context()
    if kind == "build":
        scene.arrays()  # the packed arrays are the scene as the program holds it
        most = scene.bounded_primitive_count()
        tree = [np.zeros(k, t) for k, t in ((12 * most, np.float32), (8 * most, np.int32), (most, np.int32), (4, np.int32))]
        return dict(st, ctx=ctx, scene=scene, tree=tree)
    params = native.RenderParams(case["width"], case["height"], case["spp"], case["depth"], 0, seed, 1, 0, 0)
    if kind == "open":
        scene.arrays()
        return dict(st, ctx=ctx, scene=scene, camera=camera_struct(camera), params=params,
                    image=np.zeros(case["width"] * case["height"] * 3, np.float32))
    if kind == "rows":
        res = ResidentScene.build(ctx, scene)
        band = torch.zeros(band_rows(case["height"], case["ranks"]) * case["width"] * 3,
                           dtype=torch.float32, device="cuda")
        cam = camera_struct(camera)
        render = device_rows_renderer(ctx, res, cam, params, stream=torch_stream_handle(torch))
        torch.cuda.synchronize()
        return dict(st, ctx=ctx, keep=(res, cam, params), band=band, render=render)
    if kind == "adjoint":
        ds = DifferentiableScene(ctx, scene, case["width"], case["height"], case["spp"], case["depth"],
                                 camera, frame_seed=seed)
        gen = torch.Generator(device="cuda").manual_seed(seed)
        grad = torch.randn(case["width"] * case["height"] * 3, device="cuda", generator=gen)
        albedo = torch.from_numpy(ds.albedo()).cuda().requires_grad_(True)
        emission = torch.from_numpy(ds.emission()).cuda().requires_grad_(True)
        return dict(st, ctx=ctx, ds=ds, function=render_function(), albedo=albedo, emission=emission,
                    grad=grad)
    raise ValueError("unknown kind %r" % (kind,))


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "frame":
        return st["tracer"].render_sample(st["image"], st["scene"], st["camera"], case["depth"], 0, st["seed"])
    if kind == "rows":
        st["render"](case["rank"], case["ranks"], st["band"])
        return st["band"]
    if kind == "trace":
        r = st["tracer"].trace_replay(st["scene"], st["rays"])
        return {"distance": r.hit_distances, "flag": r.hit_flags, "material": r.hit_material_indices,
                "normal": r.hit_normals, "order": r.hit_primitive_orders}
    if kind == "build":
        ctx = st["ctx"]
        bounds, nodes, refs, roots = st["tree"]
        res = ResidentScene.build(ctx, st["scene"], bins=case["bins"])
        ctx.check(ctx.lib.rtb_scene_download_bvh(ctx.handle, res.handle, native.fptr(bounds), native.iptr(nodes),
                                                 native.iptr(refs), native.iptr(roots)))
        res.close()
        return st["tree"]
    if kind == "open":
        ctx = st["ctx"]
        res = ResidentScene.build(ctx, st["scene"])
        ctx.check(ctx.lib.rtb_render_sample(ctx.handle, res.handle, C.byref(st["camera"]),
                                            C.byref(st["params"]), native.fptr(st["image"])))
        res.close()
        return st["image"]
    if kind == "adjoint":
        image = st["function"].apply(st["albedo"], st["emission"], st["ds"])
        ga, ge = torch.autograd.grad(image, (st["albedo"], st["emission"]), st["grad"])
        return {"image": image.detach(), "grad_albedo": ga, "grad_emission": ge}
    st["batch"].render(torch_stream_handle(torch))
    return st["outs"]


def _path_work(samples, depth, n, planes):
    """Operations of `samples` paths of `depth` segments over n primitives: one descent of
    the tree (two slab tests of 18 operations a level), one primitive, the planes, the
    shading."""
    return samples * depth * (36.0 * math.log2(n + 2) + 40.0 + 10.0 * planes + 100.0)


def work(case):
    kind = case["kind"]
    n = case["primitives"]
    planes = 5 if case["scene"] == "glass" else 6
    scene = n * BYTES_PER_PRIMITIVE + min(n, PALETTE) * 52
    if kind == "batch":
        b = f = 0.0
        for m, side, spp in _batch_views(case, 0):
            b += m * BYTES_PER_PRIMITIVE + min(m, PALETTE) * 52 + side * side * 12
            f += _path_work(side * side * spp, case["depth"], m, planes)
        return {"bytes": b, "flops": f}
    if kind == "trace":
        return {"bytes": scene + case["rays"] * (24 + 28), "flops": _path_work(case["rays"], 1, n, planes)}
    if kind == "build":
        # a sort and, on every level, one pass over the primitives' boxes on three axes
        return {"bytes": scene + 2 * n * 44, "flops": n * math.log2(n + 2) * 3 * 30.0}
    pixels = case["width"] * case["height"]
    if kind == "rows":
        pixels = case["width"] * len(range(case["rank"], case["height"], case["ranks"]))
    f = _path_work(pixels * case["spp"], case["depth"], n, planes)
    b = scene + pixels * 12
    if kind == "open":
        f += n * math.log2(n + 2) * 3 * 30.0
    if kind == "adjoint":
        f *= 2.0  # the backward pass traces the paths again
        b += pixels * 12 + min(n, PALETTE) * 48
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------------------- 64-bit values

def _chunk_hits(o, d, scene):
    """Nearest distances of rays o + t d (t > 1e-4) against every record of the scene, in
    64 bits from the packed 32-bit records."""
    eps = 1e-4
    inf = torch.full((1,), math.inf, dtype=torch.float64, device=o.device)
    best = torch.full((len(o),), math.inf, dtype=torch.float64, device=o.device)

    def quadratic(oc, dd, c):
        a = (dd * dd).sum(-1)
        mid = -(oc * dd).sum(-1) / a
        rest = oc + dd * mid[..., None]
        h2 = c - (rest * rest).sum(-1)
        h = torch.sqrt(torch.clamp(h2, min=0.0) / a)
        t = torch.where(mid - h > eps, mid - h, mid + h)
        return torch.where((h2 > 0) & (t > eps), t, inf)

    def slabs(oo, dd, lo, hi):
        a, b = (lo - oo) / dd, (hi - oo) / dd
        near = torch.minimum(a, b).amax(-1)
        far = torch.maximum(a, b).amin(-1)
        t = torch.where(near > eps, near, far)
        return torch.where((near < far) & (t > eps), t, inf)

    def records(data, k):
        return torch.from_numpy(np.asarray(data, np.float64).reshape(-1, k)).to(o.device)

    s = records(scene.sphere_data(), 5)
    if len(s):
        t = quadratic(o[:, None, :] - s[None, :, 0:3], d[:, None, :], s[None, :, 3] ** 2)
        best = torch.minimum(best, t.amin(1))
    x = records(scene.box_data(), 7)
    if len(x):
        t = slabs(o[:, None, :], d[:, None, :], x[None, :, 0:3], x[None, :, 3:6])
        best = torch.minimum(best, t.amin(1))
    for data, box in ((scene.affine_sphere_data(), False), (scene.affine_box_data(), True)):
        x = records(data, 22)
        if not len(x):
            continue
        m = x[:, :12].reshape(-1, 3, 4)
        lo = torch.einsum("kij,rkj->rki", m[:, :, :3], o[:, None, :] - m[None, :, :, 3])
        ld = torch.einsum("kij,rj->rki", m[:, :, :3], d)
        t = slabs(lo, ld, -1.0, 1.0) if box else quadratic(lo, ld, 1.0)
        best = torch.minimum(best, t.amin(1))
    p = records(scene.plane_data(), 26)
    if len(p):
        t = -(o @ p[:, 0:3].T + p[:, 3]) / (d @ p[:, 0:3].T)
        t = torch.where(torch.isfinite(t) & (t > eps), t, inf)
        best = torch.minimum(best, t.amin(1))
    return best


def exact(case, seed):
    """Closest-hit distances in 64 bits, where testing every ray against every primitive is
    quick.  A path's random choices turn on single bits of its hits, so frames and their
    gradients have no value that 64 bits would give, and trees are held as whole numbers."""
    if case["kind"] != "trace" or case["rays"] * case["primitives"] > 2e8:
        return None
    scene, camera = _scene(case["scene"], case["primitives"], seed)
    rays = torch.from_numpy(_rays(case, camera, seed)).double().cuda()
    step = max(1, int(2e7 // case["primitives"]))
    best = torch.cat([_chunk_hits(rays[i:i + step, :3], rays[i:i + step, 3:], scene)
                      for i in range(0, len(rays), step)])
    return {"distance": best.cpu().numpy(), "flag": None, "material": None, "normal": None, "order": None}
