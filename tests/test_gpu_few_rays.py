"""Ray queries and small frames whose rays are spread over few lanes of many warps: counts at
the edges of the rule (one ray a warp on every SM, two, a full warp, one more than each),
against the FP32 restatement (hits) and the wavefront form (frames), in every field."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle
from rtb200 import native as N
from rtb200 import synth
from rtb200.tracer import Context, GpuRayTracer, ResidentScene, camera_struct

pytestmark = pytest.mark.gpu
WARPS = 148 * 8  # warps that take rays before any takes a second


@pytest.mark.parametrize("n", [1, 31, WARPS, WARPS + 1, 2 * WARPS + 1, 31 * WARPS + 1, 32 * WARPS + 1])
def test_spread_rays_equal_the_restatement(n):
    scene = synth.hetero_scene(500, 3, synth.WORKLOAD_IDS["test"], 2)
    rays = synth.random_rays(n, 11)
    bvh = oracle.build_bvh(scene)
    with GpuRayTracer(1, 1, 1) as t:
        got = t.trace_replay(scene, rays, bvh=bvh)
    want = oracle.trace(scene, rays, bvh)
    np.testing.assert_array_equal(got.hit_primitive_orders, want["order"])
    np.testing.assert_array_equal(got.hit_distances.view(np.int32), want["t"].view(np.int32))


@pytest.mark.parametrize("width,height,spp", [(1, 1, 1), (37, 32, 1), (37, 33, 1), (64, 37, 2), (200, 190, 1)])
def test_spread_frames_equal_the_wavefront(width, height, spp):
    torch = pytest.importorskip("torch")
    ctx = Context(0)
    res = ResidentScene.build(ctx, synth.hetero_scene(500, 3, synth.WORKLOAD_IDS["test"], 2))
    try:
        p = N.RenderParams(width, height, spp, 4, 1, 9, 1, 0, 0)
        cam = camera_struct(synth.camera_looking_z((0.0, 0.0, -2.9), width / height))
        out = []
        for fn in (ctx.lib.rtb_render_device, ctx.lib.rtb_render_device_wavefront):
            img = torch.full((width * height * 3,), float("nan"), device="cuda")
            ctx.check(fn(ctx.handle, res.handle, C.byref(cam), C.byref(p), C.c_void_p(img.data_ptr()), None))
            torch.cuda.synchronize()
            out.append(img.cpu().numpy().view(np.int32))
        np.testing.assert_array_equal(*out)
    finally:
        res.close()
        ctx.close()
