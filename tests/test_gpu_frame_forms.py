"""The two forms of the frame kernel -- phases over path slots in memory, one path a lane -- and
the line between them, against the wavefront form (its own launches and order of work): the
same frames bit for bit just below and above the line, with one sample a pixel, with whole
pixels beside single samples, with every stack split, and with a tree whose rays overflow
their node budget (every primitive is tested for them then)."""
import copy
import ctypes as C

import numpy as np
import pytest

from oracle import oracle
from rtb200 import native as N
from rtb200 import synth
from rtb200.tracer import Context, ResidentScene, camera_struct

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def _scene(n):
    return synth.hetero_scene(n, 23, synth.WORKLOAD_IDS["test"], 4)


def _frame(ctx, fn, res, width, height, spp, depth, use_bvh=1, stack=0):
    torch = pytest.importorskip("torch")
    img = torch.full((width * height * 3,), float("nan"), device="cuda")
    p = N.RenderParams(width, height, spp, depth, 2, 77, use_bvh, 0, stack)
    cam = camera_struct(synth.camera_looking_z((0.05, 0.0, -2.9), width / height))
    ctx.check(fn(ctx.handle, res.handle, C.byref(cam), C.byref(p), C.c_void_p(img.data_ptr()), None))
    torch.cuda.synchronize()
    return img.cpu().numpy().view(np.int32)


# 2 samples per resident thread of 148 SMs are 303,104
@pytest.mark.parametrize("n,width,height,spp,depth,stack", [
    (600, 551, 550, 1, 3, 0), (600, 552, 550, 1, 3, 0), (600, 317, 319, 3, 5, 8), (600, 318, 318, 3, 5, 16),
    (600, 69, 69, 64, 4, -1), (600, 1024, 601, 2, 2, 0), (600, 1024, 601, 2, 3, 0), (5000, 333, 457, 2, 32, 0), (40, 552, 550, 1, 3, 0),
    (600, 552, 550, 2, 0, 0)])
def test_frame_forms_equal_the_wavefront(ctx, n, width, height, spp, depth, stack):
    res = ResidentScene.build(ctx, _scene(n))
    try:
        got = _frame(ctx, ctx.lib.rtb_render_device, res, width, height, spp, depth, stack=stack)
        want = _frame(ctx, ctx.lib.rtb_render_device_wavefront, res, width, height, spp, depth)
        np.testing.assert_array_equal(got, want)
    finally:
        res.close()


@pytest.mark.parametrize("width,height", [(40, 30), (640, 480)])
def test_rays_over_their_node_budget_test_every_primitive(ctx, width, height):
    scene = _scene(300)
    bvh = copy.copy(oracle.build_bvh(scene))
    nd = np.array(bvh.node_data, np.int32)
    deep = [i for i in range(len(nd) // 4) if nd[4 * i] >= 0][-1]
    nd[4 * deep + 1] = 0  # back to the root
    bvh.node_data = nd
    res = ResidentScene.upload(ctx, scene, bvh)
    try:
        got = _frame(ctx, ctx.lib.rtb_render_device, res, width, height, 1, 3)
        want = _frame(ctx, ctx.lib.rtb_render_device, res, width, height, 1, 3, use_bvh=0)
        np.testing.assert_array_equal(got, want)
    finally:
        res.close()
