"""The counting build of the frame kernel in phases: the same image as without counting, the same
paths as the linear mode counts (segments and plane tests; that mode runs in the other form),
and counts that agree among themselves, with every stack split and with a tree whose rays
overflow their node budget."""
import copy
import ctypes as C

import numpy as np
import pytest

from oracle import oracle
from rtb200 import native as N
from rtb200 import synth
from rtb200.tracer import Context, ResidentScene, camera_struct

pytestmark = pytest.mark.gpu
NAMES = ["rays", "aabb", "prim", "sphere", "box", "plane", "asphere", "abox", "overflow",
         "max_stack", "internal", "leaf", "homogeneous", "mixed"]
WIDTH, HEIGHT = 552, 550  # with two samples twice the two samples per resident thread of the line


def _frame(ctx, res, spp, depth, use_bvh=1, metrics=1, stack=0):
    img = np.full(WIDTH * HEIGHT * 3, np.nan, np.float32)
    p = N.RenderParams(WIDTH, HEIGHT, spp, depth, 2, 77, use_bvh, metrics, stack)
    cam = camera_struct(synth.camera_looking_z((0.05, 0.0, -2.9), WIDTH / HEIGHT))
    ctx.check(ctx.lib.rtb_render_sample(ctx.handle, res.handle, C.byref(cam), C.byref(p), N.fptr(img)))
    st = N.FrameStats()
    ctx.check(ctx.lib.rtb_last_frame_stats(ctx.handle, C.byref(st)))
    return img.view(np.int32), dict(zip(NAMES, st.counters))


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def _consistent(c):
    assert c["prim"] == c["sphere"] + c["box"] + c["plane"] + c["asphere"] + c["abox"], c
    assert c["aabb"] == 2 * c["internal"] and c["leaf"] == c["homogeneous"] + c["mixed"], c


@pytest.mark.parametrize("spp,depth,stack", [(1, 3, 0), (2, 4, -1), (2, 4, 8), (2, 4, 16), (3, 6, 0)])
def test_counts_of_the_phases(ctx, spp, depth, stack):
    scene = synth.hetero_scene(600, 23, synth.WORKLOAD_IDS["test"], 4)
    res = ResidentScene.build(ctx, scene)
    try:
        img, c = _frame(ctx, res, spp, depth, stack=stack)
        plain, none = _frame(ctx, res, spp, depth, metrics=0, stack=stack)
        linear_img, linear = _frame(ctx, res, spp, depth, use_bvh=0)
    finally:
        res.close()
    np.testing.assert_array_equal(img, plain)
    np.testing.assert_array_equal(img, linear_img)
    assert not any(none.values()), none
    _consistent(c)
    for k in ("rays", "plane"):
        assert c[k] == linear[k], (k, c[k], linear[k])
    n = scene.bounded_primitive_count()
    planes = linear["plane"] // linear["rays"]
    assert linear["prim"] == linear["rays"] * (n + planes)
    # every segment visits the top node, and the stack was used
    assert c["rays"] > WIDTH * HEIGHT * spp and c["internal"] > c["rays"] and c["max_stack"] > 1, c
    assert c["overflow"] == 0 and 0 < c["leaf"] <= c["prim"] - c["plane"] < linear["prim"] - linear["plane"], c


def test_counts_of_rays_over_their_node_budget(ctx):
    scene = synth.hetero_scene(300, 23, synth.WORKLOAD_IDS["test"], 4)
    bvh = copy.copy(oracle.build_bvh(scene))
    nd = np.array(bvh.node_data, np.int32)
    deep = [i for i in range(len(nd) // 4) if nd[4 * i] >= 0][-1]
    nd[4 * deep + 1] = 0  # back to the root
    bvh.node_data = nd
    res = ResidentScene.upload(ctx, scene, bvh)
    try:
        img, c = _frame(ctx, res, 2, 3)
        linear_img, linear = _frame(ctx, res, 2, 3, use_bvh=0)
    finally:
        res.close()
    np.testing.assert_array_equal(img, linear_img)
    _consistent(c)
    assert (c["rays"], c["plane"]) == (linear["rays"], linear["plane"]) and 0 < c["overflow"] <= c["rays"], c
