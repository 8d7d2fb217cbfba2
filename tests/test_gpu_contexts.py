"""A context's buffers across its streams, its life and other contexts: they grow from a frame on one
stream to a larger one on another and to a replay, a context ends while its frame still runs on
a caller's stream, and two contexts build, trace and render in two threads at once; every result
equals that of a context that did nothing else."""
import ctypes as C
import threading

import numpy as np
import pytest

from rtb200 import native as N
from rtb200 import synth
from rtb200.tracer import Context, GpuRayTracer, ResidentScene, camera_struct

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
SMALL, MIDDLE, LARGE = (64, 36, 1), (640, 500, 2), (1280, 710, 3)  # the last two run in phases


def _scene():
    return synth.hetero_scene(600, 23, synth.WORKLOAD_IDS["test"], 4)


def _render(ctx, res, size, stream):
    w, h, spp = size
    with torch.cuda.stream(stream):
        img = torch.full((w * h * 3,), float("nan"), device="cuda")
    p = N.RenderParams(w, h, spp, 4, 2, 77, 1, 0, 0)
    cam = camera_struct(synth.camera_looking_z((0.05, 0.0, -2.9), w / h))
    ctx.check(ctx.lib.rtb_render_device(ctx.handle, res.handle, C.byref(cam), C.byref(p), C.c_void_p(img.data_ptr()),
                                        C.c_void_p(stream.cuda_stream)))
    return img


def _replay(ctx, res, size, materials, stream):
    w, h, spp = size
    with torch.cuda.stream(stream):
        adj = torch.ones(w * h * 3, device="cuda")
        grads = [torch.empty(3 * materials, device="cuda") for _ in range(2)]
    p = N.RenderParams(w, h, spp, 4, 2, 77, 1, 0, 0)
    cam = camera_struct(synth.camera_looking_z((0.05, 0.0, -2.9), w / h))
    ctx.check(ctx.lib.rtb_render_backward(ctx.handle, res.handle, C.byref(cam), C.byref(p), C.c_void_p(adj.data_ptr()),
                                          C.c_void_p(grads[0].data_ptr()), C.c_void_p(grads[1].data_ptr()),
                                          C.c_void_p(stream.cuda_stream)))
    return [adj] + grads


@pytest.fixture(scope="module")
def alone():
    """Each result by a context of its own."""
    scene = _scene()
    out = {}
    for size in (SMALL, MIDDLE, LARGE):
        ctx = Context(0)
        res = ResidentScene.build(ctx, scene)
        img = _render(ctx, res, size, torch.cuda.current_stream())
        torch.cuda.synchronize()
        out[size] = img.cpu().numpy().view(np.int32)
        res.close()
        ctx.close()
    return out


def test_buffers_grow_across_streams(alone):
    scene = _scene()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    ctx = Context(0)
    try:
        res = ResidentScene.build(ctx, scene)
        m = scene.material_count()
        jobs = [(SMALL, a), (MIDDLE, b), (LARGE, a), (MIDDLE, b)]
        images = [(s, _render(ctx, res, s, st)) for s, st in jobs]
        first = _replay(ctx, res, MIDDLE, m, b)
        images.append((LARGE, _render(ctx, res, LARGE, a)))
        second = _replay(ctx, res, MIDDLE, m, a)
        images.append((MIDDLE, _render(ctx, res, MIDDLE, b)))
        torch.cuda.synchronize()
        for size, img in images:
            np.testing.assert_array_equal(img.cpu().numpy().view(np.int32), alone[size])
        # the same terms added in another order: 640,000 samples, a few thousand to a material
        for x, y in zip(first[1:], second[1:]):
            np.testing.assert_allclose(x.cpu().numpy(), y.cpu().numpy(), rtol=1e-4, atol=1e-4 * float(x.abs().max()))
        res.close()
    finally:
        ctx.close()


def test_a_context_ends_while_its_frame_runs(alone):
    stream = torch.cuda.Stream()
    scene = _scene()
    for _ in range(3):
        ctx = Context(0)
        res = ResidentScene.build(ctx, scene)
        images = [_render(ctx, res, LARGE, stream) for _ in range(4)]
        res.close()
        ctx.close()
        stream.synchronize()
        for img in images:
            np.testing.assert_array_equal(img.cpu().numpy().view(np.int32), alone[LARGE])


def test_two_contexts_in_two_threads(alone):
    rays = synth.random_rays(700, 5)
    hits, errors = {}, []

    def work(k):
        try:
            stream = torch.cuda.Stream()
            scene = _scene()
            for i in range(3):
                ctx = Context(0)
                res = ResidentScene.build(ctx, scene)
                img = [(s, _render(ctx, res, s, stream)) for s in ((MIDDLE, LARGE) if k else (LARGE, SMALL))]
                stream.synchronize()
                for size, x in img:
                    np.testing.assert_array_equal(x.cpu().numpy().view(np.int32), alone[size])
                res.close()
                ctx.close()
                with GpuRayTracer(64, 36, 1) as t:
                    hits[k, i] = t.trace_replay(scene, rays).hit_distances.view(np.int32).copy()
                    hits[k, i, "image"] = np.array(t.render_sample(None, scene, synth.camera_looking_z((0.0, 0.0, -2.9)),
                                                                   4, 0, 7))
        except BaseException as e:  # noqa: BLE001 -- reported by the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for i in range(3):
        for k in range(2):
            np.testing.assert_array_equal(hits[k, i], hits[0, 0])
            np.testing.assert_array_equal(hits[k, i, "image"], hits[0, 0, "image"])
