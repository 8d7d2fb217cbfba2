"""An abort stops a frame at a small fraction of its time, on the frame kernel in phases: also
the first frame of a context, whose buffers and code are not there yet, and a replay's.  The
unaborted time is taken from frames of fewer samples on the same device, so that the bound
follows the kernel's speed."""
import ctypes as C
import threading
import time

import numpy as np
import pytest

from oracle import oracle
from rtb200 import native as N
from rtb200 import synth
from rtb200.tracer import Context, ResidentScene, camera_struct

pytestmark = pytest.mark.gpu
SPP = 2048  # some six seconds at 1024 x 1024, a replay nine


def _params(w, spp, frame):
    return N.RenderParams(w.width, w.height, spp, w.max_depth, frame, w.frame_seed & 0xFFFFFFFFFFFFFFFF, 1, 0, 0)


def _frame(ctx, res, w, spp, frame=1):
    img = np.full(w.width * w.height * 3, np.nan, np.float32)
    cam = camera_struct(w.camera)
    t = time.perf_counter()
    st = ctx.lib.rtb_render_sample(ctx.handle, res.handle, C.byref(cam), C.byref(_params(w, spp, frame)), N.fptr(img))
    return st, time.perf_counter() - t


def _backward(ctx, res, w, spp):
    pixels = w.width * w.height
    adj = np.ones(3 * pixels, np.float32)
    grads = [np.zeros(3 * w.scene.material_count(), np.float32) for _ in range(2)]
    cam = camera_struct(w.camera)
    t = time.perf_counter()
    st = ctx.lib.rtb_render_backward_sample(ctx.handle, res.handle, C.byref(cam), C.byref(_params(w, spp, 1)),
                                            N.fptr(adj), N.fptr(grads[0]), N.fptr(grads[1]))
    return st, time.perf_counter() - t


def _aborted(ctx, call):
    timer = threading.Timer(0.2, lambda: ctx.lib.rtb_request_abort(ctx.handle))
    timer.start()
    st, elapsed = call()
    timer.join()
    assert st == 7, N.STATUS_NAMES.get(st, st)  # RTB_ERR_WATCHDOG
    return elapsed


@pytest.fixture(scope="module")
def workload():
    w = synth.hetero_workload()
    return w, oracle.build_bvh(w.scene)


@pytest.mark.parametrize("first", [True, False])
@pytest.mark.parametrize("call", [_frame, _backward])
def test_abort_stops_early(workload, first, call):
    w, bvh = workload
    ctx = Context(0)
    try:
        res = ResidentScene.upload(ctx, w.scene, bvh)
        if not first:
            assert call(ctx, res, w, 1)[0] == N.RTB_OK
        elapsed = _aborted(ctx, lambda: call(ctx, res, w, SPP))
        # the whole frame's time by the samples of a shorter one
        assert call(ctx, res, w, 32)[0] == N.RTB_OK
        whole = call(ctx, res, w, 64)[1] * (SPP / 64)
        print("%s first %d: %.3f s of %.2f s" % (call.__name__, first, elapsed, whole))
        assert whole > 2.0 and elapsed < 0.35 * whole, (elapsed, whole)
        res.close()
    finally:
        ctx.close()
