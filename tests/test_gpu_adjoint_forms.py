"""The adjoint kernel's two forms against each other: frames above the line of the two-phase
form, and the same frames with the tree off, which one path a lane replays (the closest hits
and so the paths are the same).  With an all-positive image adjoint every added term is
positive, so a sum of n terms in FP32 is off by at most n 2^-24 relatively whatever its order;
the longest here, a wall's, adds at most some 2,000 terms (a block's share of the hits in its
shared table, then the blocks): 1.2e-4 for each form, 2.5e-4 between the two."""

import numpy as np
import pytest

from rtb200 import native as N
from rtb200 import synth
from rtb200.diff import DifferentiableScene
from rtb200.tracer import Context

pytestmark = pytest.mark.gpu


# 2 samples per resident thread of 148 SMs are 303,104
@pytest.mark.parametrize("width,height,spp,depth", [(552, 550, 1, 3), (69, 69, 64, 4), (333, 457, 2, 1), (333, 457, 2, 3),
                                                    (318, 318, 3, 32)])
def test_adjoint_forms_agree(width, height, spp, depth):
    torch = pytest.importorskip("torch")
    ctx = Context(0)
    scene = synth.hetero_scene(600, 41, synth.WORKLOAD_IDS["test"], 30)
    ds = DifferentiableScene(ctx, scene, width, height, spp, depth,
                             synth.camera_looking_z((0.0, 0.0, -2.9), width / height), frame_seed=5)
    try:
        gen = torch.Generator(device="cuda").manual_seed(3)
        adj = torch.rand(width * height * 3, device="cuda", generator=gen) + 0.5
        grads = []
        for use_bvh in (1, 0):
            ds.params = N.RenderParams(width, height, spp, depth, 0, 5, use_bvh, 0, 0)
            ga = torch.full((ds.count * 3,), float("nan"), device="cuda")
            ge = torch.full((ds.count * 3,), float("nan"), device="cuda")
            torch.cuda.synchronize()
            ds.backward_into(adj.data_ptr(), ga.data_ptr(), ge.data_ptr())
            torch.cuda.synchronize()
            grads.append((ga.cpu().numpy(), ge.cpu().numpy()))
        for got, want in zip(*grads):
            assert np.isfinite(got).all() and (depth == 1 or got.max() > 0.0)
            np.testing.assert_allclose(got, want, rtol=2.5e-4, atol=0.0)
    finally:
        ds.close()
        ctx.close()
