"""Device builds at the limits of their numbers: weights whose sums overflow a double, so that a
node's split costs are infinite or NaN.  No split is cheaper than that: the node becomes a leaf
of all its primitives, by a warp, by a block and in the level loop."""
import numpy as np
import pytest

from oracle import oracle
from rtb200 import synth
from rtb200.scene import BvhBuildConfig, BvhBuildMode
from rtb200.tracer import Context, ResidentScene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n", [20, 40, 600, 3000])
def test_weights_whose_sums_overflow_give_one_leaf(ctx, n):
    scene = synth.hetero_scene(n, 7, synth.WORKLOAD_IDS["test"], 1)
    cfg = BvhBuildConfig(BvhBuildMode.WEIGHTED_SAH, 4, 1.0, 1e308, 1e308, 1e308, 1e308, 1.0)
    total = scene.bounded_primitive_count()
    want = oracle.build_bvh(scene)  # the root's bounds and the references of any tree
    res = ResidentScene.build(ctx, scene, cfg)
    try:
        nb, nd, refs, roots = res.download_bvh()
        np.testing.assert_array_equal(np.asarray(nd).reshape(-1, 4)[:, 1:], [[-1, 0, total]])
        np.testing.assert_array_equal(np.asarray(nb).reshape(-1), np.asarray(want.node_bounds).reshape(-1)[:6])
        np.testing.assert_array_equal(np.sort(refs), np.sort(want.refs))
        assert list(roots) == [0] and res.stats.leaf_count == 1
    finally:
        res.close()
