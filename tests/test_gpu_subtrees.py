"""Device trees at the sizes where the builder hands a node on: from the level loop to a block
(512 primitives), from the block to a warp (32), from a warp's 32 lanes an axis to eight (8), and
leaf sizes beside and across them; node for node against the oracle's restatement of the Java
builder, with unit, calibrated and undyadic weights and per-type forests."""
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


@pytest.mark.parametrize("mode", [BvhBuildMode.UNIFORM_SAH, BvhBuildMode.WEIGHTED_SAH,
                                  BvhBuildMode.PER_TYPE_WEIGHTED_SAH])
@pytest.mark.parametrize("leaf", [1, 4, 9, 40])
@pytest.mark.parametrize("n", [1, 7, 8, 31, 32, 33, 511, 512, 1100])
def test_trees_at_the_hand_over_sizes(ctx, mode, leaf, n):
    # hetero_scene adds a light to its primitives
    scene = synth.hetero_scene(n, 100 + n, synth.WORKLOAD_IDS["test"], 1)
    cfg = BvhBuildConfig.weighted(leaf_size=leaf, mode=mode, lam=0.7) if mode != BvhBuildMode.UNIFORM_SAH \
        else BvhBuildConfig(mode, leaf)
    want = oracle.build_bvh(scene, cfg)
    res = ResidentScene.build(ctx, scene, cfg)
    try:
        nb, nd, refs, roots = res.download_bvh()
        np.testing.assert_array_equal(nb.view(np.int32), want.node_bounds.view(np.int32))
        np.testing.assert_array_equal(nd, want.node_data)
        np.testing.assert_array_equal(refs, want.refs)
        np.testing.assert_array_equal(roots, want.roots)
        st = res.stats
        assert (st.node_count, st.leaf_count, st.max_depth, st.min_leaf_occupancy, st.max_leaf_occupancy) == \
            (want.node_count, want.leaf_count, want.max_depth, want.min_leaf, want.max_leaf)
        assert (st.uniform_sah_cost, st.weighted_sah_cost, st.generalized_sah_cost) == \
            (want.uniform_sah, want.weighted_sah, want.generalized_sah)
    finally:
        res.close()
