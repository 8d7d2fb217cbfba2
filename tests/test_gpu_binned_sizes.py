"""Binned device trees at the sizes where the builder hands a node on: from blocks over chunks of
2,048 positions to one block a node, from a block to a warp (128 primitives), from that to a warp
of its own (32), leaf sizes beside and across them, and coincident centroids at each; node for
node against the oracle's restatement."""
import numpy as np
import pytest

from oracle import oracle
from rtb200 import synth
from rtb200.scene import BvhBuildConfig, BvhBuildMode, GpuScene, MaterialData
from rtb200.tracer import Context, ResidentScene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = Context(0)
    yield c
    c.close()


def _same_tree(ctx, scene, cfg, bins):
    want = oracle.build_bvh(scene, cfg, bins=bins)
    res = ResidentScene.build(ctx, scene, cfg, bins=bins)
    try:
        nb, nd, refs, roots = res.download_bvh()
        np.testing.assert_array_equal(nb.view(np.int32), want.node_bounds.view(np.int32))
        np.testing.assert_array_equal(nd, want.node_data)
        np.testing.assert_array_equal(refs, want.refs)
        np.testing.assert_array_equal(roots, want.roots)
        st = res.stats
        assert (st.node_count, st.leaf_count, st.max_depth, st.min_leaf_occupancy, st.max_leaf_occupancy) == \
            (want.node_count, want.leaf_count, want.max_depth, want.min_leaf, want.max_leaf)
    finally:
        res.close()


@pytest.mark.parametrize("mode", [BvhBuildMode.WEIGHTED_SAH, BvhBuildMode.PER_TYPE_SAH])
@pytest.mark.parametrize("bins,leaf", [(2, 1), (17, 4), (32, 40), (32, 200)])
@pytest.mark.parametrize("n", [1, 31, 32, 127, 128, 129, 2047, 2048, 4099, 9000])
def test_binned_trees_at_the_hand_over_sizes(ctx, mode, bins, leaf, n):
    scene = synth.hetero_scene(n, 300 + n, synth.WORKLOAD_IDS["test"], 1)
    cfg = BvhBuildConfig.weighted(leaf_size=leaf, mode=mode) if mode.uses_primitive_weights() \
        else BvhBuildConfig(mode, leaf)
    _same_tree(ctx, scene, cfg, bins)


@pytest.mark.parametrize("n", [2, 128, 129, 2500])
def test_coincident_primitives_split_in_halves(ctx, n):
    m = MaterialData.matte((0.5, 0.5, 0.5))
    scene = GpuScene(BvhBuildConfig(BvhBuildMode.UNIFORM_SAH, 2))
    for _ in range(n):
        scene.add_sphere((0.25, -0.5, 1.0), 0.3, m)
    _same_tree(ctx, scene, scene.config, 8)
