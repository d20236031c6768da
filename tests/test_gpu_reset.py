"""resetMap clears what the map used: a map filled, reset and filled differently
(through pool growth, after a section's values, in fast mode's order) equals one
that was never used."""
import numpy as np
import pytest

from test_gpu_parity import assert_same_map, pair, ref_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("initial_leaf_capacity", [64, 65536])
def test_reset_leaves_nothing(vdbg, oracle, initial_leaf_capacity):
    rng = np.random.default_rng(initial_leaf_capacity)
    g, o = pair(vdbg, oracle, 0.1, ref_config(max_range=30.0),
                initial_leaf_capacity=initial_leaf_capacity)
    for k, n in enumerate((3000, 200, 6000)):
        g.resetMap()
        o.resetMap()
        assert g.leafCount() == 0
        for _ in range(2):
            pts = (rng.normal(size=(n, 3)) * [8.0, 8.0, 1.0] + 3.0 * k).astype(np.float32)
            for m in (g, o):
                m.insertPointCloud(pts, (0.1 * k, 0.2, 0.3), "s")
        assert_same_map(g.exportLeaves(), o.exportLeaves(), f"fill {k}")
        so, sv, sm = o.getMapSection((-40, -40, -40), (40, 40, 40), full=True)
        far = (so + np.int32(4096)).astype(np.int32)
        for m in (g, o):
            m.applyMapSectionValues(far, sv, sm)
        assert_same_map(g.exportLeaves(), o.exportLeaves(), f"values {k}")
