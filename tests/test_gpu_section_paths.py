"""getMapSection on both sides of the sizes where its path changes: a box of at most
2^15 leaf cells (written at once), of at most 2^20 (counted first), larger (listed),
full and active only, with the box's faces inside leaves. Equal to the oracle."""
import numpy as np
import pytest

from test_gpu_parity import assert_same_map, pair, ref_config
from test_gpu_sections import built_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(1, 1, 1), (32, 32, 31), (32, 32, 32), (33, 32, 32), (128, 128, 64), (129, 128, 64)])
def test_box_sizes(vdbg, oracle, cells):
    g, o = built_pair(vdbg, oracle)
    for shift in (0, 3):
        lo = np.array([-8 * (c // 2) + shift for c in cells])
        hi = lo + 8 * np.array(cells) - 1 - 2 * shift
        for full in (False, True):
            assert_same_map(g.getMapSection(lo, hi, full=full), o.getMapSection(lo, hi, full=full), f"{cells} {full}")


def test_under_a_budget(vdbg, oracle):
    """A budget that the map fits, and not much more: sections, change sets and
    morphology take what they need, and keep none of it from the pools."""
    g, o = pair(vdbg, oracle, 0.1, ref_config(max_range=8.0), max_device_bytes=192 << 20)
    g.trackChanges(True)
    rng = np.random.default_rng(3)
    pts = (rng.normal(size=(4000, 3)) * [3.0, 3.0, 0.5]).astype(np.float32)
    for k in range(3):
        for m in (g, o):
            m.insertPointCloud(pts + np.float32(0.3 * k), (0.1, 0.2, 0.3), "s")
        held = g.deviceBytes()
        for a, b in zip(g.exportChanges(), o.exportChanges()):
            assert np.array_equal(a, b)
        lo, hi = (-127, -127, -127), (127, 127, 127)
        assert_same_map(g.getMapSection(lo, hi, full=True), o.getMapSection(lo, hi, full=True), "section")
        so, _, sm = o.getMapSection(lo, hi)
        for a, b in zip(g.sectionMorphology(so, sm, "close", 2), o_morphology(oracle, so, sm)):
            assert np.array_equal(a, b)
        assert g.deviceBytes() == held
    assert_same_map(g.exportLeaves(), o.exportLeaves(), "map")


def o_morphology(oracle, origins, masks):
    return oracle.morphology(origins, masks, "close", 2)
