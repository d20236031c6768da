"""Sections of a box with far more cells than the map has leaves, under a budget that
holds the map's leaves but not a table of the box's cells: read, and written back, as
without a budget."""
import numpy as np
import pytest

from test_gpu_parity import assert_same_map, pair, ref_config
from test_gpu_sections import same_section

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells, room", [((128, 128, 64), 4 << 20), ((64, 64, 64), 2 << 20), ((32, 32, 25), 160 << 10)])
def test_more_cells_than_room(vdbg, oracle, cells, room):
    rng = np.random.default_rng(3)
    pts = (rng.normal(size=(60, 3)) * [0.6, 0.6, 0.3]).astype(np.float32)
    held = None
    for budget in (0, 1):
        g, o = pair(vdbg, oracle, 0.1, ref_config(max_range=8.0), max_device_bytes=held + room if budget else 0)
        for m in (g, o):
            m.insertPointCloud(pts, (0.1, 0.2, 0.3), "s")
        lo = -8 * (np.array(cells) // 2)
        hi = lo + 8 * np.array(cells) - 1
        if not budget:
            held = g.deviceBytes()
        for full in (False, True):
            same_section(g.getMapSection(lo, hi, full), o.getMapSection(lo, hi, full), f"{cells} {full}")
        so, _, sm = o.getMapSection(lo, hi, full=True)
        for m in (g, o):
            m.applyMapSectionStates(lo + 9, hi, so, sm & np.uint64(0x5555555555555555))
        assert_same_map(g.exportLeaves(), o.exportLeaves(), "states")
        assert not budget or g.deviceBytes() <= held + room
        g.close()
