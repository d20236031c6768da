"""Map sections over boxes that are large for the leaves in them: the box's cells are
looked up, or the map's leaves listed, whichever is less, and states are applied
without the order that only a read needs. Equal to the oracle around the rule's
lines, and a large box takes no multiple of a small one's time."""
import time

import numpy as np
import pytest

from test_gpu_parity import assert_same_map, pair, ref_config
from test_gpu_sections import same_section

pytestmark = pytest.mark.gpu


def blob(vdbg, oracle, n, spread, res=0.1):
    g, o = pair(vdbg, oracle, res, ref_config(max_range=60.0)) if oracle else (None, None)
    if g is None:
        g = vdbg.OccupancyVDBMapping(res)
        g.setConfig(ref_config(max_range=60.0))
        g.addInputSource("s", 60.0, 0)
    rng = np.random.default_rng(n)
    pts = (rng.normal(size=(n, 3)) * spread).astype(np.float32)
    for m in (g, o):
        if m is not None:
            m.insertPointCloud(pts, (0.1, 0.2, 0.3), "s")
    return g, o


def box(cells, at=(0, 0, 0)):
    lo = 8 * (np.array(at) - np.array(cells) // 2)
    return lo, lo + 8 * np.array(cells) - 1


def best(f, n=7):
    t = []
    for _ in range(n):
        t0 = time.perf_counter()
        f()
        t.append(time.perf_counter() - t0)
    return min(t[1:])


@pytest.mark.parametrize("n, spread", [(40, (0.5, 0.5, 0.3)), (3000, (3.0, 3.0, 1.0)), (20000, (12.0, 12.0, 4.0))])
def test_reads_and_states(vdbg, oracle, n, spread):
    g, o = blob(vdbg, oracle, n, spread)
    rng = np.random.default_rng(7)
    for cells in ((32, 32, 25), (30, 30, 30), (64, 32, 32), (65, 32, 32), (100, 100, 40), (128, 128, 64), (110, 110, 90)):
        for at in ((0, 0, 0), (-60, 20, 0), (3000, 3000, 3000)):
            lo, hi = box(cells, at)
            for full in (False, True):
                same_section(g.getMapSection(lo + 3, hi - 2, full), o.getMapSection(lo + 3, hi - 2, full),
                             f"{cells} {at} {full}")
        lo, hi = box(cells, (5, 0, 0))
        so, _, sm = o.getMapSection(lo, hi, full=True)
        sm = sm & rng.integers(0, 1 << 63, sm.shape, dtype=np.uint64)
        for m in (g, o):
            m.applyMapSectionStates(lo + 5, hi - 6, so, sm)
        assert_same_map(g.exportLeaves(), o.exportLeaves(), f"states {cells}")


def test_time_of_states_over_a_large_box(vdbg):
    g, _ = blob(vdbg, None, 60000, (9.0, 9.0, 3.0), 0.05)
    empty = np.zeros((0, 3), np.int32), np.zeros((0, 8), np.uint64)
    small = best(lambda: g.applyMapSectionStates(*box((60, 60, 60)), *empty))
    large = best(lambda: g.applyMapSectionStates(*box((160, 160, 160)), *empty))
    assert large < 20.0 * small, (small, large)


@pytest.mark.parametrize("cells", [(40, 40, 20), (64, 64, 64), (100, 100, 100)])
def test_time_of_reads_with_few_leaves(vdbg, cells):
    g, _ = blob(vdbg, None, 300, (1.0, 1.0, 0.4))
    for at in ((0, 0, 0), (3000, 3000, 3000)):
        small = best(lambda: g.getMapSection(*box((8, 8, 8), at), full=True))
        large = best(lambda: g.getMapSection(*box(cells, at), full=True))
        assert large < 10.0 * small, (at, small, large)
