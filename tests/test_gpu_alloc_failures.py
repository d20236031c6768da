"""A device that refuses an allocation: the calls that go on without it (a workspace
without the room to spare, or another path) give the oracle's results, and the error of
the refused allocation is not taken for that of a later launch. The refusals are made
with the test hook vdbg_test_fail_allocs."""
import numpy as np
import pytest

from vdb_mapping_gb300 import VdbgError
from vdb_mapping_gb300.mapping import Config

from test_gpu_changes import FLIPPY, same_changes
from test_gpu_parity import assert_same_map, pair
from test_gpu_sections import same_section

pytestmark = pytest.mark.gpu

BOX = ((-100, -90, -40), (99, 95, 44))


def inserted(vdbg, oracle, track=False):
    g, o = pair(vdbg, oracle, 0.1, Config(max_range=30.0, **FLIPPY))
    if track:
        g.trackChanges(True)
    rng = np.random.default_rng(11)
    for k in range(3):
        pts = (rng.normal(size=(3000, 3)) * [4.0, 4.0, 1.0]).astype(np.float32)
        for m in (g, o):
            m.insertPointCloud(pts, (0.1, 0.2, 0.3), "s")
    return g, o


def refuse(g, skip, count):
    assert g._lib.vdbg_test_fail_allocs(g._h, skip, count) == 0


@pytest.mark.parametrize("skip, count", [(0, 1), (0, 2), (1, 1), (1, 2), (2, 1)])
@pytest.mark.parametrize("full", [False, True])
def test_section(vdbg, oracle, skip, count, full):
    g, o = inserted(vdbg, oracle)
    refuse(g, skip, count)
    same_section(g.getMapSection(*BOX, full=full), o.getMapSection(*BOX, full=full))


@pytest.mark.parametrize("skip, count", [(0, 1), (0, 2), (1, 1)])
def test_section_states_are_applied(vdbg, oracle, skip, count):
    g, o = inserted(vdbg, oracle)
    rng = np.random.default_rng(5)
    so, _, sm = o.getMapSection(*BOX, full=True)
    sm = sm & rng.integers(0, 1 << 63, sm.shape, dtype=np.uint64)
    refuse(g, skip, count)
    try:
        g.applyMapSectionStates(*BOX, so, sm)
        o.applyMapSectionStates(*BOX, so, sm)
    except VdbgError as e:  # without room for the section nothing of it is applied
        assert "OUT_OF_MEMORY" in str(e) and count > 1
    refuse(g, 0, 0)
    assert_same_map(g.exportLeaves(), o.exportLeaves(), "states")


@pytest.mark.parametrize("count", [1, 2])
def test_morphology(vdbg, oracle, count):
    g, o = inserted(vdbg, oracle)
    so, _, sm = o.getMapSection(*BOX)
    refuse(g, 0, count)
    for a, b in zip(g.sectionMorphology(so, sm, "close", 2), oracle.morphology(so, sm, "close", 2)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("count", [1, 2])
def test_change_set(vdbg, oracle, count):
    g, o = inserted(vdbg, oracle, track=True)
    refuse(g, 0, count)
    same_changes(g.exportChanges(), o.exportChanges(), "changes")


def test_the_next_call(vdbg, oracle):
    """A call that fails for want of memory leaves nothing for the next one to trip over."""
    g, o = inserted(vdbg, oracle)
    pts = np.full((200000, 3), 1.0, np.float32)
    refuse(g, 0, 1)
    with pytest.raises(VdbgError) as e:
        g.insertPointCloud(pts, (0.1, 0.2, 0.3), "s")
    assert "OUT_OF_MEMORY" in str(e.value)
    for m in (g, o):
        m.insertPointCloud(pts, (0.1, 0.2, 0.3), "s")
    assert_same_map(g.exportLeaves(), o.exportLeaves(), "after a refused call")


@pytest.mark.parametrize("skip", [0, 1, 2])
def test_bytes_after_a_refused_insert(vdbg, skip):
    """device bytes count what a refused call gave back."""
    pts = np.full((200000, 3), 1.0, np.float32)
    held = []
    for refused in (False, True):
        g = vdbg.OccupancyVDBMapping(0.1)
        g.setConfig(Config(max_range=30.0, **FLIPPY))
        g.addInputSource("s", 30.0, 0)
        if refused:
            refuse(g, skip, 1)
            with pytest.raises(VdbgError):
                g.insertPointCloud(pts, (0.1, 0.2, 0.3), "s")
        g.insertPointCloud(pts, (0.1, 0.2, 0.3), "s")
        held.append(g.deviceBytes())
    assert held[0] == held[1]


@pytest.mark.parametrize("skip", range(12))
def test_bytes_after_a_refused_morphology(vdbg, oracle, skip):
    """Leaves too far apart for one grid: the hashed sets, one allocation of which is
    refused (the others go back, at their size)."""
    g, _ = inserted(vdbg, oracle)
    so = np.array([[0, 0, 0], [8 * 900, 8 * 900, 8 * 900]], np.int32)
    sm = np.full((2, 8), 0x00FF00FF00FF00FF, np.uint64)
    held = g.deviceBytes()
    refuse(g, skip, 1)
    with pytest.raises(VdbgError) as e:
        g.sectionMorphology(so, sm, "close", 2)
    assert "OUT_OF_MEMORY" in str(e.value)
    assert g.deviceBytes() == held
    for a, b in zip(g.sectionMorphology(so, sm, "close", 2), oracle.morphology(so, sm, "close", 2)):
        assert np.array_equal(a, b)
    assert g.deviceBytes() == held
