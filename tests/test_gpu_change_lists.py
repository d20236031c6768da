"""Change sets of every length class: ordered on the device in the first go, after
asking for more room, and on the host; per map of a batch; after an accumulated
window (closed by its sweep). Equal to the oracle's."""
import numpy as np
import pytest

from vdb_mapping_gb300.mapping import Config

from test_gpu_changes import FLIPPY, same_changes

pytestmark = pytest.mark.gpu


def clouds(n, seed):
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3))
    return (40.0 * d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)


@pytest.mark.parametrize("n, least, most", [(1, 1, 300), (20, 300, 2048), (80, 2049, 16384), (700, 16385, 1 << 20)])
def test_change_list_lengths(vdbg, oracle, n, least, most):
    cfg = Config(max_range=100.0, **FLIPPY)
    g = vdbg.OccupancyVDBMapping(0.1)
    g.trackChanges(True)
    o = oracle.OracleMap(0.1)
    for m in (g, o):
        m.setConfig(cfg)
        m.addInputSource("s", 100.0, 0)
    pts = clouds(n, n)
    # every voxel of the leaves the rays cross active at value 0, so that their
    # misses turn them off
    path = oracle.OracleMap(0.1)
    path.setConfig(cfg)
    path.addInputSource("s", 100.0, 0)
    path.insertPointCloud(pts, (0.05, 0.05, 0.05), "s")
    lo, hi = np.array([-410, -410, -410]), np.array([410, 410, 410])
    so, _, sm = path.getMapSection(lo, hi, full=True)
    for m in (g, o):
        m.applyMapSectionStates(lo, hi, so, np.full_like(sm, ~np.uint64(0)))
        m.accumulateUpdate(pts, (0.05, 0.05, 0.05), "s")
        m.accumulateUpdate(clouds(3, 5), (0.05, 0.05, 0.05), "s")
        m.integrateUpdate()
    gc = g.exportChanges()
    assert least <= len(gc[0]) <= most, len(gc[0])
    same_changes(gc, o.exportChanges(), f"{n} rays")


def test_change_lists_of_a_batch(vdbg, oracle):
    cfg = Config(max_range=100.0, **FLIPPY)
    b = vdbg.MapBatch([0.1, 0.1, 0.2])
    b.trackChanges(True)
    o = [oracle.OracleMap(r) for r in (0.1, 0.1, 0.2)]
    for i, m in enumerate(o):
        b.setConfig(i, cfg)
        m.setConfig(cfg)
        m.addInputSource("s", 100.0, 0)
    parts = [clouds(50 + i, i) for i in range(3)]
    b.insert(parts, [(0.05, 0.05, 0.05)] * 3)
    for i, m in enumerate(o):
        m.insertPointCloud(parts[i], (0.05, 0.05, 0.05), "s")
        same_changes(b.exportChanges(i), m.exportChanges(), f"map {i}")
