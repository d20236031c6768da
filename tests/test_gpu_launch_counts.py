"""timings()["launches"]: the kernels that a call launches, counted one by one.
Insertion: prep, scan of the buckets (three kernels when several maps' buckets need
several blocks), scatter, hits, walk, sweep."""
import numpy as np
import pytest

from vdb_mapping_gb300 import workloads as W

from test_gpu_parity import ref_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("n_maps", [2, 5])
def test_batch_step(vdbg, graph, n_maps):
    wl = W.BatchedWorkload(seed=61, n_maps=n_maps, n_steps=4, n_min=500, n_max=3000)
    b = vdbg.MapBatch(wl.resolutions, initial_leaf_capacity=1 << 18)
    for i, c in enumerate(wl.configs):
        b.setConfig(i, c)
    b.useGraph(graph)
    for _ in range(3):
        scans = wl.step(0)
        b.insert([p for p, _ in scans], [o for _, o in scans])
    assert b.timings()["launches"] == 8
    assert (b.graphStats()["replays"] > 0) == graph


def test_single_map(vdbg):
    m = vdbg.OccupancyVDBMapping(0.1)
    m.setConfig(ref_config(max_range=10.0))
    m.addInputSource("s", 10.0, 0)
    for _ in range(2):
        m.insertPointCloud(np.ones((100, 3), np.float32), (0.0, 0.0, 0.0), "s")
    assert m.timings()["launches"] == 6
