"""Budgets that leave no room for what only speeds a call up."""
import numpy as np
import pytest

from test_gpu_parity import assert_same_map, pair, ref_config

pytestmark = pytest.mark.gpu

TABLE = 16384 * 10 * 24 + 16384 * 8  # the walk's table of crossing times


def test_a_map_without_room_for_the_table(vdbg, oracle):
    """The pools fit and the table does not: the map is made, and inserts as any other."""
    g = vdbg.OccupancyVDBMapping(0.1, initial_leaf_capacity=1024, initial_block_capacity=1024)
    g.addInputSource("s", 5000.0, 0)
    held = g.deviceBytes()
    g.close()
    rng = np.random.default_rng(4)
    pts = (rng.normal(size=(500, 3)) * [4.0, 4.0, 1.0]).astype(np.float32)
    far = np.concatenate([pts, pts * np.float32(40.0)])
    cfg = ref_config(max_range=5000.0)
    g, o = pair(vdbg, oracle, 0.1, cfg, max_device_bytes=held - TABLE + (64 << 10), initial_leaf_capacity=1024,
                initial_block_capacity=1024)
    assert g.deviceBytes() <= held - TABLE + (64 << 10)
    for m in (g, o):
        m.insertPointCloud(pts[:40] * np.float32(0.2), (0.1, 0.2, 0.3), "s")
    assert_same_map(g.exportLeaves(), o.exportLeaves(), "tight")
    g, o = pair(vdbg, oracle, 0.1, cfg, max_device_bytes=1 << 30)
    for k in range(2):
        for m in (g, o):
            m.insertPointCloud(far, (0.1, 0.2 + k, 0.3), "s")
    assert_same_map(g.exportLeaves(), o.exportLeaves(), "roomy")


def test_the_call_that_allocates_nothing(vdbg, oracle):
    """With a budget the table is made by the first regular insert: before it the walk
    computes what the table holds, for short rays and for rays beyond its range."""
    from vdb_mapping_gb300 import _lib

    cfg = ref_config(max_range=5000.0)
    g, o = pair(vdbg, oracle, 0.1, cfg, max_device_bytes=4 << 30, initial_leaf_capacity=1 << 19,
                initial_block_capacity=1 << 17)
    lib = _lib.load()
    rng = np.random.default_rng(6)
    for n, spread in ((300, 3.0), (12000, 3.0), (40, 900.0)):
        pts = np.zeros((n, 4), np.float32)
        pts[:, :3] = rng.normal(size=(n, 3)) * spread
        assert lib.vdbg_insert_point_cloud_noalloc(g._h, pts.ctypes.data, n, 16, (_lib.C.c_double * 3)(0.1, 0.2, 0.3),
                                                   b"s", 0, None, None) == 0
        o.insertPointCloud(np.ascontiguousarray(pts[:, :3]), (0.1, 0.2, 0.3), "s")
        assert_same_map(g.exportLeaves(), o.exportLeaves(), f"{n}")


def test_room_of_a_raytrace(vdbg, oracle):
    """A query takes 87 bytes of inputs, answers and order and 64 of span record."""
    from test_gpu_raytrace import same_trace

    g, o = pair(vdbg, oracle, 0.1, ref_config(max_range=8.0))
    for m in (g, o):
        m.insertPointCloud(np.ones((10, 3), np.float32), (0.1, 0.2, 0.3), "s")
    n = 100000
    held = g.deviceBytes()
    d = np.random.default_rng(1).normal(size=(n, 3))
    ln = np.full(n, 5.0)
    same_trace(g.raytrace(np.zeros((n, 3)), d, ln), o.raytrace(np.zeros((n, 3)), d, ln))
    nodes = 2 * 1024 * 16
    assert g.deviceBytes() - held <= n * (87 + 64) + nodes + (64 << 10)


@pytest.mark.parametrize("count", [0, 1])
def test_fast_mode_without_room_for_its_pieces(vdbg, oracle, count):
    """The room for the pieces of every ray's windows is refused: the scan goes on with a
    piece a span."""
    from test_gpu_raytrace import active_pair

    vox = [(x, y, z) for x in range(0, 4000, 24) for y in (-4, 3) for z in (1, 9)]
    g, o = active_pair(vdbg, oracle, vox)
    n = 2000
    rng = np.random.default_rng(8)
    far = np.stack([rng.uniform(3000.0, 4100.0, n), rng.uniform(-3.9, 3.9, n), rng.uniform(0.0, 12.0, n)], 1)
    near = np.tile(np.array([[-3.2, 0.6, 4.6]]), (n, 1))
    cfg = ref_config(max_range=5000.0)
    for fast in (False, True):  # (leaves all along the rays, so that their spans are long)
        cfg.fast_mode = fast
        for m in (g, o):
            m.setConfig(cfg)
            if not fast:
                m.addInputSource("s", 5000.0, 0)
                m.insertPointCloud(far.astype(np.float32), (-3.5, 0.5, 4.5), "s")
    # (the first scan has a fast scan's other buffers made)
    for k, pts in enumerate((near, far, far + [0.0, 0.7, 0.2])):
        if k == 1:
            held = g.deviceBytes()
            assert g._lib.vdbg_test_fail_allocs(g._h, 0, count) == 0
        for m in (g, o):
            m.insertPointCloud(pts.astype(np.float32), (-3.5, 0.5, 4.5), "s")
        if k == 1:
            # more pieces than the first guess has room for, or the refusal did not matter
            assert (g.deviceBytes() > held + 32 * (2 * n + 4096)) == (count == 0)
        for key in ("rays", "visits", "hits", "updates"):
            assert g.last_stats[key] == o.last_stats[key], (k, key)
        assert_same_map(g.exportLeaves(), o.exportLeaves(), f"fast {k}")
