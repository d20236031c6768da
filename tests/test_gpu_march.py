"""The insertion's walk on the GPU where its chunks begin and end: scans of a
single ray, of full and ragged groups of 32, at both sides of the sizes where
the chunk length changes, and rays longer than the crossing-time table. Maps
and statistics equal the oracle's bit for bit."""
import numpy as np
import pytest

from test_gpu_parity import assert_same_map, pair, ref_config

pytestmark = pytest.mark.gpu


def compare(g, o, pts, org):
    for m in (g, o):
        m.insertPointCloud(pts, org, "s")
    for key in ("rays", "visits", "hits", "updates"):
        assert g.last_stats[key] == o.last_stats[key], key


@pytest.mark.parametrize("n", [1, 31, 32, 33, 8191, 8192, 99999, 100000])
def test_scan_sizes(vdbg, oracle, n):
    rng = np.random.default_rng(n)
    g, o = pair(vdbg, oracle, 0.1, ref_config(max_range=12.0))
    pts = np.zeros((n, 3), np.float32)
    pts[:] = rng.normal(size=(n, 3)) * rng.choice([0.1, 1.0, 4.0, 20.0], size=(n, 1)) * [1.0, 1.0, 0.1]
    if n > 2:
        pts[n // 2] = (0.31, -0.22, 0.4)  # an endpoint in the sensor voxel
        pts[n // 3] = (np.nan, 0.0, 1.0)
    compare(g, o, pts, (0.31, -0.22, 0.4))
    assert_same_map(g.exportLeaves(), o.exportLeaves(), f"{n} points")


@pytest.mark.parametrize("res", [0.001, 0.0004])
def test_rays_beyond_the_table(vdbg, oracle, res):
    # up to 32,000 and 80,000 voxels on one axis, ties and an axis-aligned ray among them
    g, o = pair(vdbg, oracle, res, ref_config(max_range=40.0))
    pts = np.array([[16.3, 0.7, 0.01], [32.0, 0.0, 0.0], [-9.0, 9.0, 0.0], [15.0, -5.0, 2.5], [0.004, 0.003, 31.0],
                    [-20.1, -3.3, -0.4], [0.02, 16.384, 0.0], [1.0, 3.0, 0.2]], np.float32)
    compare(g, o, pts, (0.0, 0.0, 0.0))
    assert g.mapDigest() == o.mapDigest()


@pytest.mark.parametrize("spread, n", [(0.02, 1), (0.5, 40), (60.0, 40), (60.0, 4000)])
@pytest.mark.parametrize("prob", [(0.7, 0.4, 0.12, 0.97), (0.9, 0.1, 0.49, 0.51), (0.6, 0.45, 0.001, 0.999)])
def test_sweep_of_few_and_many_leaves(vdbg, oracle, spread, n, prob):
    """One leaf, few leaves per warp, leaves spread over many blocks, full
    planes; thresholds inside and outside the clamp limits; repeated scans, so
    that voxels are clamped and states flip both ways (with the change set)."""
    cfg = ref_config(max_range=80.0)
    cfg.prob_hit, cfg.prob_miss, cfg.prob_thres_min, cfg.prob_thres_max = prob
    g, o = pair(vdbg, oracle, 0.2, cfg)
    g.trackChanges()
    rng = np.random.default_rng(n)
    base = (rng.normal(size=(n, 3)) * spread * [1.0, 1.0, 0.2]).astype(np.float32)
    for k in range(14):
        pts = base if k < 7 else base * np.float32(1.5)  # first hit, then passed through
        compare(g, o, np.ascontiguousarray(pts), (0.05, 0.05, 0.05))
    assert_same_map(g.exportLeaves(), o.exportLeaves(), f"{n} points, spread {spread}")
