"""Spans and their walks on the GPU where the work is cut: one ray to more than a
warp takes per lane, rays with more windows than a thread keeps and more pieces
than the first buffer holds, solid leaves, leaves without an active voxel. Fast
mode's maps and statistics and raytrace's answers equal the oracle's bit for bit."""
import numpy as np
import pytest

from test_gpu_parity import assert_same_map, ref_config
from test_gpu_raytrace import active_pair, same_trace

pytestmark = pytest.mark.gpu


def striped(vdbg, oracle, kind):
    """Slabs of leaves along x, and a floor of leaves without an active voxel."""
    vox = []
    step = {"sparse": 72, "touching": 8, "gaps": 32}[kind]
    for x in range(0, 3600 if kind == "sparse" else 600, step):
        for y in range(-8, 8, 8):
            for z in (0, 8):
                if kind == "touching":
                    vox += [(x + i, y + 3, z + 2) for i in range(8)]
                else:
                    vox += [(x + i, y + i, z + (3 * i & 7)) for i in range(0, 8, 3)]
    return active_pair(vdbg, oracle, vox)


@pytest.mark.parametrize("kind", ["sparse", "touching", "gaps"])
@pytest.mark.parametrize("n", [1, 33, 300])
def test_fast_mode(vdbg, oracle, kind, n):
    g, o = striped(vdbg, oracle, kind)
    cfg = ref_config(max_range=5000.0)
    cfg.fast_mode = True
    rng = np.random.default_rng(n)
    pts = np.stack([rng.uniform(300.0, 3700.0, n), rng.uniform(-7.0, 7.0, n), rng.uniform(0.0, 15.0, n)], 1)
    pts[: n // 2, 1] = np.round(pts[: n // 2, 1]) + 0.5
    pts[: n // 4, 2] = 4.5
    for m in (g, o):
        m.setConfig(cfg)
        m.addInputSource("s", 5000.0, 0)
    for origin in ((-3.5, 0.5, 4.5), (3650.2, -1.3, 7.7)):
        for m in (g, o):
            m.insertPointCloud(pts.astype(np.float32), origin, "s")
        for key in ("rays", "visits", "hits", "updates"):
            assert g.last_stats[key] == o.last_stats[key], key
    assert_same_map(g.exportLeaves(), o.exportLeaves(), kind)


@pytest.mark.parametrize("n", [1, 31, 4864, 4865, 20000])
def test_raytrace(vdbg, oracle, n):
    for kind in ("sparse", "touching"):
        g, o = striped(vdbg, oracle, kind)
        rng = np.random.default_rng(n)
        org = np.stack([rng.uniform(-20.0, 600.0, n), rng.uniform(-12.0, 12.0, n), rng.uniform(-4.0, 20.0, n)], 1)
        d = rng.normal(size=(n, 3)) * [1.0, 0.02, 0.02]
        d[: n // 3, 1:] = 0.0
        d[n // 3: n // 2, 1] = d[n // 3: n // 2, 0]
        ln = rng.uniform(1.0, 3000.0, n)
        same_trace(g.raytrace(org, d, ln), o.raytrace(org, d, ln), kind)
