"""The walk's chunks at each length with one and the same scans: a batch's step takes the
length for the largest step its scratch has held, so small scans after a first step of
300, 9,000 or 110,000 points are walked in chunks of 32, 64 and 128. Every map equals the
oracle's, and so do single maps of the same scans."""
import numpy as np
import pytest

from vdb_mapping_gb300.mapping import Config

from test_gpu_changes import FLIPPY
from test_gpu_parity import assert_same_map

pytestmark = pytest.mark.gpu

RES = (0.1, 0.03)


def clouds(seed, counts):
    rng = np.random.default_rng(seed)
    out = []
    for n in counts:
        p = rng.normal(size=(n, 3)) * [6.0, 6.0, 1.5]
        p[: n // 4] = np.round(p[: n // 4])        # ties and axis directions
        p[n // 4: n // 3] *= 8.0                   # clipped
        out.append((p.astype(np.float32), tuple(rng.uniform(-1.0, 1.0, 3))))
    return out


@pytest.mark.parametrize("first", [300, 9000, 110000])
def test_small_scans_after(vdbg, oracle, first):
    cfg = Config(max_range=20.0, **FLIPPY)
    b = vdbg.MapBatch(list(RES), initial_leaf_capacity=1 << 18)
    single = [vdbg.OccupancyVDBMapping(r) for r in RES]
    maps = [oracle.OracleMap(r) for r in RES]
    for i in range(2):
        b.setConfig(i, cfg)
        for m in (single[i], maps[i]):
            m.setConfig(cfg)
            m.addInputSource("s", 20.0, 0)
    for k, counts in enumerate(((first - 100, 100), (250, 40), (1, 280), (33, 31))):
        scans = clouds(first + k, counts)
        b.insert([p for p, _ in scans], [o for _, o in scans])
        for i, (p, o) in enumerate(scans):
            single[i].insertPointCloud(p, o, "s")
            maps[i].insertPointCloud(p, o, "s")
        for i in range(2):
            want = maps[i].exportLeaves()
            assert_same_map(b.exportLeaves(i), want, f"batch {first} {k} {i}")
            assert_same_map(single[i].exportLeaves(), want, f"single {first} {k} {i}")
