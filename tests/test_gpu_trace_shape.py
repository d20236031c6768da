"""Raytrace on both sides of the lines where its launch shape changes: a query a warp,
some queries a warp, whole warps, with and without the sorts. Answers equal the
oracle's; the sorts' launches are there only where warps are more than half full."""
import dataclasses

import numpy as np
import pytest

from vdb_mapping_gb300 import workloads as W

from test_gpu_raytrace import same_trace
from test_gpu_spans import striped

pytestmark = pytest.mark.gpu

SMS = 152


@pytest.mark.parametrize("n, launches", [
    (7, 4), (8 * SMS, 4), (8 * SMS + 1, 4), (16 * SMS, 4), (16 * SMS + 1, 4), (10000, 4), (8 * SMS * 16, 4),
    (8 * SMS * 16 + 1, 11), (8 * SMS * 32 + 1, 11)])
def test_answers_and_launches(vdbg, oracle, n, launches):
    g, o = striped(vdbg, oracle, "gaps")
    rng = np.random.default_rng(n)
    org = np.stack([rng.uniform(-20.0, 600.0, n), rng.uniform(-12.0, 12.0, n), rng.uniform(-4.0, 20.0, n)], 1)
    d = rng.normal(size=(n, 3)) * [1.0, 0.02, 0.02]
    d[: n // 3, 1:] = 0.0
    ln = rng.uniform(1.0, 900.0, n)
    same_trace(g.raytrace(org, d, ln), o.raytrace(org, d, ln), f"{n}")
    assert g.timings()["launches"] == launches


@pytest.mark.parametrize("n, launches", [(16 * SMS, 4), (32 * SMS, 4), (32 * SMS + 1, 11), (10000, 11)])
def test_a_map_of_many_leaves(vdbg, oracle, n, launches):
    """More than 2^20 leaves, most of them where no query goes (and without an active
    voxel, so that the intersector's box is that of the others)."""
    g, o = striped(vdbg, oracle, "gaps")
    g.setConfig(dataclasses.replace(W.get("small").config, max_range=4000.0))
    g.addInputSource("far", 4000.0, 0)
    d = np.random.default_rng(2).normal(size=(4000, 3))
    pts = 20000.0 + 3000.0 * d / np.linalg.norm(d, axis=1, keepdims=True)
    g.insertPointCloud(pts.astype(np.float32), (20000.0,) * 3, "far")
    assert g.leafCount() > 1 << 20
    rng = np.random.default_rng(n)
    org = np.stack([rng.uniform(-20.0, 600.0, n), rng.uniform(-12.0, 12.0, n), rng.uniform(-4.0, 20.0, n)], 1)
    d = rng.normal(size=(n, 3)) * [1.0, 0.02, 0.02]
    ln = rng.uniform(1.0, 900.0, n)
    same_trace(g.raytrace(org, d, ln), o.raytrace(org, d, ln), f"{n}")
    assert g.timings()["launches"] == launches
