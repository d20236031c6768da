"""The workspaces of the section reads are kept between calls: repeated reads of a box
of any size that is written at once allocate nothing, and a batch goes on replaying its
captured step between them."""
import numpy as np
import pytest

from vdb_mapping_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(8, 8, 8), (32, 32, 25), (32, 32, 26), (32, 32, 32)])
def test_reads_between_steps(vdbg, cells):
    wl = W.BatchedWorkload(seed=61, n_maps=2, n_steps=6, n_min=500, n_max=3000)
    b = vdbg.MapBatch(wl.resolutions, initial_leaf_capacity=1 << 17)
    for i, c in enumerate(wl.configs):
        b.setConfig(i, c)
    lo = -8 * (np.array(cells) // 2)
    hi = lo + 8 * np.array(cells) - 1
    captures, held = [], []
    for k in range(6):
        scans = wl.step(0)
        b.insert([p for p, _ in scans], [o for _, o in scans])
        for i in range(2):
            b.getMapSection(i, lo, hi, full=True)
        captures.append(b.graphStats()["captures"])
        held.append(b.deviceBytes())
    # (the first read makes the workspaces, which moves the layout once)
    assert captures[2:] == captures[2:3] * 4, captures
    assert held[2:] == held[2:3] * 4, held
