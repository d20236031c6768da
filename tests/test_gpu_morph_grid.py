"""The morphology's two paths (a dense grid of leaf cells, and a hashed set where
the cells are too many) on both sides of the rule between them, and where the
dense grid ends: steps that just reach its outermost leaves. Leaves, masks and
their order equal the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(g, oracle, o, m, op, it, keep):
    go, gm = g.sectionMorphology(o, m, op, it, keep_leaves=keep)
    oo, om = oracle.morphology(o, m, op, it, keep_leaves=keep)
    assert np.array_equal(go, oo), (op, it, keep, len(go), len(oo))
    assert np.array_equal(gm, om), (op, it, keep)


@pytest.mark.parametrize("op", ["dilate", "erode", "close", "open"])
@pytest.mark.parametrize("keep", [False, True])
@pytest.mark.parametrize("x_cells", [1, 4093, 4094, 4095, 4096, 4097])
def test_grid_or_set(vdbg, oracle, op, keep, x_cells):
    # one iteration adds a cell on each side: 8 x 8 x 4096 cells are the most
    # taken as a grid (x_cells 4094; 4096 for the erosion, which adds none)
    rng = np.random.default_rng(x_cells)
    g = vdbg.OccupancyVDBMapping(0.1)
    rows = 6 if op != "erode" else 8
    o = np.stack([8 * rng.integers(0, x_cells, 40), 8 * rng.integers(0, rows, 40), 8 * rng.integers(0, rows, 40)], 1)
    o[0] = (0, 0, 0)
    o[1] = (8 * (x_cells - 1), 8 * (rows - 1), 8 * (rows - 1))
    o = (o + [-16384, 64, -96]).astype(np.int32)
    o[5] = o[0]  # a repeated origin
    m = rng.integers(0, 1 << 63, (40, 8), dtype=np.uint64) | rng.integers(0, 1 << 63, (40, 8), dtype=np.uint64)
    m[1] = ~np.uint64(0)
    m[7] = 0     # a leaf without an active voxel
    check(g, oracle, o, m, op, 1, keep)


@pytest.mark.parametrize("op", ["dilate", "close", "open"])
@pytest.mark.parametrize("it", [0, 7, 8, 9, 16, 17])
def test_steps_reach_the_last_leaves(vdbg, oracle, op, it):
    g = vdbg.OccupancyVDBMapping(0.1)
    o = np.array([[-8, 0, 8], [0, 0, 8]], np.int32)
    m = np.zeros((2, 8), np.uint64)
    m[0, 0] = 1                      # the leaf's first corner
    m[1, 7] = np.uint64(1) << 63     # and the other's last
    for keep in (False, True):
        check(g, oracle, o, m, op, it, keep)
