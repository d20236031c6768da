"""getMapSection on both sides of the sizes where its path changes: a box of at most
2^15 leaf cells (written at once), of at most 2^20 (counted first), larger (listed),
full and active only, with the box's faces inside leaves. Equal to the oracle."""
import numpy as np
import pytest

from test_gpu_parity import assert_same_map
from test_gpu_sections import built_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(1, 1, 1), (32, 32, 31), (32, 32, 32), (33, 32, 32), (128, 128, 64), (129, 128, 64)])
def test_box_sizes(vdbg, oracle, cells):
    g, o = built_pair(vdbg, oracle)
    for shift in (0, 3):
        lo = np.array([-8 * (c // 2) + shift for c in cells])
        hi = lo + 8 * np.array(cells) - 1 - 2 * shift
        for full in (False, True):
            assert_same_map(g.getMapSection(lo, hi, full=full), o.getMapSection(lo, hi, full=full), f"{cells} {full}")
