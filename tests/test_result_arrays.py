"""The arrays that sections, change sets and morphology return hold the rows returned,
not all of the room the call was given: a program that keeps its results keeps at most
eight times them. The library is a stand-in that writes a few rows."""
import ctypes as C

import numpy as np
import pytest

from vdb_mapping_gb300 import mapping as M


class Lib:
    def __init__(self, rows):
        self.rows = rows

    def _fill(self, cap, n, *arrays):
        n._obj.value = self.rows
        if self.rows > cap:
            from vdb_mapping_gb300 import _lib

            return _lib.STATUS_CODE["VDBG_ERR_BUFFER_TOO_SMALL"]
        for at, nbytes in arrays:
            C.memset(at, 1, nbytes * self.rows)
        return 0

    def vdbg_export_section(self, h, i, lo, hi, full, cap, o, v, m, n):
        return self._fill(cap, n, (o, 12), (v, 2048), (m, 64))

    def vdbg_export_changes(self, h, i, cap, o, a, v, n):
        return self._fill(cap, n, (o, 12), (a, 64), (v, 64))

    def vdbg_section_morphology(self, h, code, it, k, o, m, cap, oo, om, n):
        return self._fill(cap, n, (oo, 12), (om, 64))


def check(status, where):
    assert status == 0


def held(a):
    while a.base is not None:
        a = a.base
    return a.nbytes


@pytest.mark.parametrize("rows", [0, 1, 700, 3000, 20000])
def test_arrays_hold_their_rows(rows):
    lib = Lib(rows)
    hi = np.array([8 * 25 - 1] * 3)
    results = [M._section_export(lib, None, -1, np.zeros(3), hi, True, check), M._export_changes(lib, None, -1, check),
               M._morphology(lib, None, np.zeros((9, 3)), np.zeros((9, 8)), "close", 1, check)]
    for arrays in results:
        for a in arrays:
            assert a.shape[0] == rows and a.flags.c_contiguous and a.flags.writeable
            assert held(a) <= 8 * a.nbytes
            assert rows == 0 or np.array_equal(np.unique(a.view(np.uint8)), [1])
