"""The public constants of the no-allocation insert: every name that the header has had
compiles, and the Python binding states the same values."""
import os
import subprocess

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

NAMES = ("VDBG_NOALLOC_MAX_POINTS", "VDBG_NOALLOC_DDA_WARPS", "VDBG_NOALLOC_RUN_SEGMENT", "VDBG_NOALLOC_SCRATCH_BYTES")


def values(tmp_path):
    src = tmp_path / "names.c"
    src.write_text("\n".join(['#include <stdio.h>', '#include "vdb_gb300.h"', "int main(void) {"] +
                             [f'  printf("%lld\\n", (long long)({n}));' for n in NAMES] + ["  return 0;", "}"]) + "\n")
    exe = tmp_path / "names"
    res = subprocess.run(["gcc", "-std=c11", "-I", os.path.join(REPO, "include"), str(src), "-o", str(exe)],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()
    return dict(zip(NAMES, map(int, out)))


def test_names_compile(tmp_path):
    v = values(tmp_path)
    assert v["VDBG_NOALLOC_DDA_WARPS"] == 256 and v["VDBG_NOALLOC_RUN_SEGMENT"] == 4096


def test_binding_agrees(tmp_path):
    from vdb_mapping_gb300 import _lib

    v = values(tmp_path)
    assert v["VDBG_NOALLOC_MAX_POINTS"] == _lib.VDBG_NOALLOC_MAX_POINTS
    assert v["VDBG_NOALLOC_SCRATCH_BYTES"] == _lib.VDBG_NOALLOC_SCRATCH_BYTES


def test_scratch_is_what_the_call_uses(tmp_path):
    """Staged points, ray records and ray order per point, two histograms of the 11,154
    sort buckets, and at most 1 MiB to spare (every GPU that loads the library holds it)."""
    v = values(tmp_path)
    used = v["VDBG_NOALLOC_MAX_POINTS"] * (16 + 16 + 4) + 2 * 11154 * 4
    assert used <= v["VDBG_NOALLOC_SCRATCH_BYTES"] <= used + (1 << 20)
