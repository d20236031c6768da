"""The chunked voxel walk of the insertion kernel (vdb_mapping_gb300/csrc/
march.cuh), compiled for the host, against the plain sequential DDA of
castRayIntoGrid in doubles, step by step: chunk starts, ties, binade changes,
walks past a chunk's end, single axes, powers of two and rays up to the index
range, for every chunk length."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_host_walk_matches_the_sequential_dda():
    src = os.path.join(HERE, "cpp", "march_host_test.cpp")
    out_dir = os.path.join(HERE, "cpp", "_build")
    os.makedirs(out_dir, exist_ok=True)
    exe = os.path.join(out_dir, "march_host_test")
    cmd = ["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-Wall", "-o", exe, src]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-3000:]
    run = subprocess.run([exe, "20"], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout[-3000:]
    assert run.stdout.strip().splitlines()[-1].startswith("ok ")
