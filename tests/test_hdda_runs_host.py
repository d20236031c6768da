"""The voxel walks over a span's windows (vdb_mapping_gb300/csrc/hdda.cuh),
compiled for the host, against the walks over every voxel of the span: raytrace
end points and the active voxels fast mode meets, bit for bit, for rays with tied
and nearly tied crossings, near-parallel rays, far origins and large coordinates."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_windows_match_the_whole_walk():
    src = os.path.join(HERE, "cpp", "hdda_runs_test.cpp")
    out_dir = os.path.join(HERE, "cpp", "_build")
    os.makedirs(out_dir, exist_ok=True)
    exe = os.path.join(out_dir, "hdda_runs_test")
    cmd = ["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-Wall", "-o", exe, src]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-3000:]
    run = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout[-3000:]
    assert run.stdout.strip().splitlines()[-1].startswith("ok ")
