"""The host threads of the set-up loops (csrc/vbd_internal.h) pass an exception on instead of ending the process."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_exceptions_reach_the_caller(tmp_path):
    out = str(tmp_path / "test_workers")
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "vbd_tetmesh_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "test_workers.cpp"), "-o", out], check=True)
    r = subprocess.run([out], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
