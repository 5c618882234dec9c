"""The tile walk's host plan (csrc/vbd_tile_plan.cpp): every list its kernels index, the chunk order,
and its exchange of published words replayed with the tiles advancing in random order
(tests/cpp/test_tile_plan.cpp; built here with the host compiler)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "vbd_tetmesh_b200", "csrc")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("tile_plan") / "test_tile_plan")
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", CSRC, os.path.join(ROOT, "tests", "cpp", "test_tile_plan.cpp"),
                    os.path.join(CSRC, "vbd_tile_plan.cpp"), "-o", out], check=True)
    return out


# lx ly lz, meshes, tiles, lanes, x = 0 face pinned, seed, warps: more tiles than some colours have
# vertices, one tile, tiles across mesh borders, an unpinned mesh, every lane and warp count
@pytest.mark.parametrize("args", [
    (5, 4, 3, 1, 7, 8, 1, 1, 8), (12, 12, 12, 1, 60, 16, 1, 2, 8), (12, 9, 7, 3, 30, 4, 0, 3, 16),
    (20, 20, 20, 1, 148, 8, 1, 4, 16), (2, 2, 2, 1, 1, 8, 0, 6, 8), (1, 1, 1, 40, 20, 4, 0, 7, 8),
])
def test_plan_and_exchange(program, args):
    r = subprocess.run([program, *map(str, args)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
