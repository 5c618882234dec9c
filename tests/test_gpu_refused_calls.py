"""Where the CUDA runtime refuses what a walk needs (its memory, its cooperative launch), the steps run as they did
without the walk, with the same bits.  The refusals come from a stand-in for the runtime's calls
(tests/cpp/fake_cuda.cpp), in a process of its own."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = """
import ctypes, sys
import numpy as np
sys.path.insert(0, {root!r})
from vbd_tetmesh_b200 import _capi, build_solver, meshgen
fake = ctypes.CDLL({fake!r})
malloc_limit = ctypes.c_size_t.in_dll(fake, "fake_malloc_limit")
cooperative_error = ctypes.c_int.in_dll(fake, "fake_cooperative_error")
G = (0.0, -9.8, 0.0)
NONE = 2**64 - 1
def same(a, b):
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    fake = str(tmp_path_factory.mktemp("fake") / "libfake_cuda.so")
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-o", fake, os.path.join(ROOT, "tests", "cpp", "fake_cuda.cpp"), "-ldl"],
                   check=True)

    def go(body):
        r = subprocess.run([sys.executable, "-c", PRELUDE.format(root=ROOT, fake=fake) + body], capture_output=True, text=True,
                           timeout=300, env=dict(os.environ, LD_PRELOAD=fake))
        assert r.returncode == 0, r.stdout + r.stderr

    return go


def test_cluster_walk_without_memory_for_its_tiles(gpu_device, run):
    run("""
m = meshgen.jittered_block(9, 6, 5, seed=3, per_tet_sigma=0.2, E=2e4)
W = np.random.default_rng(3).normal(size=(m.num_verts, 3))
out = []
for refuse in (False, True):
    s = build_solver(m, lanes=8, layout=4)
    s.set_option(_capi.OPT_CLUSTER_RESIDENT, 0)
    s.set_option(_capi.OPT_PERSISTENT, 2)
    s.record(2)  # the schedules and adjoint buffers are allocated before
    for _ in range(3):
        s.step(1 / 60, 10, G, True, 0.9)
    s.backward(W, None, 12, 0.9)
    if refuse:
        malloc_limit.value = 50000  # more than a checkpoint takes, less than the tiles' records
    s.set_option(_capi.OPT_CLUSTER_RESIDENT, 1)
    s.set_option(_capi.OPT_PERSISTENT, 2)
    s.record(2)
    for _ in range(3):
        s.step(1 / 60, 10, G, True, 0.9)
    res = [s.get_positions(), *s.backward(W, None, 12, 0.9)]
    s.set_option(_capi.OPT_LANES, 16)
    s.step(1 / 60, 10, G, True, 0.9)
    out.append(res + [s.get_positions(), s.get_velocities()])
    malloc_limit.value = NONE
    s.close()
same(*out)
""")


def test_steps_without_memory_for_the_walk(gpu_device, run):
    run("""
m = meshgen.jittered_block(9, 6, 5, seed=3, per_tet_sigma=0.2)
out = []
for refuse in (False, True):
    s = build_solver(m, lanes=16, layout=4)
    s.step(1 / 60, 10, G, True, 0.9)
    if refuse:
        malloc_limit.value = 1
    s.set_option(_capi.OPT_LANES, 4)  # more chunks for the few vertices of a tile and colour
    l0 = s.kernel_launches()
    s.step(1 / 60, 10, G, True, 0.9)
    assert (s.kernel_launches() - l0 > 10) == refuse
    out.append([s.get_positions(), s.get_velocities()])
    malloc_limit.value = NONE
    s.close()
same(*out)
""")
