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
memory = ctypes.c_size_t.in_dll(fake, "fake_memory")
memory_limit = ctypes.c_size_t.in_dll(fake, "fake_memory_limit")
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


# VBDsolver and VBD_GPU_Solver semantics; the first launch of a handle, and one between accepted ones
@pytest.mark.parametrize("semantics", [0, 1])
def test_steps_without_the_cooperative_launch(gpu_device, run, semantics):
    run(f"""
m = meshgen.jittered_block(9, 6, 5, seed=3, per_tet_sigma=0.2, E=2e4)
W = np.random.default_rng(3).normal(size=(m.num_verts, 3))
out = []
for refuse in ((), (0, 1, 2, 3), (1, 2)):
    s = build_solver(m, lanes=8, layout=4)
    s.set_option(_capi.OPT_SEMANTICS, {semantics})
    res = []
    for k in range(4):
        cooperative_error.value = 720 if k in refuse else 0  # cudaErrorCooperativeLaunchTooLarge
        s.set_option(_capi.OPT_LANES, 16 if k % 2 else 8)
        s.set_option(_capi.OPT_ENERGY_EVERY, 4 if k == 2 else 0)
        s.step(1 / 60, 10, G, True, 0.9, 2)
        res += [s.get_positions(), s.get_velocities(), s.energy_history()]
        s.update_inertia_from_cpu(m.x)
        s.solve_vbd(6, 3600.0, True, 0.9, k % 2)
        res.append(s.get_positions())
        if not {semantics}:
            s.record(2)
            for _ in range(3):
                s.step(1 / 60, 5, G, True, 0.9)
            res += s.backward(W, None, 8, 0.9)
            s.record(0)
    out.append(res)
    s.close()
same(out[0], out[1])
same(out[0], out[2])
""")


def test_walks_after_a_refused_launch_wait_as_long_as_before(gpu_device, run):
    """The count of started CTAs does not run ahead: a wait that runs out ends after its limit, not after the time
    that a CTA may take to start."""
    run("""
import time
m = meshgen.jittered_block(9, 6, 5, seed=3)
s = build_solver(m, lanes=8, layout=4)
s.step(1 / 60, 5, G, True, 0.9)
cooperative_error.value = 720
s.step(1 / 60, 5, G, True, 0.9)
cooperative_error.value = 0
s.set_option(_capi.OPT_LANES, 16)  # the walk is tried again, on the same lists
out = ctypes.c_int32(0)
t = time.perf_counter()
_capi.call("vbd_solver_walk_selftest", s._h, 5000, ctypes.byref(out))
assert out.value == 1 and time.perf_counter() - t < 5.0
""")


# about 4,200 and 7,200 free vertices a tile: the vectors and ids of the tile and its ghosts and two chunks per warp fit
# in an SM's shared memory for the smaller
@pytest.mark.parametrize("n,walks", [(40, True), (48, False)])
def test_tiles_larger_than_shared_memory(gpu_device, n, walks):
    """A mesh with too many vertices per SM takes the per-colour launches (here on a stream of 16 SMs)."""
    import numpy as np
    import torch

    from vbd_tetmesh_b200 import _capi, build_solver, meshgen

    driver = pytest.importorskip("cuda.bindings.driver")
    torch.zeros(1, device="cuda")  # the primary context

    def ok(r):
        assert r[0] == driver.CUresult.CUDA_SUCCESS, r[0]
        return r[1:] if len(r) > 2 else r[1] if len(r) == 2 else None

    sms = ok(driver.cuDeviceGetDevResource(0, driver.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups, _, _ = ok(driver.cuDevSmResourceSplitByCount(1, sms, 0, 16))
    desc = ok(driver.cuDevResourceGenerateDesc(groups, 1))
    ctx = ok(driver.cuGreenCtxCreate(desc, 0, driver.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream = ok(driver.cuGreenCtxStreamCreate(ctx, driver.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    m = meshgen.cube(n)
    out = []
    for persistent in (None, 0):
        s = build_solver(m, lanes=8, layout=4, stream=int(stream))
        if persistent is not None:
            s.set_option(_capi.OPT_PERSISTENT, persistent)
        l0 = s.kernel_launches()
        s.step(1 / 120, 3, (0.0, -9.8, 0.0), True, 0.9)
        s.sync()
        assert (s.kernel_launches() - l0 == 1) == (walks and persistent is None)
        out.append((s.get_positions(), s.get_velocities()))
        s.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    ok(driver.cuStreamDestroy(stream))
    ok(driver.cuGreenCtxDestroy(ctx))


def test_a_stream_of_fewer_sms(gpu_device):
    """On a green context's stream the walk takes as many tiles as that context has SMs."""
    import numpy as np
    import torch

    from vbd_tetmesh_b200 import _capi, build_solver, meshgen

    driver = pytest.importorskip("cuda.bindings.driver")
    torch.zeros(1, device="cuda")  # the primary context

    def ok(r):
        assert r[0] == driver.CUresult.CUDA_SUCCESS, r[0]
        return r[1:] if len(r) > 2 else r[1] if len(r) == 2 else None

    sms = ok(driver.cuDeviceGetDevResource(0, driver.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups, _, _ = ok(driver.cuDevSmResourceSplitByCount(1, sms, 0, 16))
    assert groups[0].sm.smCount < sms.sm.smCount
    desc = ok(driver.cuDevResourceGenerateDesc(groups, 1))
    ctx = ok(driver.cuGreenCtxCreate(desc, 0, driver.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream = ok(driver.cuGreenCtxStreamCreate(ctx, driver.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    m = meshgen.jittered_block(20, 12, 11, seed=3)  # more than 16 tiles on the whole device
    out = []
    for st in (None, int(stream)):
        s = build_solver(m, lanes=8, layout=4, stream=st)
        l0 = s.kernel_launches()
        s.step(1 / 60, 10, (0.0, -9.8, 0.0), True, 0.9)
        s.sync()
        assert s.kernel_launches() - l0 == 1
        out.append((s.get_positions(), s.get_velocities()))
        s.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    ok(driver.cuStreamDestroy(stream))
    ok(driver.cuGreenCtxDestroy(ctx))


def test_recording_buffers_give_way(gpu_device, run):
    """Buffers kept from a long recording are no reason to refuse another recording or its backward pass, and a new
    mesh and the end of recording give them back."""
    run("""
from vbd_tetmesh_b200 import color_vertices, mesh_mass, precompute_tets
m = meshgen.jittered_block(9, 6, 5, seed=3, per_tet_sigma=0.2, E=2e4)
W = np.random.default_rng(3).normal(size=(m.num_verts, 3))
def recorded(s, every, steps):
    s.set_positions(m.x)
    s.set_velocities(m.v)
    s.record(every)
    for _ in range(steps):
        s.step(1 / 60, 5, G, True, 0.9)
    return s.backward(W, None, 8, 0.9)
s = build_solver(m, lanes=8, layout=4)
want = recorded(s, 16, 20)
s.close()
s = build_solver(m, lanes=8, layout=4)
s.step(1 / 60, 5, G, True, 0.9)
before = memory.value
s.record(1)
for _ in range(60):
    s.step(1 / 60, 5, G, True, 0.9)
memory_limit.value = memory.value  # what the long recording took is all there is
same(want, recorded(s, 16, 20))
memory_limit.value = NONE
s.record(0)
kept = memory.value
s.record(1)
for _ in range(60):
    s.step(1 / 60, 5, G, True, 0.9)
s.record(1)
_, offs, verts = color_vertices(m.num_verts, m.tets)
dminv, v0 = precompute_tets(m.rest, m.tets)
s.init_from_cpu(m.x, mesh_mass(m.rest, m.tets, m.density)[0], m.fixed, m.tets, offs, verts, dminv, v0, m.mu, m.lam)
assert memory.value <= kept + 4 * 32 * m.num_verts, (memory.value, kept)
s.close()
""")


def test_options_give_unused_walk_memory_back(gpu_device, run):
    run("""
m = meshgen.jittered_block(20, 12, 11, seed=3, per_tet_sigma=0.2)
def steps(s):
    s.set_positions(m.x)
    s.set_velocities(m.v)
    s.step(1 / 60, 5, G, True, 0.9)
    return s.get_positions(), s.get_velocities()
s = build_solver(m, lanes=8, layout=4)
made = memory.value
s.set_option(_capi.OPT_PERSISTENT, 0)
base = memory.value
assert base < made - 44 * 4 * m.num_tets * 0.8, (base, made)  # the records, less those of pinned vertices
graph = steps(s)
s.close()
s = build_solver(m, lanes=8, layout=4)
s.set_option(_capi.OPT_SEMANTICS, 1)  # the other semantics' set instead of, not beside, the one made at init
assert memory.value - base < 2.2 * (made - base), (memory.value, base, made)
wrapper = steps(s)
s.set_option(_capi.OPT_SEMANTICS, 0)
same(steps(s), graph)
both = memory.value
s.set_option(_capi.OPT_SEMANTICS, 1)  # both have run: kept
assert memory.value == both
same(steps(s), wrapper)
s.close()
""")
