"""What the walks (csrc/vbd_tile.cuh, csrc/vbd_cluster.cuh) keep between calls: schedules, captured launches,
packed records and wait states stay right when the calls around them change."""
import ctypes as C

import numpy as np
import pytest

from vbd_tetmesh_b200 import _capi, build_solver, meshgen

pytestmark = pytest.mark.gpu

G = (0.0, -9.8, 0.0)


# tiles in the cluster's CTAs, whole-mesh copies
@pytest.mark.parametrize("resident", [1, 0])
def test_backward_with_a_longer_schedule_between(gpu_device, resident):
    """A longer adjoint schedule moves the weights to a larger buffer: a captured launch of the shorter one
    must not read the old buffer."""
    m = meshgen.jittered_block(8, 5, 4, seed=2, per_tet_sigma=0.2, E=2e4)
    W = np.random.default_rng(2).normal(size=(m.num_verts, 3))

    def recorded():
        s = build_solver(m, lanes=8, layout=4)
        s.set_option(_capi.OPT_PERSISTENT, 2)
        s.set_option(_capi.OPT_CLUSTER_RESIDENT, resident)
        s.record(2)
        for _ in range(3):
            s.step(1 / 60, 10, G, True, 0.9)
        return s

    one = recorded()
    for sweeps in (10, 50, 10, 200, 50):
        fresh = recorded()
        want = fresh.backward(W, None, sweeps, 0.9)
        fresh.close()
        for a, b in zip(one.backward(W, None, sweeps, 0.9), want):
            np.testing.assert_array_equal(a, b)
    one.close()


def give_up(s, wait_us=5000):
    """One walk of `s` whose waits run out."""
    out = C.c_int32(0)
    _capi.call("vbd_solver_walk_selftest", s._h, wait_us, C.byref(out))
    return out.value


# 8 warps with resident and streamed chunks, 16 warps with one and two rounds of a group, VBD_GPU_Solver semantics
# with 8 and 16 warps
@pytest.mark.parametrize("mesh,lanes,semantics", [
    (lambda: meshgen.jittered_block(7, 6, 5, seed=5), 16, 0), (lambda: meshgen.cube(24), 8, 0),
    (lambda: meshgen.cube(32), 16, 0), (lambda: meshgen.cube(44), 8, 0), (lambda: meshgen.cube(40), 4, 0),
    (lambda: meshgen.jittered_block(7, 6, 5, seed=5), 8, 1), (lambda: meshgen.cube(26), 8, 1),
], ids=["block", "cube24", "cube32", "cube44", "cube40", "wrapper block", "wrapper cube26"])
def test_a_wait_that_runs_out_ends_the_walk(gpu_device, mesh, lanes, semantics):
    m = mesh()
    out = []
    for fail in (False, True):
        s = build_solver(m, lanes=lanes)
        s.set_option(_capi.OPT_SEMANTICS, semantics)
        s.step(1 / 120, 4, G, True, 0.9)
        if fail:
            assert give_up(s) == 1
            with pytest.raises(_capi.VBDError) as e:
                s.sync()
            assert e.value.code == 6  # VBD_ERR_TIMEOUT
        l0 = s.kernel_launches()
        s.step(1 / 120, 4, G, True, 0.9)
        s.sync()
        assert s.kernel_launches() - l0 <= 2  # still the walk
        out.append((s.get_positions(), s.get_velocities(), np.array(s.status())))
        s.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_walk_selftest_refuses_what_is_no_walk(gpu_device):
    s = build_solver(meshgen.jittered_block(7, 6, 5, seed=5))
    for wait in (0, 1000001):
        with pytest.raises(_capi.VBDError) as e:
            give_up(s, wait)
        assert e.value.code == 1  # VBD_ERR_INVALID_ARG
    s.set_option(_capi.OPT_PERSISTENT, 0)
    with pytest.raises(_capi.VBDError) as e:
        give_up(s)
    assert e.value.code == 3  # VBD_ERR_STATE
    s.close()


@pytest.mark.parametrize("call", [
    lambda s: s.get_positions(), lambda s: s.get_velocities(), lambda s: s.get_inertia(), lambda s: s.energy(0, 1 / 60),
    lambda s: s.energy(2, 1 / 60), lambda s: s.energy_history(), lambda s: s.status(), lambda s: s.status(True),
    lambda s: s.sync(), lambda s: s.record(2), lambda s: s.backward(np.ones((s.num_verts, 3)), None, 5, 0.9),
    lambda s: s.autotune(1 / 60, 2, 1),
], ids=["positions", "velocities", "inertia", "energy", "residual", "history", "status", "status reset", "sync", "record",
        "backward", "autotune"])
def test_a_wait_that_ran_out_is_reported_once(gpu_device, call):
    """By the first call that waits for a result; the steps after the report are right again."""
    m = meshgen.jittered_block(7, 6, 5, seed=5)
    s = build_solver(m)
    s.set_option(_capi.OPT_ENERGY_EVERY, 2)
    s.record(2)
    s.step(1 / 60, 4, G, True, 0.9)
    x = s.get_positions()
    assert give_up(s) == 1
    with pytest.raises(_capi.VBDError) as e:
        call(s)
    assert e.value.code == 6  # VBD_ERR_TIMEOUT
    s.sync()
    np.testing.assert_array_equal(s.get_positions(), x)
    s.step(1 / 60, 4, G, True, 0.9)
    fresh = build_solver(m)
    for _ in range(2):
        fresh.step(1 / 60, 4, G, True, 0.9)
    np.testing.assert_array_equal(s.get_positions(), fresh.get_positions())
    s.close()
    fresh.close()


def test_a_wait_of_full_length_is_reported_between_reads(gpu_device):
    """The record is not read after every step: a wait that gave up lasts longer than the time between two looks."""
    s = build_solver(meshgen.jittered_block(7, 6, 5, seed=5))
    s.get_positions()  # looks
    assert give_up(s, 400000) == 1
    with pytest.raises(_capi.VBDError) as e:
        s.get_positions()
    assert e.value.code == 6  # VBD_ERR_TIMEOUT
    s.get_positions()
    s.close()


def test_the_barrier_selftest_leaves_a_walks_report(gpu_device):
    s = build_solver(meshgen.jittered_block(7, 6, 5, seed=5))
    assert give_up(s) == 1
    out = C.c_int32(0)
    _capi.call("vbd_solver_barrier_selftest", s._h, 2000, C.byref(out))
    assert out.value == 1
    with pytest.raises(_capi.VBDError) as e:
        s.get_positions()
    assert e.value.code == 6  # VBD_ERR_TIMEOUT
    s.sync()
    s.close()


def test_a_new_mesh_starts_without_the_last_ones_report(gpu_device):
    from vbd_tetmesh_b200 import color_vertices, mesh_mass, precompute_tets

    m = meshgen.jittered_block(7, 6, 5, seed=5)
    s = build_solver(m)
    assert give_up(s) == 1
    _, offs, verts = color_vertices(m.num_verts, m.tets)
    dminv, v0 = precompute_tets(m.rest, m.tets)
    s.init_from_cpu(m.x, mesh_mass(m.rest, m.tets, m.density)[0], m.fixed, m.tets, offs, verts, dminv, v0, m.mu, m.lam)
    s.step(1 / 60, 4, G, True, 0.9)
    assert np.isfinite(s.get_positions()).all()
    s.close()


def on_stream(m, lanes=8, ctas=0):
    """A solver with the cluster walk on a torch stream, after one step."""
    import torch

    st = torch.cuda.Stream()
    s = build_solver(m, lanes=lanes, layout=4, stream=st.cuda_stream)
    s.set_option(_capi.OPT_CLUSTER_CTAS, ctas)
    s.set_option(_capi.OPT_PERSISTENT, 2)
    s.step(1 / 60, 9, G, True, 0.9)
    s.sync()
    return s, st


def capture_step(s, st):
    import torch

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        s.step(1 / 60, 9, G, True, 0.9)
    return g


def replay(g, s, st):
    import torch

    with torch.cuda.stream(st):
        g.replay()
    s.sync()
    return s.get_positions()


def plain(m, what):
    """Positions after each of the steps `what` names by their (lanes, material factor), one launch per colour."""
    s = build_solver(m, layout=4)
    s.set_option(_capi.OPT_PERSISTENT, 0)
    out = []
    for lanes, factor in what:
        s.set_option(_capi.OPT_LANES, lanes)
        s.set_materials(m.mu * np.float32(factor), m.lam * np.float32(factor))
        s.step(1 / 60, 9, G, True, 0.9)
        out.append(s.get_positions())
    s.close()
    return out


def test_captured_cluster_step_follows_new_materials(gpu_device):
    m = meshgen.jittered_block(9, 6, 5, seed=3, per_tet_sigma=0.2)
    s, st = on_stream(m)
    g = capture_step(s, st)
    want = plain(m, [(8, 1), (8, 1), (8, 3), (8, 5), (8, 5)])
    np.testing.assert_array_equal(replay(g, s, st), want[1])
    s.set_materials(m.mu * np.float32(3), m.lam * np.float32(3))
    np.testing.assert_array_equal(replay(g, s, st), want[2])
    # a step captured right after new materials and never launched leaves them to be packed
    s.set_materials(m.mu * np.float32(5), m.lam * np.float32(5))
    unused = capture_step(s, st)
    s.step(1 / 60, 9, G, True, 0.9)
    np.testing.assert_array_equal(s.get_positions(), want[3])
    np.testing.assert_array_equal(replay(unused, s, st), want[4])
    del g, unused
    s.close()


def test_captured_cluster_step_keeps_its_records_beside_other_shapes(gpu_device):
    """Other lane and CTA counts afterwards, and the first again: what the captured step reads stays in place, and
    follows new materials."""
    m = meshgen.jittered_block(9, 6, 5, seed=3, per_tet_sigma=0.2)
    s, st = on_stream(m)
    g8 = capture_step(s, st)
    s.set_option(_capi.OPT_LANES, 16)
    want = plain(m, [(8, 1), (16, 1), (8, 1), (16, 1), (16, 2), (8, 2), (16, 2), (8, 2), (8, 2)])
    s.step(1 / 60, 9, G, True, 0.9)
    np.testing.assert_array_equal(s.get_positions(), want[1])
    np.testing.assert_array_equal(replay(g8, s, st), want[2])
    g16 = capture_step(s, st)
    np.testing.assert_array_equal(replay(g16, s, st), want[3])
    s.set_option(_capi.OPT_CLUSTER_CTAS, 5)
    s.set_materials(m.mu * np.float32(2), m.lam * np.float32(2))
    s.step(1 / 60, 9, G, True, 0.9)
    np.testing.assert_array_equal(s.get_positions(), want[4])
    np.testing.assert_array_equal(replay(g8, s, st), want[5])
    np.testing.assert_array_equal(replay(g16, s, st), want[6])
    s.set_option(_capi.OPT_LANES, 8)
    s.set_option(_capi.OPT_CLUSTER_CTAS, 0)
    s.step(1 / 60, 9, G, True, 0.9)
    np.testing.assert_array_equal(s.get_positions(), want[7])
    np.testing.assert_array_equal(replay(g8, s, st), want[8])
    del g8, g16
    s.close()


def test_backward_beside_captured_cluster_steps(gpu_device):
    """The library's own captured adjoint launches follow the sets that come and go."""
    m = meshgen.jittered_block(9, 6, 5, seed=3, per_tet_sigma=0.2, E=2e4)
    W = np.random.default_rng(3).normal(size=(m.num_verts, 3))
    s, st = on_stream(m)
    keep = []
    for lanes in (8, 16, 8, 4, 16, 8):
        s.set_option(_capi.OPT_LANES, lanes)
        s.set_positions(m.x)
        s.set_velocities(m.v)
        s.record(2)
        for _ in range(3):
            s.step(1 / 60, 9, G, True, 0.9)
        got = s.backward(W, None, 12, 0.9)
        s.record(0)
        if lanes == 8:
            keep.append(capture_step(s, st))
        ref = build_solver(m, lanes=lanes, layout=4)
        ref.set_option(_capi.OPT_PERSISTENT, 0)
        ref.record(2)
        for _ in range(3):
            ref.step(1 / 60, 9, G, True, 0.9)
        for a, b in zip(got, ref.backward(W, None, 12, 0.9)):
            np.testing.assert_array_equal(a, b)
        ref.close()
    del keep
    s.close()


def test_cluster_step_captured_after_another_shape_was_set(gpu_device):
    m = meshgen.jittered_block(9, 6, 5, seed=3, per_tet_sigma=0.2)
    s, st = on_stream(m)
    s.set_option(_capi.OPT_LANES, 4)
    g = capture_step(s, st)
    np.testing.assert_array_equal(replay(g, s, st), plain(m, [(8, 1), (4, 1)])[1])
    del g
    s.close()


@pytest.mark.parametrize("semantics", [0, 1])
@pytest.mark.parametrize("warm_up", [True, False])
def test_default_step_and_solve_captured_by_the_caller(gpu_device, semantics, warm_up):
    """The walk that a default step takes cannot be captured; the per-colour launches are captured in its place,
    whether or not a step has run before."""
    import torch

    m = meshgen.jittered_block(9, 6, 5, seed=3, per_tet_sigma=0.2)
    out = []
    for captured in (True, False):
        st = torch.cuda.Stream()
        s = build_solver(m, lanes=8, layout=4, stream=st.cuda_stream)
        s.set_option(_capi.OPT_SEMANTICS, semantics)
        if not captured:
            s.set_option(_capi.OPT_PERSISTENT, 0)
        if warm_up:
            s.step(1 / 60, 9, G, True, 0.9)
        s.sync()

        def steps():
            s.step(1 / 60, 9, G, True, 0.9, 2)
            s.solve_vbd(7, 3600.0, True, 0.9, 0)

        if captured:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=st):
                steps()
            for _ in range(2):
                x = replay(g, s, st)
            del g
        else:
            steps()
            steps()
            x = s.get_positions()
        out.append((x, s.get_velocities()))
        s.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_changing_schedules_are_queued_without_waiting(gpu_device):
    """A step with another schedule than the one before returns while that one is still at work, as with the same
    schedule: schedules used before, and a new one."""
    import torch

    st = torch.cuda.Stream()
    s = build_solver(meshgen.cube(32), stream=st.cuda_stream)
    for n, accel, rho in ((2000, True, 0.9), (20, False, 0.9), (25, True, 0.95)):
        s.step(1 / 120, n, G, accel, rho)
    s.sync()
    for n, accel, rho in ((20, False, 0.9), (25, True, 0.95), (30, True, 0.8)):
        s.step(1 / 120, 2000, G, True, 0.9)  # about 5 ms
        before = torch.cuda.Event()
        before.record(st)
        s.step(1 / 120, n, G, accel, rho)
        assert not before.query()
        s.sync()
    s.close()


@pytest.mark.parametrize("persistent", [None, 1, 2])
def test_many_schedules_equal_the_graph(gpu_device, persistent):
    """More schedules than are kept, prefixes of one another, with and without blending, in turn."""
    m = meshgen.jittered_block(9, 6, 5, seed=3, per_tet_sigma=0.2)
    shapes = [(n, accel, rho) for n in (3, 12, 7) for accel, rho in ((True, 0.9), (True, 0.95), (False, 0.0), (True, 0.5))]
    order = np.random.default_rng(1).integers(0, len(shapes), 40)
    out = []
    for p in (persistent, 0):
        s = build_solver(m, lanes=8, layout=4)
        if p is not None:
            s.set_option(_capi.OPT_PERSISTENT, p)
        for k in order:
            n, accel, rho = shapes[k]
            s.step(1 / 60, n, G, accel, rho)
        out.append((s.get_positions(), s.get_velocities()))
        s.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("persistent", [1, 2])
def test_captured_step_keeps_its_schedule(gpu_device, persistent):
    m = meshgen.jittered_block(9, 6, 5, seed=3, per_tet_sigma=0.2)
    s, st = on_stream(m)
    s.set_option(_capi.OPT_PERSISTENT, persistent)
    s.step(1 / 60, 9, G, True, 0.9)
    g = capture_step(s, st)
    ref = build_solver(m, lanes=8, layout=4)
    ref.set_option(_capi.OPT_PERSISTENT, 0)
    for _ in range(2):
        ref.step(1 / 60, 9, G, True, 0.9)
    for k in range(10):
        for t in (s, ref):
            t.step(1 / 60, 9, G, True, 0.5 + 0.04 * k)
    ref.step(1 / 60, 9, G, True, 0.9)
    np.testing.assert_array_equal(replay(g, s, st), ref.get_positions())
    del g
    s.close()
    ref.close()
