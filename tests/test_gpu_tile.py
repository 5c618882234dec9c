"""The tile walk (csrc/vbd_tile.cuh), which vbd_solver_step / _solve / _backward take for meshes of a few
hundred vertices and more until VBD_OPT_PERSISTENT is set: the same bits as the captured graph of
per-colour launches (VBD_OPT_PERSISTENT 0)."""
import numpy as np
import pytest

from vbd_tetmesh_b200 import _capi, build_batch_solver, build_solver, meshgen

pytestmark = pytest.mark.gpu

G = (0.0, -9.8, 0.0)


def both(make, run):
    """run(solver) on the tile walk and on the graph; checks that the first took fewer launches."""
    out, launches = [], []
    for graph in (False, True):
        s = make()
        if graph:
            s.set_option(_capi.OPT_PERSISTENT, 0)
        l0 = s.kernel_launches()
        out.append(run(s))
        s.sync()
        launches.append(s.kernel_launches() - l0)
        s.close()
    assert launches[0] < launches[1]
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def step(s, dt, iterations, accel, rho=0.9, substeps=1, steps=2):
    for _ in range(steps):
        s.step(dt, iterations, G, accel, rho, substeps)
    return s.get_positions(), s.get_velocities()


# the smallest mesh with a plan, one tile, ragged tiles; lanes 4 to 16; stored and derived det M; a pinned
# face inside and none; with and without acceleration (blended words, both buffers), sub-steps
@pytest.mark.parametrize("dims,lanes,layout,pin,accel,substeps,iterations", [
    ((7, 6, 5), 16, 4, "x0", True, 1, 9), ((7, 6, 5), 4, 3, "z1", False, 2, 3), ((13, 7, 5), 8, 4, "y0", True, 2, 1),
    ((15, 14, 13), 4, 4, "x1", True, 1, 12), ((15, 14, 13), 8, 3, "y1", True, 1, 12), ((30, 9, 8), 16, 4, "x0", False, 1, 7),
])
def test_tile_walk_equals_graph(gpu_device, dims, lanes, layout, pin, accel, substeps, iterations):
    m = meshgen.jittered_block(*dims, seed=5, pin_face=pin, per_tet_sigma=0.2)
    both(lambda: build_solver(m, lanes=lanes, layout=layout), lambda s: step(s, 1 / 60, iterations, accel, 0.9, substeps))


@pytest.mark.parametrize("n", [16, 40, 56])  # 8 warps with both buffers, 16 warps with and without them
def test_tile_walk_cubes_equal_graph(gpu_device, n):
    m = meshgen.cube(n)
    both(lambda: build_solver(m), lambda s: step(s, 1 / 120, 10, True))


def test_tile_walk_batch_equals_graph(gpu_device):
    b = meshgen.concat(meshgen.batched_blocks(num_meshes=24, lo=2, hi=14, seed=7))
    both(lambda: build_batch_solver(b), lambda s: step(s, 1 / 60, 10, True))


@pytest.mark.parametrize("mode", [0, 1])
def test_tile_solve_energy_and_new_materials_equal_graph(gpu_device, mode):
    m = meshgen.jittered_block(14, 13, 12, seed=1, per_tet_sigma=0.2)
    y = (m.x + np.random.default_rng(0).normal(0, 1e-3, m.x.shape) * (m.fixed == 0)[:, None]).astype(np.float32)

    def run(s):
        s.update_inertia_from_cpu(y)
        s.solve_vbd(11, 3600.0, True, 0.9, mode)
        out = [s.get_positions()]
        s.set_materials(m.mu * 3, m.lam * 2)
        s.set_option(_capi.OPT_ENERGY_EVERY, 4)
        s.step(1 / 60, 10, G, True, 0.9)
        out += [s.energy_history(), *step(s, 1 / 60, 5, True)]
        s.set_option(_capi.OPT_LANES, 4)  # another lane count: other groups and chunks
        return out + [*step(s, 1 / 60, 5, True)]

    both(lambda: build_solver(m), run)


@pytest.mark.parametrize("dims,lanes,layout,adj_rho", [((9, 6, 5), 8, 4, 0.9), ((9, 6, 5), 16, 3, 0.0), ((40, 24, 22), 4, 4, 0.9)])
def test_tile_backward_equals_graph(gpu_device, dims, lanes, layout, adj_rho):
    m = meshgen.jittered_block(*dims, seed=3, per_tet_sigma=0.2, E=2e4)
    W = np.random.default_rng(3).normal(size=(m.num_verts, 3))

    def run(s):
        s.record(2)
        for _ in range(3):
            s.step(1 / 60, 10, G, True, 0.9)
        return s.backward(W, None, 12, adj_rho)

    both(lambda: build_solver(m, lanes=lanes, layout=layout), run)


def test_non_finite_positions_spread_as_in_the_graph(gpu_device):
    """Padding records add exact zeros whatever the positions hold: a NaN and an infinity reach the
    same vertices as on the graph path."""
    m = meshgen.jittered_block(14, 13, 12, seed=2)
    m.x = m.x.copy()
    m.x[1000, 1], m.x[1500, 0] = np.nan, np.inf
    both(lambda: build_solver(m), lambda s: [np.isfinite(a) for a in step(s, 1 / 60, 2, True, steps=1)])


def test_two_solvers_on_two_threads(gpu_device):
    """Tile walks of two handles on two streams, launched from two threads at once, give what each gives
    alone."""
    import threading

    meshes = [meshgen.cube(20), meshgen.cube(24)]
    alone = []
    for m in meshes:
        s = build_solver(m)
        alone.append(step(s, 1 / 120, 20, True, steps=30))
        s.close()
    solvers = [build_solver(m) for m in meshes]
    out = [None, None]

    def work(k):
        out[k] = step(solvers[k], 1 / 120, 20, True, steps=30)
        solvers[k].sync()

    ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    for k in range(2):
        solvers[k].close()
        for a, b in zip(alone[k], out[k]):
            np.testing.assert_array_equal(a, b)
