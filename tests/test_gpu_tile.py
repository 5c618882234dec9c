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


def delaunay(n, seed, around=60):
    """A Delaunay mesh of n random points and a centre with `around` points about it: valences from 4 to 40 and,
    at the centre, to twice `around`."""
    from scipy.spatial import Delaunay

    rng = np.random.default_rng(seed)
    shell = rng.normal(size=(around, 3))
    shell = 0.5 + 0.12 * shell / np.linalg.norm(shell, axis=1)[:, None]
    pts = np.concatenate([rng.uniform(0, 1, (n, 3)), shell, [[0.5, 0.5, 0.5]]])
    pts = pts[(np.linalg.norm(pts - 0.5, axis=1) > 0.119) | (np.arange(len(pts)) == len(pts) - 1)]
    tets = Delaunay(pts).simplices.astype(np.int32)
    e = pts[tets[:, 1:]] - pts[tets[:, :1]]
    vol = np.linalg.det(e) / 6
    tets[vol < 0, 2:] = tets[vol < 0, 3:1:-1]
    tets = tets[np.abs(vol) > 2e-6]
    p = pts.astype(np.float32)
    mu, lam = meshgen.lame(1e5, 0.3)
    t = len(tets)
    return meshgen.Mesh(p.copy(), p.copy(), np.zeros_like(p), tets, (p[:, 0] < 0.1).astype(np.uint8),
                        np.full(t, mu, np.float32), np.full(t, lam, np.float32))


# more incidences per vertex than one round holds, at every lane count
@pytest.mark.parametrize("lanes,around", [(4, 60), (8, 60), (16, 60), (16, 12)])
def test_tile_walk_high_valence_equals_graph(gpu_device, lanes, around):
    m = delaunay(900, 1, around)
    assert np.bincount(m.tets.ravel()).max() > 32

    def run(s):
        out = step(s, 1 / 240, 6, True)
        s.record(2)
        s.step(1 / 240, 5, G, True, 0.9)
        return [*out, *s.backward(np.ones((m.num_verts, 3)), None, 6, 0.9)]

    both(lambda: build_solver(m, lanes=lanes), run)


# VBD_GPU_Solver semantics: 8 and 16 warps, records resident and streamed, two rounds per vertex, ragged groups,
# large initial velocities (the corotated steps have work to do), a batch
@pytest.mark.parametrize("make", [
    lambda: meshgen.jittered_block(7, 6, 5, seed=5, per_tet_sigma=0.3), lambda: meshgen.cube(18), lambda: meshgen.cube(26),
    lambda: delaunay(900, 2), lambda: meshgen.concat(meshgen.batched_blocks(num_meshes=9, lo=2, hi=9, seed=4)),
], ids=["block", "cube18", "cube26", "delaunay", "batch"])
def test_wrapper_semantics_tile_equals_graph(gpu_device, make):
    m = make()

    def run(s):
        s.set_option(_capi.OPT_SEMANTICS, 1)
        out = [*step(s, 1 / 120, 10, True)]
        s.set_materials(m.mu * 2, m.lam * 3)
        out += [*step(s, 1 / 120, 7, False, substeps=2, steps=1)]
        s.update_inertia_from_cpu(m.x)
        for mode in (0, 1):
            s.solve_vbd(6, 14400.0, True, 0.9, mode)
            out.append(s.get_positions())
        return out

    both(lambda: build_batch_solver(m) if isinstance(m, meshgen.Batch) else build_solver(m), run)


def test_wrapper_semantics_degenerate_elements_equal_graph(gpu_device):
    """Elements whose rotation steps stop at |det| < 1e-8 (flattened cells) and non-finite positions."""
    m = meshgen.jittered_block(9, 8, 7, seed=6)
    m.x = m.x.copy()
    m.x[(m.ijk[:, 0] >= 4) & (m.ijk[:, 0] <= 6), 0] = 0.25
    m.x[100] = m.x[101]
    m.x[300, 2], m.x[301, 1] = np.nan, np.inf

    def run(s):
        s.set_option(_capi.OPT_SEMANTICS, 1)
        s.update_inertia_from_cpu(m.x)
        s.solve_vbd(2, 3600.0, True, 0.9, 0)
        x = s.get_positions()
        return x, np.array(s.status())

    both(lambda: build_solver(m), run)
