"""What the walks (csrc/vbd_tile.cuh, csrc/vbd_cluster.cuh) keep between calls: schedules, captured launches,
packed records and wait states stay right when the calls around them change."""
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
