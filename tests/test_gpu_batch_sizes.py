"""Batches on both sides of the sizes where their launches change form (overlapping or not, levels of the ghost update
alone or chained, the clusters' sizes), with and without periodic axes: instance by instance what the serial calls
give, bit for bit; and the instances' own launches afterwards."""
import numpy as np
import pytest

from advection_cases import ball_3d, shapes_2d

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sg():
    from samurai_gb300 import build

    build.build()
    import samurai_gb300

    return samurai_gb300


def problem(sg, dim, maxl, seed, periodic):
    s = sg.AdvectionSim(dim, 2, maxl, periodic=[periodic] * dim)
    lv, co, _ = s.cells()
    s.set_cell_values((shapes_2d(seed, 3, 3) if dim == 2 else ball_3d(seed))(lv, co))
    return s


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("dim,maxl", [(2, 7), (3, 5)])
@pytest.mark.parametrize("n", [1, 3, 4, 11, 12, 16])
def test_batch_of_n_matches_serial(sg, dim, maxl, periodic, n):
    mine, serial = ([problem(sg, dim, maxl - k % 2, 50 + k, periodic) for k in range(n)] for _ in range(2))
    a = [[1.0, -0.6, 0.4][:dim], [-0.7, 0.5, -0.9][:dim]]
    shapes = [s.mesh.launch_shape() for s in mine]
    batch = sg.Batch(mine, n_threads=3)
    for _ in range(3):
        passes = batch.step(1e-3, 1.0, [a[k % 2] for k in range(n)], [0.3 / (1 << maxl)] * n).copy()
        for k, s in enumerate(serial):
            assert s.adapt(1e-3, 1.0) == passes[k]
            s.update_ghost()
            s.upwind(a[k % 2], 0.3 / (1 << maxl))
    batch.synchronize()
    batch.update_ghost()
    batch.synchronize()
    batch.close()
    for k, (x, y) in enumerate(zip(mine, serial)):
        y.update_ghost()
        for p, q in zip(x.cells(), y.cells()):
            assert np.array_equal(p, q), k
        assert np.array_equal(x.field(), y.field()), k
    assert shapes == [s.mesh.launch_shape() for s in mine]
