"""The adjoint under launch shapes of large blocks (SG_BLOCK, or a tuned shape): the transposed kernels hold linear forms
in registers, and their blocks are bounded by that; dot-product test of the recorded map, 2D and 3D."""
import numpy as np
import pytest

from advection_cases import ball_3d, shapes_2d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block", [64, 512, 1024])
@pytest.mark.parametrize("dim,maxl", [(2, 6), (3, 4)])
def test_dot_product_with_large_blocks(monkeypatch, dim, maxl, block):
    import samurai_gb300 as sg

    monkeypatch.setenv("SG_BLOCK", str(block))
    s = sg.AdvectionSim(dim, 2, maxl)
    lv, co, _ = s.cells()
    s.set_cell_values((shapes_2d(31, 3, 3) if dim == 2 else ball_3d(4))(lv, co))
    s.adapt(1e-3, 1.0)
    assert s.mesh.launch_shape()["block"] == block
    adj = sg.Adjoint(s.u, checkpoint_every=2)
    a = [0.9, -0.6, 0.4][:dim]
    adj.record(s.cell_values(), 5, 1e-3, 1.0, a, 0.3 / (1 << maxl))
    n0, nT, _ = adj.counts()
    rng = np.random.default_rng(7)
    v, w = rng.standard_normal(n0), rng.standard_normal(nT)
    lhs = float(adj.replay(v, a) @ w)
    rhs = float(v @ adj.backward(w)[0])
    # sums of nT and n0 products of order 1, each product within some tens of roundings of 5 steps
    assert abs(lhs - rhs) <= 1e-13 * (np.abs(w).sum() + np.abs(v).sum())
