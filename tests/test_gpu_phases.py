"""The phases of the step alone and chained, against the oracle, bit for bit: meshes whose phases all join one
chain, whose phases all launch alone, and mixed ones; one and two levels; blocks that are no power of two (the
items of a block are found by bisection); more fields than one phase takes; meshes whose word count is around a
chunk of the scan.  No tolerance: meshes, tags, details and values are equal."""
import numpy as np
import pytest

from advection_cases import ball_3d, centers, shapes_2d
from gpu_util import compare_cells, compare_fields, compare_meshes
from oracle.pyoracle import OracleSim

pytestmark = pytest.mark.gpu

SHAPES = [
    {"SG_CHAIN_BLOCKS": "0"},
    {"SG_CHAIN_BLOCKS": "2"},
    {"SG_CHAIN_BLOCKS": "16", "SG_FUSE_WORDS": "1000000", "SG_FUSE_WORDS_FIELD": "1000000", "SG_FUSE_WORDS_MAX": "1000000"},
    {"SG_BLOCK": "96", "SG_MAX_BLOCKS": "3"},
    {"SG_OVERLAP_LAUNCHES": "0"},
]


@pytest.fixture(scope="module")
def sg():
    from samurai_gb300 import build

    build.build()
    import samurai_gb300

    return samurai_gb300


def advance(sg, g, o, dim, maxl, eps, reg, steps):
    a = [0.9, -0.6, 0.4][:dim]
    dt = 0.3 / (1 << maxl)
    lv, co, _ = o.cells()
    vals = (shapes_2d(11, 5, 5) if dim == 2 else ball_3d(7))(lv, co)
    g.set_cell_values(vals)
    o.set_cell_values(vals)
    for it in range(steps):
        where = "it %d" % it
        assert g.adapt(eps, reg) == o.adapt(eps, reg), where
        compare_cells(g, o, where)
        g.update_ghost()
        o.update_ghost()
        compare_fields(g, o, where + " ghosts")
        g.upwind(a, dt)
        o.upwind(a, dt)
        compare_fields(g, o, where + " upwind", cells_only=True)
    compare_meshes(g, o, maxl, "final")


@pytest.mark.parametrize("env", SHAPES, ids=["alone", "two blocks", "all chained", "odd blocks", "not overlapped"])
@pytest.mark.parametrize("dim,minl,maxl,radius,pred", [(2, 1, 2, 1, 1), (2, 4, 4, 1, 1), (2, 2, 7, 2, 1), (2, 3, 9, 1, 0), (3, 1, 3, 1, 1), (3, 2, 5, 2, 1)])
def test_phases_against_oracle(sg, monkeypatch, env, dim, minl, maxl, radius, pred):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    g = sg.AdvectionSim(dim, minl, maxl, radius, pred)
    o = OracleSim(dim, minl, maxl, radius, pred)
    advance(sg, g, o, dim, maxl, 1e-3, 1.0, 3)


@pytest.mark.parametrize("env", SHAPES[:3], ids=["alone", "two blocks", "all chained"])
def test_details_and_tags_of_a_converged_pass(sg, monkeypatch, env):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    g, o = sg.AdvectionSim(2, 2, 7), OracleSim(2, 2, 7)
    lv, co, _ = o.cells()
    vals = shapes_2d(23, 4, 4)(lv, co)
    g.set_cell_values(vals)
    o.set_cell_values(vals)
    for ite in range(5):
        done = o.harten(ite, 1e-3, 1.0)
        assert g.harten(ite, 1e-3, 1.0) == done
        if done:
            break
    assert done
    do, dg = o.detail(), g.detail()
    ok = ~np.isnan(do)
    assert np.array_equal(do[ok], dg[ok]) and np.array_equal(o.tag(), g.tag())


@pytest.mark.parametrize("env", [SHAPES[0], SHAPES[2]], ids=["alone", "all chained"])
def test_more_fields_than_one_phase_takes(sg, monkeypatch, env):
    """nine components adapted together, on relative details, with a field carried along"""
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    n = 9
    mesh = sg.MRMesh(2, 2, 6)
    v = sg.make_vector_field("v", mesh, n)
    w = sg.make_scalar_field("w", mesh)
    bcs = [0.1 * k - 0.3 for k in range(n)]
    sg.make_bc(sg.Dirichlet(1), v, *bcs)
    sg.make_bc(sg.Dirichlet(1), w, 0.5)
    o = OracleSim(2, 2, 6, 1, 1, 1, bcs[0])
    ks = [0] + [o.add_field(b) for b in bcs[1:]]
    kw = o.add_field(0.5)
    lv, co, _ = o.cells()
    vals = np.stack([(1.0 + k) * shapes_2d(30 + k, 1, 1)(lv, co) for k in range(n)], axis=1)
    carried = np.sin(5.0 * centers(lv, co)[:, 0])
    v.set_cells(vals)
    w.set_cells(carried)
    for c, k in enumerate(ks):
        o.set_cell_values_k(k, vals[:, c])
    o.set_cell_values_k(kw, carried)
    cfg = sg.mra_config().epsilon(1e-3).regularity(1.0).relative_detail(True)
    adapt = sg.make_MRAdapt(v)
    assert adapt(cfg, w) == o.adapt_fields(1e-3, 1.0, n, 1, relative_detail=True)
    lg, cg, _ = mesh.cells()
    lo, coo, _ = o.cells()
    assert np.array_equal(lg, lo) and np.array_equal(cg, coo)
    got = v.cell_values()
    for c, k in enumerate(ks):
        assert np.array_equal(got[:, c], o.cell_values_k(k)), c
    assert np.array_equal(w.cell_values(), o.cell_values_k(kw))


@pytest.mark.parametrize("minl,maxl", [(4, 4), (2, 6)])
@pytest.mark.parametrize("a", [[0.9, -0.6], [0.0, 1.0]])
def test_flux_form_of_values_that_are_not_finite(sg, minl, maxl, a):
    """a term with a zero coefficient may be left out only where its value is finite: 0 * inf is NaN in the oracle"""
    g, o = sg.AdvectionSim(2, minl, maxl), OracleSim(2, minl, maxl)
    lv, co, _ = o.cells()
    vals = shapes_2d(5, 3, 3)(lv, co)
    g.set_cell_values(vals)
    o.set_cell_values(vals)
    if minl < maxl:
        assert g.adapt(1e-3, 1.0) == o.adapt(1e-3, 1.0)
    n = len(o.cells()[0])
    vals = np.cos(np.arange(n))
    vals[n // 5], vals[n // 2], vals[4 * n // 5] = np.inf, -np.inf, np.nan
    g.set_cell_values(vals)
    o.set_cell_values(vals)
    g.update_ghost()
    o.update_ghost()
    g.upwind(a, 0.3 / (1 << maxl), 2)
    o.upwind(a, 0.3 / (1 << maxl), 2)
    idx = o.cells()[2]
    got, want = g.field()[idx], o.field()[idx]
    assert np.isnan(want).any() and np.isfinite(want).any()
    assert np.array_equal(got, want, equal_nan=True)
