"""Details and tags of single Harten passes read in the numbering of the mesh that the pass leaves: a cell reads what
the last pass that had it in its reference mesh found there, 0 where that pass examined no parent of it and 0 where no
pass ever had it; also after a pass that changed the mesh.  Against the oracle, pass by pass, bit for bit."""
import numpy as np
import pytest

from advection_cases import ball_3d, shapes_2d
from oracle import pyoracle
from oracle.pyoracle import OracleSim

pytestmark = pytest.mark.gpu

PAD = 8  # cells stored around the box


@pytest.fixture(scope="module")
def sg():
    from samurai_gb300 import build

    build.build()
    import samurai_gb300

    return samurai_gb300


def reference_cells(o):
    """per level the coordinates of the reference cells, rows in storage order"""
    out = []
    for level in range(o.max_level + 1):
        rows = o.intervals("reference", level)
        n = rows[:, 1] - rows[:, 0]
        x = np.concatenate([np.arange(a, b) for a, b in rows[:, :2]]) if len(rows) else np.empty(0, np.int64)
        out.append(np.column_stack([x] + [np.repeat(rows[:, 2 + d], n) for d in range(o.dim - 1)]).astype(np.int64))
    return out


class History:
    """what the passes so far found, per stored cell"""

    def __init__(self, o):
        shape = lambda level: ((1 << level) + 2 * PAD,) * o.dim  # noqa: E731
        self.detail = [np.zeros(shape(level)) for level in range(o.max_level + 1)]
        self.tag = [np.zeros(shape(level), np.uint8) for level in range(o.max_level + 1)]

    def take(self, o, cells):
        """the pass just made on the reference cells `cells` (the oracle's arrays are still numbered by them)"""
        n = sum(len(c) for c in cells)
        det, tag = np.empty(n), np.empty(n, np.uint8)
        pyoracle.lib().oracle_get_detail(o.h, pyoracle._ptr(det))
        pyoracle.lib().oracle_get_tag(o.h, pyoracle._ptr(tag))
        first = 0
        for level, c in enumerate(cells):
            at = tuple((c + PAD).T)
            self.detail[level][at] = det[first:first + len(c)]
            self.tag[level][at] = tag[first:first + len(c)]
            first += len(c)

    def read(self, cells):
        at = [tuple((c + PAD).T) for c in cells]
        return np.concatenate([d[a] for d, a in zip(self.detail, at)]), np.concatenate([t[a] for t, a in zip(self.tag, at)])


@pytest.mark.parametrize("dim,minl,maxl,radius,per", [(2, 2, 7, 1, 0), (2, 3, 7, 2, 0), (2, 2, 6, 1, 3), (3, 2, 5, 1, 0)])
def test_every_pass_reads_as_it_was_made(sg, dim, minl, maxl, radius, per):
    periodic = [bool(per >> d & 1) for d in range(3)]
    g = sg.AdvectionSim(dim, minl, maxl, radius, 1, 1, 0.0, periodic=periodic[:dim])
    o = OracleSim(dim, minl, maxl, radius, 1, 1, 0.0, periodic=periodic)
    lv, co, _ = o.cells()
    vals = (shapes_2d(19, 4, 4) if dim == 2 else ball_3d(9))(lv, co)
    g.set_cell_values(vals)
    o.set_cell_values(vals)
    seen, changed, leftover = History(o), 0, 0
    a, dt = [1.0, -0.7, 0.5][:dim], 0.45 / (1 << maxl)
    for it in range(4):
        for ite in range(maxl - minl):
            old = reference_cells(o)
            done = o.harten(ite, 1e-3, 1.0)
            assert g.harten(ite, 1e-3, 1.0) == done
            before = [d.copy() for d in seen.detail]
            seen.take(o, old)
            new = reference_cells(o)
            det, tag = seen.read(new)
            ok = ~np.isnan(det)
            got = g.detail()
            where = "step %d, pass %d" % (it, ite)
            assert np.array_equal(got[ok], det[ok]), where + ": %d details differ" % np.count_nonzero(got[ok] != det[ok])
            assert np.array_equal(g.tag(), tag), where + ": tags"
            changed += not done
            # cells with a detail from an earlier pass that this one had in its reference without examining them
            leftover += sum(int(np.count_nonzero((b != 0.0) & (s == 0.0))) for b, s in zip(before, seen.detail))
            if done:
                break
        for _ in range(3):  # the solution moves on an old mesh, so that the next pass refines and coarsens
            g.update_ghost()
            o.update_ghost()
            g.upwind(a, dt)
            o.upwind(a, dt)
    assert changed > 4 and leftover > 0


@pytest.mark.parametrize("dim,minl,maxl,radius", [(2, 2, 8, 1), (2, 2, 8, 2), (3, 2, 6, 1)])
def test_a_pass_that_keeps_the_mesh_leaves_carried_fields_alone(sg, dim, minl, maxl, radius):
    """a mesh refined along the boundary only: the criteria coarsen every ring inside, and the graduation refines them
    again, ring after ring (with radius 2 in more than two of its passes), until the cells are the old ones.  Fields carried along
    get new ghosts only when the mesh changes (mr/adapt.hpp:380-386)."""
    mesh = sg.MRMesh(dim, minl, maxl, radius, 1, 1)
    mesh.set_refine_boundary(True)
    u, w = sg.make_scalar_field("u", mesh), sg.make_scalar_field("w", mesh)
    for f in (u, w):
        sg.make_bc(sg.Dirichlet(1), f, 0.0)
    u.fill(0.0)
    adapt = sg.make_MRAdapt(u)
    cfg = sg.mra_config().epsilon(1e-4).regularity(0.0)
    for _ in range(2 * maxl):
        if adapt(cfg) == 1:
            break
    before = mesh.cells()
    assert set(before[0]) >= set(range(maxl - 3, maxl + 1))
    values = np.random.default_rng(3).uniform(1.0, 2.0, mesh.nb_cells("reference"))
    w.set_array(values)
    assert adapt(cfg, w) == 1
    after = mesh.cells()
    assert all(np.array_equal(x, y) for x, y in zip(before, after))
    assert np.array_equal(w.array(), values)


def test_timers_count_the_phases_of_the_mesh_that_changed(sg):
    """an adaptation whose first pass keeps the mesh builds no mesh and moves no field"""
    s = sg.AdvectionSim(2, 2, 7)
    lv, co, _ = s.cells()
    s.set_cell_values(shapes_2d(5, 3, 3)(lv, co))
    while s.adapt(1e-3, 1.0) > 1:
        pass
    s.mesh.timers(enable=True, reset=True)
    assert s.adapt(1e-3, 1.0) == 1
    s.mesh.synchronize()
    t = s.mesh.timers(enable=False)
    assert t["mesh adaptation"][1] == 1 and t["detail computation"][1] == 1
    assert t["mesh construction"] == (0.0, 0) and t["fields update"] == (0.0, 0)
