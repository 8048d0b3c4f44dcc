"""The phases of meshes with periodic axes, alone and chained (the phases of small levels run in a chain's first block,
exchanges stand between the levels, both sides of an axis exchange tags together or in turn), against the oracle, bit
for bit: one to three axes, both stencil radii, boxes narrower than two ghost widths, meshes of one level."""
import pytest

from gpu_util import compare_cells, compare_fields, compare_meshes
from oracle.pyoracle import OracleSim
from test_gpu_periodic import near_boundary

pytestmark = pytest.mark.gpu

FORMS = {
    "alone": {"SG_CHAIN_BLOCKS": "0"},
    "one block": {"SG_CHAIN_BLOCKS": "1"},
    "two blocks": {"SG_CHAIN_BLOCKS": "2"},
    "at most twelve blocks": {"SG_CHAIN_BLOCKS": "12"},
    "all chained": {"SG_CHAIN_BLOCKS": "16", "SG_FUSE_WORDS": "1000000", "SG_FUSE_WORDS_FIELD": "1000000", "SG_FUSE_WORDS_MAX": "1000000"},
    "levels alone": {"SG_FUSE_WORDS_FIELD": "0"},
    "odd blocks": {"SG_BLOCK": "96", "SG_MAX_BLOCKS": "3"},
    "not overlapped": {"SG_OVERLAP_LAUNCHES": "0"},
}
CASES = [
    (2, 1, 7, 1, (1, 0)),
    (2, 2, 8, 1, (1, 1)),
    (2, 3, 8, 2, (0, 1)),
    (2, 3, 7, 2, (1, 1)),
    (2, 5, 5, 1, (1, 1)),
    (3, 1, 4, 1, (1, 0, 1)),
    (3, 2, 5, 1, (1, 1, 1)),
    (3, 3, 5, 2, (1, 1, 0)),
]


@pytest.fixture(scope="module")
def sg():
    from samurai_gb300 import build

    build.build()
    import samurai_gb300

    return samurai_gb300


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("dim,minl,maxl,radius,per", CASES)
def test_periodic_phases_against_oracle(sg, monkeypatch, form, dim, minl, maxl, radius, per):
    for k, v in FORMS[form].items():
        monkeypatch.setenv(k, v)
    per = tuple(bool(p) for p in per) + (False,) * (3 - dim)
    g = sg.AdvectionSim(dim, minl, maxl, radius, 1, 1, 0.25, periodic=per[:dim])
    o = OracleSim(dim, minl, maxl, radius, 1, 1, 0.25, periodic=per)
    lv, co, _ = o.cells()
    vals = near_boundary(lv, co, dim)
    g.set_cell_values(vals)
    o.set_cell_values(vals)
    a = [-1.0, 0.5, 0.75][:dim]
    for it in range(3):
        where = "it %d" % it
        assert g.adapt(1e-3, 1.0) == o.adapt(1e-3, 1.0), where
        compare_cells(g, o, where)
        g.update_ghost()
        o.update_ghost()
        compare_fields(g, o, where + " ghosts")
        g.upwind(a, 0.3 / (1 << maxl))
        o.upwind(a, 0.3 / (1 << maxl))
        compare_fields(g, o, where + " upwind", cells_only=True)
    compare_meshes(g, o, maxl, "final")
