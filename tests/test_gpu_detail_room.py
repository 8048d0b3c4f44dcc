"""Adapting many fields on a mesh needs a detail slab per field; where the device has no room for them the call is
refused and the mesh adapts as before: no captured launch and no pointer to the freed slabs is left, the refusal is
reported once, and the same call succeeds when there is room again."""
import pytest

from advection_cases import shapes_2d
from gpu_util import compare_cells, compare_fields
from oracle.pyoracle import OracleSim

pytestmark = pytest.mark.gpu

MINL, MAXL, N = 3, 11, 23  # a slab is 48 MB


@pytest.mark.parametrize("graphed", [False, True])
def test_refused_details_leave_the_mesh_as_it_was(monkeypatch, graphed):
    torch = pytest.importorskip("torch")
    import samurai_gb300 as sg

    if graphed:
        monkeypatch.setenv("SG_GRAPHED_ADAPT", "1")
    g, o = sg.AdvectionSim(2, MINL, MAXL), OracleSim(2, MINL, MAXL)
    v = [sg.make_scalar_field("v%d" % k, g.mesh) for k in range(N)]
    for f in v:
        f.fill(0.0)
    lv, co, _ = o.cells()
    vals = shapes_2d(7, 3, 3)(lv, co)
    g.set_cell_values(vals)
    o.set_cell_values(vals)
    alone, together = sg.make_MRAdapt(g.u), sg.make_MRAdapt(g.u, *v)

    def step(where):
        # the spare buffers of every field and the launches of one field's details exist after the first of these
        assert alone(1e-3, 1.0, *v, relative_detail=True) == o.adapt(1e-3, 1.0, relative_detail=True), where
        compare_cells(g, o, where)
        g.update_ghost()
        o.update_ghost()
        compare_fields(g, o, where)
        g.upwind([0.8, -0.5], 0.4 / (1 << MAXL))
        o.upwind([0.8, -0.5], 0.4 / (1 << MAXL))

    for k in range(3):
        step("before, step %d" % k)
    g.mesh.synchronize()
    keep = 400 << 20  # less than the slabs of all fields take
    fill = []
    try:
        for chunk in (16 << 30, 1 << 30, 64 << 20):
            while torch.cuda.mem_get_info()[0] > keep + chunk:
                fill.append(torch.empty(chunk, dtype=torch.uint8, device="cuda"))
        with pytest.raises(sg.SamuraiGpuError, match="cudaMalloc"):
            together(1e-3, 1.0)
        for k in range(3):
            step("without room, step %d" % k)
    finally:
        fill.clear()
        torch.cuda.empty_cache()
    assert together(1e-3, 1.0) >= 1
    g.update_ghost()
